// fp32 pipeline of the chunked HDLA operator for rank 2 and head dims up to 128, forward and backward: five launches.
//
// It serves fp32 inputs (whose 1e-4 tolerance tensor-core operand rounding cannot meet) and the bf16 calls whose decay is
// beyond the tensor-core pipeline.  The result does not depend on the chunk size, so it works in chunks of 16 tokens
// whatever was asked for: a whole chunk's operands and scores then live in one CTA's shared memory, the inverse is a
// 32 x 32 substitution in one warp, and 16-token chunks make four times as many independent tiles as 64.
//
//   tile_fwd   per tile   decay sums, the four gated score matrices, M = (I - Aab)^-1, w = M ag, u = M Aak v
//   scan<fwd>  per (batch, head, 16 state columns), serial over chunks:
//                  v2 = w S + u ;  o = qg S + Aqk v + Aqb v2 ;  S <- decay (.) S + kg^T v + bg^T v2
//   scan<rev>  the same, backwards:
//                  dv2 = bg dS + Aqb^T dO ;  dS <- decay (.) dS + qg^T dO + w^T dv2
//   tile_bwd   per tile   everything else.  With Y = [dO; dP], Z = [v; v2], dP = M^T dv2, the scores' gradient is the one
//                  masked product Y Z^T and the state's shares are Y S^T and Z dS^T.  (The reference goes through the
//                  WY factors, HRDPLR/bwd_triton.py:489-612: dw = dv2 S^T, dM = dv2 P^T + dw ag^T, M^T dM M^T.  With
//                  M P + w S = v2 these collapse: M^T dw = dP S^T, M^T dM M^T = dP (u + w S)^T = dP v2^T.)
//   (other stages: HRDPLR/naive.py:107-263, HRDPLR/bwd_triton.py:17-487, 761-947)
//
// What bounds them (B2 T1000 H8 K=V=128: 1008 tiles, 128 scan CTAs): the tile kernels issue fp32 arithmetic and shared loads
// from 8 warps per SM (77 and 266 us), the scans are the serial chain of 63 steps of 2.4 us from one warp per scheduler
// (155 us each).  Checkpoints are kept transposed, [v][k], so that a scan thread's four state rows move as 16 bytes next
// to its neighbours' (element by element they took two thirds of the scans' shared/global access slots, 262 us each).
//
// Decay-weighted products take the exponent difference per element (exp(g_i - g_j) with g_i <= g_j on the causal mask),
// so nothing can overflow however strong the decay is.
#include "common.cuh"
#include "f32x2.cuh"
#include "sm100.cuh"

namespace hdla {
namespace {

constexpr int CT = 16, M2 = 32, RR = 48;     // tokens of a tile, low-rank rows, stacked rows ([q|k|v] 16 + [a|b|v2] 32)
constexpr int VS = 16;                       // state columns of a scan CTA

// Status words of these kernels (include/hdla.h, hdla_fp32_status_words), one set per device: they are only written when a
// time-limited wait has run out.  (Words in the workspace, copied out after every call, cost 13 us of a training step of
// 107.)
__device__ int g_f32_status[4] = {0, 0, 0x7fc00000, 0};

// Waits with a limit and records `code` if it runs out; the waits after one that ran out have a shorter limit, so that a
// kernel whose copies never arrive ends.  (Out of line: inline, the scans' code gets worse, and B2 T1000 H8 K=V=128 forward
// and backward takes 683 us instead of 630.)
__device__ __noinline__ void wait_or_record(uint64_t* bar, uint32_t parity, int code) {
    const bool lost = *reinterpret_cast<volatile int*>(&g_f32_status[0]) != 0;
    if (!sm100::mbar_wait(bar, parity, lost ? 200000 : sm100::kWaitBudgetNs)) atomicExch(&g_f32_status[0], code);
}
__device__ __forceinline__ void wait_copy(uint64_t* bar, uint32_t parity, int code) {
    if (!sm100::mbar_try_wait(bar, parity)) wait_or_record(bar, parity, code);
}
// before a CTA leaves: copies that were late when they were waited for have arrived, or are waited for once more
__device__ __forceinline__ void wait_late(uint64_t* bar, uint32_t parity) {
    if (*reinterpret_cast<volatile int*>(&g_f32_status[0]) != 0) wait_or_record(bar, parity, g_f32_status[0]);
}

// ------------------------------------------------------------------------------------------ workspace
// Per tile, padded to KP x VP channels: a record [WQ | KB | decay | A2 | M | Aak] with WQ = [w; qg], KB = [kg; bg] (48 x KP),
// A2 = [Aqk | Aqb] (16 x 48); UV = [v; u, replaced by v2] (48 x VP); state checkpoints; backward: dv2, dS, shares of dgl.
struct F32Plan {
    int KP, VP, NT, BH, nslice;
    long long G;
    long long rec, uv, h, dv2, dE, dglp;     // float offsets
    long long rec_floats;
    long long total_fwd, total;
};
int pad_dim(int d) { return d <= 64 ? 64 : 128; }
F32Plan make_f32_plan(const HdlaDims& d) {
    F32Plan p{};
    p.KP = pad_dim(d.K); p.VP = pad_dim(d.V);
    p.NT = (d.T + CT - 1) / CT;
    p.BH = d.B * d.H;
    p.G = (long long)p.BH * p.NT;
    p.nslice = p.VP / VS;
    p.rec_floats = 2 * RR * p.KP + p.KP + CT * RR + M2 * M2 + M2 * CT;
    long long off = 0;
    auto take = [&](long long n) { long long o = off; off += (n + 63) / 64 * 64; return o; };
    p.rec = take(p.rec_floats * p.G);
    p.uv = take((long long)RR * p.VP * p.G);
    p.total_fwd = off;
    p.h = take((long long)p.KP * p.VP * (p.NT + 1) * p.BH);
    p.dv2 = take((long long)M2 * p.VP * p.G);
    p.dE = take((long long)p.KP * p.VP * p.G);
    p.dglp = take((long long)p.KP * p.nslice * p.G);
    p.total = off;
    return p;
}

struct TileP {
    const void *q, *k, *v, *a, *b, *gk, *d_o;
    float *rec, *uv;
    const float *h, *dv2, *dE, *dglp;
    void *dq, *dk, *dv, *da, *db, *dgk;
    float scale;
    int T, H, K, V, NT, dt, gdt, nslice, vec_k, vec_v;
    long long rec_floats;
};

// Raw inputs of a tile in shared memory: q (scaled), k, a, b as [row][KP + 4], and gx[0] = 0, gx[i + 1] = inclusive decay sum
// of token i: ge_i = gx[i], gi_i = gx[i + 1].  Positions outside the sequence or the head's channels are zero.
template <int KP>
struct Raw {
    static constexpr int KS = KP + 4;
    float q[CT][KS], k[CT][KS], a[M2][KS], b[M2][KS], gx[CT + 1][KS];
};

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float a, float b, float c, float d) { *reinterpret_cast<float4*>(p) = make_float4(a, b, c, d); }

// Elements c .. c + N - 1 (N = 2 or 4) of the row of `lim` elements that starts at element `row`; zeros beyond it.  `vec`: rows
// are a multiple of four elements and aligned, so the group exists as a whole or not at all and moves in one access.
template <int N>
__device__ __forceinline__ void ld_row(float (&x)[N], const void* base, size_t row, int c, int lim, int dt, int vec) {
#pragma unroll
    for (int j = 0; j < N; ++j) x[j] = 0.f;
    if (c >= lim) return;
    if (!vec) {
#pragma unroll
        for (int j = 0; j < N; ++j) if (c + j < lim) x[j] = ld_elem(base, row + c + j, dt);
    } else if (dt == HDLA_F32) {
        const float* p = static_cast<const float*>(base) + row + c;
        if constexpr (N == 4) { const float4 t = ld4(p); x[0] = t.x; x[1] = t.y; x[2] = t.z; x[3] = t.w; }
        else { const float2 t = *reinterpret_cast<const float2*>(p); x[0] = t.x; x[1] = t.y; }
    } else {
        const __nv_bfloat16* p = static_cast<const __nv_bfloat16*>(base) + row + c;
        uint32_t w[N / 2];
        if constexpr (N == 4) { const uint2 t = *reinterpret_cast<const uint2*>(p); w[0] = t.x; w[1] = t.y; }
        else w[0] = *reinterpret_cast<const uint32_t*>(p);
#pragma unroll
        for (int j = 0; j < N / 2; ++j) { x[2 * j] = __uint_as_float(w[j] << 16); x[2 * j + 1] = __uint_as_float(w[j] & 0xffff0000u); }
    }
}
template <int N>
__device__ __forceinline__ void st_row(const float (&x)[N], void* base, size_t row, int c, int lim, int dt, int vec) {
    if (c >= lim) return;
    if (!vec) {
#pragma unroll
        for (int j = 0; j < N; ++j) if (c + j < lim) st_elem(base, row + c + j, dt, x[j]);
    } else if (dt == HDLA_F32) {
        float* p = static_cast<float*>(base) + row + c;
        if constexpr (N == 4) st4(p, x[0], x[1], x[2], x[3]);
        else *reinterpret_cast<float2*>(p) = make_float2(x[0], x[1]);
    } else {
        __nv_bfloat16* p = static_cast<__nv_bfloat16*>(base) + row + c;
        if constexpr (N == 4) *reinterpret_cast<uint2*>(p) = make_uint2(sm100::pack_bf16(x[0], x[1]), sm100::pack_bf16(x[2], x[3]));
        else *reinterpret_cast<uint32_t*>(p) = sm100::pack_bf16(x[0], x[1]);
    }
}

template <int KP>
__device__ __forceinline__ void load_raw(const TileP& p, Raw<KP>& s, int b, int h, int t0, int valid) {
    constexpr int NI = CT * (KP / 4) / 256;                   // groups of four channels per thread (256 threads)
    float x[NI][7][4];                                        // every load is issued before the first value is stored
#pragma unroll
    for (int it = 0; it < NI; ++it) {
        const int e = threadIdx.x + it * 256, i = e / (KP / 4), c = (e % (KP / 4)) * 4;
        const size_t tok = (size_t)b * p.T + t0 + min(i, valid - 1);
        const size_t src = (tok * p.H + h) * p.K, sa = (tok * 2 * p.H + h) * p.K, sb = sa + (size_t)p.H * p.K;
        const int lim = i < valid ? p.K : 0;
        ld_row<4>(x[it][0], p.q, src, c, lim, p.dt, p.vec_k);
        ld_row<4>(x[it][1], p.k, src, c, lim, p.dt, p.vec_k);
        ld_row<4>(x[it][2], p.gk, src, c, lim, p.gdt, p.vec_k);
        ld_row<4>(x[it][3], p.a, sa, c, lim, p.dt, p.vec_k);
        ld_row<4>(x[it][4], p.a, sb, c, lim, p.dt, p.vec_k);
        ld_row<4>(x[it][5], p.b, sa, c, lim, p.dt, p.vec_k);
        ld_row<4>(x[it][6], p.b, sb, c, lim, p.dt, p.vec_k);
    }
#pragma unroll
    for (int it = 0; it < NI; ++it) {
        const int e = threadIdx.x + it * 256, i = e / (KP / 4), c = (e % (KP / 4)) * 4;
        auto put = [&](float* dst, const float (&y)[4], float f) { st4(dst + c, f * y[0], f * y[1], f * y[2], f * y[3]); };
        put(s.q[i], x[it][0], p.scale); put(s.k[i], x[it][1], 1.f); put(s.gx[i + 1], x[it][2], 1.f);
        put(s.a[2 * i], x[it][3], 1.f); put(s.a[2 * i + 1], x[it][4], 1.f);
        put(s.b[2 * i], x[it][5], 1.f); put(s.b[2 * i + 1], x[it][6], 1.f);
    }
    __syncthreads();
    if (threadIdx.x < KP) {
        float run = 0.f, g[CT];
#pragma unroll
        for (int i = 0; i < CT; ++i) g[i] = s.gx[i + 1][threadIdx.x];
        s.gx[0][threadIdx.x] = 0.f;
#pragma unroll
        for (int i = 0; i < CT; ++i) { run += g[i]; s.gx[i + 1][threadIdx.x] = run; }
    }
    __syncthreads();
}

// ------------------------------------------------------------------------------------------ tile_fwd
// One thread per token pair (i, j) computes the nine scores between {q_i, a_i0, a_i1} and {k_j, b_j0, b_j1}: they share
// the two exponentials per channel.
template <int KP, int VP>
struct FwdSmem {
    Raw<KP> x;
    float v[CT][VP + 4], P[M2][VP + 4];
    float A[RR][52];                         // scores: rows q_i, then a_{i,r}; columns k_j, then b_{j,r}
    float MT[M2][M2 + 4];                    // M transposed: MT[c][r]
};

template <int KP, int VP>
__global__ void __launch_bounds__(256) f32_tile_fwd_kernel(TileP p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    FwdSmem<KP, VP>& s = *reinterpret_cast<FwdSmem<KP, VP>*>(smem_raw);
    const long long g = blockIdx.x;
    const int bh = (int)(g / p.NT), n = (int)(g % p.NT);
    const int b = bh / p.H, h = bh % p.H;
    const int t0 = n * CT, valid = min(CT, p.T - t0);
    const int tid = threadIdx.x;
    float* rec = p.rec + g * p.rec_floats;
    float* uv = p.uv + g * RR * VP;
    for (int e = tid; e < CT * (VP / 4); e += 256) {
        const int i = e / (VP / 4), c = (e % (VP / 4)) * 4;
        float x[4];
        ld_row<4>(x, p.v, (((size_t)b * p.T + t0 + min(i, valid - 1)) * p.H + h) * p.V, c, i < valid ? p.V : 0, p.dt, p.vec_v);
        st4(&s.v[i][c], x[0], x[1], x[2], x[3]);
        st4(uv + i * VP + c, x[0], x[1], x[2], x[3]);
    }
    load_raw<KP>(p, s.x, b, h, t0, valid);
    {   // scores
        const int i = tid >> 4, j = tid & 15;
        float acc[3][3] = {};
        if (j <= i) {
#pragma unroll 2
            for (int c = 0; c < KP; c += 4) {
                const float4 gi = ld4(&s.x.gx[i + 1][c]), ge = ld4(&s.x.gx[i][c]), gj = ld4(&s.x.gx[j + 1][c]);
                const float4 xq = ld4(&s.x.q[i][c]), x0 = ld4(&s.x.a[2 * i][c]), x1 = ld4(&s.x.a[2 * i + 1][c]);
                const float4 yk = ld4(&s.x.k[j][c]), y0 = ld4(&s.x.b[2 * j][c]), y1 = ld4(&s.x.b[2 * j + 1][c]);
                auto step = [&](float gi_, float ge_, float gj_, float q, float a0, float a1, float k, float b0, float b1) {
                    const float e1 = __expf(gi_ - gj_), e2 = j < i ? __expf(ge_ - gj_) : 0.f;
                    q *= e1; a0 *= e2; a1 *= e2;
                    acc[0][0] = fmaf(q, k, acc[0][0]);  acc[0][1] = fmaf(q, b0, acc[0][1]);  acc[0][2] = fmaf(q, b1, acc[0][2]);
                    acc[1][0] = fmaf(a0, k, acc[1][0]); acc[1][1] = fmaf(a0, b0, acc[1][1]); acc[1][2] = fmaf(a0, b1, acc[1][2]);
                    acc[2][0] = fmaf(a1, k, acc[2][0]); acc[2][1] = fmaf(a1, b0, acc[2][1]); acc[2][2] = fmaf(a1, b1, acc[2][2]);
                };
                step(gi.x, ge.x, gj.x, xq.x, x0.x, x1.x, yk.x, y0.x, y1.x);
                step(gi.y, ge.y, gj.y, xq.y, x0.y, x1.y, yk.y, y0.y, y1.y);
                step(gi.z, ge.z, gj.z, xq.z, x0.z, x1.z, yk.z, y0.z, y1.z);
                step(gi.w, ge.w, gj.w, xq.w, x0.w, x1.w, yk.w, y0.w, y1.w);
            }
        }
        const int rows[3] = {i, CT + 2 * i, CT + 2 * i + 1}, cols[3] = {j, CT + 2 * j, CT + 2 * j + 1};
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c) s.A[rows[r]][cols[c]] = acc[r][c];
    }
    __syncthreads();
    // record parts that need no further products; ag = a e^{ge} replaces a
    for (int e = tid; e < CT * (KP / 4); e += 256) {
        const int i = e / (KP / 4), c = (e % (KP / 4)) * 4;
        const float4 gi = ld4(&s.x.gx[i + 1][c]), ge = ld4(&s.x.gx[i][c]), gl = ld4(&s.x.gx[CT][c]);
        const float4 ei = make_float4(__expf(gi.x), __expf(gi.y), __expf(gi.z), __expf(gi.w));
        const float4 ee = make_float4(__expf(ge.x), __expf(ge.y), __expf(ge.z), __expf(ge.w));
        const float4 el = make_float4(__expf(gl.x - gi.x), __expf(gl.y - gi.y), __expf(gl.z - gi.z), __expf(gl.w - gi.w));
        auto mul = [](float4 x, float4 y) { return make_float4(x.x * y.x, x.y * y.y, x.z * y.z, x.w * y.w); };
        float4* wq = reinterpret_cast<float4*>(rec + (M2 + i) * KP + c);
        float4* kb = reinterpret_cast<float4*>(rec + RR * KP);
        *wq = mul(ld4(&s.x.q[i][c]), ei);
        kb[(i * KP + c) / 4] = mul(ld4(&s.x.k[i][c]), el);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            kb[((CT + 2 * i + r) * KP + c) / 4] = mul(ld4(&s.x.b[2 * i + r][c]), el);
            *reinterpret_cast<float4*>(&s.x.a[2 * i + r][c]) = mul(ld4(&s.x.a[2 * i + r][c]), ee);
        }
        if (i == 0)
            *reinterpret_cast<float4*>(rec + 2 * RR * KP + c) = make_float4(__expf(gl.x), __expf(gl.y), __expf(gl.z), __expf(gl.w));
    }
    float* rA2 = rec + 2 * RR * KP + KP;
    for (int e = tid; e < CT * RR; e += 256) rA2[e] = s.A[e / RR][e % RR];
    for (int e = tid; e < M2 * CT; e += 256) rA2[CT * RR + M2 * M2 + e] = s.A[CT + e / CT][e % CT];
    if (tid < 32) {
        // M = (I - Aab)^-1 by forward substitution: lane = column, its entries in registers
        float m[M2];
#pragma unroll
        for (int i = 0; i < M2; ++i) {
            float acc0 = i == tid ? 1.f : 0.f, acc1 = 0.f;
#pragma unroll
            for (int j = 0; j < M2; j += 4)
                if (j < i) {
                    const float4 l = ld4(&s.A[CT + i][CT + j]);          // (entries at or right of the diagonal are zero)
                    acc0 = fmaf(l.x, m[j], acc0);
                    if (j + 1 < i) acc1 = fmaf(l.y, m[j + 1], acc1);
                    if (j + 2 < i) acc0 = fmaf(l.z, m[j + 2], acc0);
                    if (j + 3 < i) acc1 = fmaf(l.w, m[j + 3], acc1);
                }
            m[i] = acc0 + acc1;
        }
#pragma unroll
        for (int i = 0; i < M2; i += 4) st4(&s.MT[tid][i], m[i], m[i + 1], m[i + 2], m[i + 3]);
        float* rM = rA2 + CT * RR;                                       // row-major M
#pragma unroll
        for (int i = 0; i < M2; ++i) rM[i * M2 + tid] = m[i];
    } else {
        for (int e = tid - 32; e < M2 * (VP / 4); e += 224) {            // P = Aak v
            const int r = e / (VP / 4), c = (e % (VP / 4)) * 4;
            float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int j = 0; j < (r >> 1); ++j) {
                const float x = s.A[CT + r][j];
                const float4 y = ld4(&s.v[j][c]);
                acc.x = fmaf(x, y.x, acc.x); acc.y = fmaf(x, y.y, acc.y); acc.z = fmaf(x, y.z, acc.z); acc.w = fmaf(x, y.w, acc.w);
            }
            *reinterpret_cast<float4*>(&s.P[r][c]) = acc;
        }
    }
    __syncthreads();
    // [w | u] = M [ag | P]: a thread owns 8 rows x 4 columns
    for (int e = tid; e < 4 * ((KP + VP) / 4); e += 256) {
        const int rg = e / ((KP + VP) / 4), cg = (e % ((KP + VP) / 4)) * 4;
        const bool is_w = cg < KP;
        float4 acc[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int j = 0; j < rg * 8 + 8; ++j) {                           // M is lower triangular
            const float4 y = is_w ? ld4(&s.x.a[j][cg]) : ld4(&s.P[j][cg - KP]);
            const float4 m0 = ld4(&s.MT[j][rg * 8]), m1 = ld4(&s.MT[j][rg * 8 + 4]);
            const float m[8] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                acc[i].x = fmaf(m[i], y.x, acc[i].x); acc[i].y = fmaf(m[i], y.y, acc[i].y);
                acc[i].z = fmaf(m[i], y.z, acc[i].z); acc[i].w = fmaf(m[i], y.w, acc[i].w);
            }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int r = rg * 8 + i;
            if (is_w) *reinterpret_cast<float4*>(rec + r * KP + cg) = acc[i];
            else *reinterpret_cast<float4*>(uv + (CT + r) * VP + cg - KP) = acc[i];
        }
    }
}

// ------------------------------------------------------------------------------------------ scans
// One CTA of 128 threads per (batch, head, 16 state columns); the columns do not depend on each other.  The state
// lives in registers (thread = 4 rows x KP / 32 columns) and, transposed, in shared memory for the product that
// contracts over its rows; the next tile's record arrives by one bulk copy while the current one is worked on.
struct ScanP {
    const float* rec;
    float* uv;                   // fwd: u in, v2 out (with `save`)
    const void* d_o;             // rev
    const float* init;           // h0 / dht, public dims, may be null
    float* fin;                  // final state / dh0, public dims, may be null
    float* h;                    // checkpoints, NT + 1 slots per (batch, head): fwd writes (with `save`), rev reads
    float *dv2, *dE, *dglp;      // rev
    void* o;                     // fwd, may be null
    int T, H, K, V, VP, NT, dt, nslice, save;
    long long rec_floats;
};

template <int KP>
struct ScanSmem {
    static constexpr int kRec = 2 * RR * KP + KP + CT * RR;              // floats of a record that the scans read
    float rec[2][kRec];
    float ST[VS][KP + 4];        // the state, transposed
    float vv[RR][VS + 4];        // fwd: v, v2; rev: dv2, dO
    float vT[VS][RR + 4];        // the same, transposed
    float red[8][KP];
    uint64_t bar[2];
};

// (three CTAs to an SM are what shared memory leaves room for with KP = 64; without the bound the compiler aims at four and
// spills, which cost 91 instead of 85 us for B2 T256 H4 K=V=64 forward and backward)
template <int KP, bool REV>
__global__ void __launch_bounds__(128, 3) f32_scan_kernel(ScanP p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    typedef ScanSmem<KP> Sm;
    Sm& s = *reinterpret_cast<Sm*>(smem_raw);
    constexpr int VPT = KP / 32;                 // columns per thread in the state update (4 k x VPT v)
    constexpr int KG = KP / 4;                   // groups of four rows
    constexpr int NA = REV ? 4 : 6;              // rows per thread of the row product: 32 (dv2) or 48 (v2, qg S)
    const int bh = blockIdx.x / p.nslice, c0 = (blockIdx.x % p.nslice) * VS;
    const int b = bh / p.H, hd = bh % p.H;
    const int tid = threadIdx.x;
    const int kg = (tid % KG) * 4, vg = (tid / KG) * VPT;               // state update: this thread's rows / columns
    const int ks = tid & 3, va = ((tid >> 2) & 3) * 4, rg = tid >> 4;   // row product: k split, column group, row rg + 8 i
    const int vcol = va + ((ks & 1) ? 2 : 0) + ((ks & 2) ? 1 : 0);      // the column whose sums this thread ends up with
    const long long g0 = (long long)bh * p.NT;
    if (tid == 0) {
        sm100::mbar_init(&s.bar[0], 1); sm100::mbar_init(&s.bar[1], 1);
        sm100::fence_mbar_init();
    }
    float S[4][VPT];                             // [row][column]
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int c = 0; c < VPT; ++c) {
            const int k = kg + j, v = c0 + vg + c;
            S[j][c] = (p.init && k < p.K && v < p.V) ? p.init[((size_t)bh * p.K + k) * p.V + v] : 0.f;
        }
    auto put_state = [&] {
#pragma unroll
        for (int c = 0; c < VPT; ++c) st4(&s.ST[vg + c][kg], S[0][c], S[1][c], S[2][c], S[3][c]);
    };
    put_state();
    __syncthreads();
    const int dn = REV ? -1 : 1, n_first = REV ? p.NT - 1 : 0;
    auto request = [&](int it) {
        const uint32_t bytes = Sm::kRec * 4;
        sm100::mbar_expect_tx(&s.bar[it & 1], bytes);
        sm100::bulk_g2s(s.rec[it & 1], p.rec + (g0 + n_first + it * dn) * p.rec_floats, bytes, &s.bar[it & 1]);
    };
    if (tid == 0) { request(0); if (p.NT > 1) request(1); }
    // values of the next tile that go through registers: two of the 16 x 16 slice of v / dO, and u
    const int er = tid >> 3, ec = (tid & 7) * 2;
    float nx[2], nu[4];
    auto fetch = [&](int n) {
        const long long g = g0 + n;
        const int t = n * CT + er;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            if (REV) {
                const int v = c0 + ec + e;
                nx[e] = (t < p.T && v < p.V) ? ld_elem(p.d_o, (((size_t)b * p.T + t) * p.H + hd) * p.V + v, p.dt) : 0.f;
            } else {
                nx[e] = p.uv[(g * RR + er) * p.VP + c0 + ec + e];
            }
        }
        if (!REV)
#pragma unroll
            for (int i = 0; i < 4; ++i) nu[i] = p.uv[(g * RR + CT + rg + 8 * i) * p.VP + c0 + vcol];
    };
    fetch(n_first);
    for (int it = 0; it < p.NT; ++it) {
        const int n = n_first + it * dn;
        const long long g = g0 + n;
        const float* rec = s.rec[it & 1];
        const float *WQ = rec, *KB = rec + RR * KP, *dec = rec + 2 * RR * KP, *A2 = dec + KP;
        constexpr int vrow = REV ? M2 : 0;       // rows of vv that the slice of v / dO takes
#pragma unroll
        for (int e = 0; e < 2; ++e) { s.vv[vrow + er][ec + e] = nx[e]; s.vT[ec + e][vrow + er] = nx[e]; }
        float u[4] = {nu[0], nu[1], nu[2], nu[3]};
        // (an output of this tile overwrites u: the next fetch reads other addresses)
        if (it + 1 < p.NT) fetch(n + dn);
        float4 hn[VPT];                          // rev: the state after this tile, for the decay gradient
#pragma unroll
        for (int c = 0; c < VPT; ++c) {          // (checkpoints are kept transposed: [v][k])
            const size_t at = (size_t)(c0 + vg + c) * KP + kg;
            if (REV) hn[c] = ld4(p.h + ((size_t)bh * (p.NT + 1) + n + 1) * KP * p.VP + at);
            if (REV) st4(p.dE + (size_t)g * KP * p.VP + at, S[0][c], S[1][c], S[2][c], S[3][c]);
            else if (p.save) st4(p.h + ((size_t)bh * (p.NT + 1) + n) * KP * p.VP + at, S[0][c], S[1][c], S[2][c], S[3][c]);
        }
        wait_copy(&s.bar[it & 1], (it >> 1) & 1, 90 + REV);
        // row product over the state's rows: fwd [w; qg] S, rev bg dS
        f2 acc[NA][4];
#pragma unroll
        for (int i = 0; i < NA; ++i)
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[i][c] = 0ull;
        const float* rows = REV ? KB + CT * KP : WQ;
#pragma unroll
        for (int j = 0; j < KP / 16; ++j) {
            const int k = j * 16 + ks * 4;
            ulonglong2 y[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) y[c] = *reinterpret_cast<const ulonglong2*>(&s.ST[va + c][k]);
#pragma unroll
            for (int i = 0; i < NA; ++i) {
                const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(rows + (rg + 8 * i) * KP + k);
#pragma unroll
                for (int c = 0; c < 4; ++c) acc[i][c] = f2_fma(x.y, y[c].y, f2_fma(x.x, y[c].x, acc[i][c]));
            }
        }
        float r[NA];
#pragma unroll
        for (int i = 0; i < NA; ++i) {           // sum over the four k splits, scattering the columns over them
            float f[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) f[c] = f2_sum(acc[i][c]);
            const bool u1 = ks & 1, u2 = ks & 2;
            const float g0_ = u1 ? f[0] : f[2], g1_ = u1 ? f[1] : f[3];
            float k0 = (u1 ? f[2] : f[0]) + __shfl_xor_sync(0xffffffffu, g0_, 1);
            float k1 = (u1 ? f[3] : f[1]) + __shfl_xor_sync(0xffffffffu, g1_, 1);
            r[i] = (u2 ? k1 : k0) + __shfl_xor_sync(0xffffffffu, u2 ? k0 : k1, 2);
        }
        if (REV) {                               // dv2 += Aqb^T dO (the slice of dO was written before the barrier below)
            __syncthreads();
            float x[CT];
#pragma unroll
            for (int t = 0; t < CT; t += 4) {
                const float4 y = ld4(&s.vT[vcol][M2 + t]);
                x[t] = y.x; x[t + 1] = y.y; x[t + 2] = y.z; x[t + 3] = y.w;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int t = 0; t < CT; ++t) r[i] = fmaf(A2[t * RR + CT + rg + 8 * i], x[t], r[i]);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int row = rg + 8 * i;
            if (!REV) r[i] += u[i];
            s.vv[(REV ? 0 : CT) + row][vcol] = r[i];
            s.vT[vcol][(REV ? 0 : CT) + row] = r[i];
            if (REV) p.dv2[((size_t)g * M2 + row) * p.VP + c0 + vcol] = r[i];
            else if (p.save) p.uv[((size_t)g * RR + CT + row) * p.VP + c0 + vcol] = r[i];
        }
        if (REV) {                               // this slice's share of dgl = rowsum(dS (.) S_{n+1})
            float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int c = 0; c < VPT; ++c) {
                x.x = fmaf(S[0][c], hn[c].x, x.x); x.y = fmaf(S[1][c], hn[c].y, x.y);
                x.z = fmaf(S[2][c], hn[c].z, x.z); x.w = fmaf(S[3][c], hn[c].w, x.w);
            }
            *reinterpret_cast<float4*>(&s.red[tid / KG][kg]) = x;
        }
        __syncthreads();
        if (REV && tid < KP) {
            float x = 0.f;
#pragma unroll
            for (int w = 0; w < 128 / KG; ++w) x += s.red[w][tid];
            p.dglp[((size_t)g * p.nslice + blockIdx.x % p.nslice) * KP + tid] = x;
        }
        // state update: S <- decay (.) S + rows^T vv
        {
            const float4 d4 = ld4(dec + kg);
            f2 x[VPT][2];
#pragma unroll
            for (int c = 0; c < VPT; ++c) {
                x[c][0] = f2_pack(d4.x * S[0][c], d4.y * S[1][c]);
                x[c][1] = f2_pack(d4.z * S[2][c], d4.w * S[3][c]);
            }
            const float* up = (REV ? WQ : KB) + kg;
#pragma unroll 8
            for (int q = 0; q < RR; ++q) {
                const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(up + q * KP);
                float w[VPT];
                if constexpr (VPT == 4) {
                    const float4 t = ld4(&s.vv[q][vg]);
                    w[0] = t.x; w[1] = t.y; w[2] = t.z; w[3] = t.w;
                } else {
                    const float2 t = *reinterpret_cast<const float2*>(&s.vv[q][vg]);
                    w[0] = t.x; w[1] = t.y;
                }
#pragma unroll
                for (int c = 0; c < VPT; ++c) {
                    const f2 d = f2_dup(w[c]);
                    x[c][0] = f2_fma(y.x, d, x[c][0]);
                    x[c][1] = f2_fma(y.y, d, x[c][1]);
                }
            }
#pragma unroll
            for (int c = 0; c < VPT; ++c) { f2_unpack(x[c][0], S[0][c], S[1][c]); f2_unpack(x[c][1], S[2][c], S[3][c]); }
        }
        if (!REV && p.o) {                       // o = qg S + [Aqk | Aqb] [v; v2]: rows rg, rg + 8 of column vcol
            f2 o0 = 0ull, o1 = 0ull;
#pragma unroll
            for (int q = 0; q < RR; q += 4) {
                const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(&s.vT[vcol][q]);
                const ulonglong2 a0 = *reinterpret_cast<const ulonglong2*>(A2 + rg * RR + q);
                const ulonglong2 a1 = *reinterpret_cast<const ulonglong2*>(A2 + (rg + 8) * RR + q);
                o0 = f2_fma(a0.y, y.y, f2_fma(a0.x, y.x, o0));
                o1 = f2_fma(a1.y, y.y, f2_fma(a1.x, y.x, o1));
            }
            const int v = c0 + vcol;
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int t = n * CT + rg + 8 * e;
                if (t < p.T && v < p.V)
                    st_elem(p.o, (((size_t)b * p.T + t) * p.H + hd) * p.V + v, p.dt, r[NA - 2 + e] + f2_sum(e ? o1 : o0));
            }
        }
        put_state();
        __syncthreads();                         // state, vv and this record buffer are free / complete
        if (tid == 0 && it + 2 < p.NT) request(it + 2);
    }
    if (tid == 0)
        for (int it = max(p.NT - 2, 0); it < p.NT; ++it) wait_late(&s.bar[it & 1], (it >> 1) & 1);
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int c = 0; c < VPT; ++c) {
            const int k = kg + j, v = c0 + vg + c;
            if (p.fin && k < p.K && v < p.V) p.fin[((size_t)bh * p.K + k) * p.V + v] = S[j][c];
            if (!REV && p.save) p.h[(((size_t)bh * (p.NT + 1) + p.NT) * p.VP + v) * KP + k] = S[j][c];
        }
}

// ------------------------------------------------------------------------------------------ tile_bwd
// Warp w owns the tokens 2w and 2w + 1 and a lane KP / 32 adjacent channels, for everything: the state's shares Y S^T and
// Z dS^T, the gated score shares and the un-gating stay in the same thread's registers, up to the decay gradient's
// running sum over the tokens.
template <int KP, int VP>
struct BwdSmem {
    union {
        struct { float S[VP][KP + 4], dE[VP][KP + 4]; } st;          // transposed, as the scans keep them
        Raw<KP> x;
    };
    float Y[RR][VP + 4], Z[RR][VP + 4];      // [dO; dv2, then dP], [v; v2];  Y later: decay gradient terms [16][KP + 4]
    float dA[RR][52];
    float M[M2][M2 + 4];
    uint64_t bar;
};

template <int N>
__device__ __forceinline__ void ld_sm(float (&x)[N], const float* p) {       // N = 2 or 4 adjacent floats
    if constexpr (N == 4) { const float4 t = ld4(p); x[0] = t.x; x[1] = t.y; x[2] = t.z; x[3] = t.w; }
    else { const float2 t = *reinterpret_cast<const float2*>(p); x[0] = t.x; x[1] = t.y; }
}

template <int KP, int VP>
__global__ void __launch_bounds__(256, KP == 128 ? 1 : 2) f32_tile_bwd_kernel(TileP p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    BwdSmem<KP, VP>& s = *reinterpret_cast<BwdSmem<KP, VP>*>(smem_raw);
    constexpr int CPT = KP / 32;
    const long long g = blockIdx.x;
    const int bh = (int)(g / p.NT), n = (int)(g % p.NT);
    const int b = bh / p.H, h = bh % p.H;
    const int t0 = n * CT, valid = min(CT, p.T - t0);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const float* rec = p.rec + g * p.rec_floats;
    const float *KB = rec + RR * KP, *A2 = rec + 2 * RR * KP + KP, *rM = A2 + CT * RR, *rAak = rM + M2 * M2;
    if (tid == 0) { sm100::mbar_init(&s.bar, 1); sm100::fence_mbar_init(); }
    __syncthreads();
    if (tid == 0) sm100::mbar_expect_tx(&s.bar, 2 * VP * KP * 4 + (RR + M2) * VP * 4);
    __syncthreads();
    {   // rows of the padded tiles, one bulk copy each
        const float* S = p.h + ((size_t)bh * (p.NT + 1) + n) * KP * VP;
        const float* dE = p.dE + (size_t)g * KP * VP;
        for (int r = tid; r < 2 * VP + RR + M2; r += 256) {
            if (r < VP) sm100::bulk_g2s(s.st.S[r], S + (size_t)r * KP, KP * 4, &s.bar);
            else if (r < 2 * VP) sm100::bulk_g2s(s.st.dE[r - VP], dE + (size_t)(r - VP) * KP, KP * 4, &s.bar);
            else if (r < 2 * VP + RR) sm100::bulk_g2s(s.Z[r - 2 * VP], p.uv + ((size_t)g * RR + r - 2 * VP) * VP, VP * 4, &s.bar);
            else sm100::bulk_g2s(s.Y[CT + r - 2 * VP - RR], p.dv2 + ((size_t)g * M2 + r - 2 * VP - RR) * VP, VP * 4, &s.bar);
        }
    }
    for (int e = tid; e < CT * (VP / 4); e += 256) {
        const int i = e / (VP / 4), c = (e % (VP / 4)) * 4;
        float x[4];
        ld_row<4>(x, p.d_o, (((size_t)b * p.T + t0 + min(i, valid - 1)) * p.H + h) * p.V, c, i < valid ? p.V : 0, p.dt, p.vec_v);
        st4(&s.Y[i][c], x[0], x[1], x[2], x[3]);
    }
    for (int e = tid; e < M2 * M2; e += 256) s.M[e / M2][e % M2] = rM[e];
    wait_copy(&s.bar, 0, 92);
    __syncthreads();
    {   // dP = M^T dv2, in place
        constexpr int VG = VP / 4, NR = M2 * VG / 256;
        const int c = (tid % VG) * 4, r0 = (tid / VG) * NR;
        float4 acc[NR];
#pragma unroll
        for (int i = 0; i < NR; ++i) acc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int r = r0; r < M2; ++r) {
            const float4 y = ld4(&s.Y[CT + r][c]);
#pragma unroll
            for (int i = 0; i < NR; ++i) {
                const float m = s.M[r][r0 + i];
                acc[i].x = fmaf(m, y.x, acc[i].x); acc[i].y = fmaf(m, y.y, acc[i].y);
                acc[i].z = fmaf(m, y.z, acc[i].z); acc[i].w = fmaf(m, y.w, acc[i].w);
            }
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < NR; ++i) *reinterpret_cast<float4*>(&s.Y[CT + r0 + i][c]) = acc[i];
    }
    __syncthreads();
    {   // dA = mask(Y Z^T), thread = token pair
        const int i = tid >> 4, j = tid & 15;
        const int rows[3] = {i, CT + 2 * i, CT + 2 * i + 1}, cols[3] = {j, CT + 2 * j, CT + 2 * j + 1};
        f2 acc[3][3];
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c) acc[r][c] = 0ull;
        if (j <= i)
#pragma unroll 4
            for (int v = 0; v < VP; v += 4) {
                ulonglong2 x[3], y[3];
#pragma unroll
                for (int r = 0; r < 3; ++r) {
                    x[r] = *reinterpret_cast<const ulonglong2*>(&s.Y[rows[r]][v]);
                    y[r] = *reinterpret_cast<const ulonglong2*>(&s.Z[cols[r]][v]);
                }
#pragma unroll
                for (int r = 0; r < 3; ++r)
#pragma unroll
                    for (int c = 0; c < 3; ++c) acc[r][c] = f2_fma(x[r].y, y[c].y, f2_fma(x[r].x, y[c].x, acc[r][c]));
            }
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c) s.dA[rows[r]][cols[c]] = (r == 0 || j < i) ? f2_sum(acc[r][c]) : 0.f;
    }
    // state shares: rows q_i, a_i0, a_i1 of Y S^T and k_i, b_i0, b_i1 of Z dS^T for this warp's tokens
    float dX[2][3][CPT], dW[2][3][CPT];
    const int ch = lane * CPT;                                   // this lane's first channel
    auto state_share = [&](const float (*L)[VP + 4], const float (*R)[KP + 4], float (&out)[2][3][CPT]) {
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
            for (int r = 0; r < 3; ++r)
#pragma unroll
                for (int c = 0; c < CPT; ++c) out[t][r][c] = 0.f;
#pragma unroll 2
        for (int v = 0; v < VP; v += 4) {
            float y[4][CPT];
#pragma unroll
            for (int e = 0; e < 4; ++e) ld_sm<CPT>(y[e], &R[v + e][ch]);
#pragma unroll
            for (int t = 0; t < 2; ++t)
#pragma unroll
                for (int r = 0; r < 3; ++r) {
                    const int i = 2 * warp + t;
                    const float4 x = ld4(&L[r == 0 ? i : CT + 2 * i + r - 1][v]);
#pragma unroll
                    for (int c = 0; c < CPT; ++c)
                        out[t][r][c] = fmaf(x.w, y[3][c], fmaf(x.z, y[2][c], fmaf(x.y, y[1][c], fmaf(x.x, y[0][c], out[t][r][c]))));
                }
        }
    };
    state_share(s.Y, s.st.S, dX);
    state_share(s.Z, s.st.dE, dW);
    {   // dv = kg dS + Aqk^T dO + Aak^T dP: this warp's tokens, columns lane + 32 e
        constexpr int NV = VP / 32;
        f2 acc[2][NV];
        float sum[2][NV];
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
            for (int e = 0; e < NV; ++e) acc[t][e] = 0ull;
        const float *k0 = KB + (2 * warp) * KP, *k1 = k0 + KP;
#pragma unroll 4
        for (int k = 0; k < KP; k += 4) {
            const ulonglong2 x0 = __ldg(reinterpret_cast<const ulonglong2*>(k0 + k)), x1 = __ldg(reinterpret_cast<const ulonglong2*>(k1 + k));
#pragma unroll
            for (int e = 0; e < NV; ++e) {
                const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(&s.st.dE[lane + 32 * e][k]);
                acc[0][e] = f2_fma(x0.y, y.y, f2_fma(x0.x, y.x, acc[0][e]));
                acc[1][e] = f2_fma(x1.y, y.y, f2_fma(x1.x, y.x, acc[1][e]));
            }
        }
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
            for (int e = 0; e < NV; ++e) sum[t][e] = f2_sum(acc[t][e]);
#pragma unroll 8
        for (int r = 0; r < RR; ++r) {
            const float2 x = __ldg(reinterpret_cast<const float2*>((r < CT ? A2 + r * RR : rAak + (r - CT) * CT) + 2 * warp));
#pragma unroll
            for (int e = 0; e < NV; ++e) {
                const float y = s.Y[r][lane + 32 * e];
                sum[0][e] = fmaf(x.x, y, sum[0][e]); sum[1][e] = fmaf(x.y, y, sum[1][e]);
            }
        }
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
            for (int e = 0; e < NV; ++e)
                if (2 * warp + t < valid && lane + 32 * e < p.V)
                    st_elem(p.dv, (((size_t)b * p.T + t0 + 2 * warp + t) * p.H + h) * p.V + lane + 32 * e, p.dt, sum[t][e]);
    }
    __syncthreads();                                             // the states have been read: the raw inputs take their place
    load_raw<KP>(p, s.x, b, h, t0, valid);
#pragma unroll
    for (int t = 0; t < 2; ++t)                                  // un-gate the state shares
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
            const int i = 2 * warp + t;
            const float gi = s.x.gx[i + 1][ch + c], ei = __expf(gi), ee = __expf(s.x.gx[i][ch + c]), el = __expf(s.x.gx[CT][ch + c] - gi);
            dX[t][0][c] *= ei; dX[t][1][c] *= ee; dX[t][2][c] *= ee;
            dW[t][0][c] *= el; dW[t][1][c] *= el; dW[t][2][c] *= el;
        }
    // score shares of the rows: tokens j <= i
    for (int j = 0; j <= 2 * warp + 1; ++j) {
        float y[3][CPT], gj[CPT];
        ld_sm<CPT>(y[0], &s.x.k[j][ch]); ld_sm<CPT>(y[1], &s.x.b[2 * j][ch]); ld_sm<CPT>(y[2], &s.x.b[2 * j + 1][ch]);
        ld_sm<CPT>(gj, &s.x.gx[j + 1][ch]);
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            const int i = 2 * warp + t;
            if (j > i) continue;
            float co[3][3];
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                const int row = r == 0 ? i : CT + 2 * i + r - 1;
                co[r][0] = s.dA[row][j];
                const float2 x = *reinterpret_cast<const float2*>(&s.dA[row][CT + 2 * j]);
                co[r][1] = x.x; co[r][2] = x.y;
            }
            float gi[CPT], ge[CPT];
            ld_sm<CPT>(gi, &s.x.gx[i + 1][ch]); ld_sm<CPT>(ge, &s.x.gx[i][ch]);
#pragma unroll
            for (int c = 0; c < CPT; ++c) {
                const float e1 = __expf(gi[c] - gj[c]), e2 = j < i ? __expf(ge[c] - gj[c]) : 0.f;
#pragma unroll
                for (int r = 0; r < 3; ++r)
                    dX[t][r][c] = fmaf(r == 0 ? e1 : e2, fmaf(co[r][0], y[0][c], fmaf(co[r][1], y[1][c], co[r][2] * y[2][c])), dX[t][r][c]);
            }
        }
    }
    // score shares of the columns: tokens i >= j
    for (int i = 2 * warp; i < CT; ++i) {
        float x[3][CPT], gi[CPT], ge[CPT];
        ld_sm<CPT>(x[0], &s.x.q[i][ch]); ld_sm<CPT>(x[1], &s.x.a[2 * i][ch]); ld_sm<CPT>(x[2], &s.x.a[2 * i + 1][ch]);
        ld_sm<CPT>(gi, &s.x.gx[i + 1][ch]); ld_sm<CPT>(ge, &s.x.gx[i][ch]);
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            const int j = 2 * warp + t;
            if (i < j) continue;
            float co[3][3];
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                const int row = r == 0 ? i : CT + 2 * i + r - 1;
                co[r][0] = s.dA[row][j];
                const float2 y = *reinterpret_cast<const float2*>(&s.dA[row][CT + 2 * j]);
                co[r][1] = y.x; co[r][2] = y.y;
            }
            float gj[CPT];
            ld_sm<CPT>(gj, &s.x.gx[j + 1][ch]);
#pragma unroll
            for (int c = 0; c < CPT; ++c) {
                const float e1 = __expf(gi[c] - gj[c]), e2 = i > j ? __expf(ge[c] - gj[c]) : 0.f;
                const float xq = x[0][c] * e1, x0 = x[1][c] * e2, x1 = x[2][c] * e2;
#pragma unroll
                for (int r = 0; r < 3; ++r) dW[t][r][c] = fmaf(co[0][r], xq, fmaf(co[1][r], x0, fmaf(co[2][r], x1, dW[t][r][c])));
            }
        }
    }
    // gradients out, and the decay gradient's running sum over the tokens
    float (*D)[KP + 4] = reinterpret_cast<float (*)[KP + 4]>(&s.Y[0][0]);
    float dge[2][CPT];
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        const int i = 2 * warp + t;
        float q[CPT], k[CPT], a0[CPT], a1[CPT], b0[CPT], b1[CPT];
        ld_sm<CPT>(q, &s.x.q[i][ch]); ld_sm<CPT>(k, &s.x.k[i][ch]);
        ld_sm<CPT>(a0, &s.x.a[2 * i][ch]); ld_sm<CPT>(a1, &s.x.a[2 * i + 1][ch]);
        ld_sm<CPT>(b0, &s.x.b[2 * i][ch]); ld_sm<CPT>(b1, &s.x.b[2 * i + 1][ch]);
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
            dge[t][c] = a0[c] * dX[t][1][c] + a1[c] * dX[t][2][c];
            D[i][ch + c] = q[c] * dX[t][0][c] - k[c] * dW[t][0][c] - b0[c] * dW[t][1][c] - b1[c] * dW[t][2][c] + dge[t][c];
            dX[t][0][c] *= p.scale;
        }
        if (i < valid) {
            const size_t tok = (size_t)b * p.T + t0 + i;
            const size_t at = (tok * p.H + h) * p.K, r0 = (tok * 2 * p.H + h) * p.K, r1 = r0 + (size_t)p.H * p.K;
            st_row<CPT>(dX[t][0], p.dq, at, ch, p.K, p.dt, p.vec_k);
            st_row<CPT>(dW[t][0], p.dk, at, ch, p.K, p.dt, p.vec_k);
            st_row<CPT>(dX[t][1], p.da, r0, ch, p.K, p.dt, p.vec_k); st_row<CPT>(dX[t][2], p.da, r1, ch, p.K, p.dt, p.vec_k);
            st_row<CPT>(dW[t][1], p.db, r0, ch, p.K, p.dt, p.vec_k); st_row<CPT>(dW[t][2], p.db, r1, ch, p.K, p.dt, p.vec_k);
        }
    }
    __syncthreads();
    if (tid < KP) {
        float run = 0.f;                                         // the gradient of the chunk-end decay, from all slices ...
        for (int w = 0; w < p.nslice; ++w) run += p.dglp[((size_t)g * p.nslice + w) * KP + tid];
#pragma unroll
        for (int i = CT - 1; i >= 0; --i) { run += D[i][tid]; D[i][tid] = run; }      // ... and the running sum
    }
    __syncthreads();
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        const int i = 2 * warp + t;
        float x[CPT];
#pragma unroll
        for (int c = 0; c < CPT; ++c) x[c] = D[i][ch + c] - dge[t][c];
        if (i < valid) st_row<CPT>(x, p.dgk, (((size_t)b * p.T + t0 + i) * p.H + h) * p.K, ch, p.K, p.gdt, p.vec_k);
    }
    if (tid == 0) wait_late(&s.bar, 0);
}

// ------------------------------------------------------------------------------------------ host side
template <typename Kern>
int allow_smem(Kern kern, size_t bytes) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return fail(HDLA_ERR_CUDA, "cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    return HDLA_OK;
}

#define TRY(x) do { int rc__ = (x); if (rc__ != HDLA_OK) return rc__; } while (0)

template <int KP, int VP>
int set_attributes() {
    static thread_local int attr_dev = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (attr_dev == dev) return HDLA_OK;
    TRY(allow_smem(f32_tile_fwd_kernel<KP, VP>, sizeof(FwdSmem<KP, VP>)));
    TRY(allow_smem(f32_tile_bwd_kernel<KP, VP>, sizeof(BwdSmem<KP, VP>)));
    TRY(allow_smem(f32_scan_kernel<KP, false>, sizeof(ScanSmem<KP>)));
    TRY(allow_smem(f32_scan_kernel<KP, true>, sizeof(ScanSmem<KP>)));
    attr_dev = dev;
    return HDLA_OK;
}

TileP tile_params(const HdlaDims& d, const F32Plan& pl, float* ws, const void* q, const void* k, const void* v,
                  const void* a, const void* b, const void* gk, float scale) {
    TileP p{};
    p.q = q; p.k = k; p.v = v; p.a = a; p.b = b; p.gk = gk;
    p.rec = ws + pl.rec; p.uv = ws + pl.uv; p.h = ws + pl.h; p.dv2 = ws + pl.dv2; p.dE = ws + pl.dE; p.dglp = ws + pl.dglp;
    p.scale = scale;
    p.T = d.T; p.H = d.H; p.K = d.K; p.V = d.V; p.NT = pl.NT; p.dt = d.dtype; p.gdt = d.gk_dtype; p.nslice = pl.nslice;
    p.rec_floats = pl.rec_floats;
    p.vec_k = d.K % 4 == 0; p.vec_v = d.V % 4 == 0;
    for (const void* x : {q, k, v, a, b, gk})
        if (reinterpret_cast<uintptr_t>(x) % 16 != 0) p.vec_k = p.vec_v = 0;
    return p;
}
ScanP scan_params(const HdlaDims& d, const F32Plan& pl, float* ws) {
    ScanP p{};
    p.rec = ws + pl.rec; p.uv = ws + pl.uv; p.h = ws + pl.h; p.dv2 = ws + pl.dv2; p.dE = ws + pl.dE; p.dglp = ws + pl.dglp;
    p.T = d.T; p.H = d.H; p.K = d.K; p.V = d.V; p.VP = pl.VP; p.NT = pl.NT; p.dt = d.dtype; p.nslice = pl.nslice;
    p.rec_floats = pl.rec_floats;
    return p;
}

template <int KP, int VP>
int fwd(const HdlaDims& d, const F32Plan& pl, const TileP& tp, ScanP sp, cudaStream_t st) {
    TRY((set_attributes<KP, VP>()));
    f32_tile_fwd_kernel<KP, VP><<<(unsigned)pl.G, 256, sizeof(FwdSmem<KP, VP>), st>>>(tp);
    HDLA_CHECK_LAUNCH("f32_tile_fwd_kernel");
    f32_scan_kernel<KP, false><<<(unsigned)(pl.BH * pl.nslice), 128, sizeof(ScanSmem<KP>), st>>>(sp);
    HDLA_CHECK_LAUNCH("f32_scan_kernel");
    return HDLA_OK;
}
template <int KP, int VP>
int bwd(const HdlaDims& d, const F32Plan& pl, const TileP& tp, ScanP sp, cudaStream_t st) {
    TRY((set_attributes<KP, VP>()));
    f32_scan_kernel<KP, true><<<(unsigned)(pl.BH * pl.nslice), 128, sizeof(ScanSmem<KP>), st>>>(sp);
    HDLA_CHECK_LAUNCH("f32_scan_kernel");
    f32_tile_bwd_kernel<KP, VP><<<(unsigned)pl.G, 256, sizeof(BwdSmem<KP, VP>), st>>>(tp);
    HDLA_CHECK_LAUNCH("f32_tile_bwd_kernel");
    return HDLA_OK;
}

}  // namespace

int f32_status_words(void** words) {
    const cudaError_t e = cudaGetSymbolAddress(words, g_f32_status);
    if (e != cudaSuccess) return fail(HDLA_ERR_CUDA, "fp32 status words: %s", cudaGetErrorString(e));
    return HDLA_OK;
}

// Rank 2, head dims up to 128; other problems stay on the general kernels of chunk_simt.cu.  So do large ones that would
// need more memory here than there: heads of a few channels, padded to 64, with a requested chunk of 16 (5.5 KB per token
// and head against 2.1 to 4.9 for K = V = 1 to 16; from 24 channels on, or with larger chunks, this pipeline needs less).
// They would fit a device there and not here, which no gain in time makes up for; up to kAlwaysBytes, a small part of any
// device that runs these kernels, the faster pipeline takes them (B4 T1024 H8 K = V = 16, chunk 16, fwd+bwd: 533 us in
// 173 MB against 2324 us in 152 MB).
constexpr size_t kAlwaysBytes = (size_t)4 << 30;
bool f32_supported(const HdlaDims& d) {
    const F32Plan pl = make_f32_plan(d);
    if (d.flags & kFlagGeneralKernels) return false;
    if (!(d.R == 2 && d.K <= 128 && d.V <= 128 && pl.G < 0x7fffffffLL && (long long)pl.BH * pl.nslice < 0x7fffffffLL))
        return false;
    return (size_t)pl.total * sizeof(float) <= kAlwaysBytes ||
           ((size_t)pl.total <= simt_workspace_floats(d, 1) && (size_t)pl.total_fwd <= simt_workspace_floats(d, 0));
}
size_t f32_workspace_floats(const HdlaDims& d, int with_backward) {
    const F32Plan pl = make_f32_plan(d);
    return (size_t)(with_backward ? pl.total : pl.total_fwd);
}

int f32_chunk_fwd(const HdlaDims& d, const void* q, const void* k, const void* v, const void* a, const void* b,
                  const void* gk, float scale, const float* h0, void* o, float* ht, float* ws, size_t ws_floats,
                  bool need_o, cudaStream_t st) {
    const F32Plan pl = make_f32_plan(d);
    const TileP tp = tile_params(d, pl, ws, q, k, v, a, b, gk, scale);
    ScanP sp = scan_params(d, pl, ws);
    sp.init = h0; sp.fin = ht; sp.o = need_o ? o : nullptr;
    sp.save = ws_floats >= (size_t)pl.total;         // a workspace sized for backward keeps what it reads
    if (pl.KP == 64) return pl.VP == 64 ? fwd<64, 64>(d, pl, tp, sp, st) : fwd<64, 128>(d, pl, tp, sp, st);
    return pl.VP == 64 ? fwd<128, 64>(d, pl, tp, sp, st) : fwd<128, 128>(d, pl, tp, sp, st);
}

int f32_chunk_bwd(const HdlaDims& d, const void* q, const void* k, const void* v, const void* a, const void* b,
                  const void* gk, float scale, const float* h0, const void* d_o, const float* dht, void* dq, void* dk,
                  void* dv, void* da, void* db, void* dgk, float* dh0, float* ws, cudaStream_t st) {
    const F32Plan pl = make_f32_plan(d);
    if (!(d.flags & HDLA_FLAG_WS_HOLDS_FWD))
        TRY(f32_chunk_fwd(d, q, k, v, a, b, gk, scale, h0, nullptr, nullptr, ws, (size_t)pl.total, false, st));
    TileP tp = tile_params(d, pl, ws, q, k, v, a, b, gk, scale);
    for (const void* x : {d_o, (const void*)dq, (const void*)dk, (const void*)dv, (const void*)da, (const void*)db, (const void*)dgk})
        if (reinterpret_cast<uintptr_t>(x) % 16 != 0) tp.vec_k = tp.vec_v = 0;
    tp.d_o = d_o; tp.dq = dq; tp.dk = dk; tp.dv = dv; tp.da = da; tp.db = db; tp.dgk = dgk;
    ScanP sp = scan_params(d, pl, ws);
    sp.d_o = d_o; sp.init = dht; sp.fin = dh0;
    if (pl.KP == 64) return pl.VP == 64 ? bwd<64, 64>(d, pl, tp, sp, st) : bwd<64, 128>(d, pl, tp, sp, st);
    return pl.VP == 64 ? bwd<128, 64>(d, pl, tp, sp, st) : bwd<128, 128>(d, pl, tp, sp, st);
}

}  // namespace hdla
