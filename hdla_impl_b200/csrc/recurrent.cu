// Fused recurrent forward of the rank-R DPLR delta rule (decode and short prefill).
//
// Follows the per-token recurrence of the reference kernel (HRDPLR/recurrent.py:75-115):
//     sa_r  = a_r^T S_{t-1}                          (one V-vector per rank)
//     S_t   = exp(g_t) (.) S_{t-1} + sum_r b_r sa_r^T + k_t v_t^T
//     o_t   = (scale q_t)^T S_t
//
// Two kernels: up to kTileTokens tokens per call the state tile passes through shared memory
// (recurrent_tile_kernel: bound by HBM, the fp32 state is read and written once); longer sequences keep it in
// registers (recurrent_reg_kernel: bound by fp32 arithmetic or by the dependent steps of the recurrence).
#include "common.cuh"
#include "f32x2.cuh"
#include "sm100.cuh"

namespace hdla {
namespace {

// Read with hdla_recurrent_read_status(): non-zero once a time-limited wait of a kernel here ran out.  None of them has
// such waits, so it stays zero.
__device__ int g_recurrent_status;

struct RecParams {
    const void *q, *k, *v, *a, *b, *gk;
    const float* h0;
    void* o;
    float* ht;
    const int64_t* cu;
    float scale;
    int T, H, K, V, dt, gdt, reverse;
};

// Sum N values over the eight row lanes of a warp (lane bits 2..4), N = 1, 2, 4 or 8: each step halves the values a lane
// still carries, so N = 8 costs 7 shuffles instead of 24.  Lane r ends with the sums of N/8 (at least one) values,
// the first of them number scatter_index<N>(r).
template <int N>
__device__ __forceinline__ void reduce_scatter(float* v, int lane) {
    int n = N;
#pragma unroll
    for (int m = 4; m <= 16; m <<= 1) {
        if (n > 1) {
            const bool up = (lane & m) != 0;
            n >>= 1;
#pragma unroll
            for (int i = 0; i < N / 2; ++i)
                if (i < n) {
                    const float give = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
                    v[i] = keep + __shfl_xor_sync(0xffffffffu, give, m);
                }
        } else {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], m);
        }
    }
}
// ... and with every lane holding all N sums (three dependent steps instead of the six of scatter and gather)
template <int N>
__device__ __forceinline__ void all_reduce(float* v) {
#pragma unroll
    for (int m = 4; m <= 16; m <<= 1)
#pragma unroll
        for (int i = 0; i < N; ++i) v[i] += __shfl_xor_sync(0xffffffffu, v[i], m);
}
template <int N>
__device__ __forceinline__ int scatter_index(int lane) {
    int n = N, at = 0;
#pragma unroll
    for (int m = 4; m <= 16; m <<= 1)
        if (n > 1) { n >>= 1; at += (lane & m) ? n : 0; }
    return at;
}

// CPT adjacent columns (from c0, a multiple of CPT) of row k of a state tile; V is a multiple of 4, so a group of up to
// four columns exists as a whole or not at all.  Rows and columns outside the tile read as zero.
template <int CPT>
__device__ __forceinline__ void ld_cols(float* x, const float* base, int nh, int k, int c0, int K, int V) {
#pragma unroll
    for (int q = 0; q < CPT; ++q) x[q] = 0.f;
    if (!base || k >= K) return;
    const float* src = base + ((size_t)nh * K + k) * V + c0;
    if constexpr (CPT == 2) {
        if (c0 < V) { const float2 t = __ldcs(reinterpret_cast<const float2*>(src)); x[0] = t.x; x[1] = t.y; }
    } else {
#pragma unroll
        for (int q = 0; q < CPT; q += 4)
            if (c0 + q < V) {
                const float4 t = __ldcs(reinterpret_cast<const float4*>(src + q));
                x[q] = t.x; x[q + 1] = t.y; x[q + 2] = t.z; x[q + 3] = t.w;
            }
    }
}
template <int CPT>
__device__ __forceinline__ void st_cols(const float* x, float* base, int nh, int k, int c0, int K, int V) {
    if (k >= K) return;
    float* dst = base + ((size_t)nh * K + k) * V + c0;
    if constexpr (CPT == 2) {
        if (c0 < V) __stcs(reinterpret_cast<float2*>(dst), make_float2(x[0], x[1]));
    } else {
#pragma unroll
        for (int q = 0; q < CPT; q += 4)
            if (c0 + q < V) __stcs(reinterpret_cast<float4*>(dst + q), make_float4(x[q], x[q + 1], x[q + 2], x[q + 3]));
    }
}

// Register-state kernel: more than a few tokens per call (kTileTokens).
//   * A column of the state depends on the other columns through nothing, so the columns are spread over warps (and,
//     while there are fewer warps than the chip runs, over CTAs): a warp owns 4 CPT columns, lane (r, c) of it the
//     rows 4 r + 32 j + {0..3} of CPT adjacent columns, in registers, as packed row pairs.
//   * Tokens are staged kRecBlock at a time: the raw K- and V-vectors of the next block arrive by asynchronous copies
//     while the current one is worked on; at the block boundary they are turned into fp32 (q scaled, decay
//     exponentiated) in shared memory once for the whole CTA.  Between two boundaries there is no CTA barrier.
//   * One pass over the state per token: the update of token t, its output q^T S, and a^T S for token t + 1.  A
//     128-bit shared load of a vector (four rows) feeds 4 CPT state elements.
// What bounds it: instruction issue with many sequences (0.55 of the issue slots, 0.31 of the fp32 pipe: 224 packed FMAs
// of 578 instructions per warp and token at K = 128; shared loads, shuffles and the block conversion are the rest),
// with few the dependent pass + shuffle sums, 0.66 us per token.  Before, every token's vectors were fetched from
// global memory between two CTA barriers: 413 tokens in 16 sequences x 16 heads of 128 took 262 us, now 66; one
// sequence of 128 tokens x 4 heads 540 us, now 85.
constexpr int kRecBlock = 8;
// Up to two tokens the tile in shared memory is the faster form (4096 heads of 128: 0.71 / 0.83 of the registers' time for 1 /
// 2 tokens), from three on the registers are (0.98 for 3, 1.25 for 6; with 64 heads 1.6 and 2.2; with so few heads they
// already are for two tokens, 1.33).  But the register kernel pads K to 32, 64, 128 or 256 rows: where a fifth or more of
// them is padding and there are two heads or more to an SM, the tile is faster up to eight tokens -- 0.66 of the time over
// 352 measured cases (K x V of 16 x 64 to 100 x 132, ranks 1 to 4, 1024 and 4096 heads, 3 to 8 tokens), up to 1.1 in four.
constexpr int kTileTokens = 2, kTileTokensPadded = 8;

template <int KR, int CPT, int R>
__global__ void __launch_bounds__(128, KR * CPT <= 32 ? 4 : KR * CPT <= 64 ? 3 : 2) recurrent_reg_kernel(RecParams p, int col_blocks, int async_ok) {
    constexpr int KP = 8 * KR, NV = 3 + 2 * R;               // padded rows; K-vectors per token: e k q a.. b..
    extern __shared__ __align__(16) float sm[];
    const int nh = blockIdx.x / col_blocks, cb = blockIdx.x % col_blocks;
    const int n = nh / p.H, h = nh % p.H;
    const int K = p.K, V = p.V, H = p.H;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int r = lane >> 2, c = lane & 3;
    const int cta_cols = (blockDim.x >> 5) * 4 * CPT;
    const int cta_c0 = cb * cta_cols;                        // first column of this CTA
    const int wc = warp * 4 * CPT + c * CPT;                 // this lane's first column within the CTA
    const int c0 = cta_c0 + wc;
    const int ncol = min(cta_cols, V - cta_c0);              // columns of this CTA that exist
    const int tok_floats = NV * KP + cta_cols;
    unsigned char* raw = reinterpret_cast<unsigned char*>(sm + kRecBlock * tok_floats);
    const int es = p.dt == HDLA_F32 ? 4 : 2, gs = p.gdt == HDLA_F32 ? 4 : 2;
    const int tok_raw = ((2 + 2 * R) * K + ncol) * es + K * gs;

    long long bos, len;
    if (p.cu) { bos = p.cu[n]; len = p.cu[n + 1] - bos; }
    else      { bos = (long long)n * p.T; len = p.T; }

    const long long stride = p.reverse ? -1 : 1, first = p.reverse ? bos + len - 1 : bos;     // token s is first + s * stride
    // Request the raw vectors of tokens [s0, s0 + kRecBlock): a thread keeps its 16-byte piece for all tokens of the block.
    auto request = [&](long long s0) {
        const int cnt = (int)min((long long)kRecBlock, len - s0);
        const int nq = K * es / 16, ng = K * gs / 16, nv = ncol * es / 16;
        const int per = nq * (2 + 2 * R) + ng + nv;
        for (int w = tid; w < per; w += blockDim.x) {
            const char* src;
            size_t step;                                          // bytes between tokens
            const size_t t0 = (size_t)(first + s0 * stride);
            if (w < ng) {
                src = static_cast<const char*>(p.gk) + (t0 * H + h) * K * gs + (size_t)w * 16;
                step = (size_t)H * K * gs;
            } else if (w < ng + nv) {
                src = static_cast<const char*>(p.v) + ((t0 * H + h) * V + cta_c0) * es + (size_t)(w - ng) * 16;
                step = (size_t)H * V * es;
            } else {
                const int vec = (w - ng - nv) / nq, at = (w - ng - nv) % nq;      // 0 k, 1 q, 2.. a, 2 + R.. b
                const char* base = static_cast<const char*>(vec == 0 ? p.k : vec == 1 ? p.q : vec < 2 + R ? p.a : p.b);
                const size_t row = vec < 2 ? t0 * H + h : (t0 * R + (vec < 2 + R ? vec - 2 : vec - 2 - R)) * H + h;
                src = base + row * K * es + (size_t)at * 16;
                step = (size_t)H * K * es * (vec < 2 ? 1 : R);
            }
            unsigned char* dst = raw + (size_t)w * 16;
            if (p.reverse) step = (size_t)0 - step;
            for (int tk = 0; tk < cnt; ++tk, src += step, dst += tok_raw) sm100::cp_async16(dst, src);
        }
        sm100::cp_async_commit();
    };
    // Turn them into fp32, four elements at a time: a thread keeps its place for all tokens of the block, so the
    // eight tokens' loads are in flight together.
    auto convert = [&](long long s0) {
        const int cnt = (int)min((long long)kRecBlock, len - s0);
        for (int i = tid; i < NV * (KP / 4) + cta_cols / 4; i += blockDim.x) {
            const int vec = i / (KP / 4);                         // 0 e, 1 k, 2 q, 3.. a, 3 + R.. b, NV: v
            const bool is_v = i >= NV * (KP / 4);
            const int kk = is_v ? (i - NV * (KP / 4)) * 4 : (i % (KP / 4)) * 4;
            const int lim = is_v ? ncol : K;
            float4* dst = reinterpret_cast<float4*>(sm + (is_v ? NV * KP : vec * KP) + kk);
            const int dt = vec == 0 ? p.gdt : p.dt;
            if (async_ok) {
                const unsigned char* rw = raw + (is_v ? K * gs : vec == 0 ? 0 : K * gs + ncol * es + (vec - 1) * K * es)
                                          + kk * (dt == HDLA_F32 ? 4 : 2);
                float4 x[kRecBlock];
#pragma unroll
                for (int tk = 0; tk < kRecBlock; ++tk) {
                    x[tk] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (tk < cnt && kk < lim) {
                        if (dt == HDLA_F32) {
                            x[tk] = *reinterpret_cast<const float4*>(rw + (size_t)tk * tok_raw);
                        } else {
                            const uint2 u = *reinterpret_cast<const uint2*>(rw + (size_t)tk * tok_raw);
                            x[tk] = make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u),
                                                __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
                        }
                        if (vec == 0) { x[tk].x = __expf(x[tk].x); x[tk].y = __expf(x[tk].y); x[tk].z = __expf(x[tk].z); x[tk].w = __expf(x[tk].w); }
                        if (vec == 2) { x[tk].x *= p.scale; x[tk].y *= p.scale; x[tk].z *= p.scale; x[tk].w *= p.scale; }
                    }
                }
#pragma unroll
                for (int tk = 0; tk < kRecBlock; ++tk) dst[tk * (tok_floats / 4)] = x[tk];
            } else {                                              // rows that asynchronous copies cannot take: element by element
                const void* base = is_v ? p.v : vec == 0 ? p.gk : vec == 1 ? p.k : vec == 2 ? p.q : vec < 3 + R ? p.a : p.b;
                for (int tk = 0; tk < cnt; ++tk) {
                    const size_t t = (size_t)(first + (s0 + tk) * stride);
                    const size_t at = is_v ? (t * H + h) * V + cta_c0
                                           : (vec < 3 ? t * H + h : (t * R + (vec < 3 + R ? vec - 3 : vec - 3 - R)) * H + h) * K;
                    float e[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        e[j] = kk + j < lim ? ld_elem(base, at + kk + j, dt) : 0.f;
                        if (vec == 0 && kk + j < lim) e[j] = __expf(e[j]);
                        if (vec == 2) e[j] *= p.scale;
                    }
                    dst[tk * (tok_floats / 4)] = make_float4(e[0], e[1], e[2], e[3]);
                }
            }
        }
    };

    if (async_ok && len > 0) request(0);
    f2 S[KR / 2][CPT];                                       // S[2 j + u][c]: rows 4 r + 32 j + 2 u + {0, 1}
#pragma unroll
    for (int j = 0; j < KR / 4; ++j)
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int k0 = 32 * j + 4 * r + 2 * u;
            float x[CPT], y[CPT];
            ld_cols<CPT>(x, p.h0, nh, k0, c0, K, V);
            ld_cols<CPT>(y, p.h0, nh, k0 + 1, c0, K, V);
#pragma unroll
            for (int q = 0; q < CPT; ++q) S[2 * j + u][q] = f2_pack(x[q], y[q]);
        }

    for (long long s0 = 0; s0 < len; s0 += kRecBlock) {
        const int cnt = (int)min((long long)kRecBlock, len - s0);
        if (async_ok) sm100::cp_async_wait<0>();
        __syncthreads();                                     // the raw block is here and the fp32 block has been read
        convert(s0);
        __syncthreads();
        if (async_ok && s0 + kRecBlock < len) request(s0 + kRecBlock);
        // a^T S for the block's first token
        float sa[R][CPT];
        {
            f2 acc[R][CPT];
#pragma unroll
            for (int rr = 0; rr < R; ++rr)
#pragma unroll
                for (int q = 0; q < CPT; ++q) acc[rr][q] = 0ull;
#pragma unroll
            for (int j = 0; j < KR / 4; ++j)
#pragma unroll
                for (int rr = 0; rr < R; ++rr) {
                    const ulonglong2 av = *reinterpret_cast<const ulonglong2*>(sm + (3 + rr) * KP + 32 * j + 4 * r);
#pragma unroll
                    for (int q = 0; q < CPT; ++q) {
                        acc[rr][q] = f2_fma(av.x, S[2 * j][q], acc[rr][q]);
                        acc[rr][q] = f2_fma(av.y, S[2 * j + 1][q], acc[rr][q]);
                    }
                }
#pragma unroll
            for (int rr = 0; rr < R; ++rr) {
#pragma unroll
                for (int q = 0; q < CPT; ++q) sa[rr][q] = f2_sum(acc[rr][q]);
                all_reduce<CPT>(sa[rr]);
            }
        }
        for (int tk = 0; tk < cnt; ++tk) {
            const float* tok = sm + tk * tok_floats;
            const float* nxt = tk + 1 < cnt ? tok + tok_floats : tok;     // (the last token's a^T S is not used)
            f2 v2[CPT], s2[R][CPT], oa[CPT], na[R][CPT];
#pragma unroll
            for (int q = 0; q < CPT; ++q) {
                v2[q] = f2_dup(tok[NV * KP + wc + q]);
#pragma unroll
                for (int rr = 0; rr < R; ++rr) s2[rr][q] = f2_dup(sa[rr][q]);
            }
#pragma unroll
            for (int j = 0; j < KR / 4; ++j) {
                const int at = 32 * j + 4 * r;
                auto vec = [&](const float* base, int i) { return *reinterpret_cast<const ulonglong2*>(base + i * KP + at); };
                const ulonglong2 e = vec(tok, 0), kv = vec(tok, 1), qv = vec(tok, 2);
                ulonglong2 bv[R], av[R];
#pragma unroll
                for (int rr = 0; rr < R; ++rr) { bv[rr] = vec(tok, 3 + R + rr); av[rr] = vec(nxt, 3 + rr); }
#pragma unroll
                for (int q = 0; q < CPT; ++q) {
                    f2 x = f2_fma(kv.x, v2[q], f2_mul(e.x, S[2 * j][q]));
                    f2 y = f2_fma(kv.y, v2[q], f2_mul(e.y, S[2 * j + 1][q]));
#pragma unroll
                    for (int rr = 0; rr < R; ++rr) { x = f2_fma(bv[rr].x, s2[rr][q], x); y = f2_fma(bv[rr].y, s2[rr][q], y); }
                    S[2 * j][q] = x; S[2 * j + 1][q] = y;
                    oa[q] = f2_fma(qv.y, y, j == 0 ? f2_mul(qv.x, x) : f2_fma(qv.x, x, oa[q]));
#pragma unroll
                    for (int rr = 0; rr < R; ++rr)
                        na[rr][q] = f2_fma(av[rr].y, y, j == 0 ? f2_mul(av[rr].x, x) : f2_fma(av[rr].x, x, na[rr][q]));
                }
            }
            if (tk + 1 < cnt) {
#pragma unroll
                for (int rr = 0; rr < R; ++rr) {
#pragma unroll
                    for (int q = 0; q < CPT; ++q) sa[rr][q] = f2_sum(na[rr][q]);
                    all_reduce<CPT>(sa[rr]);
                }
            }
            float o[CPT];
#pragma unroll
            for (int q = 0; q < CPT; ++q) o[q] = f2_sum(oa[q]);
            reduce_scatter<CPT>(o, lane);
            // with fewer values than row lanes several lanes hold the same sum: one of them stores it
            const int col = c0 + scatter_index<CPT>(lane);
            const bool mine = CPT >= 8 || (CPT == 4 ? (r & 4) == 0 : (r & 6) == 0);
            if (mine && col < V) {
                const long long t = first + (s0 + tk) * stride;
                st_elem(p.o, ((size_t)t * H + h) * V + col, p.dt, o[0]);
            }
        }
    }

    if (p.ht) {
#pragma unroll
        for (int j = 0; j < KR / 4; ++j)
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int k0 = 32 * j + 4 * r + 2 * u;
                float x[CPT], y[CPT];
#pragma unroll
                for (int q = 0; q < CPT; ++q) f2_unpack(S[2 * j + u][q], x[q], y[q]);
                st_cols<CPT>(x, p.ht, nh, k0, c0, K, V);
                st_cols<CPT>(y, p.ht, nh, k0 + 1, c0, K, V);
            }
    }
}

// an element as it is stored, and its value
__device__ __forceinline__ uint32_t ld_raw(const void* p, size_t i, int dt) {
    return dt == HDLA_F32 ? static_cast<const uint32_t*>(p)[i] : static_cast<const unsigned short*>(p)[i];
}
__device__ __forceinline__ float raw_float(uint32_t x, int dt) { return __uint_as_float(dt == HDLA_F32 ? x : x << 16); }

// ------------------------------------------------------------------------------------------
// Decode variant (a few tokens per call): the state tile is staged in shared memory.
//   * one CTA per (sequence, head) brings the whole contiguous fp32 [K,V] tile (64 KB at K=V=128) into shared memory by
//     16-byte asynchronous copies, so the bytes in flight per SM are set by how many tiles fit in shared memory (three),
//     not by the register file;
//   * a token's vectors are asked for a step ahead, the first one's before the tile, and stay as they came until they are
//     needed: behind the tile's copies, or converted at once, they cost 25 to 50 us of 165 (256 sequences x 32 heads);
//   * lane l of a warp owns rows l/8 + 4s of 4 adjacent columns, a warp 32 columns (128-bit, conflict-free accesses;
//     reductions by register sums and two shuffles); a token updates the tile in place, the last one writes it to global
//     memory from the registers (whole 128-byte lines), which drains while the next CTA's tile is on its way.
// Bound by HBM, the fp32 state being read and written once: 256 sequences x 32 heads of 128 take 165 us for one token,
// 6.6 TB/s; two tokens 226.
// (Before, one bulk copy brought the tile in, counted on an mbarrier, and one took it back: 184 and 267 us.  That form ended
// in a launch failure with 28 CTAs of 256-byte tiles on an SM -- K = V = 8, 4096 heads, two tokens -- with every address,
// size and alignment in order; larger tiles, which leave room for fewer CTAs, never showed it.)
// ------------------------------------------------------------------------------------------
template <int R>
__global__ void __launch_bounds__(256) recurrent_tile_kernel(RecParams p) {
    extern __shared__ __align__(16) float sS[];                 // [K][V], then the token's vectors
    const int nh = blockIdx.x;
    const int n = nh / p.H, h = nh % p.H;
    const int K = p.K, V = p.V, H = p.H;
    float* s_q = sS + (size_t)K * V;
    float* s_k = s_q + K;
    float* s_e = s_k + K;
    float* s_a = s_e + K;
    float* s_b = s_a + R * K;
    float* s_v = s_b + R * K;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r = lane >> 3;
    const int c4 = (warp * 8 + (lane & 7)) * 4;
    const bool col_ok = c4 < V;

    long long bos, len;
    if (p.cu) { bos = p.cu[n]; len = p.cu[n + 1] - bos; }
    else      { bos = (long long)n * p.T; len = p.T; }

    const int tid = threadIdx.x;
    uint32_t raw[4 + 2 * R];                                     // element tid of q k gk v and of every a, b
    auto ask = [&](long long step) {
        const long long t = p.reverse ? (bos + len - 1 - step) : (bos + step);
        const size_t tk = ((size_t)t * H + h) * K + tid;
        if (tid < K) {
            raw[0] = ld_raw(p.q, tk, p.dt); raw[1] = ld_raw(p.k, tk, p.dt); raw[2] = ld_raw(p.gk, tk, p.gdt);
#pragma unroll
            for (int rr = 0; rr < R; ++rr) {
                const size_t ta = (((size_t)t * R + rr) * H + h) * K + tid;
                raw[4 + 2 * rr] = ld_raw(p.a, ta, p.dt); raw[5 + 2 * rr] = ld_raw(p.b, ta, p.dt);
            }
        }
        if (tid < V) raw[3] = ld_raw(p.v, ((size_t)t * H + h) * V + tid, p.dt);
    };
    if (len > 0) ask(0);
    const size_t tile = (size_t)nh * K * V;
    if (p.h0) {
        const float* src = p.h0 + tile;
#pragma unroll 8
        for (int i = tid * 4; i < K * V; i += blockDim.x * 4) sm100::cp_async16(sS + i, src + i);
    } else {
        for (int i = tid * 4; i < K * V; i += blockDim.x * 4)
            *reinterpret_cast<float4*>(sS + i) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    sm100::cp_async_commit();

    for (long long step = 0; step < len; ++step) {
        const bool last = step + 1 == len;
        const long long t = p.reverse ? (bos + len - 1 - step) : (bos + step);
        const size_t tk = ((size_t)t * H + h) * K;
        if (tid < K) {
            s_q[tid] = raw_float(raw[0], p.dt) * p.scale; s_k[tid] = raw_float(raw[1], p.dt);
            s_e[tid] = __expf(raw_float(raw[2], p.gdt));
#pragma unroll
            for (int rr = 0; rr < R; ++rr) {
                s_a[rr * K + tid] = raw_float(raw[4 + 2 * rr], p.dt); s_b[rr * K + tid] = raw_float(raw[5 + 2 * rr], p.dt);
            }
        }
        if (tid < V) s_v[tid] = raw_float(raw[3], p.dt);
        for (int i = tid + blockDim.x; i < K; i += blockDim.x) { // (heads with more rows than the CTA has threads)
            s_q[i] = ld_elem(p.q, tk + i, p.dt) * p.scale;
            s_k[i] = ld_elem(p.k, tk + i, p.dt);
            s_e[i] = __expf(ld_elem(p.gk, tk + i, p.gdt));
#pragma unroll
            for (int rr = 0; rr < R; ++rr) {
                const size_t ta = (((size_t)t * R + rr) * H + h) * K;
                s_a[rr * K + i] = ld_elem(p.a, ta + i, p.dt);
                s_b[rr * K + i] = ld_elem(p.b, ta + i, p.dt);
            }
        }
        sm100::cp_async_wait<0>();                               // the tile (first step)
        __syncthreads();
        if (!last) ask(step + 1);

        float sa[R][4];
#pragma unroll
        for (int rr = 0; rr < R; ++rr) { sa[rr][0] = sa[rr][1] = sa[rr][2] = sa[rr][3] = 0.f; }
        if (col_ok) {
            for (int kk = r; kk < K; kk += 4) {
                const float4 x = *reinterpret_cast<const float4*>(sS + (size_t)kk * V + c4);
#pragma unroll
                for (int rr = 0; rr < R; ++rr) {
                    const float av = s_a[rr * K + kk];
                    sa[rr][0] = fmaf(av, x.x, sa[rr][0]); sa[rr][1] = fmaf(av, x.y, sa[rr][1]);
                    sa[rr][2] = fmaf(av, x.z, sa[rr][2]); sa[rr][3] = fmaf(av, x.w, sa[rr][3]);
                }
            }
        }
#pragma unroll
        for (int rr = 0; rr < R; ++rr)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                sa[rr][j] += __shfl_xor_sync(0xffffffffu, sa[rr][j], 8);
                sa[rr][j] += __shfl_xor_sync(0xffffffffu, sa[rr][j], 16);
            }
        float oa[4] = {0.f, 0.f, 0.f, 0.f};
        if (col_ok) {
            const float vv[4] = {s_v[c4], s_v[c4 + 1], s_v[c4 + 2], s_v[c4 + 3]};
            float* out = last && p.ht ? p.ht + tile + c4 : nullptr;
            for (int kk = r; kk < K; kk += 4) {
                float4* ps = reinterpret_cast<float4*>(sS + (size_t)kk * V + c4);
                const float4 x = *ps;
                const float e = s_e[kk], kv = s_k[kk], qv = s_q[kk];
                float y[4] = {fmaf(kv, vv[0], e * x.x), fmaf(kv, vv[1], e * x.y), fmaf(kv, vv[2], e * x.z),
                              fmaf(kv, vv[3], e * x.w)};
#pragma unroll
                for (int rr = 0; rr < R; ++rr) {
                    const float bv = s_b[rr * K + kk];
#pragma unroll
                    for (int j = 0; j < 4; ++j) y[j] = fmaf(bv, sa[rr][j], y[j]);
                }
                const float4 z = make_float4(y[0], y[1], y[2], y[3]);
                if (!last) *ps = z;
                else if (out) *reinterpret_cast<float4*>(out + (size_t)kk * V) = z;
#pragma unroll
                for (int j = 0; j < 4; ++j) oa[j] = fmaf(qv, y[j], oa[j]);
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            oa[j] += __shfl_xor_sync(0xffffffffu, oa[j], 8);
            oa[j] += __shfl_xor_sync(0xffffffffu, oa[j], 16);
        }
        if (r == 0 && col_ok) {
            const size_t to = ((size_t)t * H + h) * V + c4;
            if (p.dt == HDLA_F32) {
                *reinterpret_cast<float4*>(static_cast<float*>(p.o) + to) = make_float4(oa[0], oa[1], oa[2], oa[3]);
            } else {
                uint2 pk;
                pk.x = sm100::pack_bf16(oa[0], oa[1]);
                pk.y = sm100::pack_bf16(oa[2], oa[3]);
                *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(p.o) + to) = pk;
            }
        }
        if (!last) __syncthreads();                              // vectors are single buffered
    }
    if (len == 0) {                                              // a sequence without tokens: its state passes through
        sm100::cp_async_wait<0>();
        if (p.ht)                                                // (each thread the pieces it brought in itself)
            for (int i = tid * 4; i < K * V; i += blockDim.x * 4)
                *reinterpret_cast<float4*>(p.ht + tile + i) = *reinterpret_cast<const float4*>(sS + i);
    }
}

template <int KR, int CPT, int R>
int launch_reg(const RecParams& p, int NH, cudaStream_t st) {
    // up to four warps (4 CPT columns each) of one head per CTA share its staged vectors
    const int warps = (p.V + 4 * CPT - 1) / (4 * CPT);
    const int per_cta = warps < 4 ? warps : 4;
    const int col_blocks = (warps + per_cta - 1) / per_cta;
    const int cols = per_cta * 4 * CPT;
    const int es = p.dt == HDLA_F32 ? 4 : 2, gs = p.gdt == HDLA_F32 ? 4 : 2;
    bool async_ok = p.K * es % 16 == 0 && p.K * gs % 16 == 0 && p.V * es % 16 == 0;
    for (const void* q : {p.q, p.k, p.v, p.a, p.b, p.gk}) async_ok = async_ok && reinterpret_cast<uintptr_t>(q) % 16 == 0;
    const size_t smem = (size_t)kRecBlock * (((3 + 2 * R) * 8 * KR + cols) * sizeof(float)
                                             + (async_ok ? ((2 + 2 * R) * p.K + cols) * es + p.K * gs : 0));
    static thread_local int attr_dev = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (attr_dev != dev) {
        cudaError_t e = cudaFuncSetAttribute(recurrent_reg_kernel<KR, CPT, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        if (e != cudaSuccess) return fail(HDLA_ERR_CUDA, "recurrent: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
        attr_dev = dev;
    }
    recurrent_reg_kernel<KR, CPT, R><<<NH * col_blocks, per_cta * 32, smem, st>>>(p, col_blocks, async_ok ? 1 : 0);
    return HDLA_OK;
}

template <int KR, int CPT>
int launch_rank(const RecParams& p, int NH, int R, cudaStream_t st) {
    switch (R) {
        case 1: return launch_reg<KR, CPT, 1>(p, NH, st);
        case 2: return launch_reg<KR, CPT, 2>(p, NH, st);
        case 3: return launch_reg<KR, CPT, 3>(p, NH, st);
        case 4: return launch_reg<KR, CPT, 4>(p, NH, st);
        default: return fail(HDLA_ERR_UNSUPPORTED, "recurrent: rank R=%d not in 1..4", R);
    }
}

}  // namespace

int recurrent_read_status(int* dst, cudaStream_t st) {
    void* sym = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&sym, g_recurrent_status);
    if (e == cudaSuccess) e = cudaMemcpyAsync(dst, sym, sizeof(int), cudaMemcpyDefault, st);
    if (e != cudaSuccess) return fail(HDLA_ERR_CUDA, "recurrent status: %s", cudaGetErrorString(e));
    return HDLA_OK;
}

int recurrent_fwd_launch(const HdlaDims& d, const void* q, const void* k, const void* v, const void* a,
                         const void* b, const void* gk, float scale, const float* h0, void* o, float* ht,
                         const int64_t* cu_seqlens, int n_seqs, int reverse, cudaStream_t st) {
    if (d.K > 256 || d.K < 1) return fail(HDLA_ERR_UNSUPPORTED, "recurrent: K=%d must be in 1..256", d.K);
    if (d.V % 4 != 0 || d.V > 256 || d.V < 4)
        return fail(HDLA_ERR_UNSUPPORTED, "recurrent: V=%d must be a multiple of 4 in 4..256", d.V);
    if (cu_seqlens && d.B != 1) return fail(HDLA_ERR_INVALID, "recurrent: cu_seqlens needs B == 1, got B=%d", d.B);
    const int N = cu_seqlens ? n_seqs : d.B;
    if (N <= 0) return fail(HDLA_ERR_INVALID, "recurrent: no sequences");
    RecParams p{q, k, v, a, b, gk, h0, o, ht, cu_seqlens, scale, d.T, d.H, d.K, d.V, d.dtype, d.gk_dtype, reverse};
    const int blocks = N * d.H;
    const int threads = 32 * ((d.V + 31) / 32);
    // few tokens per call: the kernel with the tile in shared memory (which it must fit)
    const size_t tile = (size_t)d.K * d.V * 4;
    const int rows = d.K <= 32 ? 32 : d.K <= 64 ? 64 : d.K <= 128 ? 128 : 256;        // of the register kernel
    const bool padded = 5 * d.K <= 4 * rows && tile > 2048 && blocks >= 2 * sm_count();
    if (d.T <= (padded ? kTileTokensPadded : kTileTokens) && tile <= 65536 && tile % 16 == 0 && d.R <= 4) {
        const size_t smem_t = tile + sizeof(float) * ((3 + 2 * d.R) * (size_t)d.K + d.V);
        static thread_local int attr_dev = -1;
        int dev = 0;
        cudaGetDevice(&dev);
        if (attr_dev != dev) {
            cudaError_t e = cudaFuncSetAttribute(recurrent_tile_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, 65536 + 16384);
            if (e == cudaSuccess) e = cudaFuncSetAttribute(recurrent_tile_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, 65536 + 16384);
            if (e == cudaSuccess) e = cudaFuncSetAttribute(recurrent_tile_kernel<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, 65536 + 16384);
            if (e == cudaSuccess) e = cudaFuncSetAttribute(recurrent_tile_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, 65536 + 16384);
            if (e != cudaSuccess) return fail(HDLA_ERR_CUDA, "recurrent: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
            attr_dev = dev;
        }
        switch (d.R) {
            case 1: recurrent_tile_kernel<1><<<blocks, threads, smem_t, st>>>(p); break;
            case 2: recurrent_tile_kernel<2><<<blocks, threads, smem_t, st>>>(p); break;
            case 3: recurrent_tile_kernel<3><<<blocks, threads, smem_t, st>>>(p); break;
            default: recurrent_tile_kernel<4><<<blocks, threads, smem_t, st>>>(p); break;
        }
        HDLA_CHECK_LAUNCH("recurrent_tile_kernel");
        return HDLA_OK;
    }
    int rc;
    const int NH = N * d.H;
    // Two columns per lane instead of four while that leaves no more than two warps to a scheduler (four per SM): the pass
    // over the state is then what a token waits for, and it is half as long.  (With more warps the wider tile wins,
    // since a shared load feeds twice the arithmetic.)
    const bool narrow = d.R == 2 && (long long)NH * ((d.V + 15) / 16) <= sm_count() * 4;
    if (narrow && d.K <= 64)       rc = launch_reg<8, 2, 2>(p, NH, st);
    else if (narrow && d.K <= 128) rc = launch_reg<16, 2, 2>(p, NH, st);
    else if (d.K <= 32)  rc = launch_rank<4, 4>(p, NH, d.R, st);
    else if (d.K <= 64)  rc = launch_rank<8, 4>(p, NH, d.R, st);
    else if (d.K <= 128) rc = launch_rank<16, 4>(p, NH, d.R, st);
    else                 rc = launch_rank<32, 4>(p, NH, d.R, st);
    if (rc != HDLA_OK) return rc;
    HDLA_CHECK_LAUNCH("recurrent_reg_kernel");
    return HDLA_OK;
}

}  // namespace hdla
