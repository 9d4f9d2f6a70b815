// Packed fp32 pairs: one FFMA2 does two fused multiply-adds, so half the instructions are issued.
#pragma once
#include <cuda_runtime.h>

namespace hdla {

typedef unsigned long long f2;
__device__ __forceinline__ f2 f2_dup(float x) { f2 r; asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(x)); return r; }
__device__ __forceinline__ f2 f2_pack(float x, float y) { f2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y)); return r; }
__device__ __forceinline__ void f2_unpack(f2 a, float& x, float& y) { asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a)); }
__device__ __forceinline__ float f2_sum(f2 a) { float x, y; f2_unpack(a, x, y); return x + y; }
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b) { f2 r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c) { f2 r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }

}  // namespace hdla
