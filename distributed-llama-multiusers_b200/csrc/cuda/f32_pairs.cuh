// Two f32 in a register pair: one instruction, two operations, each rounded as the scalar one does.
#pragma once

typedef unsigned long long pair_f;
__device__ __forceinline__ pair_f pair_of(float lo, float hi) { pair_f r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi)); return r; }
__device__ __forceinline__ void pair_get(pair_f v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ float pair_sum(pair_f v) { float lo, hi; pair_get(v, lo, hi); return lo + hi; }
__device__ __forceinline__ pair_f fma2(pair_f x, pair_f y, pair_f z) { pair_f r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(x), "l"(y), "l"(z)); return r; }
__device__ __forceinline__ pair_f mul2(pair_f x, pair_f y) { pair_f r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(x), "l"(y)); return r; }
__device__ __forceinline__ pair_f add2(pair_f x, pair_f y) { pair_f r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(x), "l"(y)); return r; }
__device__ __forceinline__ pair_f ld_pair(const float* p) { return *reinterpret_cast<const pair_f*>(p); }
__device__ __forceinline__ void st_pair(float* p, pair_f v) { *reinterpret_cast<pair_f*>(p) = v; }
