// Arithmetic shared by the fused scan kernels.
#pragma once
#include "common.cuh"

namespace mb200 {

// Two float32 in one 64-bit register pair.  Kept as a 64-bit value from definition to use (and across loops), the pair needs no
// moves to stay aligned; as float2 the compiler spends up to one move per packed instruction on re-pairing.
typedef unsigned long long f2;
__device__ __forceinline__ f2 pk(float lo, float hi) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpk(f2 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ float lo(f2 v) {
  float a, b;
  unpk(v, a, b);
  return a;
}
__device__ __forceinline__ float hi(f2 v) {
  float a, b;
  unpk(v, a, b);
  return b;
}
__device__ __forceinline__ f2 pfma(f2 a, f2 b, f2 c) {
  f2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ f2 pmul(f2 a, f2 b) {
  f2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f2 padd(f2 a, f2 b) {
  f2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f2 pex2(f2 v) {
  float a, b;
  unpk(v, a, b);
  return pk(ex2f(a), ex2f(b));
}

// softplus_fast without a branch: the lanes of a warp see both sides of it all the time.
__device__ __forceinline__ float softplus_sel(float x) {
  const float e = __expf(x);
  const float small = e * (1.f - e * (0.5f - e * (1.f / 3.f))), big = __logf(1.f + e);
  const float r = e < 1e-2f ? small : big;
  return x > 20.f ? x : r;
}

}  // namespace mb200
