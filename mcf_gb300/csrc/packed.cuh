// packed.cuh -- pairs of FP32 numbers in one 64-bit register and Blackwell's
// packed arithmetic on them (add, mul, fma .f32x2, sm_100 and later): each
// half rounds as the scalar operation does, at half the issue slots.  The
// FP32 sweeps are bound by instruction issue, so this is where they gain.
#pragma once
#include <cuda_runtime.h>

namespace mcfg {

struct F2 {
  unsigned long long u;
};

__device__ __forceinline__ F2 pack2(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.u) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ F2 splat2(float a) { return pack2(a, a); }
__device__ __forceinline__ void unpack2(F2 a, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a.u));
}
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
  F2 r;
  asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r.u) : "l"(a.u), "l"(b.u));
  return r;
}
__device__ __forceinline__ F2 sub2(F2 a, F2 b) {
  F2 r;
  asm("sub.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r.u) : "l"(a.u), "l"(b.u));
  return r;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r.u) : "l"(a.u), "l"(b.u));
  return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(r.u) : "l"(a.u), "l"(b.u), "l"(c.u));
  return r;
}

// A separation at which the packed sweeps put their padding: outside every
// support whose kernel constants FP32 holds (coef goes with 1/h^2 at least, so
// h is below 1e18), its square finite.  (From the cut-off, a constant of the
// launch, instead of an immediate: the density 12 us of 490 slower.)
constexpr float kBeyond = 1e19f;

// max(a - s, 0) per half: a truncated power's base
__device__ __forceinline__ F2 base2(float a, F2 s) {
  float lo, hi;
  unpack2(sub2(splat2(a), s), lo, hi);
  return pack2(fmaxf(lo, 0.0f), fmaxf(hi, 0.0f));
}

// a + b and its rounding error
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
  s = a + b;
  const float bb = s - a;
  e = (a - (s - bb)) + (b - bb);
}

// The Kahan sums of the two halves, and over a group of S lanes in lane order,
// as a sum hi and its remainder lo.
template <int S>
__device__ __forceinline__ void join_sums(F2 acc, F2 cmp, unsigned gmask, float& hi, float& lo) {
  float p0, p1, c0, c1;
  unpack2(acc, p0, p1);
  unpack2(cmp, c0, c1);
  two_sum(p0, p1, hi, lo);
  lo -= c0 + c1;
  if (S > 1) {
    const int base = (threadIdx.x & 31) & ~(S - 1);
    const float ph = hi, pl = lo;
    hi = __shfl_sync(gmask, ph, base);
    lo = __shfl_sync(gmask, pl, base);
#pragma unroll
    for (int w = 1; w < S; ++w) {
      const float oh = __shfl_sync(gmask, ph, base + w), ol = __shfl_sync(gmask, pl, base + w);
      float e;
      two_sum(hi, oh, hi, e);
      lo += ol + e;
    }
  }
}

}  // namespace mcfg
