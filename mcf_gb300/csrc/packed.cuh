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

}  // namespace mcfg
