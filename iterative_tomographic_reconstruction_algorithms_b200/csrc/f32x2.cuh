// Packed pairs of floats (sm_100a): one instruction, two results, each rounded
// as the scalar one.  The pipe takes as long as for two scalar instructions,
// so pairs pay where a loop is bound by instruction issue, not by FP32 itself.
// A product that goes into an add2 is contracted into one fma (ptxas 12.9,
// explicit rounding notwithstanding, also through a multiplication by 1): where
// the product has to be rounded, unpack it and go on with scalar operations.
// As the addend of an fma2 it is safe.
#pragma once

#include <cuda_runtime.h>

namespace tomo {
namespace {

struct F2 {
  unsigned long long v;
};
__device__ __forceinline__ F2 f2(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ F2 f2(float a) { return f2(a, a); }
__device__ __forceinline__ float2 unpack(F2 a) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a.v));
  return r;
}
#define TOMO_F2_OP2(name, op)                                             \
  __device__ __forceinline__ F2 name(F2 a, F2 b) {                        \
    F2 r;                                                                 \
    asm(op ".f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));        \
    return r;                                                             \
  }
TOMO_F2_OP2(add2, "add.rn")
TOMO_F2_OP2(add2_rd, "add.rm")
TOMO_F2_OP2(add2_ru, "add.rp")
TOMO_F2_OP2(mul2, "mul.rn")
#undef TOMO_F2_OP2
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ F2 fma2_rd(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rm.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ F2 fma2_ru(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rp.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
// c - a, rounded once
__device__ __forceinline__ F2 rsub2(F2 a, F2 c) { return fma2(a, f2(-1.0f), c); }

}  // namespace
}  // namespace tomo
