// Two f32 operations per instruction (sm_100a), each half rounded as the scalar operation rounds it.  They run at the scalar
// ones' rate per value (128 a clock and SM) and so leave half of the issue slots to loads and address arithmetic.
#pragma once

#include <cstdint>

namespace cmld {

__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// The rounded products of two pairs.  Packed multiplications are contracted with a packed addition that follows, although
// both name their rounding, and so are fused forms with a constant zero: the addend is -0 (a product's own sign of zero stays)
// and comes from the launch, so that it is a value like any other.
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b, uint64_t neg_zero) { return fma2(a, b, neg_zero); }
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t both(float x) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ uint64_t pair(float x, float y) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float2 halves(uint64_t v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}

}  // namespace cmld
