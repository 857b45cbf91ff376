// fp32 values as three bf16 planes that add up to them: x = h + m + l.
#pragma once
#include "ptx.cuh"

namespace sd3 {

// two floats as bf16 rounded to nearest, of magnitude at most the largest finite bf16 (x0 in the low half)
__device__ __forceinline__ uint32_t pack_bf16x2_finite(float x0, float x1) {
  uint32_t r;
  asm("cvt.rn.satfinite.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(x1), "f"(x0));
  return r;
}

// Each plane is the remainder so far rounded to nearest (8 significant bits), so the
// subtractions are exact and 8 + 8 + 8 bits with signs hold the whole 24-bit significand
// (values whose last bits lie under bf16's smallest denormal, 2^-133, excepted).  The first two planes
// stop at the largest finite bf16, 3.3895e38: finite floats above it (up to 3.4028e38) still add up, and of
// an infinity only the last plane is infinite, so that no inf - inf arises here.  A NaN is one in every
// plane.  Two values per 32-bit word, x0 in the low half.
// The subtractions are packed (fma.f32x2: x - h exactly).
__device__ __forceinline__ void split3_x2(float x0, float x1, uint32_t& h, uint32_t& m, uint32_t& l) {
  const float2 minus = make_float2(-1.0f, -1.0f);
  h = pack_bf16x2_finite(x0, x1);
  const float2 r =
      __ffma2_rn(make_float2(__uint_as_float(h << 16), __uint_as_float(h & 0xffff0000u)), minus, make_float2(x0, x1));
  m = pack_bf16x2_finite(r.x, r.y);
  const float2 q = __ffma2_rn(make_float2(__uint_as_float(m << 16), __uint_as_float(m & 0xffff0000u)), minus, r);
  l = pack_bf16x2(q.x, q.y);
}

}  // namespace sd3
