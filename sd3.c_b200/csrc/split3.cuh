// fp32 values as three bf16 planes that add up to them: x = h + m + l.
#pragma once
#include "ptx.cuh"

namespace sd3 {

// Each plane is the remainder so far rounded to nearest (8 significant bits), so the
// subtractions are exact and 8 + 8 + 8 bits with signs hold the whole 24-bit significand
// (values whose last bits lie under bf16's smallest denormal, 2^-133, excepted).  A value that is
// not finite gives a NaN in the middle plane.  Two values per 32-bit word, x0 in the low half.
__device__ __forceinline__ void split3_x2(float x0, float x1, uint32_t& h, uint32_t& m, uint32_t& l) {
  h = pack_bf16x2(x0, x1);
  const float r0 = x0 - __uint_as_float(h << 16), r1 = x1 - __uint_as_float(h & 0xffff0000u);
  m = pack_bf16x2(r0, r1);
  l = pack_bf16x2(r0 - __uint_as_float(m << 16), r1 - __uint_as_float(m & 0xffff0000u));
}

}  // namespace sd3
