// Division by a stored divisor: from its rounded reciprocal, host and device.
#pragma once

#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <cstring>

namespace sl3dgpu {

// x / d rounded to nearest from d's rounded reciprocal y: a quotient and its
// exact remainder, whose share corrects it (Markstein's division). A division
// proper costs about ten instructions, six a point in the strain; FP64 ones
// are 19 cycles an SM each. In FP64 one correction leaves the rounding wrong
// for one value in 2^52 at most; in FP32, where that would be one in 2^23, a
// second leaves none. The remainder is exact for |x| from 2^-100 (FP32) and
// 2^-968 (FP64); below, the quotient is within its last place. Zero,
// subnormal and non-finite quotients are x y.
__host__ __device__ inline double DivideBy(double x, double d, double y) {
  const double q = x * y;
#ifdef __CUDA_ARCH__
  const uint32_t high = static_cast<uint32_t>(__double2hiint(q));
#else
  uint64_t bits;
  std::memcpy(&bits, &q, 8);
  const uint32_t high = static_cast<uint32_t>(bits >> 32);
#endif
  const uint32_t e = (high >> 20) & 0x7FFu;
  return e - 1u >= 0x7FEu ? q : fma(fma(-q, d, x), y, q);
}
__host__ __device__ inline float DivideBy(float x, float d, float y) {
  float q = x * y;
#ifdef __CUDA_ARCH__
  const uint32_t bits = __float_as_uint(q);
#else
  uint32_t bits;
  std::memcpy(&bits, &q, 4);
#endif
  const uint32_t e = (bits >> 23) & 0xFFu;
  if (e - 1u >= 0xFEu) return q;
  q = fmaf(fmaf(-q, d, x), y, q);
  return fmaf(fmaf(-q, d, x), y, q);
}

}  // namespace sl3dgpu
