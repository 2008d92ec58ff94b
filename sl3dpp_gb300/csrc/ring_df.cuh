// The FP64 rings of a grid that asked for the emulation, in double-float: the
// values and their conversions (host and device, so that the conversions are
// checked on the CPU too).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "ring_fixed.cuh"
#include "ring_stages.cuh"

namespace sl3dgpu {

// A double-float value, hi + lo with |lo| <= ulp(hi) / 2 (about 48
// significant bits): the FP64 ring transforms' arithmetic on the FP32 pipe
// when the grid emulates FP64 (the FP64 pipe is GB300's slow one). Dekker's
// and Knuth's error-free transformations -- TwoSum, FastTwoSum and the
// FMA-based TwoProduct -- in their usual double-single forms: a sum's
// error is bounded by about 2^-46 (|a| + |b|) (the "sloppy" addition, whose
// bound is normwise, which is what a transform's error analysis uses), a
// product's by about 2^-46 |a b|. The _rn intrinsics keep the compiler from
// contracting the error terms into FMAs.
struct Df {
  float hi, lo;
  __host__ __device__ constexpr Df() : hi(0.0f), lo(0.0f) {}
  __host__ __device__ constexpr Df(float h, float l) : hi(h), lo(l) {}
  // the nearest double-float of a literal constant (folded by the compiler;
  // run-time values go through FromDouble)
  __host__ __device__ constexpr Df(double d)
      : hi(static_cast<float>(d)), lo(static_cast<float>(d - static_cast<double>(static_cast<float>(d)))) {}
  __host__ __device__ constexpr Df(int i) : Df(static_cast<double>(i)) {}
};
struct Df2 {
  Df x, y;
};
template <>
struct Real<Df2> {
  using type = Df;
};

// FastTwoSum of s and an error term e (|s| >= |e| or s = 0)
__device__ inline Df Renormalise(float s, float e) {
  const float h = __fadd_rn(s, e);
  return Df(h, __fsub_rn(e, __fsub_rn(h, s)));
}
__device__ inline Df operator+(Df a, Df b) {
  const float s = __fadd_rn(a.hi, b.hi);
  const float bb = __fsub_rn(s, a.hi);
  const float e = __fadd_rn(__fsub_rn(a.hi, __fsub_rn(s, bb)), __fsub_rn(b.hi, bb));  // TwoSum's error
  return Renormalise(s, __fadd_rn(e, __fadd_rn(a.lo, b.lo)));
}
__device__ inline Df operator-(Df a) { return Df(-a.hi, -a.lo); }
__device__ inline Df operator-(Df a, Df b) { return a + (-b); }
__device__ inline Df operator*(Df a, Df b) {
  const float p = __fmul_rn(a.hi, b.hi);
  float e = __fmaf_rn(a.hi, b.hi, -p);  // TwoProduct's error
  e = __fmaf_rn(a.hi, b.lo, e);
  e = __fmaf_rn(a.lo, b.hi, e);
  return Renormalise(p, e);
}

// -- conversions ---------------------------------------------------------------------------
//
// hi = d rounded to FP32, lo = (d - hi) rounded to FP32, and hi + lo rounded to
// FP64, each exactly as the FP64 instructions give them, by integer
// arithmetic on the bits: a conversion between FP64 and FP32 is an FP64-pipe
// instruction (19 cycles an SM for a warp on GB300), and the four in and
// three out a value were half of the ring kernel's time. Values outside the
// range where the integer form is exact take the FP64 instructions.

__host__ __device__ inline uint32_t FloatBits(float v) {
#ifdef __CUDA_ARCH__
  return __float_as_uint(v);
#else
  uint32_t b;
  __builtin_memcpy(&b, &v, 4);
  return b;
#endif
}
__host__ __device__ inline float FloatOf(uint32_t b) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(b);
#else
  float v;
  __builtin_memcpy(&v, &b, 4);
  return v;
#endif
}
__host__ __device__ inline unsigned long long DoubleBits(double v) {
#ifdef __CUDA_ARCH__
  return static_cast<unsigned long long>(__double_as_longlong(v));
#else
  unsigned long long b;
  __builtin_memcpy(&b, &v, 8);
  return b;
#endif
}
__host__ __device__ inline double DoubleOf(unsigned long long b) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double(static_cast<long long>(b));
#else
  double v;
  __builtin_memcpy(&v, &b, 8);
  return v;
#endif
}

__host__ __device__ inline Df FromDouble(double d) {
  const unsigned long long bits = DoubleBits(d);
  const int e = static_cast<int>((bits >> 52) & 0x7FF) - 1023;
  if (e < -74 || e > 126) {  // zero, and values whose parts could leave FP32's normal range
    if ((bits << 1) == 0) return Df(FloatOf(static_cast<uint32_t>(bits >> 32)), 0.0f);
    const float hi = static_cast<float>(d);
    return Df(hi, static_cast<float>(d - static_cast<double>(hi)));
  }
  const uint32_t sign = static_cast<uint32_t>(bits >> 32) & 0x80000000u;
  const uint32_t top = static_cast<uint32_t>(bits >> 29) & 0x7FFFFFu;  // the 23 fraction bits kept
  const uint32_t low = static_cast<uint32_t>(bits) & 0x1FFFFFFFu;      // the 29 below
  const uint32_t half = 1u << 28;
  const uint32_t up = (low > half || (low == half && (top & 1u))) ? 1u : 0u;
  const uint32_t hi = sign | ((static_cast<uint32_t>(e + 127) << 23) + top + up);  // a carry moves the exponent
  const int rest = static_cast<int>(low) - static_cast<int>(up << 29);
  const float unit = FloatOf(sign | (static_cast<uint32_t>(e - 52 + 127) << 23));
  return Df(FloatOf(hi), rest == 0 ? 0.0f : static_cast<float>(rest) * unit);
}

__host__ __device__ inline double ToDouble(Df v) {
  const uint32_t h = FloatBits(v.hi), l = FloatBits(v.lo);
  const int eh = static_cast<int>((h >> 23) & 0xFF), el = static_cast<int>((l >> 23) & 0xFF);
  // hi normal, lo zero or normal and below half a unit of hi
  const bool none = (l << 1) == 0;
  if (eh < 1 || eh > 254 || (!none && (el < 1 || el > eh - 24)))
    return static_cast<double>(v.hi) + static_cast<double>(v.lo);
  // |hi| in units of 2^(eh - 127 - 61): the 24-bit significand at bits 61 .. 38
  unsigned long long m = static_cast<unsigned long long>((h & 0x7FFFFFu) | 0x800000u) << 38;
  if (!none) {
    const unsigned long long f = static_cast<unsigned long long>((l & 0x7FFFFFu) | 0x800000u);
    const int shift = el - eh + 38;  // at most 14
    unsigned long long part;
    if (shift >= 0)
      part = f << shift;
    else if (shift > -25)
      part = (f >> -shift) | ((f & ((1ULL << -shift) - 1)) != 0 ? 1ULL : 0ULL);  // the rest as a sticky bit
    else
      part = 1ULL;
    m = ((h ^ l) >> 31) != 0 ? m - part : m + part;
  }
  // the leading bit is 61, or 60 after a subtraction at a power of two
  int e = eh - 127;
  if ((m >> 61) == 0) {
    m <<= 1;
    --e;
  }
  // to 53 bits (9 below), nearest, ties to even
  const unsigned long long kept = m >> 9, rem = m & 511ULL;
  const unsigned long long up = rem > 256ULL || (rem == 256ULL && (kept & 1ULL)) ? 1ULL : 0ULL;
  const unsigned long long sign = static_cast<unsigned long long>(h & 0x80000000u) << 32;
  return DoubleOf(sign | ((static_cast<unsigned long long>(e + 1022) << 52) + kept + up));
}

// The ring passes in double-float (the fixed-point ones' interface); the plan
// has the radices 4, 2, 3, 5.
int LaunchDfRings(const FxPlan& plan, FxRingArgs args, cudaStream_t stream);

}  // namespace sl3dgpu
