// Division by a stored reciprocal (csrc/divide.cuh) against division, on the
// host: every FP32 significand under divisors of the kinds the strain has (3 r,
// 2 sqrt(2) r, r) and random ones, FP64 at random, then every exponent.
#include <cstdio>
#include <random>
#include <vector>

#include "divide.cuh"

using sl3dgpu::DivideBy;

namespace {
float Float(uint32_t b) {
  float v;
  std::memcpy(&v, &b, 4);
  return v;
}
double Double(uint64_t b) {
  double v;
  std::memcpy(&v, &b, 8);
  return v;
}
uint32_t Bits(float v) {
  uint32_t b;
  std::memcpy(&b, &v, 4);
  return b;
}
uint64_t Bits(double v) {
  uint64_t b;
  std::memcpy(&b, &v, 8);
  return b;
}
}  // namespace

int main() {
  std::mt19937_64 rng(3);
  long long wrong = 0, far = 0;
  std::vector<float> divisors;
  for (float r : {0.55f, 0.8931f, 1.0f})
    for (float c : {3.0f, 2.0f * 1.41421356f, 1.0f}) divisors.push_back(c * r);
  for (uint32_t m : {0u, 1u, 0x7FFFFFu, 0x7FFFFEu, 0x400000u}) divisors.push_back(Float((127u << 23) | m));
  for (int i = 0; i < 10; ++i) divisors.push_back(Float((127u << 23) | (rng() & 0x7FFFFFu)));
  for (float d : divisors)
    for (uint32_t m = 0; m < (1u << 23); ++m) {
      const float x = Float((127u << 23) | m);
      wrong += DivideBy(x, d, 1.0f / d) != x / d;
    }
  std::printf("FP32 significands: %lld wrong\n", wrong);
  for (int i = 0; i < 20000000; ++i) {
    const double d = Double((1023ull << 52) | (rng() >> 12)), x = Double((1023ull << 52) | (rng() >> 12));
    wrong += DivideBy(x, d, 1.0 / d) != x / d;
  }
  std::printf("and FP64 ones: %lld wrong\n", wrong);
  // every exponent, zeros, subnormals, infinities and NaN; the divisors are radii
  for (int i = 0; i < 20000000; ++i) {
    const uint64_t r = rng();
    const float x = Float(static_cast<uint32_t>(r)), d = Float((static_cast<uint32_t>(120 + r % 12) << 23) | (rng() & 0x7FFFFFu));
    const float q = DivideBy(x, d, 1.0f / d), want = x / d;
    if (std::isnan(want) ? !std::isnan(q) : Bits(q) != Bits(want)) {
      if (std::fabs(x) >= std::ldexp(1.0f, -100) && std::isfinite(x * (1.0f / d))) ++wrong;
      if (std::isfinite(want) && std::isfinite(q) ? std::llabs(static_cast<long long>(Bits(q)) - Bits(want)) > 1 : std::isfinite(x * (1.0f / d))) ++far;
    }
    const double X = Double(rng()), D = Double(((1016ull + r % 12) << 52) | (rng() >> 12));
    const double Q = DivideBy(X, D, 1.0 / D), Want = X / D;
    if (std::isnan(Want) ? !std::isnan(Q) : Bits(Q) != Bits(Want)) {
      if (std::fabs(X) >= std::ldexp(1.0, -968) && std::isfinite(X * (1.0 / D))) ++wrong;
      if (std::isfinite(Want) && std::isfinite(Q) ? std::llabs(static_cast<long long>(Bits(Q) - Bits(Want))) > 1 : std::isfinite(X * (1.0 / D))) ++far;
    }
  }
  std::printf("and every exponent: %lld wrong, %lld further off than the last place\n", wrong, far);
  return wrong == 0 && far == 0 ? 0 : 1;
}
