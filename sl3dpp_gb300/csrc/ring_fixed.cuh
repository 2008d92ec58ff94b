// The FP64 longitude transforms in block fixed point (ring_fixed.cu): the
// arithmetic, host and device, and the launch.
//
// A ring's values are 64-bit integers under one power of two: |value| times
// 2^scale is below 2^61 even summed over the ring (the scale comes from the
// ring's sum of magnitudes), so no intermediate of the transform can
// overflow. A product with a root of unity (Q62) is three 32 x 32 -> 64
// multiplications and is within about one unit of the exact one; a unit is
// 2^-61 of the ring's sum of magnitudes, so the transform's error is below
// an FP64 transform's (whose roundings are 2^-53 of its running values).
#pragma once

#include <cstdint>
#include <vector>

#include "common.cuh"

namespace sl3dgpu {

// A complex fixed-point value.
struct Fx2 {
  long long x, y;
};
// A root of unity in Q62, each part split as h 2^32 + l with l signed.
struct FxRoot {
  int ch, cl, sh, sl;
};

// The stages of a ring's transform: radices in order, and per stage the
// division by Ns (the product of the radices before it) as a multiplication.
constexpr int kFxMaxStages = 12;
struct FxPlan {
  int n = 0;
  int stages = 0;
  int radix[kFxMaxStages] = {};
  uint32_t divNs[kFxMaxStages] = {};    // ceil(2^32 / Ns): x / Ns = mulhi(x, divNs) (Ns > 1, x Ns < 2^32)
  uint32_t divM[kFxMaxStages] = {};     // ceil(2^32 / (n / radix)): which ring a butterfly belongs to
};

// x / d for the d that `magic` was made for (x d < 2^32), d > 1.
__host__ __device__ inline uint32_t FxDivide(uint32_t x, uint32_t magic) {
#ifdef __CUDA_ARCH__
  return __umulhi(x, magic);
#else
  return static_cast<uint32_t>((static_cast<uint64_t>(x) * magic) >> 32);
#endif
}

// Plans for a 5-smooth n (false: n has another factor or too many stages):
// composite radices (10, 12, 8, 6) where they save a stage, the odd ones
// first, whose stores step over the shared-memory banks.
bool MakeFxPlan(int n, FxPlan* plan);
// The plan of given radices (their product n).
FxPlan FxPlanOf(int n, const int* radices, int stages);
// e^{2 pi i k / n} in Q62, k < n.
std::vector<FxRoot> MakeFxRoots(int n);

__host__ __device__ inline long long FxProduct(int ah, int al, int wh, int wl) {
  const long long p = static_cast<long long>(ah) * wl + (1LL << 29) + static_cast<long long>(al) * wh;
  return (static_cast<long long>(ah) * wh) * 4 + (p >> 30);
}
__host__ __device__ inline void FxSplit(long long a, int& h, int& l) {
  l = static_cast<int>(static_cast<uint32_t>(static_cast<unsigned long long>(a)));
  h = static_cast<int>(static_cast<unsigned long long>(a) >> 32) - (l >> 31);
}
// a w for a constant w in (-1, 1] given as Q62 (|a| < 2^61).
template <long long W>
__host__ __device__ inline long long FxConst(long long a) {
  constexpr int wl = static_cast<int>(static_cast<uint32_t>(static_cast<unsigned long long>(W)));
  constexpr int wh = static_cast<int>((W - wl) >> 32);
  int h, l;
  FxSplit(a, h, l);
  return FxProduct(h, l, wh, wl);
}
__host__ __device__ inline Fx2 FxAdd(Fx2 a, Fx2 b) { return {a.x + b.x, a.y + b.y}; }
__host__ __device__ inline Fx2 FxSub(Fx2 a, Fx2 b) { return {a.x - b.x, a.y - b.y}; }
__host__ __device__ inline Fx2 FxI(Fx2 a) { return {-a.y, a.x}; }  // i a
template <long long W>
__host__ __device__ inline Fx2 FxScale(Fx2 a) {
  return {FxConst<W>(a.x), FxConst<W>(a.y)};
}
// a w
__host__ __device__ inline Fx2 FxRotate(Fx2 a, FxRoot w) {
  int xh, xl, yh, yl;
  FxSplit(a.x, xh, xl);
  FxSplit(a.y, yh, yl);
  const int msh = -w.sh, msl = -w.sl;
  using L = long long;
  const L rh = static_cast<L>(xh) * w.ch + static_cast<L>(yh) * msh;
  const L rl = static_cast<L>(xh) * w.cl + (1LL << 29) + static_cast<L>(xl) * w.ch + static_cast<L>(yh) * msl +
               static_cast<L>(yl) * msh;
  const L ih = static_cast<L>(xh) * w.sh + static_cast<L>(yh) * w.ch;
  const L il = static_cast<L>(xh) * w.sl + (1LL << 29) + static_cast<L>(xl) * w.sh + static_cast<L>(yh) * w.cl +
               static_cast<L>(yl) * w.ch;
  return {rh * 4 + (rl >> 30), ih * 4 + (il >> 30)};
}

// Q62 constants: sqrt(3)/2, sqrt(1/2), sqrt(5)/4, sin 72 deg, sin 72 - sin 36,
// and sin 72 + sin 36 - 1.
constexpr long long kFxRoot3Half = 3993837246235628775LL;
constexpr long long kFxRootHalf = 3260954456333195553LL;
constexpr long long kFxRoot5Quarter = 2578010857022246787LL;
constexpr long long kFxSin72 = 4385974038932618941LL;
constexpr long long kFxSin72Less36 = 1675293009097605857LL;
constexpr long long kFxSin72Plus36Less1 = 2484969050340244120LL;

// The DFT of R values in registers, y_u = sum_q v_q e^{2 pi i q u / R}.
template <int R>
__host__ __device__ inline void FxButterfly(Fx2 (&v)[R]) {
  if constexpr (R == 2) {
    const Fx2 a = v[0];
    v[0] = FxAdd(a, v[1]);
    v[1] = FxSub(a, v[1]);
  } else if constexpr (R == 3) {
    const Fx2 t = FxAdd(v[1], v[2]);
    const Fx2 d = FxI(FxScale<kFxRoot3Half>(FxSub(v[1], v[2])));
    const Fx2 a = {v[0].x - ((t.x + 1) >> 1), v[0].y - ((t.y + 1) >> 1)};
    v[0] = FxAdd(v[0], t);
    v[1] = FxAdd(a, d);
    v[2] = FxSub(a, d);
  } else if constexpr (R == 4) {
    const Fx2 a0 = FxAdd(v[0], v[2]), a1 = FxSub(v[0], v[2]);
    const Fx2 b0 = FxAdd(v[1], v[3]), b1 = FxI(FxSub(v[1], v[3]));
    v[0] = FxAdd(a0, b0);
    v[1] = FxAdd(a1, b1);
    v[2] = FxSub(a0, b0);
    v[3] = FxSub(a1, b1);
  } else if constexpr (R == 5) {
    const Fx2 t1 = FxAdd(v[1], v[4]), t2 = FxAdd(v[2], v[3]);
    const Fx2 d1 = FxSub(v[1], v[4]), d2 = FxSub(v[2], v[3]);
    const Fx2 s = FxAdd(t1, t2), b = FxScale<kFxRoot5Quarter>(FxSub(t1, t2));
    const Fx2 a = {v[0].x - ((s.x + 2) >> 2), v[0].y - ((s.y + 2) >> 2)};
    const Fx2 a1 = FxAdd(a, b), a2 = FxSub(a, b);
    const Fx2 p = FxScale<kFxSin72>(FxAdd(d1, d2));
    const Fx2 e1 = FxI(FxSub(p, FxScale<kFxSin72Less36>(d2)));
    const Fx2 e2 = FxI(FxSub(FxAdd(d1, FxScale<kFxSin72Plus36Less1>(d1)), p));
    v[0] = FxAdd(v[0], s);
    v[1] = FxAdd(a1, e1);
    v[4] = FxSub(a1, e1);
    v[2] = FxAdd(a2, e2);
    v[3] = FxSub(a2, e2);
  } else if constexpr (R == 8) {
    Fx2 a[4] = {v[0], v[2], v[4], v[6]}, b[4] = {v[1], v[3], v[5], v[7]};
    FxButterfly<4>(a);
    FxButterfly<4>(b);
    const Fx2 b1 = FxScale<kFxRootHalf>({b[1].x - b[1].y, b[1].x + b[1].y});
    const Fx2 b2 = FxI(b[2]);
    const Fx2 b3 = FxScale<kFxRootHalf>({-b[3].x - b[3].y, b[3].x - b[3].y});
    v[0] = FxAdd(a[0], b[0]);
    v[4] = FxSub(a[0], b[0]);
    v[1] = FxAdd(a[1], b1);
    v[5] = FxSub(a[1], b1);
    v[2] = FxAdd(a[2], b2);
    v[6] = FxSub(a[2], b2);
    v[3] = FxAdd(a[3], b3);
    v[7] = FxSub(a[3], b3);
  } else {
    // R = A B with A and B coprime: the prime-factor form, no rotations
    // between the two (input (B q_A + A q_B) mod R; output u with u = u_A
    // mod A and u = u_B mod B)
    static_assert(R == 6 || R == 10 || R == 12, "a radix of the plans");
    constexpr int A = R == 12 ? 4 : 2, B = R / A;
    Fx2 w[A][B];
#pragma unroll
    for (int qa = 0; qa < A; ++qa) {
      Fx2 t[B];
#pragma unroll
      for (int qb = 0; qb < B; ++qb) t[qb] = v[(B * qa + A * qb) % R];
      FxButterfly<B>(t);
#pragma unroll
      for (int qb = 0; qb < B; ++qb) w[qa][qb] = t[qb];
    }
#pragma unroll
    for (int ub = 0; ub < B; ++ub) {
      Fx2 t[A];
#pragma unroll
      for (int qa = 0; qa < A; ++qa) t[qa] = w[qa][ub];
      FxButterfly<A>(t);
#pragma unroll
      for (int ua = 0; ua < A; ++ua) {
        // the root of u's product is (q_A / A + q_B / B) u: output u takes
        // u mod A of the one and u mod B of the other
        int u = 0;
#pragma unroll
        for (int x = 0; x < R; ++x)
          if (x % A == ua && x % B == ub) u = x;
        v[u] = t[ua];
      }
    }
  }
}

// One Stockham butterfly of radix R: reads in[b + q m], rotates by
// e^{2 pi i q k / (Ns R)}, writes out[(b / Ns) Ns R + k + u Ns], shifted down
// by `down` bits (rounded).
template <int R>
__host__ __device__ inline void FxStageButterfly(const Fx2* in, Fx2* out, int b, int m, int Ns, uint32_t divNs,
                                                 int stride, const FxRoot* roots, int down) {
  const int blk = Ns > 1 ? static_cast<int>(FxDivide(static_cast<uint32_t>(b), divNs)) : b;
  const int k = b - blk * Ns;
  Fx2 v[R];
#pragma unroll
  for (int q = 0; q < R; ++q) v[q] = in[b + q * m];
  if (Ns > 1) {
#pragma unroll
    for (int q = 1; q < R; ++q) v[q] = FxRotate(v[q], roots[q * k * stride]);
  }
  FxButterfly<R>(v);
  if (down > 0) {
    const long long half = 1LL << (down - 1);
#pragma unroll
    for (int u = 0; u < R; ++u) v[u] = Fx2{(v[u].x + half) >> down, (v[u].y + half) >> down};
  }
  Fx2* o = out + blk * Ns * R + k;
#pragma unroll
  for (int u = 0; u < R; ++u) o[u * Ns] = v[u];
}

// -- FP64 values to and from fixed point ---------------------------------------------------

constexpr int kFxSumBits = 16;  // the magnitude sum's resolution below the largest exponent

// The biased exponent of v's bits (0x7FF: not finite).
__host__ __device__ inline int FxExponent(unsigned long long bits) { return static_cast<int>((bits >> 52) & 0x7FF); }
// An upper bound of |v| in units of 2^(emax - 1023 - kFxSumBits).
__host__ __device__ inline uint32_t FxMagnitude(unsigned long long bits, int emax) {
  const uint32_t top = (static_cast<uint32_t>(bits >> (52 - kFxSumBits)) & ((1u << kFxSumBits) - 1)) | (1u << kFxSumBits);
  const int d = emax - FxExponent(bits);
  return d > kFxSumBits ? 1u : (top >> d) + 1u;
}
// The scale of a ring whose magnitudes sum to below `sum` such units (the
// transform then stays below 2^61): values are X 2^-scale.
__host__ __device__ inline int FxScaleOf(int emax, uint32_t sum) {
#ifdef __CUDA_ARCH__
  const int bits = 32 - __clz(sum);
#else
  const int bits = sum ? 32 - __builtin_clz(sum) : 0;
#endif
  return 61 - bits - (emax - 1023 - kFxSumBits);
}
// The bits a ring's early stages may keep above that scale. A stage's values
// are sums of Ns of the inputs, below 2 Ns of their largest, so until the
// last stage they may carry more bits than the whole sum allows: `room` is
// 61 less the largest input's bits less `scale`, and FxHeadAt the bits kept
// through the stage that makes sums of Ns. Where the ring's sum is far above
// its largest value most of a transform's error would otherwise be its
// inputs' rounding. `doubled`: the inputs are sums of two values.
__host__ __device__ inline int FxRoom(int emax, int scale, bool doubled) {
  return 61 - (doubled ? 1 : 0) - (emax - 1022) - scale;
}
__host__ __device__ inline int FxHeadAt(int room, int Ns) {
#ifdef __CUDA_ARCH__
  const int bits = 32 - __clz(2 * Ns - 1);
#else
  const int bits = 32 - __builtin_clz(static_cast<unsigned>(2 * Ns - 1));
#endif
  return room > bits ? room - bits : 0;
}
// round(v 2^scale), below 2^61 for the ring's values.
__host__ __device__ inline long long FxFrom(unsigned long long bits, int scale) {
  const int e = FxExponent(bits);
  const long long mantissa = static_cast<long long>((bits & ((1ULL << 52) - 1)) | (1ULL << 52));
  const int shift = e - 1023 - 52 + scale;  // at most 9
  long long X;
  if (shift >= 0)
    X = mantissa << shift;
  else
    X = shift < -54 ? 0 : (mantissa + (1LL << (-shift - 1))) >> -shift;
  if (e == 0) X = 0;  // zero, or subnormal: below the unit of any ring held in fixed point
  return bits >> 63 ? -X : X;
}
// X 2^-scale as a double, rounded to nearest.
__host__ __device__ inline double FxTo(long long X, int scale) {
  if (X == 0) return 0.0;
  const unsigned long long sign = static_cast<unsigned long long>(X) & (1ULL << 63);
  unsigned long long m = X < 0 ? 0ULL - static_cast<unsigned long long>(X) : static_cast<unsigned long long>(X);
#ifdef __CUDA_ARCH__
  const int lead = __clzll(static_cast<long long>(m));
#else
  const int lead = __builtin_clzll(m);
#endif
  m <<= lead;
  const unsigned long long mantissa = (m >> 11) + ((m >> 10) & 1);  // 2^52 .. 2^53
  const int exponent = 1023 + 63 - lead - scale;                     // of the leading bit, biased
  if (exponent < 1 || exponent > 2045) {
    const double v = ldexp(static_cast<double>(mantissa), exponent - 1023 - 52);
    return sign ? -v : v;
  }
  const unsigned long long bits = sign | ((static_cast<unsigned long long>(exponent - 1) << 52) + mantissa);
#ifdef __CUDA_ARCH__
  return __longlong_as_double(static_cast<long long>(bits));
#else
  double v;
  __builtin_memcpy(&v, &bits, 8);
  return v;
#endif
}

// The ring passes on FP64 values (Grid::RingSynthesis, RingAnalysis and
// RingWeighted): `mode` 0 spectra -> fields, 1 fields (times a weight) ->
// spectra, 2 spectra -> weighted fields -> spectra. One launch takes up to
// three batches of `count` fields (a tensor's spin components), spin (complex)
// or real, under the same point weights.
struct FxRingPart {
  bool real;
  const double2* spectraIn;  // [order][colatitude][field]
  const void* fieldsIn;      // [field][colatitude][longitude]
  void* fieldsOut;
  double2* spectraOut;
};
struct FxRingArgs {
  int mode, lmax, ntheta, count;
  const FxRoot* roots;     // n
  const double2* twiddle;  // n, FP64 (the double-float rings', and the rings that fall back to FP64)
  const double* weights;   // per colatitude
  const double* pointWeight;
  int parts;
  FxRingPart part[3];
  int blocks[3];  // CTAs of each part along x (the launch fills them)
};
// This CTA's part, and its place among the part's CTAs.
__device__ __forceinline__ const FxRingPart& FxPartOf(const FxRingArgs& a, int& x) {
  x = static_cast<int>(blockIdx.x);
  int p = 0;
  while (p + 1 < a.parts && x >= a.blocks[p]) x -= a.blocks[p++];
  return a.part[p];
}
// The parts' CTAs at G rings each; their sum.
inline int FxBlocks(FxRingArgs& a, int G) {
  int total = 0;
  for (int p = 0; p < a.parts; ++p) {
    const int rings = a.part[p].real ? (a.count + 1) / 2 : a.count;  // real fields go two to a ring
    a.blocks[p] = (rings + G - 1) / G;
    total += a.blocks[p];
  }
  return total;
}
// The most rings of a part.
inline int FxRings(const FxRingArgs& a) {
  int rings = 1;
  for (int p = 0; p < a.parts; ++p)
    rings = rings > (a.part[p].real ? (a.count + 1) / 2 : a.count) ? rings : (a.part[p].real ? (a.count + 1) / 2 : a.count);
  return rings;
}
int LaunchFxRings(const FxPlan& plan, FxRingArgs args, cudaStream_t stream);

}  // namespace sl3dgpu
