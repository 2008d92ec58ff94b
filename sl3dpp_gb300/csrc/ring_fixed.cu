// The longitude transforms of FP64 values in block fixed point.
//
// Why. GB300's FP64 unit issues one warp instruction in 64 cycles a
// sub-partition (19 an SM, whatever lanes are active), conversions between
// FP64 and FP32 included, while a 64-bit integer addition takes about half a
// cycle an SM and a 61 x 62 bit product about four. A ring transform is mostly
// additions, so the same transform in 64-bit integers under one scale a
// ring (ring_fixed.cuh) does a fraction of the work, and its error is below
// the FP64 transform's (measured against quadruple precision on white and
// decaying spectra, 72 to 800 longitudes). Both transforms of 45 spin -2 fields
// at lmax 128 went from 1.28 to 0.63 ms with it, the rings from the larger
// part of that to half.
//
// How. One CTA per (colatitude, G consecutive fields; G a power of two so that
// a thread's values belong to one ring). The raw FP64 bits go to shared
// memory; each thread's largest exponent and then its sum of magnitudes are
// reduced over the ring to its scale; the values are converted in place and
// the Stockham stages run over the CTA's butterflies, ping-ponging between
// two buffers a ring. Radices up to 12 keep it to three stages at the
// configurations' 400 and 800 longitudes. The opposite direction swaps real
// and imaginary parts at the conversions. Weighted rings multiply in fixed
// point between the two transforms (the weights under their ring's largest)
// and rescale. Real fields go two to a ring, as its real and imaginary parts.
//
// A ring holding an infinity or a NaN, or whose largest value is within 2^128
// of the ends of the FP64 range (its scale would leave it), is transformed in
// FP64, with its CTA's other rings.
#include <algorithm>
#include <cmath>
#include <string>
#include <vector>

#include "profile.cuh"
#include "ring_fixed.cuh"

namespace sl3dgpu {

namespace {

enum { kFxSynth = 0, kFxAnalyse = 1, kFxWeighted = 2 };

constexpr int kFxThreads = 256;
constexpr int kFxMaxRings = 8;
constexpr int kFxExponentLow = 128, kFxExponentHigh = 2046 - 128;

// -- the FP64 form -------------------------------------------------------------------------

__device__ double2 Rotate64(double2 a, double2 w) {
  return make_double2(a.x * w.x - a.y * w.y, a.x * w.y + a.y * w.x);
}

// One ring's plain Stockham transform by one warp in FP64, sign +1 or -1:
// radix by radix as the direct sums (a rare path: a few instructions matter
// more than its speed). Returns the buffer holding the result.
__device__ __noinline__ double2* Ring64(double2* a, double2* b, const FxPlan& plan, const double2* tw, int sign,
                                        int lane) {
  const int n = plan.n;
  int Ns = 1;
  for (int s = 0; s < plan.stages; ++s) {
    const int R = plan.radix[s], m = n / R, stride = n / (Ns * R);
    for (int e = lane; e < n; e += kWarp) {
      const int u = e / m, idx = e % m, blk = idx / Ns, k = idx % Ns;
      double2 sum = make_double2(0.0, 0.0);
      for (int q = 0; q < R; ++q) {
        // e^{2 pi i (q k / (Ns R) + q u / R)}
        double2 w = tw[(q * k * stride + (q * u % R) * m) % n];
        if (sign < 0) w.y = -w.y;
        const double2 v = Rotate64(a[idx + q * m], w);
        sum.x += v.x;
        sum.y += v.y;
      }
      b[blk * Ns * R + k + u * Ns] = sum;
    }
    __syncwarp();
    double2* t = a;
    a = b;
    b = t;
    Ns *= R;
  }
  return a;
}

// The CTA's rings in FP64 from the inputs again.
__device__ __noinline__ void Rings64(const FxPlan& plan, const FxRingArgs& A, const FxRingPart& Q, int x,
                                      double2* bufs, int G) {
  const int n = plan.n, perRing = Q.real ? 2 : 1, j = blockIdx.y;
  const int mcount = Q.real ? A.lmax + 1 : 2 * A.lmax + 1;
  const int lane = threadIdx.x % kWarp;
  const double scale = 2.0 * 3.14159265358979323846 / n * A.weights[j];
  for (int g = threadIdx.x / kWarp; g < G; g += blockDim.x / kWarp) {
    const int f0 = (x * G + g) * perRing;
    if (f0 >= A.count) break;
    const bool second = Q.real && f0 + 1 < A.count;
    const long long row0 = (static_cast<long long>(f0) * A.ntheta + j) * n, row1 = row0 + static_cast<long long>(A.ntheta) * n;
    double2* a = bufs + static_cast<long long>(g) * 2 * n;
    double2* b = a + n;
    if (A.mode != kFxAnalyse) {
      for (int k = lane; k < n; k += kWarp) a[k] = make_double2(0.0, 0.0);
      __syncwarp();
      for (int mi = lane; mi < mcount; mi += kWarp) {
        const long long at = (static_cast<long long>(mi) * A.ntheta + j) * A.count + f0;
        const double2 v = Q.spectraIn[at];
        if (!Q.real) {
          const int m = mi - A.lmax;
          a[m < 0 ? m + n : m] = v;
          continue;
        }
        const double2 u = second ? Q.spectraIn[at + 1] : make_double2(0.0, 0.0);
        if (mi == 0) {
          a[0] = make_double2(v.x, u.x);
        } else {
          a[mi] = make_double2(v.x - u.y, v.y + u.x);
          a[n - mi] = make_double2(v.x + u.y, u.x - v.y);
        }
      }
      __syncwarp();
      double2* res = Ring64(a, b, plan, A.twiddle, 1, lane);
      if (A.mode == kFxSynth) {
        for (int k = lane; k < n; k += kWarp) {
          if (Q.real) {
            static_cast<double*>(Q.fieldsOut)[row0 + k] = res[k].x;
            if (second) static_cast<double*>(Q.fieldsOut)[row1 + k] = res[k].y;
          } else {
            static_cast<double2*>(Q.fieldsOut)[row0 + k] = res[k];
          }
        }
        continue;
      }
      b = res == a ? b : a;
      a = res;
      for (int k = lane; k < n; k += kWarp) {
        const double w0 = A.pointWeight[row0 + k], w1 = Q.real ? (second ? A.pointWeight[row1 + k] : 0.0) : w0;
        a[k] = make_double2(a[k].x * w0, a[k].y * w1);
      }
    } else {
      for (int k = lane; k < n; k += kWarp) {
        double2 v = Q.real ? make_double2(static_cast<const double*>(Q.fieldsIn)[row0 + k],
                                          second ? static_cast<const double*>(Q.fieldsIn)[row1 + k] : 0.0)
                           : static_cast<const double2*>(Q.fieldsIn)[row0 + k];
        if (A.pointWeight != nullptr) {
          const double w0 = A.pointWeight[row0 + k], w1 = Q.real ? (second ? A.pointWeight[row1 + k] : 0.0) : w0;
          v = make_double2(v.x * w0, v.y * w1);
        }
        a[k] = v;
      }
    }
    __syncwarp();
    const double2* res = Ring64(a, b, plan, A.twiddle, -1, lane);
    for (int mi = lane; mi < mcount; mi += kWarp) {
      const long long at = (static_cast<long long>(mi) * A.ntheta + j) * A.count + f0;
      if (!Q.real) {
        const int m = mi - A.lmax;
        const double2 z = res[m < 0 ? m + n : m];
        Q.spectraOut[at] = make_double2(z.x * scale, z.y * scale);
        continue;
      }
      const double2 z = res[mi], w = res[mi == 0 ? 0 : n - mi];
      Q.spectraOut[at] = make_double2(0.5 * (z.x + w.x) * scale, 0.5 * (z.y - w.y) * scale);
      if (second) Q.spectraOut[at + 1] = make_double2(0.5 * (z.y + w.y) * scale, 0.5 * (w.x - z.x) * scale);
    }
  }
}

// -- the fixed-point form ------------------------------------------------------------------

template <int R>
__device__ __forceinline__ void FxStage(Fx2* bufs, const FxPlan& plan, int s, int from, int Ns, int G,
                                        const FxRoot* roots, const int* room) {
  const int n = plan.n, m = n / R;
  const bool last = s + 1 == plan.stages;
  const uint32_t divM = plan.divM[s], divNs = plan.divNs[s];
  const int stride = m / Ns;
  for (int e = threadIdx.x; e < G * m; e += blockDim.x) {
    const int g = m > 1 ? static_cast<int>(FxDivide(static_cast<uint32_t>(e), divM)) : e;
    const Fx2* in = bufs + g * (2 * n + 1) + from * n;
    Fx2* out = bufs + g * (2 * n + 1) + (1 - from) * n;
    // the bits above the scale given up after this stage
    const int down = FxHeadAt(room[g], Ns * R) - (last ? 0 : FxHeadAt(room[g], Ns * R * plan.radix[s + 1]));
    FxStageButterfly<R>(in, out, e - g * m, m, Ns, divNs, stride, roots, down);
  }
}

// The CTA's rings through the plan's stages, from buffer `from` of each ring;
// the buffer holding the result. The inputs carry FxHeadAt(room, first radix)
// bits above their ring's scale, the result none. Synchronises before (the
// inputs) and after every stage.
__device__ int FxTransform(Fx2* bufs, const FxPlan& plan, int from, int G, const FxRoot* roots, const int* room) {
  int Ns = 1;
  __syncthreads();
  for (int s = 0; s < plan.stages; ++s) {
    const int R = plan.radix[s];
    switch (R) {
      case 2: FxStage<2>(bufs, plan, s, from, Ns, G, roots, room); break;
      case 3: FxStage<3>(bufs, plan, s, from, Ns, G, roots, room); break;
      case 4: FxStage<4>(bufs, plan, s, from, Ns, G, roots, room); break;
      case 5: FxStage<5>(bufs, plan, s, from, Ns, G, roots, room); break;
      case 6: FxStage<6>(bufs, plan, s, from, Ns, G, roots, room); break;
      case 8: FxStage<8>(bufs, plan, s, from, Ns, G, roots, room); break;
      case 10: FxStage<10>(bufs, plan, s, from, Ns, G, roots, room); break;
      default: FxStage<12>(bufs, plan, s, from, Ns, G, roots, room); break;
    }
    from = 1 - from;
    Ns *= R;
    __syncthreads();
  }
  return from;
}

// A value reduced over the threads of its ring (thread t's ring is t % G):
// `shared` holds kFxThreads / 32 x kFxMaxRings values; every thread gets its
// ring's. Two barriers.
template <class Op>
__device__ __forceinline__ uint32_t OverRing(uint32_t v, uint32_t* shared, int G, Op op) {
  for (int off = 16; off >= G; off >>= 1) v = op(v, __shfl_xor_sync(0xffffffffu, v, off));
  const int lane = threadIdx.x % kWarp, warp = threadIdx.x / kWarp;
  __syncthreads();  // the last use of `shared`
  if (lane < G) shared[warp * kFxMaxRings + lane] = v;
  __syncthreads();
  const int g = threadIdx.x % G;
  v = shared[g];
  for (int w = 1; w < static_cast<int>(blockDim.x) / kWarp; ++w) v = op(v, shared[w * kFxMaxRings + g]);
  return v;
}

__device__ __forceinline__ uint32_t Most(uint32_t a, uint32_t b) { return max(a, b); }
__device__ __forceinline__ uint32_t Sum(uint32_t a, uint32_t b) { return a + b; }

__device__ __forceinline__ unsigned long long Bits(double v) {
  return static_cast<unsigned long long>(__double_as_longlong(v));
}

// The largest exponent of a thread's values: 0 for zeros alone, subnormal values
// counting as 1, so that a ring (or its weights) of nothing larger takes the
// FP64 form. Kept as the largest upper word and the lower words together: two
// instructions a value.
struct LargestExponent {
  uint32_t upper = 0, lower = 0;
  __device__ __forceinline__ void See(unsigned long long bits) {
    upper = max(upper, static_cast<uint32_t>(bits >> 32) & 0x7FFFFFFFu);
    lower |= static_cast<uint32_t>(bits);
  }
  __device__ __forceinline__ uint32_t Exponent() const { return max(upper >> 20, (upper | lower) != 0 ? 1u : 0u); }
};

// Whether an exponent keeps a ring's scale inside the FP64 range (a ring of
// zeros has none).
__device__ __forceinline__ bool FxCarries(uint32_t emax) {
  return emax == 0 || (emax >= kFxExponentLow && emax <= kFxExponentHigh);
}

__global__ void __launch_bounds__(kFxThreads, 2) FxRingKernel(const __grid_constant__ FxPlan plan,
                                                              const __grid_constant__ FxRingArgs A, int G) {
  extern __shared__ __align__(16) unsigned char fxSmem[];
  __shared__ uint32_t shared[kFxThreads / kWarp * kFxMaxRings];
  __shared__ int ringScale[kFxMaxRings], ringRoom[kFxMaxRings];
  __shared__ int fallback;
  const int n = plan.n, tid = threadIdx.x, T = blockDim.x;
  FxRoot* roots = reinterpret_cast<FxRoot*>(fxSmem);
  Fx2* bufs = reinterpret_cast<Fx2*>(roots + n);  // [ring][2][n], a value between the rings' (their banks apart)
  int px;  // this CTA among its part's
  const FxRingPart& Q = FxPartOf(A, px);
  const int perRing = Q.real ? 2 : 1;
  const int j = blockIdx.y, f0 = px * G * perRing;
  const int mcount = Q.real ? A.lmax + 1 : 2 * A.lmax + 1;
  const int g = tid % G, lead = tid / G, step = T / G;  // this thread's ring, and its share of the ring's values
  const int fa = f0 + g * perRing;                      // its (first) field
  const bool live = fa < A.count, second = Q.real && fa + 1 < A.count;
  const long long row0 = (static_cast<long long>(fa) * A.ntheta + j) * n;
  const long long row1 = row0 + static_cast<long long>(A.ntheta) * n;
  Fx2* ring = bufs + g * (2 * n + 1);
  auto raw = reinterpret_cast<ulonglong2*>(ring);
  for (int e = tid; e < n; e += T) roots[e] = A.roots[e];
  if (tid == 0) fallback = 0;

  // The raw values: a complex field's order m at m (or n + m); a real pair's
  // order m at m and the second field's at n - m (order 0 of both at 0).
  // Only this thread's own entries until the transform.
  LargestExponent largest;
  auto seen = [&](unsigned long long bits) { largest.See(bits); };
  const bool synth = A.mode != kFxAnalyse;
  if (synth) {
    const double2* in = Q.spectraIn + static_cast<long long>(j) * A.count + fa;
    const long long order = static_cast<long long>(A.ntheta) * A.count;
    const int zeros = Q.real ? n - (2 * A.lmax + 1) : n - mcount;  // the orders beyond lmax
    for (int k = lead; k < zeros; k += step) ring[A.lmax + 1 + k] = Fx2{0, 0};
#pragma unroll 4
    for (int mi = lead; mi < mcount; mi += step) {
      const double2 v = live ? in[mi * order] : make_double2(0.0, 0.0);
      ulonglong2 a = make_ulonglong2(Bits(v.x), Bits(v.y));
      if (!Q.real) {
        const int m = mi - A.lmax;
        raw[m < 0 ? m + n : m] = a;
      } else {
        const double2 w = second ? in[mi * order + 1] : make_double2(0.0, 0.0);
        const ulonglong2 b = make_ulonglong2(Bits(w.x), Bits(w.y));
        if (mi == 0) {
          raw[0] = make_ulonglong2(a.x, b.x);  // a real field's order 0 is real
          a.y = b.x;
        } else {
          raw[mi] = a;
          raw[n - mi] = b;
          seen(b.x);
          seen(b.y);
        }
      }
      seen(a.x);
      seen(a.y);
    }
  } else {
#pragma unroll 4
    for (int k = lead; k < n; k += step) {
      double2 v = make_double2(0.0, 0.0);
      if (live) {
        if (Q.real)
          v = make_double2(static_cast<const double*>(Q.fieldsIn)[row0 + k],
                           second ? static_cast<const double*>(Q.fieldsIn)[row1 + k] : 0.0);
        else
          v = static_cast<const double2*>(Q.fieldsIn)[row0 + k];
        if (A.pointWeight != nullptr) {
          const double w0 = A.pointWeight[row0 + k], w1 = Q.real ? (second ? A.pointWeight[row1 + k] : 0.0) : w0;
          v = make_double2(v.x * w0, v.y * w1);
        }
      }
      const ulonglong2 a = make_ulonglong2(Bits(v.x), Bits(v.y));
      raw[k] = a;
      seen(a.x);
      seen(a.y);
    }
  }
  const uint32_t emax = OverRing(largest.Exponent(), shared, G, Most);
  if (!FxCarries(emax)) fallback = 1;
  // The ring's sum of magnitudes, and its scale.
  uint32_t sum = 0;
  const int e0 = static_cast<int>(emax);
  if (e0 > 0) {
    if (synth) {
      for (int mi = lead; mi < mcount; mi += step) {
        if (!Q.real) {
          const int m = mi - A.lmax;
          const ulonglong2 a = raw[m < 0 ? m + n : m];
          sum += FxMagnitude(a.x, e0) + FxMagnitude(a.y, e0);
        } else {
          const ulonglong2 a = raw[mi];
          sum += FxMagnitude(a.x, e0) + FxMagnitude(a.y, e0);
          if (mi > 0) {
            const ulonglong2 b = raw[n - mi];
            sum += FxMagnitude(b.x, e0) + FxMagnitude(b.y, e0);
          }
        }
      }
    } else {
      for (int k = lead; k < n; k += step) {
        const ulonglong2 a = raw[k];
        sum += FxMagnitude(a.x, e0) + FxMagnitude(a.y, e0);
      }
    }
  }
  sum = OverRing(sum, shared, G, Sum);
  if (fallback) {  // uniform: set before the barriers above
    Rings64(plan, A, Q, px, reinterpret_cast<double2*>(bufs), G);
    return;
  }
  // a real pair's order m enters twice, at m and n - m
  int scale = FxScaleOf(e0, sum) - (synth && Q.real ? 1 : 0);
  const int first = plan.stages > 0 ? plan.radix[0] : n;
  const int room = e0 > 0 && plan.stages > 0 ? FxRoom(e0, scale, synth && Q.real) : 0;
  const int head = FxHeadAt(room, first);
  if (lead == 0) {
    ringScale[g] = scale;
    ringRoom[g] = room;
  }
  // To fixed point in place; the forward sum's sign by swapping the parts.
  if (synth) {
    for (int mi = lead; mi < mcount; mi += step) {
      if (!Q.real) {
        const int m = mi - A.lmax;
        const int at = m < 0 ? m + n : m;
        const ulonglong2 a = raw[at];
        ring[at] = Fx2{FxFrom(a.x, scale + head), FxFrom(a.y, scale + head)};
      } else {
        const ulonglong2 a = raw[mi];
        const Fx2 v{FxFrom(a.x, scale + head), FxFrom(a.y, scale + head)};
        if (mi == 0) {
          ring[0] = v;
        } else {
          const ulonglong2 b = raw[n - mi];
          const Fx2 u{FxFrom(b.x, scale + head), FxFrom(b.y, scale + head)};
          ring[mi] = Fx2{v.x - u.y, v.y + u.x};
          ring[n - mi] = Fx2{v.x + u.y, u.x - v.y};
        }
      }
    }
  } else {
    for (int k = lead; k < n; k += step) {
      const ulonglong2 a = raw[k];
      ring[k] = Fx2{FxFrom(a.y, scale + head), FxFrom(a.x, scale + head)};  // swapped
    }
  }
  int at = FxTransform(bufs, plan, 0, G, roots, ringRoom);
  if (A.mode == kFxSynth) {
    // by ring, longitudes adjacent
    for (int r = 0; r < G; ++r) {
      const int f = f0 + r * perRing;
      if (f >= A.count) break;
      const Fx2* res = bufs + r * (2 * n + 1) + at * n;
      const int sc = ringScale[r];
      const long long row = (static_cast<long long>(f) * A.ntheta + j) * n;
      if (Q.real) {
        auto* out = static_cast<double*>(Q.fieldsOut);
        const bool two = f + 1 < A.count;
        const long long next = row + static_cast<long long>(A.ntheta) * n;
        for (int k = tid; k < n; k += T) {
          out[row + k] = FxTo(res[k].x, sc);
          if (two) out[next + k] = FxTo(res[k].y, sc);
        }
      } else {
        auto* out = static_cast<double2*>(Q.fieldsOut);
        for (int k = tid; k < n; k += T) out[row + k] = make_double2(FxTo(res[k].x, sc), FxTo(res[k].y, sc));
      }
    }
    return;
  }
  if (A.mode == kFxWeighted) {
    // The weights under the ring's largest, in Q62 below 1; the products
    // (swapped for the analysis) and their sum of magnitudes; the rescale.
    Fx2* res = ring + at * n;
    LargestExponent weights;
    if (live)
      for (int k = lead; k < n; k += step) {
        weights.See(Bits(A.pointWeight[row0 + k]));
        if (second) weights.See(Bits(A.pointWeight[row1 + k]));
      }
    const uint32_t wmax = OverRing(weights.Exponent(), shared, G, Most);
    if (!FxCarries(wmax) || (wmax > 0 && e0 > 0 && !FxCarries(static_cast<uint32_t>(max(1, e0 + static_cast<int>(wmax) - 1023)))))
      fallback = 1;
    const int wscale = 62 - (static_cast<int>(wmax) - 1022);  // |w| 2^wscale < 2^62
    uint32_t total = 0;  // in units of 2^44, rounded up: at most 2^17 + 1 a value
    for (int k = lead; k < n; k += step) {
      const Fx2 v = res[k];
      long long a = 0, b = 0;
      if (live && wmax > 0) {
        int vh, vl, wh, wl;
        FxSplit(FxFrom(Bits(A.pointWeight[row0 + k]), wscale), wh, wl);
        FxSplit(v.x, vh, vl);
        a = FxProduct(vh, vl, wh, wl);
        if (Q.real) FxSplit(second ? FxFrom(Bits(A.pointWeight[row1 + k]), wscale) : 0, wh, wl);
        FxSplit(v.y, vh, vl);
        b = FxProduct(vh, vl, wh, wl);
      }
      res[k] = Fx2{b, a};
      total += static_cast<uint32_t>(llabs(a) >> 44) + static_cast<uint32_t>(llabs(b) >> 44) + 2;
    }
    total = OverRing(total, shared, G, Sum);
    if (fallback) {  // uniform, as above
      Rings64(plan, A, Q, px, reinterpret_cast<double2*>(bufs), G);
      return;
    }
    // the sum is below 2^61 after a shift down by `whole`, each value before it
    const int whole = 32 - __clz(total) + 44 - 61, down = whole - (plan.stages > 0 ? FxHeadAt(whole, first) : 0);
    if (lead == 0) ringRoom[g] = plan.stages > 0 ? whole : 0;
    scale += wscale - 62 - whole;
    if (down > 0) {
      const long long half = 1LL << (down - 1);
      for (int k = lead; k < n; k += step) res[k] = Fx2{(res[k].x + half) >> down, (res[k].y + half) >> down};
    } else if (down < 0) {
      for (int k = lead; k < n; k += step) res[k] = Fx2{res[k].x << -down, res[k].y << -down};
    }
    at = FxTransform(bufs, plan, at, G, roots, ringRoom);
  }
  // The orders to lmax, times 2 pi w / n, the parts swapped back.
  if (!live) return;
  const double factor = 2.0 * 3.14159265358979323846 / n * A.weights[j];
  const unsigned long long fbits = Bits(factor);
  const int fshift = FxExponent(fbits) - 1022;                  // factor = fq 2^(fshift - 62), fq < 2^62
  const long long fq = FxFrom(fbits, 62 - fshift);
  int fh, fl;
  FxSplit(fq, fh, fl);
  const int outScale = scale - fshift;
  auto scaled = [&](long long a) {
    int h, l;
    FxSplit(a, h, l);
    return FxTo(FxProduct(h, l, fh, fl), outScale);
  };
  const Fx2* res = ring + at * n;
  double2* out = Q.spectraOut + static_cast<long long>(j) * A.count + fa;
  const long long order = static_cast<long long>(A.ntheta) * A.count;
#pragma unroll 2
  for (int mi = lead; mi < mcount; mi += step) {
    if (!Q.real) {
      const int m = mi - A.lmax;
      const Fx2 z = res[m < 0 ? m + n : m];
      out[mi * order] = make_double2(scaled(z.y), scaled(z.x));
    } else {
      // X_m = (Z_m + conj Z_{n-m}) / 2, Y_m = (Z_m - conj Z_{n-m}) / 2i
      const Fx2 z = res[mi], w = res[mi == 0 ? 0 : n - mi];  // (imaginary, real)
      const long long xr = (z.y + w.y) >> 1, xi = (z.x - w.x) >> 1, yr = (z.x + w.x) >> 1, yi = (w.y - z.y) >> 1;
      out[mi * order] = make_double2(scaled(xr), scaled(xi));
      if (second) out[mi * order + 1] = make_double2(scaled(yr), scaled(yi));
    }
  }
}

}  // namespace

std::vector<FxRoot> MakeFxRoots(int n) {
  auto q62 = [](long double v, int* h, int* l) {
    long long w = std::llrint(v * 4611686018427387904.0L);  // 2^62
    if (static_cast<int>(static_cast<uint32_t>(static_cast<unsigned long long>(w))) == INT32_MIN) ++w;  // -l stays in range
    *l = static_cast<int>(static_cast<uint32_t>(static_cast<unsigned long long>(w)));
    *h = static_cast<int>((w - *l) >> 32);
  };
  const long double pi = 3.14159265358979323846264338327950288L;
  // By the octant, so that the quarter turns are exact. The angle within it is
  // a multiple `at` <= n / 2 of 2 pi / 4n that up to eight roots share; its
  // cosine and sine are taken once (a long double is software arithmetic on Arm:
  // 400 roots took 246 us one by one, 56 so, the same bits).
  struct Angle {
    bool made = false;
    long double c = 0, s = 0;
  };
  std::vector<Angle> angles(n / 2 + 1);
  std::vector<FxRoot> roots(n);
  for (int k = 0; k < n; ++k) {
    const int octant = static_cast<int>(8LL * k / n);
    const long long at = octant % 2 ? (octant + 1) / 2 * static_cast<long long>(n) - 4LL * k
                                    : 4LL * k - octant / 2 * static_cast<long long>(n);
    Angle& a = angles[at];
    if (!a.made) {
      const long double t = 2.0L * pi * (static_cast<long double>(at) / 4) / n;
      a = Angle{true, std::cos(t), std::sin(t)};
    }
    const long double c = a.c, s = a.s;
    long double x = 0, y = 0;
    switch (octant) {
      case 0: x = c; y = s; break;
      case 1: x = s; y = c; break;
      case 2: x = -s; y = c; break;
      case 3: x = -c; y = s; break;
      case 4: x = -c; y = -s; break;
      case 5: x = -s; y = -c; break;
      case 6: x = s; y = -c; break;
      default: x = c; y = -s; break;
    }
    q62(x, &roots[k].ch, &roots[k].cl);
    q62(y, &roots[k].sh, &roots[k].sl);
  }
  return roots;
}

FxPlan FxPlanOf(int n, const int* radices, int stages) {
  FxPlan plan;
  plan.n = n;
  plan.stages = stages;
  int Ns = 1;
  auto magic = [](int d) { return d > 1 ? static_cast<uint32_t>(((1ULL << 32) + d - 1) / d) : 0u; };
  for (int s = 0; s < stages; ++s) {
    plan.radix[s] = radices[s];
    plan.divNs[s] = magic(Ns);
    plan.divM[s] = magic(n / radices[s]);
    Ns *= radices[s];
  }
  return plan;
}

bool MakeFxPlan(int n, FxPlan* plan) {
  // the fewest stages, by radices in the order a first stage stores best
  // (the odd and twice-odd strides miss the banks least), the largest last
  static constexpr int kRadix[] = {5, 10, 3, 6, 12, 8, 4, 2};
  std::vector<int> best;
  auto search = [&](auto&& self, int left, int from, std::vector<int>& taken) -> void {
    if (left == 1) {
      if (best.empty() || taken.size() < best.size()) best = taken;
      return;
    }
    if (taken.size() >= kFxMaxStages || (!best.empty() && taken.size() + 1 >= best.size())) return;
    for (int i = from; i < 8; ++i)
      if (left % kRadix[i] == 0) {
        taken.push_back(kRadix[i]);
        self(self, left / kRadix[i], i, taken);
        taken.pop_back();
      }
  };
  std::vector<int> taken;
  search(search, n, 0, taken);
  if (n > 1 && best.empty()) return false;
  *plan = FxPlanOf(n, best.data(), static_cast<int>(best.size()));
  return true;
}

int LaunchFxRings(const FxPlan& plan, FxRingArgs args, cudaStream_t stream) {
  if (args.count == 0) return SL3DGPU_OK;
  const int n = plan.n;
  // Rings a CTA: up to eight, two CTAs an SM while that leaves them two
  // (twiddles and two buffers a ring: 115 KB at four rings of 800).
  const int rings = FxRings(args);
  auto bytes = [n](int g) { return (n + static_cast<size_t>(g) * (2 * n + 1)) * 16; };
  int G = 1;
  while (G < kFxMaxRings && G < rings && bytes(2 * G) <= 115300) G *= 2;
  if (bytes(G) > 224 * 1024) {
    SetError("rings: " + std::to_string(n) + " longitudes exceed shared memory");
    return SL3DGPU_ERR_ARGUMENT;
  }
  int T = 64;  // a power of two: a multiple of G
  while (T < kFxThreads && T < G * n / 8) T *= 2;
  SL3D_CUDA(AllowDynamicSmem(FxRingKernel));
  FxRingKernel<<<dim3(FxBlocks(args, G), args.ntheta), T, bytes(G), stream>>>(plan, args, G);
  SL3D_CHECK_LAUNCH();
  return SL3DGPU_OK;
}

}  // namespace sl3dgpu
