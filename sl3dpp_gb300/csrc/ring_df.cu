// The longitude transforms of FP64 values in double-float, for the grids that
// asked for the FP64 emulation (the mixed form's FP64 passes).
//
// Why beside the fixed-point rings (ring_fixed.cu): the mixed form stops its
// iteration at its tolerance, where the FP32 corrections' path has left an
// error of a few 1e-9 in the strain at lmax 256, and another rounding takes
// another path; these rings keep the form's results as they are, bit for
// bit. They are also no slower: the FP32 pipe does the sums at a quarter of a
// cycle an SM, and their conversions are integer arithmetic (ring_df.cuh;
// both transforms of 55 spin -1 fields at lmax 256 went from 3.29 to 2.62 ms
// when the FP64 unit no longer made them).
//
// One CTA per (colatitude, G consecutive fields); the values are converted as
// they are read, and the Stockham stages run over the CTA's butterflies,
// ping-ponging between two buffers a ring. The modes, layouts and real pairs
// are the fixed-point kernel's.
#include <algorithm>

#include "profile.cuh"
#include "ring_df.cuh"

namespace sl3dgpu {

namespace {

enum { kDfSynth = 0, kDfAnalyse = 1, kDfWeighted = 2 };

constexpr int kDfThreads = 256;
constexpr int kDfMaxRings = 8;

__device__ __forceinline__ Df2 FromDouble2(double2 v) {
  Df2 r;
  r.x = FromDouble(v.x);
  r.y = FromDouble(v.y);
  return r;
}

template <int R>
__device__ __forceinline__ void DfStage(Df2* bufs, const FxPlan& plan, int s, int from, int Ns, int G, const Df2* tw,
                                        int sign) {
  const int n = plan.n, m = n / R, stride = m / Ns;
  const uint32_t divM = plan.divM[s], divNs = plan.divNs[s];
  for (int e = threadIdx.x; e < G * m; e += blockDim.x) {
    const int g = m > 1 ? static_cast<int>(FxDivide(static_cast<uint32_t>(e), divM)) : e;
    const int idx = e - g * m;
    const int blk = Ns > 1 ? static_cast<int>(FxDivide(static_cast<uint32_t>(idx), divNs)) : idx;
    const int k = idx - blk * Ns;
    const Df2* in = bufs + g * (2 * n + 1) + from * n;
    Df2* out = bufs + g * (2 * n + 1) + (1 - from) * n;
    Df2 v[R];
#pragma unroll
    for (int q = 0; q < R; ++q) v[q] = in[idx + q * m];
    if (k > 0) {
#pragma unroll
      for (int q = 1; q < R; ++q) {
        Df2 w = tw[q * k * stride];
        if (sign < 0) w.y = -w.y;
        v[q] = Mul(v[q], w);
      }
    }
    Butterfly<Df2, R>(v, sign);
    const int base = blk * Ns * R + k;
#pragma unroll
    for (int u = 0; u < R; ++u) out[base + u * Ns] = v[u];
  }
}

// The CTA's rings through the plan's stages, from buffer `from`; the buffer
// holding the result.
__device__ int DfTransform(Df2* bufs, const FxPlan& plan, int from, int G, const Df2* tw, int sign) {
  int Ns = 1;
  __syncthreads();
  for (int s = 0; s < plan.stages; ++s) {
    const int R = plan.radix[s];
    if (R == 4)
      DfStage<4>(bufs, plan, s, from, Ns, G, tw, sign);
    else if (R == 2)
      DfStage<2>(bufs, plan, s, from, Ns, G, tw, sign);
    else if (R == 3)
      DfStage<3>(bufs, plan, s, from, Ns, G, tw, sign);
    else
      DfStage<5>(bufs, plan, s, from, Ns, G, tw, sign);
    from = 1 - from;
    Ns *= R;
    __syncthreads();
  }
  return from;
}

__global__ void __launch_bounds__(kDfThreads, 2) DfRingKernel(const __grid_constant__ FxPlan plan,
                                                              const __grid_constant__ FxRingArgs A, int G) {
  extern __shared__ __align__(16) unsigned char dfSmem[];
  const int n = plan.n, tid = threadIdx.x, T = blockDim.x;
  Df2* tw = reinterpret_cast<Df2*>(dfSmem);
  Df2* bufs = tw + n;  // [ring][2][n], a value between the rings' (their banks apart)
  int px;  // this CTA among its part's
  const FxRingPart& Q = FxPartOf(A, px);
  const int perRing = Q.real ? 2 : 1;
  const int j = blockIdx.y, f0 = px * G * perRing;
  const int mcount = Q.real ? A.lmax + 1 : 2 * A.lmax + 1;
  const int g = tid % G, lead = tid / G, step = T / G;
  const int fa = f0 + g * perRing;
  const bool live = fa < A.count, second = Q.real && fa + 1 < A.count;
  const long long rows = static_cast<long long>(A.ntheta) * n;  // a field's values
  Df2* ring = bufs + g * (2 * n + 1);
  const Df zero(0.0f, 0.0f);
  const Df2 zero2 = Make<Df2>(zero, zero);
  for (int e = tid; e < n; e += T) tw[e] = FromDouble2(A.twiddle[e]);
  int at = 0;
  const double2* in = Q.spectraIn + static_cast<long long>(j) * A.count + fa;
  const long long order = static_cast<long long>(A.ntheta) * A.count;
  if (A.mode != kDfAnalyse) {
    const int zeros = n - (2 * A.lmax + 1);  // the orders beyond lmax
    for (int k = lead; k < zeros; k += step) ring[A.lmax + 1 + k] = zero2;
#pragma unroll 4
    for (int mi = lead; mi < mcount; mi += step) {
      const Df2 v = live ? FromDouble2(in[mi * order]) : zero2;
      if (!Q.real) {
        const int m = mi - A.lmax;
        ring[m < 0 ? m + n : m] = v;
      } else {
        const Df2 u = second ? FromDouble2(in[mi * order + 1]) : zero2;
        if (mi == 0) {
          ring[0] = Make<Df2>(v.x, u.x);
        } else {
          ring[mi] = Make<Df2>(v.x - u.y, v.y + u.x);      // v + i u
          ring[n - mi] = Make<Df2>(v.x + u.y, u.x - v.y);  // conj(v) + i conj(u)
        }
      }
    }
    at = DfTransform(bufs, plan, 0, G, tw, 1);
    // by ring, longitudes adjacent
    for (int r = 0; r < G; ++r) {
      const int f = f0 + r * perRing;
      if (f >= A.count) break;
      Df2* res = bufs + r * (2 * n + 1) + at * n;
      const long long row = static_cast<long long>(f) * rows + static_cast<long long>(j) * n, next = row + rows;
      const bool two = Q.real && f + 1 < A.count;
      if (A.mode == kDfWeighted) {
#pragma unroll 2
        for (int k = tid; k < n; k += T) {
          const Df w0 = FromDouble(A.pointWeight[row + k]);
          const Df w1 = Q.real ? (two ? FromDouble(A.pointWeight[next + k]) : zero) : w0;
          const Df2 v = res[k];
          res[k] = Make<Df2>(v.x * w0, v.y * w1);
        }
      } else if (Q.real) {
        auto* out = static_cast<double*>(Q.fieldsOut);
        for (int k = tid; k < n; k += T) {
          out[row + k] = ToDouble(res[k].x);
          if (two) out[next + k] = ToDouble(res[k].y);
        }
      } else {
        auto* out = static_cast<double2*>(Q.fieldsOut);
        for (int k = tid; k < n; k += T) out[row + k] = make_double2(ToDouble(res[k].x), ToDouble(res[k].y));
      }
    }
    if (A.mode == kDfSynth) return;
  } else {
    for (int r = 0; r < G; ++r) {
      const int f = f0 + r * perRing;
      Df2* to = bufs + r * (2 * n + 1);
      const long long row = static_cast<long long>(f) * rows + static_cast<long long>(j) * n, next = row + rows;
      const bool one = f < A.count, two = Q.real && f + 1 < A.count;
#pragma unroll 2
      for (int k = tid; k < n; k += T) {
        Df2 v = zero2;
        if (one) {
          if (Q.real)
            v = Make<Df2>(FromDouble(static_cast<const double*>(Q.fieldsIn)[row + k]),
                          two ? FromDouble(static_cast<const double*>(Q.fieldsIn)[next + k]) : zero);
          else
            v = FromDouble2(static_cast<const double2*>(Q.fieldsIn)[row + k]);
          if (A.pointWeight != nullptr) {
            const Df w0 = FromDouble(A.pointWeight[row + k]);
            const Df w1 = Q.real ? (two ? FromDouble(A.pointWeight[next + k]) : zero) : w0;
            v = Make<Df2>(v.x * w0, v.y * w1);
          }
        }
        to[k] = v;
      }
    }
  }
  at = DfTransform(bufs, plan, at, G, tw, -1);
  if (!live) return;
  const Df scale = FromDouble(2.0 * 3.14159265358979323846 / n * A.weights[j]), half(0.5);
  const Df2* res = ring + at * n;
  double2* out = Q.spectraOut + static_cast<long long>(j) * A.count + fa;
#pragma unroll 2
  for (int mi = lead; mi < mcount; mi += step) {
    if (!Q.real) {
      const int m = mi - A.lmax;
      const Df2 v = res[m < 0 ? m + n : m];
      out[mi * order] = make_double2(ToDouble(v.x * scale), ToDouble(v.y * scale));
    } else {
      // X_m = (Z_m + conj Z_{n-m}) / 2, Y_m = (Z_m - conj Z_{n-m}) / 2i
      const Df2 z = res[mi], w = res[mi == 0 ? 0 : n - mi];
      out[mi * order] =
          make_double2(ToDouble((half * (z.x + w.x)) * scale), ToDouble((half * (z.y - w.y)) * scale));
      if (second)
        out[mi * order + 1] =
            make_double2(ToDouble((half * (z.y + w.y)) * scale), ToDouble((half * (w.x - z.x)) * scale));
    }
  }
}

}  // namespace

int LaunchDfRings(const FxPlan& plan, FxRingArgs args, cudaStream_t stream) {
  if (args.count == 0) return SL3DGPU_OK;
  const int n = plan.n;
  // Rings a CTA as the fixed-point kernel takes them: up to eight, two CTAs an SM.
  const int rings = FxRings(args);
  auto bytes = [n](int g) { return (n + static_cast<size_t>(g) * (2 * n + 1)) * 16; };
  int G = 1;
  while (G < kDfMaxRings && G < rings && bytes(2 * G) <= 115300) G *= 2;
  if (bytes(G) > 224 * 1024) {
    SetError("rings: " + std::to_string(n) + " longitudes exceed shared memory");
    return SL3DGPU_ERR_ARGUMENT;
  }
  int T = 64;
  while (T < kDfThreads && T < G * n / 4) T *= 2;
  SL3D_CUDA(AllowDynamicSmem(DfRingKernel));
  DfRingKernel<<<dim3(FxBlocks(args, G), args.ntheta), T, bytes(G), stream>>>(plan, args, G);
  SL3D_CHECK_LAUNCH();
  return SL3DGPU_OK;
}

}  // namespace sl3dgpu
