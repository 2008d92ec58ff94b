// The FP64 Legendre contraction emulated on the tcgen05 tensor cores (see
// tc_gemm.cuh): C(i, n) (+)= sum_k A(i, k) B(k, n) in FP64 from exact BF16
// slice products (the Ozaki splitting).
//
// Splitting. Row i of A has the exponent e_i with max_k |A(i, k)| < 2^{e_i},
// column n of B the exponent f_n likewise; x = A(i, k) 2^{-e_i} (|x| < 1) is
// rounded to X = round(x 2^{7 S}) for S slices, an integer read off the
// double's bits, and X is written in balanced base-2^7 digits,
// X = sum_{p < S} s_p 2^{7 (S - 1 - p)}, |s_p| <= 64 for p > 0 and
// |s_0| <= 128: x = sum_p s_p 2^{-7 (p + 1)} to within 2^{-7 S - 1}. Integer
// arithmetic only (the FP64 units of this part are slow); the digits are
// exact in BF16.
//
// Two widths. S = 7 (49 bits, 28 slice products a step) serves a grid that
// asked for the emulation; S = 8 (56 bits, 36 products) is the default FP64
// contraction: a value within a factor eight of its row's (column's) largest
// enters with all its 53 bits and the products below 2^-63 of the row and
// column maxima are dropped, so that its error stays below the FP64 units'
// own rounding (measured against quadruple precision at lmax 33 to 256, white
// and decaying coefficients: 0.1 to 0.45 of theirs in the 2-norm). That is so in
// the norm and not value by value: at lmax 128, order 40, a column that falls
// tenfold over eight degrees leaves a result of 4e-12 of the largest with six
// digits, one that falls tenfold over three degrees those below 1e-20 with none
// (FP64 sums: fifteen). Against
// the FP64 units' register-tiled product, bound by GB300's 1.2 TF/s FP64
// pipe: 45 spin -2 fields at lmax 128, 1.12 ms a contraction there; both
// transforms of these fields, rings included, take 0.50 ms here.
//
// Products. Level d = p + q gathers sum_k s_p(A) s_q(B) over p + q = d, at
// most (d + 3) 2^12 per k in magnitude, so below 2^24 -- exact in the FP32
// accumulator -- for K <= 455 at S = 7 (d = 6) and K <= 409 at S = 8 (d = 7).
// The levels d < S are kept and joined exactly as integers, the upper ones
// into H, the last four into L, and C(i, n) = 2^{e_i + f_n} 2^{-7 (S + 1)}
// (H 2^28 + L) is rounded once to FP64 from that exact integer, by integer
// arithmetic.
//
// Infinities and NaN. A column of B holding one has no exponent; it is
// marked, and its outputs are the plain FP64 sum over k from the table and B
// themselves, as the FP64 units would give them (the packed digits of such a
// column are not used). A wait that gives up leaves NaN in its tile.
//
// Kernel. One CTA of eight warps per (32-column tile, 128-row tile, item),
// two an SM, so that one's epilogue runs beside the other's products (with 64
// columns the levels filled tensor memory and every CTA's epilogue, a third
// to a half of its time, left the tensor pipe idle); the column tiles of a row
// tile are adjacent in the launch so that its A panel is read from HBM once.
// One elected thread runs the K loop as the FP32 contraction does
// (tc_gemm.cu): it arms a stage's "full" mbarrier, issues two TMA bulk copies
// (A's S slices, 4 KB each; B's, 1 KB each), and when they have landed issues
// the step's tcgen05.mma kind::f16 into the level accumulators
// (tensor-memory columns 32 d .. 32 d + 31 of 256) and commits them to the
// stage's "empty" mbarrier. B's slices are stored as one operand of 32 S rows,
// slice q in rows 32 q .. 32 q + 31, so that one MMA of N = 32 (S - p)
// multiplies A's slice p by the slices 0 .. S - 1 - p into the consecutive
// levels p ..: a step takes S MMAs. Every wait has an iteration limit. The
// epilogue reads the levels with tcgen05.ld, two warps per lane quarter (a
// column half each), joins them and stores (or adds) the rows in range.
#include <climits>
#include <cstdint>

#include "profile.cuh"
#include "tc_gemm.cuh"

namespace sl3dgpu {
namespace {

constexpr int kTileN = kTc64TileN;
constexpr int kStages = 2;     // a CTA; two CTAs an SM
constexpr int kThreads = 256;  // eight warps: two per tensor-memory lane quarter in the epilogue
constexpr int kATile = kTcTileM * kTcTileK;  // BF16 values of one slice of an A tile: 2048 (4 KB)
constexpr int kBTile = kTileN * kTcTileK;    // of a B tile: 512 (1 KB)
constexpr int kBSlice = kTileN * 8;          // BF16 offset of the next slice's rows (4 row groups of 64)
constexpr uint32_t kTmemColumns = 256;       // up to 8 levels x 32 columns: two CTAs an SM
constexpr int kNonFinite = INT_MIN;           // the exponent of a column that holds an infinity or a NaN

static_assert(kTc64Slices * kTileN <= static_cast<int>(kTmemColumns) &&
                  kTc64SlicesFull * kTileN <= static_cast<int>(kTmemColumns),
              "the levels fit in tensor memory");

// Instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both
// K-major, N and M.
__host__ __device__ constexpr uint32_t InstrDescriptorBf16(int n, int m) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(n >> 3) << 17) |
         (static_cast<uint32_t>(m >> 4) << 24);
}

// The float of an integer of magnitude at most 256, whose upper half is its BF16
// (exact: at most eight significant bits). The integer goes in as the low bits
// of 1.5 2^23: the conversion instruction runs at a quarter of the rate.
__device__ inline uint32_t FloatBits(int integer) {
  return __float_as_uint(__uint_as_float(0x4B400000u + static_cast<uint32_t>(integer)) - 12582912.0f);
}
// The upper halves of two floats, the first lowest.
__device__ inline uint32_t UpperHalves(uint32_t a, uint32_t b) { return __byte_perm(a, b, 0x7632); }

// The exponent e with |v| < 2^e for the largest |v| of a set, from the
// largest magnitude's bits (0 for zero; subnormals count as below 2^-1022).
__device__ inline int ExponentAbove(unsigned long long magnitudeBits) {
  if (magnitudeBits == 0) return 0;
  const int biased = static_cast<int>(magnitudeBits >> 52);
  if (biased == 0x7FF) return kNonFinite;
  return biased == 0 ? -1022 : biased - 1022;
}

// v (|v| < 2^e) as S balanced base-2^7 digits of round(v 2^{7 S - e}),
// as their floats' bits. (A non-finite column's digits are arbitrary: its
// outputs do not use them.)
template <int S>
__device__ inline void Split(double v, int e, uint32_t (&s)[S]) {
  const unsigned long long bits = static_cast<unsigned long long>(__double_as_longlong(v));
  const int biased = static_cast<int>((bits >> 52) & 0x7FF);
  const long long mantissa = static_cast<long long>(bits & ((1ULL << 52) - 1)) | (biased ? (1LL << 52) : 0LL);
  // v = mantissa 2^{E - 52}, so X = mantissa 2^{E - e + 7 S - 52}: a right
  // shift by t, rounded to nearest, or with S = 8 a left one, by at most 3 where
  // E <= e - 1, and by 4 in a row (column) of subnormal values, whose E and e
  // are both -1022 and whose mantissas are below 2^52
  const int E = biased ? biased - 1023 : -1022;
  const int t = e - E + 52 - 7 * S;
  long long X = 0;
  if (7 * S < 53 || t > 0) {
    if (t < 63) X = (mantissa + (1LL << (t - 1))) >> t;
  } else {
    X = mantissa << min(-t, 4);
  }
  if (bits >> 63) X = -X;
#pragma unroll
  for (int p = S - 1; p > 0; --p) {
    int r = static_cast<int>(X & 127);
    if (r >= 64) r -= 128;
    s[p] = FloatBits(r);
    X = (X - r) >> 7;
  }
  s[0] = FloatBits(static_cast<int>(X));
}

// (H 2^28 + L) 2^scale as a double, rounded to nearest even, by
// integer arithmetic (the exact 128-bit integer's top 53 bits and its
// exponent written into the bits); values outside the normal range take the
// slow path through ldexp.
__device__ inline double JoinToDouble(long long H, long long L, int scale) {
  const __int128 T = (static_cast<__int128>(H) << 28) + L;
  if (T == 0) return 0.0;
  const bool negative = T < 0;
  const unsigned __int128 m = negative ? -static_cast<unsigned __int128>(T) : static_cast<unsigned __int128>(T);
  const unsigned long long top = static_cast<unsigned long long>(m >> 64), low = static_cast<unsigned long long>(m);
  const int bits = top ? 128 - __clzll(top) : 64 - __clzll(low);  // the integer's bit length
  const int shift = bits - 53;
  unsigned long long mantissa;
  int exponent = bits - 1 + scale;
  if (shift > 0) {
    const unsigned __int128 q = m >> shift;
    const unsigned __int128 rem = m - (q << shift), half = static_cast<unsigned __int128>(1) << (shift - 1);
    mantissa = static_cast<unsigned long long>(q);
    if (rem > half || (rem == half && (mantissa & 1))) ++mantissa;
    if (mantissa >> 53) {
      mantissa >>= 1;
      ++exponent;
    }
  } else {
    mantissa = static_cast<unsigned long long>(m) << -shift;
  }
  if (exponent < -1022 || exponent > 1023) {
    const double v = ldexp(static_cast<double>(mantissa), exponent - 52);
    return negative ? -v : v;
  }
  const unsigned long long out = (negative ? (1ULL << 63) : 0ULL) |
                                 (static_cast<unsigned long long>(exponent + 1023) << 52) |
                                 (mantissa & ((1ULL << 52) - 1));
  return __longlong_as_double(static_cast<long long>(out));
}

// Offset (in BF16 values) of element (row, k) of a K-major 16-deep tile of
// `rows` rows in the core-matrix layout [k / 8][row / 8][row % 8][k % 8].
__device__ inline int Tile16Index(int row, int k, int rows) {
  return (k >> 3) * (rows * 8) + (row >> 3) * 64 + (row & 7) * 8 + (k & 7);
}

// Eight consecutive values of one row split and stored as one 16-byte
// core-matrix row per slice; two values at a time, so that their digits are
// joined in pairs as they are made and not sixty-four registers later.
template <int S, class Value>
__device__ inline void StoreSplit(uint16_t* tile, int sliceStride, int at, int e, Value value) {
  uint32_t words[4][S];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    uint32_t a[S], b[S];
    Split<S>(value(2 * q), e, a);
    Split<S>(value(2 * q + 1), e, b);
#pragma unroll
    for (int p = 0; p < S; ++p) words[q][p] = UpperHalves(a[p], b[p]);
  }
#pragma unroll
  for (int p = 0; p < S; ++p)
    *reinterpret_cast<uint4*>(tile + p * sliceStride + at) =
        make_uint4(words[0][p], words[1][p], words[2][p], words[3][p]);
}

// One output as the FP64 units sum it, for a column holding an infinity or a
// NaN.
__device__ __noinline__ double PlainSum(const GemmItem& g, const double* table, const double* B, int i, int n) {
  double sum = 0.0;
  for (int k = 0; k < g.K; ++k)
    sum = fma(table[g.a + static_cast<long long>(i) * g.sAi + static_cast<long long>(k) * g.sAk],
              B[g.b + static_cast<long long>(k) * g.ldb + n], sum);
  return sum;
}

// Row exponents of A, one thread per (item, row): the maximum over the
// item's depth.
__global__ void RowExpKernel(const GemmItem* items, const Tc64Item* tcItems, const double* table, int* rowExp) {
  const GemmItem g = items[blockIdx.y];
  const Tc64Item it = tcItems[blockIdx.y];
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < g.M; i += gridDim.x * blockDim.x) {
    unsigned long long mx = 0;
    for (int k = 0; k < g.K; ++k) {
      const double v = table[g.a + static_cast<long long>(i) * g.sAi + static_cast<long long>(k) * g.sAk];
      mx = max(mx, static_cast<unsigned long long>(__double_as_longlong(v)) & 0x7FFFFFFFFFFFFFFFULL);
    }
    rowExp[it.rowExp + i] = ExponentAbove(mx);
  }
}

// A's panel: one thread per (item, tile, 8-deep K group, row).
template <int S>
__global__ void PanelA64Kernel(const GemmItem* items, const Tc64Item* tcItems, const double* table,
                               const int* rowExp, uint16_t* panels) {
  const GemmItem g = items[blockIdx.y];
  const Tc64Item it = tcItems[blockIdx.y];
  const long long total = static_cast<long long>(it.mTiles) * it.kSteps * 2 * kTcTileM;
  for (long long t = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; t < total;
       t += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int r = static_cast<int>(t % kTcTileM);
    const long long rest = t / kTcTileM;
    const int kg = static_cast<int>(rest % 2);
    const long long tile = rest / 2;
    const int ks = static_cast<int>(tile % it.kSteps), mt = static_cast<int>(tile / it.kSteps);
    const int i = mt * kTcTileM + r, k0 = ks * kTcTileK + 8 * kg;
    const int e = i < g.M ? rowExp[it.rowExp + i] : 0;
    StoreSplit<S>(panels + (it.aPanel + tile) * S * kATile, kATile, Tile16Index(r, 8 * kg, kTcTileM), e, [&](int q) {
      const int k = k0 + q;
      return (i < g.M && k < g.K)
                 ? table[g.a + static_cast<long long>(i) * g.sAi + static_cast<long long>(k) * g.sAk]
                 : 0.0;
    });
  }
}

// B's column exponents and packed slices, one CTA of 256 threads per
// (column tile, item): 32 columns x 8 lanes along k. The exponents first
// (each lane's maximum over its k, then over the eight lanes), then the
// slices, 8-deep k groups in turn; a warp's reads of one k are 32
// consecutive columns and its stores of one slice 512 contiguous bytes.
// Latency bounds it, and so the threads an SM holds: at 64 registers, four CTAs
// (92 fields at lmax 64 for three spins, 37 -> 32 us; reading a group ahead
// took 98 registers and 51 us).
constexpr int kPackThreads = 256, kPackLanes = kPackThreads / kTileN;

template <int S>
__global__ void __launch_bounds__(kPackThreads, 4) PackB64Kernel(const Tc64Item* tcItems, const double* B, int* colExp,
                                                              uint16_t* packed) {
  const Tc64Item it = tcItems[blockIdx.y];
  const int nt = blockIdx.x;
  if (nt >= it.nTiles) return;
  __shared__ unsigned long long largest[kPackLanes][kTileN];
  const int nn = threadIdx.x % kTileN, lane = threadIdx.x / kTileN;
  const int n = nt * kTileN + nn;
  const double* col = B + it.b + n;
  unsigned long long mx = 0;
  if (n < it.N)
    for (int k = lane; k < it.K; k += kPackLanes)
      mx = max(mx, static_cast<unsigned long long>(__double_as_longlong(col[static_cast<long long>(k) * it.ldb])) &
                       0x7FFFFFFFFFFFFFFFULL);
  largest[lane][nn] = mx;
  __syncthreads();
  for (int q = 0; q < kPackLanes; ++q) mx = max(mx, largest[q][nn]);
  const int e = ExponentAbove(mx);
  if (lane == 0 && n < it.N) colExp[it.colExp + n] = e;
  uint16_t* base = packed + (it.bPack + static_cast<long long>(nt) * it.kSteps) * S * kBTile;
  for (int group = lane; group < 2 * it.kSteps; group += kPackLanes) {
    const int ks = group / 2, kg = group % 2, k0 = 8 * group;
    double v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int k = k0 + q;
      v[q] = (n < it.N && k < it.K) ? col[static_cast<long long>(k) * it.ldb] : 0.0;
    }
    StoreSplit<S>(base + static_cast<long long>(ks) * S * kBTile, kBSlice, Tile16Index(nn, 8 * kg, S * kTileN), e,
                  [&](int q) { return v[q]; });
  }
}

template <int S>
__global__ void __launch_bounds__(kThreads, 2) TcGemm64Kernel(const GemmItem* items, const Tc64Item* tcItems,
                                                           const Tc64Tables tables, const double* B,
                                                           const uint16_t* panels, const uint16_t* packed,
                                                           const int* rowExp, const int* colExp, double* C,
                                                           bool accumulate, int* errorFlag) {
  constexpr int kSlices = S;
  constexpr int kBRows = kSlices * kTileN;  // B's slices as one operand
  const Tc64Item it = tcItems[blockIdx.z];
  const int nt = blockIdx.x, mt = blockIdx.y;
  if (mt >= it.mTiles || nt >= it.nTiles) return;  // the whole CTA, before any tensor-memory work
  const int i0 = mt * kTcTileM, n0 = nt * kTileN;
  const int nCols = min(kTileN, it.N - n0);
  constexpr uint32_t aBytes = kSlices * kATile * 2, bBytes = kSlices * kBTile * 2;

  extern __shared__ __align__(128) unsigned char tc64Smem[];
  uint16_t* sA = reinterpret_cast<uint16_t*>(tc64Smem);  // kStages x kSlices x kATile
  uint16_t* sB = sA + kStages * kSlices * kATile;          // kStages x kSlices x kBTile
  uint64_t* full = reinterpret_cast<uint64_t*>(sB + kStages * kSlices * kBTile);
  uint64_t* empty = full + kStages;
  uint32_t* tmemSlot = reinterpret_cast<uint32_t*>(empty + kStages);
  __shared__ int okShared;
  // the epilogue's staging, each warp's 32 x 16 block padded, in the stages'
  // memory (every MMA has read them by then)
  auto rowsOut = reinterpret_cast<double (*)[32][17]>(tc64Smem);
  const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(SmemAddr(tmemSlot)),
                 "r"(kTmemColumns)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(SmemAddr(full + s)), "r"(1) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(SmemAddr(empty + s)), "r"(1) : "memory");
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmemSlot;

  if (tid == 0) {
    const uint16_t* aSrc = panels + (it.aPanel + static_cast<long long>(mt) * it.kSteps) * kSlices * kATile;
    const uint16_t* bSrc = packed + (it.bPack + static_cast<long long>(nt) * it.kSteps) * kSlices * kBTile;
    uint32_t phaseFull[kStages] = {}, phaseEmpty[kStages] = {};
    bool ok = true;
    int issued = 0, landed = 0;  // steps whose copies were started, and waited for
    auto issue = [&](int ks) {
      const int buf = ks % kStages;
      if (ks >= kStages) {
        ok = ok && WaitParity(SmemAddr(empty + buf), phaseEmpty[buf]);
        phaseEmpty[buf] ^= 1u;
      }
      if (!ok) return;
      const uint32_t bar = SmemAddr(full + buf);
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(aBytes + bBytes)
                   : "memory");
      asm volatile(
          "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
              SmemAddr(sA + buf * kSlices * kATile)),
          "l"(aSrc + static_cast<long long>(ks) * kSlices * kATile), "r"(aBytes), "r"(bar)
          : "memory");
      asm volatile(
          "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
              SmemAddr(sB + buf * kSlices * kBTile)),
          "l"(bSrc + static_cast<long long>(ks) * kSlices * kBTile), "r"(bBytes), "r"(bar)
          : "memory");
      ++issued;
    };
    for (int ks = 0; ks < min(kStages - 1, it.kSteps); ++ks) issue(ks);
    for (int ks = 0; ks < it.kSteps && ok; ++ks) {
      if (ks + kStages - 1 < it.kSteps) issue(ks + kStages - 1);
      if (!ok) break;
      const int buf = ks % kStages;
      ok = WaitParity(SmemAddr(full + buf), phaseFull[buf]);
      phaseFull[buf] ^= 1u;
      if (!ok) break;
      ++landed;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t aBase = SmemAddr(sA + buf * kSlices * kATile);
      const uint32_t bBase = SmemAddr(sB + buf * kSlices * kBTile);
      constexpr uint32_t aLbo = kTcTileM * 16, bLbo = kBRows * 16, sbo = 128;
      // A's slice p against B's slices 0 .. S - 1 - p (N = 32 (S - p)), levels
      // p .. S - 1; p = 0 writes every level first.
#pragma unroll
      for (int p = 0; p < kSlices; ++p) {
        const uint64_t dA = Descriptor(aBase + p * kATile * 2, aLbo, sbo);
        const uint64_t dB = Descriptor(bBase, bLbo, sbo);
        const uint32_t enable = (ks > 0 || p > 0) ? 1u : 0u;
        asm volatile(
            "{\n\t.reg .pred r;\n\t"
            "setp.ne.b32 r, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, r;\n\t}" ::"r"(tmem + p * kTileN),
            "l"(dA), "l"(dB), "r"(InstrDescriptorBf16((kSlices - p) * kTileN, kTcTileM)), "r"(enable)
            : "memory");
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                       SmemAddr(empty + buf))
                   : "memory");
    }
    // The last step's commit covers every MMA before it.
    if (ok && it.kSteps > 0) {
      const int last = (it.kSteps - 1) % kStages;
      ok = WaitParity(SmemAddr(empty + last), phaseEmpty[last]);
    }
    // having given up, wait (bounded) for the copies still in flight
    if (!ok)
      for (int ks = landed; ks < issued; ++ks)
        WaitParity(SmemAddr(full + ks % kStages), phaseFull[ks % kStages]);
    okShared = ok ? 1 : 0;
    if (!ok) ReportGiveUp(errorFlag);
  }
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const bool good = okShared != 0;
  {
    // Epilogue: this warp's lane quarter (32 rows) and column half, 16
    // columns at a time, the levels joined as integers and rounded once to
    // FP64.
    const int quarter = warp % 4, half = warp / 4;
    const int i = i0 + 32 * quarter + lane;
    const int e = i < it.M ? rowExp[it.rowExp + i] : 0;
    for (int c0 = half * (kTileN / 2); c0 < (half + 1) * (kTileN / 2); c0 += 16) {
      uint32_t r[kSlices][16];
#pragma unroll
      for (int d = 0; d < kSlices; ++d) {
        const uint32_t addr =
            tmem + (static_cast<uint32_t>(32 * quarter) << 16) + static_cast<uint32_t>(d * kTileN + c0);
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
            "%14, %15}, [%16];"
            : "=r"(r[d][0]), "=r"(r[d][1]), "=r"(r[d][2]), "=r"(r[d][3]), "=r"(r[d][4]), "=r"(r[d][5]),
              "=r"(r[d][6]), "=r"(r[d][7]), "=r"(r[d][8]), "=r"(r[d][9]), "=r"(r[d][10]), "=r"(r[d][11]),
              "=r"(r[d][12]), "=r"(r[d][13]), "=r"(r[d][14]), "=r"(r[d][15])
            : "r"(addr)
            : "memory");
      }
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      // the joined values of this lane's row, then out through shared memory
      // so that a store instruction writes two rows' 16 consecutive columns
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        const int n = c0 + q;
        double v = 0.0;
        if (i < it.M && n < nCols) {
          long long acc[kSlices];
#pragma unroll
          for (int d = 0; d < kSlices; ++d) acc[d] = __float2int_rn(__uint_as_float(r[d][q]));
          long long H = 0, L = 0;
#pragma unroll
          for (int d = 0; d < kSlices - 4; ++d) H += acc[d] << (7 * (kSlices - 5 - d));
#pragma unroll
          for (int d = kSlices - 4; d < kSlices; ++d) L += acc[d] << (7 * (kSlices - 1 - d));
          v = JoinToDouble(H, L, e + colExp[it.colExp + n0 + n] - 7 * (kSlices + 1));
        }
        rowsOut[warp][lane][q] = v;
      }
      // a non-finite column among these 16 (or a wait that gave up): rare
      const bool marked = lane < 16 && c0 + lane < nCols && colExp[it.colExp + n0 + c0 + lane] == kNonFinite;
      const unsigned columns = __ballot_sync(0xffffffffu, marked);
      if (!good || columns != 0) {
        for (int q = 0; q < 16; ++q)
          if (!good)
            rowsOut[warp][lane][q] = __longlong_as_double(0x7FF8000000000000LL);
          else if (((columns >> q) & 1u) && i < it.M)
            rowsOut[warp][lane][q] = PlainSum(items[blockIdx.z], tables.of[items[blockIdx.z].table], B, i, n0 + c0 + q);
      }
      __syncwarp();
      const int n = c0 + (lane & 15);
      // this lane's 16 rows' old values first (loads in flight together), then the stores
      double old[16];
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        const int row = i0 + 32 * quarter + 2 * q + (lane >> 4);
        old[q] = (accumulate && row < it.M && n < nCols) ? C[it.c + static_cast<long long>(row) * it.ldc + n0 + n]
                                                         : 0.0;
      }
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        const int rr = 2 * q + (lane >> 4), row = i0 + 32 * quarter + rr;
        if (row < it.M && n < nCols)
          C[it.c + static_cast<long long>(row) * it.ldc + n0 + n] = old[q] + rowsOut[warp][rr][lane & 15];
      }
      __syncwarp();
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemColumns) : "memory");
}

}  // namespace

namespace {
template <int S>
int Run(const GemmItem* items, const Tc64Item* tcItems, int count, int maxMTiles, int maxNTiles, const Tc64Tables& tables,
        const Tc64Panel& panel, const double* B, uint16_t* packed, int* colExp, double* C, bool accumulate,
        int* errorFlag, cudaStream_t stream) {
  constexpr size_t smem = static_cast<size_t>(kStages) * S * (kATile + kBTile) * sizeof(uint16_t) +
                          2 * kStages * sizeof(uint64_t) + 16;
  static_assert(smem <= 226 * 1024, "the stages fit in shared memory");
  static_assert(smem >= kThreads / 32 * 32 * 17 * sizeof(double), "the epilogue's staging fits in the stages");
  SL3D_CUDA(AllowDynamicSmem(TcGemm64Kernel<S>));
  dim3 grid(static_cast<unsigned>(maxNTiles), static_cast<unsigned>(maxMTiles), static_cast<unsigned>(count));
  TcGemm64Kernel<S><<<grid, kThreads, smem, stream>>>(items, tcItems, tables, B, panel.slices, packed, panel.rowExp,
                                                      colExp, C, accumulate, errorFlag);
  SL3D_CHECK_LAUNCH();
  return SL3DGPU_OK;
}
}  // namespace

void LaunchPanelA64(int slices, const GemmItem* items, const Tc64Item* tcItems, int count, int maxM, int maxATiles,
                    const double* table, const Tc64Panel& panel, cudaStream_t stream) {
  if (count == 0) return;
  RowExpKernel<<<dim3(static_cast<unsigned>((maxM + 127) / 128), count), 128, 0, stream>>>(items, tcItems, table,
                                                                                          panel.rowExp);
  const long long perItem = static_cast<long long>(maxATiles) * 2 * kTcTileM;
  const dim3 grid(static_cast<unsigned>(std::min<long long>((perItem + 255) / 256, 4096)), count);
  if (slices == kTc64SlicesFull)
    PanelA64Kernel<kTc64SlicesFull><<<grid, 256, 0, stream>>>(items, tcItems, table, panel.rowExp, panel.slices);
  else
    PanelA64Kernel<kTc64Slices><<<grid, 256, 0, stream>>>(items, tcItems, table, panel.rowExp, panel.slices);
}

void LaunchPackB64(int slices, const Tc64Item* tcItems, int count, int maxNTiles, const double* B, int* colExp,
                   uint16_t* packed, cudaStream_t stream) {
  if (count == 0 || maxNTiles == 0) return;
  const dim3 grid(static_cast<unsigned>(maxNTiles), count);
  if (slices == kTc64SlicesFull)
    PackB64Kernel<kTc64SlicesFull><<<grid, kPackThreads, 0, stream>>>(tcItems, B, colExp, packed);
  else
    PackB64Kernel<kTc64Slices><<<grid, kPackThreads, 0, stream>>>(tcItems, B, colExp, packed);
}

int RunGemm64Tc(int slices, const GemmItem* items, const Tc64Item* tcItems, int count, int maxMTiles, int maxNTiles,
                const Tc64Tables& tables, const Tc64Panel& panel, const double* B, uint16_t* packed, int* colExp,
                double* C, bool accumulate, int* errorFlag, cudaStream_t stream) {
  if (count == 0 || maxMTiles == 0 || maxNTiles == 0) return SL3DGPU_OK;
  return slices == kTc64SlicesFull
             ? Run<kTc64SlicesFull>(items, tcItems, count, maxMTiles, maxNTiles, tables, panel, B, packed, colExp, C,
                                    accumulate, errorFlag, stream)
             : Run<kTc64Slices>(items, tcItems, count, maxMTiles, maxNTiles, tables, panel, B, packed, colExp, C,
                                accumulate, errorFlag, stream);
}

}  // namespace sl3dgpu
