// The device spherical-harmonic grid: Gauss-Legendre colatitudes, uniform
// longitudes, the stored spin-N Legendre (Wigner-d) tables and the FFT plan,
// with the batched transforms between coefficients and grid values.
//
// Basis (docs/design.md:245-250 of the reference): Y^N_lm =
// sqrt((2l+1)/4pi) d^l_{Nm}(theta) e^{i m phi}, d^l_{0m} the Condon-Shortley
// associated Legendre function; forward transform the integral of conj(Y) f.
// Reference index layouts (include/sl3dpp/SurfaceGrid.hpp:110-118, 191-200):
// spin N complex, l^2 - N^2 + (m + l) over l = |N|..lmax and every m; real
// spin 0, l(l+1)/2 + m over m >= 0. Grid values colatitude-major, longitude
// k at 2 pi k / nphi.
//
// Device ("m-major") layouts, what the kernels read and write: a batch of
// `count` fields keeps, per spin, the coefficients of order m and degree l at
// row RowOffset(m) + (l - l0(m)) of a [row][count] complex array (the node
// fastest), so that one order's degrees over the batch are one dense matrix;
// ring spectra are [m][j][count] complex.
#pragma once

#include <array>
#include <climits>
#include <cstdint>
#include <functional>
#include <map>
#include <memory>
#include <mutex>
#include <vector>

#include "common.cuh"
#include "ring_fixed.cuh"

namespace sl3dgpu {

struct FftPlan {
  int n = 0;
  int stages = 0;
  int radix[16] = {};
};

// One spin's table: for each order m in [-lmax, lmax] (index m + lmax) a
// block of (lmax - l0 + 1) rows of ntheta values, rows = degrees.
struct SpinTable {
  int N = 0;
  std::vector<int> rowOffset;  // 2 lmax + 2 entries, cumulative rows by m index
  double* values = nullptr;    // device
  int* dRowOffset = nullptr;   // device copy of rowOffset
  int Rows(int m, int lmax) const { return rowOffset[m + lmax + 1] - rowOffset[m + lmax]; }
};

struct GemmItem {
  int M, N, K;
  int table;  // which of its batch's tables A is in
  long long a, b, c;
  int sAi, sAk, ldb, ldc;
};

// One item of the FP64 contraction emulated on the tensor cores: 128-row
// tiles of A, 32-column tiles of B, 16-deep steps.
struct Tc64Item {
  int M, N, K, mTiles;
  int kSteps, nTiles, ldc, ldb;
  long long aPanel;  // tiles: the item's panel, [mTile][kStep] of [slice][128 x 16]
  long long bPack;   // tiles: its packed B, [nTile][kStep] of [slice][32 x 16]
  long long b, c;    // FP64 offsets of B's source and of C
  long long rowExp;  // ints: the power-of-two exponents of its M rows of A
  long long colExp;  // ints: those of its N columns of B (per call)
};

// A batch's FP64 tables (a tensor's three spins, or one).
struct Tc64Tables {
  const double* of[3] = {nullptr, nullptr, nullptr};
};

// The table split into FP64 slices for one direction: its slice panels and
// row exponents.
struct Tc64Panel {
  uint16_t* slices = nullptr;
  int* rowExp = nullptr;
};

// A tensor-core item's host description (mirrors TcItem in tc_gemm.cuh).
struct TcItemHost {
  int M, N, K, mTiles;
  int kSteps, nTiles, ldc, ldb;
  long long aPanel, bPack;
  long long b, c;
};

class Grid {
 public:
  static int Create(int lmax, int nmax, double oversampling, std::unique_ptr<Grid>& out);
  ~Grid();

  int lmax = 0, nmax = 0, band = 0, ntheta = 0, nphi = 0;
  // The FP64 contractions run as slice products on the tensor cores
  // (tc_gemm64.cu): eight slices, at least the FP64 units' accuracy in the norm,
  // or, with this set, seven (about 49 bits) and the rings in double-float. Batches of
  // few columns and ones deeper than the slices' exactness bound keep the
  // FP64 units.
  bool emulateFp64 = false;
  std::vector<double> theta, weights;  // host copies
  double* dTheta = nullptr;
  double* dWeights = nullptr;
  double2* dTwiddle = nullptr;
  float2* dTwiddle32 = nullptr;
  FxRoot* dRoots = nullptr;  // the fixed-point rings' roots of unity
  FxPlan fxPlan, dfPlan;
  FftPlan plan;

  // The table of spin N, built on first use (device kernel).
  int Table(int N, const SpinTable** out);
  // Rows of one spin's coefficients per field (its (l, m) count).
  long long SpinRows(int N) const { return static_cast<long long>(lmax + 1) * (lmax + 1) - N * N; }
  // Rows of a real spin-0 field (m >= 0).
  long long RealRows() const { return static_cast<long long>(lmax + 1) * (lmax + 2) / 2; }

  // -- transforms in the device layouts -------------------------------------------
  // Spin N: coefficients [row][P] complex (columns p0 .. p0 + count of them
  // taking part) -> spectra [m][j][count] -> fields [count][j][k] complex;
  // and back. Real spin 0 likewise with m >= 0 rows. The analysis may add its
  // result to what the coefficients hold (the memory force's fixed part).
  int LegendreSynthesis(int N, bool real, const double* coeffs, int P, int p0, int count,
                        double* spectra, cudaStream_t stream);
  int LegendreAnalysis(int N, bool real, const double* spectra, int P, int p0, int count,
                       double* coeffs, bool accumulate, cudaStream_t stream);
  int LegendreSynthesis(int N, bool real, const double* coeffs, int count, double* spectra,
                        cudaStream_t stream) {
    return LegendreSynthesis(N, real, coeffs, count, 0, count, spectra, stream);
  }
  int LegendreAnalysis(int N, bool real, const double* spectra, int count, double* coeffs,
                       cudaStream_t stream) {
    return LegendreAnalysis(N, real, spectra, count, 0, count, coeffs, false, stream);
  }
  // fixedPoint: small batches in fixed point too (larger ones always are).
  int RingSynthesis(bool real, const double* spectra, int count, double* fields, cudaStream_t stream,
                    bool fixedPoint = false);
  // Optional pointwise weight (a real field over the same values) applied
  // before the analysis.
  int RingAnalysis(bool real, const double* fields, int count, double* spectra, cudaStream_t stream,
                   const double* weight = nullptr, bool fixedPoint = false);
  // Synthesis, the pointwise weight and the analysis of each ring in one
  // pass through shared memory: the grid values never reach HBM.
  int RingWeighted(bool real, const double* spectraIn, int count, const double* weight,
                   double* spectraOut, cudaStream_t stream);

  // The same contraction and ring passes in FP32 (the mixed form's
  // correction passes): FP32 copies of the table and twiddles, made once.
  int LegendreSynthesisF(int N, bool real, const float* coeffs, int P, int p0, int count, float* spectra,
                         cudaStream_t stream);
  // Whether a tensor-core contraction gave up waiting (SL3DGPU_ERR_WAIT, once):
  // in the work of `stream` and before (synchronises it), or in what has ended
  // so far, which costs a read of host memory.
  int TensorCoreStatus(cudaStream_t stream);
  int TensorCoreStatus();
  // The flag those waits set, made on first use.
  int GiveUpFlag(int** flag);
  int LegendreAnalysisF(int N, bool real, const float* spectra, int P, int p0, int count, float* coeffs,
                        bool accumulate, cudaStream_t stream);

  // The same for a tensor's three components at once, spins -2 and -1 and the
  // real spin 0, in one launch each where the one-component calls would take
  // three: coefficients the components' rows one after another
  // ([row][P] each), spectra theirs ([m][j][count] each, TripleStride(count)
  // complex values apart). One launch fills the SMs at small sizes and has
  // one last wave at large ones (a pass at lmax 45 558 -> 453 us, at lmax 128
  // 2583 -> 2417). lmax >= 2, so every order of every component
  // has degrees.
  long long TripleStride(int count) const { return static_cast<long long>(2 * lmax + 1) * ntheta * count; }
  // Complex values a triple's spectra take.
  static long long TripleSize(int lmax, int ntheta, int count) {
    return (2LL * (2 * lmax + 1) + lmax + 1) * ntheta * count;
  }
  int LegendreSynthesis3(const double* coeffs, int P, int p0, int count, double* spectra, cudaStream_t stream);
  int LegendreAnalysis3(const double* spectra, int P, int p0, int count, double* coeffs, bool accumulate,
                        cudaStream_t stream);
  int RingSynthesis3(const double* spectra, int count, double2* f0, double2* f1, double* fr, cudaStream_t stream);
  int RingAnalysis3(const double2* f0, const double2* f1, const double* fr, int count, double* spectra,
                    cudaStream_t stream, const double* weight = nullptr);
  int RingWeighted3(const double* spectraIn, int count, const double* weight, double* spectraOut, cudaStream_t stream);
  int LegendreSynthesis3F(const float* coeffs, int count, float* spectra, cudaStream_t stream);
  int LegendreAnalysis3F(const float* spectra, int count, float* coeffs, cudaStream_t stream);
  int RingWeighted3F(const float* spectraIn, int count, const float* weight, float* spectraOut, cudaStream_t stream);

  // The Legendre sum between the reference layout's coefficients and the
  // spectra, where one kernel does both (few fields on the FP64 units, every
  // order with degrees); `done` says whether.
  int LegendreInReferenceLayout(int N, bool real, bool analysis, const double* in, int count, double* out,
                                cudaStream_t stream, bool* done);

  // Reference layout <-> device layout permutations.
  int ToDevice(int N, bool real, const double* ref, int count, double* dev, cudaStream_t stream);
  int FromDevice(int N, bool real, const double* dev, int count, double* ref, cudaStream_t stream);

  // Scratch owned by the grid for the reference-layout batch calls.
  int Scratch(size_t spectraDoubles, size_t coeffDoubles, double** spectra, double** coeffs);

 private:
  std::map<int, SpinTable> tables_;
  // The components a batch's contraction covers: a spin's, or a tensor's three
  // (N = kTriple), each an item range with its own table.
  static constexpr int kTriple = INT_MAX;  // no grid has this spin
  struct Part {
    int N = 0;
    bool real = false;
    int first = 0, count = 0;  // items
  };
  struct Batch {
    std::vector<Part> parts;
    GemmItem* items = nullptr;
    int count = 0, maxM = 0, maxN = 0;
    bool analysis = false;
    double flops = 0.0;    // 2 M N K summed over the items
    double outputs = 0.0, inputs = 0.0, tableValues = 0.0;  // M N, K N and M K summed over the items
    // the tensor-core form (FP32): its items, tile width and extents, the
    // packed B (made on first use) and the key of its table panel
    std::vector<TcItemHost> tcHost;
    void* tcItems = nullptr;
    int tileN = 0, maxMTiles = 0, maxNTiles = 0, maxATiles = 0, maxBTiles = 0;
    long long panelFloats = 0, packedFloats = 0;
    float* packed = nullptr;
    std::vector<int4> tcTiles;  // {item, row tile, column tile}, column tiles of a row tile adjacent
    int4* dTcTiles = nullptr;
    int maxK = 0;
    // the FP64 slices' form: items (made on first use) and extents
    std::vector<Tc64Item> tc64Host;
    Tc64Item* tc64Items = nullptr;
    int maxNTiles64 = 0;
    long long panel64 = 0, packed64 = 0;  // tiles of the panel and of the packed B
    long long rowExps = 0, colExps = 0;
  };
  // The table split for the FP64 slices per (spin, real, direction, slices).
  std::map<std::array<int, 4>, Tc64Panel> panels64_;
  // Where a call's packed B and column exponents come from, stream-ordered:
  // calls on several streams each have their own, and the memory stays with
  // the grid between them.
  cudaMemPool_t pool_ = nullptr;
  bool UseSlices64(const Batch& b) const;
  int Tables(const Batch& b, Tc64Tables* out);
  // The complex rows before a triple's component, and its spin.
  long long TripleRows(int component) const {
    return component == 0 ? 0 : component == 1 ? SpinRows(-2) : SpinRows(-2) + SpinRows(-1);
  }
  int RunGemm64(int N, bool real, Batch& b, const double* B, double* C, bool accumulate, cudaStream_t stream);
  int Contract64(const Batch& b, int slices, const Tc64Tables& tables, const Tc64Panel& panel, const double* B,
                 double* C, bool accumulate, int* giveUp, cudaStream_t stream);
  // The table pre-tiled for the tensor cores per (spin, real, direction).
  std::map<std::array<int, 3>, float*> panels_;
  std::map<std::array<long long, 6>, Batch> batches_;
  // A panel is made on the stream of the call that first wants it (under a
  // capture, on a stream made for it, whose work is waited for). Calls on other
  // streams wait for the last one made, on their streams (in a capture, on the
  // host), until one finds it finished. No stream is kept: with one more in the
  // process the sea-level equation's solves on the default stream took 3% longer.
  cudaEvent_t panelsMade_ = nullptr;
  bool panelsPending_ = false;
  int MakePanel(cudaStream_t stream, const std::function<int(cudaStream_t)>& launch);
  int AwaitPanels(cudaStream_t stream);
  int BatchFor(int N, bool real, bool analysis, int P, int p0, int count, const Batch** out);
  Batch* MutableBatch(int N, bool real, bool analysis, int P, int p0, int count);
  double* scratchSpectra_ = nullptr;
  size_t scratchSpectraSize_ = 0;
  double* scratchCoeffs_ = nullptr;
  size_t scratchCoeffsSize_ = 0;
  int RunGemm(const Batch& b, const double* A, const double* B, double* C, bool accumulate,
              cudaStream_t stream);
  // The FP32 contraction on the tensor cores (tc_gemm.cu): the spin's table
  // panel (made on first use), B packed, the contraction.
  int RunGemmF(int N, bool real, Batch& b, const float* B, float* C, bool accumulate, cudaStream_t stream);
  int* giveUp_ = nullptr;  // set by a tensor-core wait that gave up (pinned)

 public:
  // The spin's table, with the FP32 twiddles made.
  int Table32(int N, const SpinTable** out);
};

// One real field's transforms with the rings in fixed point (the sea-level
// solver's), the coefficients in the reference layout or, with `device`, in
// the transforms' own (an order's degrees together).
int SynthesiseFixed(sl3dgpu_grid* grid, const double* coeffs, double* field, cudaStream_t stream, bool device = false);
int ExpandFixed(sl3dgpu_grid* grid, const double* field, double* coeffs, cudaStream_t stream, bool device = false);

// What another part of the library keeps with a grid handle (released with it).
struct GridAttachment {
  std::mutex lock;
  std::shared_ptr<void> workspace;
};
GridAttachment& AttachmentOf(sl3dgpu_grid* grid);
Grid& GridOf(sl3dgpu_grid* grid);

// Smallest 2^a 3^b 5^c at or above n.
int FftFriendly(int n);

}  // namespace sl3dgpu
