// The FP64 Cholesky solves by blocks of rows (band_block.cu): a flavour's
// factorised systems rewritten once so that a solve advances a block of rows
// at a time.
#pragma once

#include <vector>

#include "common.cuh"

namespace sl3dgpu {

// One system of a blocked solve.
struct BlockSystem {
  int n, kd, nrhs, blocks;
  long long forward, backward;  // doubles: its blocks' coefficients, [block][(kd + B) x B]
  long long rhs, scale;         // as sl3dgpu_band_system's
  int second;                   // which of the two right-hand-side arrays
};

struct BlockSolver {
  int block = 0;  // rows a block (8 or 16); 0: the row-by-row solve is the faster
  int kd = 0;     // the largest bandwidth
  int itemCount = 0;
  BlockSystem* systems = nullptr;
  int2* items = nullptr;  // (system, first column)
  double* data = nullptr;
  // the FP32 form (the mixed form's correction solves): the coefficients
  // rounded, and its items (more columns a CTA)
  int firstCount = 0;  // systems of the first list
  int itemCount32 = 0;
  int2* items32 = nullptr;
  float* data32 = nullptr;
  BlockSolver() = default;
  BlockSolver(const BlockSolver&) = delete;
  BlockSolver& operator=(const BlockSolver&) = delete;
  ~BlockSolver() {
    cudaFree(systems);
    cudaFree(items);
    cudaFree(data);
    cudaFree(items32);
    cudaFree(data32);
  }
};

// Chooses the form for two lists of factorised Cholesky systems (the second
// list's right-hand sides in the second array) and makes a blocked form's
// coefficients from their factors.
int BuildBlockSolver(const std::vector<sl3dgpu_band_system>& first, const std::vector<sl3dgpu_band_system>& second,
                     const double* bands, const double* scales, bool fp32, BlockSolver& out, cudaStream_t stream);
// Solves every system in place (out.block > 0).
int RunBlockSolver(const BlockSolver& b, double* first, double* second, const double* scales, cudaStream_t stream);

// The FP32 solves over row windows (windowsFirst, windowsSecond: {lo, hi} a
// system, the right-hand side zero outside): rows lo .. n - 1 of both
// substitutions, as BandSolveWindowF's (which completes the rows below).
int RunBlockSolver32(const BlockSolver& b, float* first, float* second, const float* scales, const int2* windowsFirst,
                     const int2* windowsSecond, cudaStream_t stream);

}  // namespace sl3dgpu
