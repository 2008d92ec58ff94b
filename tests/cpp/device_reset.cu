// A program that resets its device (its own context) between two uses of the
// library: kernels whose shared-memory limits the first context had raised, and
// the fixed scratch of the solver that allocates nothing.
#include <cstdio>
#include <cmath>
#include <vector>

#include <cuda_runtime.h>
#include <sl3dgpu.h>

namespace {

// Twelve fields' synthesis and expansion at 625 longitudes, whose rings take
// about 100 KB of shared memory a CTA; the largest error of the round trip.
double RoundTrip() {
  const int lmax = 200, count = 12;
  sl3dgpu_grid* grid = nullptr;
  int nt = 0, nphi = 0;
  if (sl3dgpu_grid_create(lmax, 0, 1.5, &grid) != 0 || sl3dgpu_grid_shape(grid, &nt, &nphi) != 0) return 1e300;
  const size_t n = static_cast<size_t>(lmax + 1) * (lmax + 2) / 2 * count * 2;
  std::vector<double> c(n), back(n, 0.0);
  for (size_t i = 0; i < n; i += 2) c[i] = std::cos(0.1 * i);  // real coefficients
  double *dc = nullptr, *df = nullptr;
  double worst = 1e300;
  if (cudaMalloc(&dc, n * sizeof(double)) == cudaSuccess &&
      cudaMalloc(&df, static_cast<size_t>(nt) * nphi * count * sizeof(double)) == cudaSuccess &&
      cudaMemcpy(dc, c.data(), n * sizeof(double), cudaMemcpyHostToDevice) == cudaSuccess &&
      sl3dgpu_synthesise_batch(grid, dc, count, df, nullptr) == 0 &&
      sl3dgpu_expand_batch(grid, df, count, dc, nullptr) == 0 &&
      cudaMemcpy(back.data(), dc, n * sizeof(double), cudaMemcpyDeviceToHost) == cudaSuccess) {
    worst = 0.0;
    for (size_t i = 0; i < n; ++i) worst = std::max(worst, std::fabs(back[i] - c[i]));
  } else {
    std::printf("%s\n", sl3dgpu_last_error());
  }
  cudaFree(dc);
  cudaFree(df);
  sl3dgpu_grid_destroy(grid);
  return worst;
}

// The solver without allocations on the factor 2 I: halves twice.
double Solve() {
  const int n = 40, kd = 3, nrhs = 5;
  std::vector<double> ab((kd + 1) * n, 0.0), b(n * nrhs);
  for (int j = 0; j < n; ++j) ab[j * (kd + 1) + kd] = 2.0;
  for (size_t i = 0; i < b.size(); ++i) b[i] = 4.0 * i;
  double *dab = nullptr, *db = nullptr, worst = 1e300;
  if (cudaMalloc(&dab, ab.size() * sizeof(double)) == cudaSuccess &&
      cudaMalloc(&db, b.size() * sizeof(double)) == cudaSuccess &&
      cudaMemcpy(dab, ab.data(), ab.size() * sizeof(double), cudaMemcpyHostToDevice) == cudaSuccess &&
      cudaMemcpy(db, b.data(), b.size() * sizeof(double), cudaMemcpyHostToDevice) == cudaSuccess &&
      sl3dgpu_band_cholesky_solve_noalloc(dab, n, kd, db, nrhs, nullptr) == 0 &&
      cudaMemcpy(b.data(), db, b.size() * sizeof(double), cudaMemcpyDeviceToHost) == cudaSuccess) {
    worst = 0.0;
    for (size_t i = 0; i < b.size(); ++i) worst = std::max(worst, std::fabs(b[i] - static_cast<double>(i)));
  } else {
    std::printf("%s\n", sl3dgpu_last_error());
  }
  cudaFree(dab);
  cudaFree(db);
  return worst;
}

}  // namespace

int main() {
  bool good = true;
  for (int use = 0; use < 3; ++use) {
    const double ring = RoundTrip(), solve = Solve();
    std::printf("use %d: round trip off %.2e, solve off %.2e\n", use, ring, solve);
    good = good && ring < 1e-12 && solve == 0.0;
    if (cudaDeviceReset() != cudaSuccess) return 2;
  }
  return good ? 0 : 1;
}
