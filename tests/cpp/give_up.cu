// A tensor-core wait that gave up, as the grid's calls report it. No wait is made
// to run out: the mark is set as the kernels set it, by a kernel of this program.
#include <cstdio>
#include <cstring>
#include <vector>

#include "sht.cuh"
#include "tc_gemm.cuh"

using namespace sl3dgpu;

namespace {
__global__ void MarkKernel(int* flag) { ReportGiveUp(flag); }
}  // namespace

int main() {
  bool good = true;
  auto check = [&](bool ok, const char* what) {
    std::printf("%s: %s\n", ok ? "ok" : "FAIL", what);
    good = good && ok;
  };
  const int lmax = 16, count = 12;
  sl3dgpu_grid* grid = nullptr;
  if (sl3dgpu_grid_create(lmax, 2, 1.5, &grid) != SL3DGPU_OK) return 2;
  Grid& g = GridOf(grid);
  const size_t rows = g.RealRows() * count * 2, values = static_cast<size_t>(g.ntheta) * g.nphi * count;
  double *c = nullptr, *f = nullptr;
  if (cudaMalloc(&c, rows * sizeof(double)) != cudaSuccess || cudaMalloc(&f, values * sizeof(double)) != cudaSuccess)
    return 2;
  if (CopyIn(c, std::vector<double>(rows, 0.25).data(), rows * sizeof(double)) != cudaSuccess) return 2;
  check(sl3dgpu_synthesise_batch(grid, c, count, f, nullptr) == SL3DGPU_OK, "a wide call");
  check(g.TensorCoreStatus(nullptr) == SL3DGPU_OK, "no mark after it");
  int* flag = nullptr;
  if (g.GiveUpFlag(&flag) != SL3DGPU_OK) return 2;
  auto mark = [&] {
    MarkKernel<<<1, 1>>>(flag);
    return cudaDeviceSynchronize() == cudaSuccess;
  };
  auto reported = [](int status) {
    return status == SL3DGPU_ERR_WAIT && std::strstr(sl3dgpu_last_error(), "gave up waiting") != nullptr;
  };
  check(mark() && reported(sl3dgpu_synthesise_batch(grid, c, count, f, nullptr)), "the next synthesis reports it");
  check(sl3dgpu_synthesise_batch(grid, c, count, f, nullptr) == SL3DGPU_OK, "once");
  check(mark() && reported(sl3dgpu_expand_batch(grid, f, count, c, nullptr)), "the next expansion reports it");
  check(mark() && reported(sl3dgpu_legendre_device(grid, 0, 1, 0, 0, c, 0, f, nullptr)), "the Legendre stage reports it");
  check(mark() && reported(g.TensorCoreStatus(nullptr)), "a status call reports it");
  check(g.TensorCoreStatus(nullptr) == SL3DGPU_OK, "once");
  check(sl3dgpu_expand_batch(grid, f, count, c, nullptr) == SL3DGPU_OK && cudaDeviceSynchronize() == cudaSuccess,
        "and calls go on");
  sl3dgpu_grid_destroy(grid);
  return good ? 0 : 1;
}
