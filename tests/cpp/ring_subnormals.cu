// Rings of subnormal values and rings under subnormal weights, through the
// grid's weighted rings (sht.cuh): a batch of ten fields, which goes through
// the fixed-point kernel, against each field alone, on the FP64 units.
// Prints the largest difference and the bound of each case; exit 1 past it.
#include <cstdio>
#include <random>
#include <vector>

#include "sht.cuh"

using namespace sl3dgpu;

namespace {

template <class T>
T* Upload(const std::vector<T>& v) {
  T* p = nullptr;
  if (cudaMalloc(&p, v.size() * sizeof(T)) != cudaSuccess || CopyIn(p, v.data(), v.size() * sizeof(T)) != cudaSuccess)
    std::exit(2);
  return p;
}

// One call's outputs, [order][colatitude][count] complex.
std::vector<double> Weighted(Grid& g, bool real, const std::vector<double>& spectra, int count,
                             const std::vector<double>& weight) {
  double *in = Upload(spectra), *w = Upload(weight), *out = Upload(std::vector<double>(spectra.size(), 0.0));
  std::vector<double> host(spectra.size());
  if (g.RingWeighted(real, in, count, w, out, nullptr) != SL3DGPU_OK) std::exit(2);
  if (cudaMemcpy(host.data(), out, host.size() * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess) std::exit(2);
  cudaFree(in);
  cudaFree(w);
  cudaFree(out);
  return host;
}

}  // namespace

int main() {
  const int lmax = 6, count = 10;
  std::unique_ptr<Grid> g;
  if (Grid::Create(lmax, 2, 1.5, g) != SL3DGPU_OK) return 2;
  const int n = g->nphi, nt = g->ntheta;
  // the exponents of the spectra and of the weights, the second the subnormal one
  const struct { int spectra, weights; } cases[] = {{-1040, 0}, {300, -1040}, {0, -1050}, {-1030, 10}};
  bool good = true;
  for (const auto& c : cases)
    for (const bool real : {false, true}) {
      const int orders = real ? lmax + 1 : 2 * lmax + 1;
      const size_t each = static_cast<size_t>(orders) * nt * 2;
      std::mt19937_64 rng(1);
      std::uniform_real_distribution<double> u(0.5, 1.0);
      std::vector<double> spectra(each * count), weight(static_cast<size_t>(count) * nt * n);
      for (auto& v : spectra) v = std::ldexp(u(rng), c.spectra);
      for (auto& v : weight) v = std::ldexp(u(rng), c.weights);
      const auto got = Weighted(*g, real, spectra, count, weight);
      double largest = 0.0, worst = 0.0;
      for (int p = 0; p < count; ++p) {
        std::vector<double> one(each), w(weight.begin() + static_cast<long long>(p) * nt * n,
                                         weight.begin() + static_cast<long long>(p + 1) * nt * n);
        for (size_t i = 0; i < each / 2; ++i)
          for (int q = 0; q < 2; ++q) one[2 * i + q] = spectra[2 * (i * count + p) + q];
        const auto want = Weighted(*g, real, one, 1, w);
        for (size_t i = 0; i < each / 2; ++i)
          for (int q = 0; q < 2; ++q) {
            // by an exact factor out of the subnormal range
            const double a = std::ldexp(got[2 * (i * count + p) + q], 600), b = std::ldexp(want[2 * i + q], 600);
            largest = std::max(largest, std::fabs(b));
            worst = std::max(worst, std::fabs(a - b));
          }
      }
      // A transform's stages each round a value's at most 12 products and their
      // sum to the spacing 2^-1074 or to 2^-53 of the value; an error of a stage
      // reaches an output at most n times over. Two transforms of 24 n
      // roundings on either side, the first's under weights and the second's
      // sums of up to n: 96 n^2 spacings, and 2^-46 of the largest.
      const double spacing = std::ldexp(1.0, -1074 + 600);
      const double bound = 96.0 * n * n * spacing * std::max(1.0, std::ldexp(1.0, c.weights)) + std::ldexp(largest, -46);
      std::printf("%s 2^%d under 2^%d: largest %.3e off %.3e bound %.3e\n", real ? "real" : "spin", c.spectra,
                  c.weights, largest, worst, bound);
      good = good && largest > 0.0 && worst <= bound && bound < 0.01 * largest;
    }
  return good ? 0 : 1;
}
