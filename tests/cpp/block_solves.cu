// The Cholesky solves by blocks of rows (csrc/band_block.cu), called directly:
// both block sizes, in FP64 and, over row windows, in FP32, on systems whose
// row counts, columns, windows and bandwidths are and are not multiples of the
// blocks.
//
// Each solution's backward error is bounded: with z = S^-1 x, the residual of
// (S A S) z = S b is at most 8 (kd + B) u kappa (|S A S| |z| + |S b|) in the
// largest norm, u the unit roundoff and kappa the largest condition of a
// B x B diagonal block of the factor (a block's rows are its inverse times
// sums of kd + B products). The row-by-row solve, whose bound lacks kappa, is
// held to the same, and its error printed beside.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

#include "band_block.cuh"
#include "systems.cuh"

using namespace sl3dgpu;

namespace {

struct System {
  sl3dgpu_band_system s;
  std::vector<double> A;  // S A S, upper band as the factor's
};

struct Batch {
  std::vector<System> first, second;
  std::vector<double> bands, scales;
  long long values[2] = {0, 0};  // right-hand sides of either list
};

// A symmetric positive definite band of overlapping elements, scaled to a
// unit diagonal, and its factor appended to the batch's.
void Add(Batch& b, int which, int n, int kd, int nrhs, int pinned, bool scaled, std::mt19937_64& rng) {
  std::normal_distribution<double> g;
  const int ld = kd + 1;
  std::vector<double> a(static_cast<size_t>(n) * ld, 0.0), scale(n);
  auto at = [&](std::vector<double>& m, int i, int j) -> double& { return m[static_cast<size_t>(j) * ld + kd + i - j]; };
  for (int e = 0; e + 1 < n || e == 0; e += std::max(1, kd)) {
    const int m = std::min(kd + 1, n - e);
    for (int r = 0; r < m; ++r) {  // a stiff element: m rank-one terms of decaying size
      std::vector<double> v(m);
      for (auto& x : v) x = g(rng);
      const double c = std::exp(-0.5 * r);
      for (int i = 0; i < m; ++i)
        for (int j = i; j < m; ++j) at(a, e + i, e + j) += c * v[i] * v[j];
    }
  }
  for (int i = 0; i < n; ++i) {
    at(a, i, i) *= 1.0 + 1e-3;
    if (i == pinned) {
      for (int t = 0; t <= kd; ++t) {
        if (i - t >= 0) at(a, i - t, i) = 0.0;
        if (i + t < n) at(a, i, i + t) = 0.0;
      }
      at(a, i, i) = 1.0;
    }
  }
  for (int i = 0; i < n; ++i) scale[i] = 1.0 / std::sqrt(at(a, i, i));
  for (int j = 0; j < n; ++j)
    for (int i = std::max(0, j - kd); i <= j; ++i) at(a, i, j) *= scale[i] * scale[j];
  if (scaled)  // the unscaled system's diagonal spans six decades
    for (int i = 0; i < n; ++i) scale[i] *= std::pow(10.0, 3.0 * std::sin(0.37 * i));
  else
    std::fill(scale.begin(), scale.end(), 1.0);
  std::vector<double> u = a;
  for (int j = 0; j < n; ++j)
    for (int i = std::max(0, j - kd); i <= j; ++i) {
      long double sum = at(a, i, j);
      for (int k = std::max(0, j - kd); k < i; ++k) sum -= static_cast<long double>(at(u, k, i)) * at(u, k, j);
      at(u, i, j) = static_cast<double>(i == j ? std::sqrt(sum) : sum / at(u, i, i));
    }
  System sys{};
  sys.A = a;
  sys.s.n = n;
  sys.s.kl = sys.s.ku = kd;
  sys.s.nrhs = nrhs;
  sys.s.band = static_cast<long long>(b.bands.size());
  sys.s.rhs = b.values[which];
  sys.s.scale = scaled ? static_cast<long long>(b.scales.size()) : -1;
  sys.s.pinned0 = pinned;
  sys.s.pinned1 = -1;
  b.bands.insert(b.bands.end(), u.begin(), u.end());
  if (scaled) b.scales.insert(b.scales.end(), scale.begin(), scale.end());
  b.values[which] += static_cast<long long>(n) * nrhs;
  (which ? b.second : b.first).push_back(sys);
}

std::vector<sl3dgpu_band_system> Plain(const std::vector<System>& systems) {
  std::vector<sl3dgpu_band_system> out;
  for (const auto& s : systems) out.push_back(s.s);
  return out;
}

// The largest condition number (largest-norm) of a block of the factor.
double BlockCondition(const Batch& b, const sl3dgpu_band_system& s, int B) {
  const int ld = s.ku + 1;
  auto U = [&](int i, int j) { return j - i > s.ku || i > j ? 0.0 : b.bands[s.band + static_cast<long long>(j) * ld + s.ku + i - j]; };
  double worst = 1.0;
  for (int j0 = 0; j0 < s.n; j0 += B) {
    const int m = std::min(B, s.n - j0);
    std::vector<double> M(m * m, 0.0);  // the inverse of L = U^T
    for (int c = 0; c < m; ++c)
      for (int r = c; r < m; ++r) {
        double sum = r == c ? 1.0 : 0.0;
        for (int k = c; k < r; ++k) sum -= U(j0 + k, j0 + r) * M[k * m + c];
        M[r * m + c] = sum / U(j0 + r, j0 + r);
      }
    for (int side = 0; side < 2; ++side) {  // L, then its transpose
      double l = 0.0, i = 0.0;
      for (int r = 0; r < m; ++r) {
        double a = 0.0, c = 0.0;
        for (int k = 0; k < m; ++k) {
          a += std::fabs(side ? U(j0 + r, j0 + k) : U(j0 + k, j0 + r));
          c += std::fabs(side ? M[k * m + r] : M[r * m + k]);
        }
        l = std::max(l, a);
        i = std::max(i, c);
      }
      worst = std::max(worst, l * i);
    }
  }
  return worst;
}

// The backward error of one system's columns over |S A S| |z| + |S b|.
template <class T>
double BackwardError(const Batch& b, const System& sys, const std::vector<T>& x, const std::vector<T>& rhs) {
  const auto& s = sys.s;
  const int ld = s.ku + 1;
  double worst = 0.0;
  for (int c = 0; c < s.nrhs; ++c) {
    double residual = 0.0, size = 0.0, norm = 0.0, z = 0.0, load = 0.0;
    for (int i = 0; i < s.n; ++i) {
      auto Z = [&](int r) {
        const double f = s.scale >= 0 ? static_cast<double>(static_cast<T>(b.scales[s.scale + r])) : 1.0;
        return static_cast<double>(x[s.rhs + static_cast<long long>(r) * s.nrhs + c]) / f;
      };
      const double f = s.scale >= 0 ? static_cast<double>(static_cast<T>(b.scales[s.scale + i])) : 1.0;
      const double right = i == s.pinned0 ? 0.0 : f * rhs[s.rhs + static_cast<long long>(i) * s.nrhs + c];
      long double sum = right;
      double row = 0.0;
      for (int k = std::max(0, i - s.ku); k <= std::min(s.n - 1, i + s.ku); ++k) {
        const double a = sys.A[static_cast<size_t>(std::max(i, k)) * ld + s.ku - std::abs(i - k)];
        sum -= static_cast<long double>(a) * Z(k);
        row += std::fabs(a);
      }
      residual = std::max(residual, std::fabs(static_cast<double>(sum)));
      norm = std::max(norm, row);
      z = std::max(z, std::fabs(Z(i)));
      load = std::max(load, std::fabs(right));
    }
    size = norm * z + load;
    worst = std::max(worst, size > 0.0 ? residual / size : residual);
  }
  return worst;
}

template <class T>
struct Device {
  Dev<T> d;
  explicit Device(const std::vector<T>& v) {
    if (d.Upload(v) != cudaSuccess) std::exit(2);
  }
  std::vector<T> Read() const {
    std::vector<T> v(d.n);
    if (cudaMemcpy(v.data(), d.p, d.n * sizeof(T), cudaMemcpyDeviceToHost) != cudaSuccess) std::exit(2);
    return v;
  }
};

bool good = true;
void Try(int status) {
  if (status != SL3DGPU_OK) {
    std::printf("%s\n", sl3dgpu_last_error());
    std::exit(2);
  }
}

template <class T>
void CheckBound(const char* form, const Batch& b, int B, const std::vector<T> x[2], const std::vector<T> rhs[2]) {
  const double u = sizeof(T) == sizeof(double) ? std::ldexp(1.0, -53) : std::ldexp(1.0, -24);
  double worst = 0.0, ratio = 0.0;
  for (int which = 0; which < 2; ++which)
    for (const auto& sys : which ? b.second : b.first) {
      const double e = BackwardError(b, sys, x[which], rhs[which]);
      const double bound = 8.0 * (sys.s.ku + B) * u * BlockCondition(b, sys.s, B);
      worst = std::max(worst, e);
      ratio = std::max(ratio, e / bound);
      if (!(e <= bound)) good = false;
    }
  std::printf("%-28s blocks of %2d: backward error %.2e, %.3f of the bound\n", form, B, worst, ratio);
}

void Check(Batch& b, int expected, std::mt19937_64& rng) {
  if (b.scales.empty()) b.scales.push_back(1.0);
  const auto first = Plain(b.first), second = Plain(b.second);
  Device<double> bands(b.bands), scales(b.scales);
  BlockSolver solver;
  Try(BuildBlockSolver(first, second, bands.d.p, scales.d.p, true, solver, nullptr));
  std::printf("%zu + %zu systems: blocks of %d\n", first.size(), second.size(), solver.block);
  if (solver.block != expected || solver.itemCount32 == 0) {
    std::printf("FAIL: expected blocks of %d and the FP32 form\n", expected);
    good = false;
    return;
  }
  std::normal_distribution<double> g;
  // FP64, every row
  {
    std::vector<double> rhs[2], x[2], rows[2];
    for (int w = 0; w < 2; ++w) {
      rhs[w].resize(std::max<long long>(b.values[w], 1));
      for (auto& v : rhs[w]) v = g(rng);
    }
    Device<double> a(rhs[0]), c(rhs[1]), ra(rhs[0]), rc(rhs[1]);
    Try(RunBlockSolver(solver, a.d.p, c.d.p, scales.d.p, nullptr));
    x[0] = a.Read();
    x[1] = c.Read();
    CheckBound("FP64", b, solver.block, x, rhs);
    for (int w = 0; w < 2; ++w) {
      const auto& systems = w ? second : first;
      if (systems.empty()) continue;
      Dev<sl3dgpu_band_system> d;
      Dev<int2> items;
      const auto list = BandWorkItems(systems.data(), static_cast<int>(systems.size()));
      if (d.Upload(systems) != cudaSuccess || items.Upload(list) != cudaSuccess) std::exit(2);
      Try(BandSolveBatch(d.p, systems.data(), static_cast<int>(systems.size()), items.p, static_cast<int>(list.size()),
                         bands.d.p, nullptr, (w ? rc : ra).d.p, scales.d.p, 0, nullptr));
      rows[w] = (w ? rc : ra).Read();
    }
    CheckBound("FP64, row by row", b, solver.block, rows, rhs);
  }
  // FP32 over windows: from the first row, from inside a block, one row, the
  // last row, and two empty ones (their right-hand sides all zero)
  std::vector<float> bands32(b.bands.begin(), b.bands.end()), scales32(b.scales.begin(), b.scales.end());
  Device<float> db(bands32), ds(scales32);
  for (int kind = 0; kind < 6; ++kind) {
    std::vector<float> rhs[2], x[2], rows[2];
    std::vector<int2> windows[2];
    for (int w = 0; w < 2; ++w) {
      rhs[w].assign(std::max<long long>(b.values[w], 1), 0.0f);
      int k = 0;
      for (const auto& sys : w ? b.second : b.first) {
        const int n = sys.s.n,
                  lo = kind == 0 ? 0 : kind == 5 ? n : std::min(n - 1, kind == 3 ? n - 1 : n / 3 + k++ % 19);
        const int hi = kind == 0 || kind == 3 ? n - 1 : kind == 2 ? lo : kind >= 4 ? lo - 1 : std::min(n - 1, lo + n / 4);
        windows[w].push_back(make_int2(lo, hi));
        for (int i = lo; i <= hi; ++i)
          for (int c = 0; c < sys.s.nrhs; ++c)
            rhs[w][sys.s.rhs + static_cast<long long>(i) * sys.s.nrhs + c] =
                static_cast<float>(g(rng) / (sys.s.scale >= 0 ? b.scales[sys.s.scale + i] : 1.0));
      }
      if (windows[w].empty()) windows[w].push_back(make_int2(0, -1));
    }
    Device<float> a(rhs[0]), c(rhs[1]), ra(rhs[0]), rc(rhs[1]);
    Device<int2> w0(windows[0]), w1(windows[1]);
    Try(RunBlockSolver32(solver, a.d.p, c.d.p, ds.d.p, w0.d.p, w1.d.p, nullptr));
    for (int w = 0; w < 2; ++w) {
      const auto half = (w ? c : a).Read();  // rows below the window are left as they were, zero
      int k = 0;
      for (const auto& sys : w ? b.second : b.first) {
        const int lo = windows[w][k++].x;
        for (long long i = 0; i < static_cast<long long>(lo) * sys.s.nrhs; ++i)
          if (half[sys.s.rhs + i] != 0.0f) good = false;
      }
      // the rows below, by the row form's completion; and the row form throughout
      const auto& systems = w ? second : first;
      if (systems.empty()) continue;
      Dev<sl3dgpu_band_system> d;
      Dev<int2> items;
      const auto list = BandWorkItems(systems.data(), static_cast<int>(systems.size()));
      if (d.Upload(systems) != cudaSuccess || items.Upload(list) != cudaSuccess) std::exit(2);
      auto solve = [&](float* v, bool completion) {
        Try(BandSolveWindowF(d.p, systems.data(), static_cast<int>(systems.size()), items.p,
                             static_cast<int>(list.size()), db.d.p, v, ds.d.p, (w ? w1 : w0).d.p, completion, nullptr));
      };
      solve((w ? c : a).d.p, true);
      solve((w ? rc : ra).d.p, false);
      solve((w ? rc : ra).d.p, true);
      x[w] = (w ? c : a).Read();
      rows[w] = (w ? rc : ra).Read();
    }
    char name[32];
    std::snprintf(name, sizeof name, "FP32, windows %d", kind);
    CheckBound(name, b, solver.block, x, rhs);
    std::snprintf(name, sizeof name, "FP32, windows %d, by rows", kind);
    CheckBound(name, b, solver.block, rows, rhs);
  }
}

}  // namespace

int main() {
  std::mt19937_64 rng(5);
  {
    // few columns: a chain of blocks bounds the solve, blocks of 16
    Batch b;
    for (int n : {1, 15, 16, 17, 33, 100, 255}) Add(b, 0, n, n == 1 ? 0 : 14, 2 * (n % 5 + 1), n == 33 ? 20 : -1, n != 17, rng);
    for (int n : {2, 31, 73}) Add(b, 1, n, 4, 6, -1, true, rng);
    Check(b, 16, rng);
  }
  {
    // the same with one list
    Batch b;
    for (int n : {47, 90}) Add(b, 0, n, 17, 10, 3, true, rng);
    Check(b, 16, rng);
  }
  {
    // many columns: the FP64 unit bounds it, blocks of 8
    Batch b;
    for (int k = 0; k < 60; ++k) Add(b, 0, 150 + k, 14, 2 * (30 + k), k == 2 ? 149 : -1, k % 7 != 0, rng);
    for (int k = 0; k < 60; ++k) Add(b, 1, 70 + k % 9, 4, 2 * (31 + k), -1, true, rng);
    Check(b, 8, rng);
  }
  return good ? 0 : 1;
}
