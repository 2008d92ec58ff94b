// The FP64 Cholesky solves by blocks of rows.
//
// Why. A row of a band substitution is a chain: kd products and the division
// by the diagonal wait for the row before, and GB300 issues one FP64 warp
// instruction in 64 cycles a sub-partition. The row-by-row solve
// (CholeskySolve64Kernel) therefore costs about (kd + 3) 64 cycles a row
// however few columns there are: 0.61 ms for an lmax-45 pass's two launches,
// most SMs idle.
//
// How. With the rows in blocks J of B, L = U^T and y_p the kd values before J,
//   y_J = L_JJ^-1 (S b_J) - (L_JJ^-1 L_Jp) y_p,
// and backward x_J = U_JJ^-1 y_J - (U_JJ^-1 U_Jn) x_n. Both coefficient
// matrices, kd x B and B x B, are made once a flavour; then every row of a
// block is an independent sum of kd + B products and the chain has one link a
// block. A warp holds B rows x 32 / B columns, a lane a value; the four warps
// of a CTA (one a sub-partition) share the staged coefficients. A row costs
// kd + B products rather than kd + 3, so the form pays where latency bounds
// the solve and not the FP64 unit; BuildBlockSolver estimates both from the
// systems and takes the faster. The block inverses are of B x B triangles of
// a factor whose system is scaled to a unit diagonal; a pass's strain moves by
// 1e-15 of itself against the row-by-row solve. Against the factor's exact
// solution (forces on every row, degrees 2 to 100 of 40- and 80-element
// models) either form is off by 2e-16 to 3e-15, the one nearer in half of the
// degrees, the other in half. Measured, spheroidal and
// toroidal together, rows -> blocks: lmax 32 0.53 -> 0.098 ms, 45 0.61 -> 0.144,
// 128 1.65 -> 0.70; at lmax 256 the rows' 20 products a row keep the FP64 unit
// busier than the blocks' 26 and stay.
#include <algorithm>

#include "band_block.cuh"
#include "profile.cuh"

namespace sl3dgpu {

namespace {

constexpr int kBlockWarps = 4;
constexpr int kBlockStages = 4;

// U(i, j) of a factor in upper band storage, 0 outside the band or the system.
__device__ inline double FactorAt(const double* ab, int n, int kd, int i, int j) {
  if (i < 0 || j >= n || i > j || j - i > kd) return 0.0;
  return ab[static_cast<long long>(j) * (kd + 1) + kd + i - j];
}

// The coefficients of one block of one system, a warp each.
template <int B>
__global__ void __launch_bounds__(kWarp) BlockCoefficientsKernel(const BlockSystem* systems,
                                                                 const sl3dgpu_band_system* bandSystems,
                                                                 const double* bands, const double* scales,
                                                                 double* data) {
  const BlockSystem s = systems[blockIdx.y];
  const int blk = blockIdx.x;
  if (blk >= s.blocks) return;
  const sl3dgpu_band_system bs = bandSystems[blockIdx.y];
  const double* ab = bands + bs.band;
  const int n = s.n, kd = s.kd, j0 = blk * B, lane = threadIdx.x;
  __shared__ double M[B][B + 1];  // L_JJ^-1, lower triangular
  // column c by lane c: L M = I, L(r, k) = U(j0 + k, j0 + r); rows past the
  // system's end are zero
  if (lane < B) {
    for (int r = 0; r < B; ++r) M[r][lane] = 0.0;
    for (int r = lane; r < B && j0 + r < n; ++r) {
      double sum = r == lane ? 1.0 : 0.0;
      for (int k = lane; k < r; ++k) sum = fma(-FactorAt(ab, n, kd, j0 + k, j0 + r), M[k][lane], sum);
      M[r][lane] = sum / FactorAt(ab, n, kd, j0 + r, j0 + r);
    }
  }
  __syncwarp();
  double* f = data + s.forward + static_cast<long long>(blk) * (kd + B) * B;
  double* b = data + s.backward + static_cast<long long>(blk) * (kd + B) * B;
  for (int e = lane; e < kd * B; e += kWarp) {
    const int t = e / B + 1, r = e % B;
    double sf = 0.0, sb = 0.0;
    for (int k = 0; k <= r; ++k) sf = fma(M[r][k], FactorAt(ab, n, kd, j0 - t, j0 + k), sf);
    for (int k = r; k < B; ++k) sb = fma(M[k][r], FactorAt(ab, n, kd, j0 + k, j0 + B - 1 + t), sb);
    f[e] = sf;
    b[e] = sb;
  }
  f += kd * B;
  b += kd * B;
  for (int e = lane; e < B * B; e += kWarp) {
    const int k = e / B, r = e % B, row = j0 + k;
    double scale = 1.0;
    if (s.scale >= 0 && row < n) scale = scales[s.scale + row];
    if (row == bs.pinned0 || row == bs.pinned1) scale = 0.0;  // a pinned dof's right-hand side is zero
    f[e] = M[r][k] * scale;
    b[e] = M[k][r];
  }
}

template <int B>
__global__ void __launch_bounds__(kBlockWarps* kWarp) BlockSolveKernel(const BlockSystem* systems, const int2* items,
                                                                      const double* data, double* first,
                                                                      double* second, const double* scales, int maxKd) {
  constexpr int C = kWarp / B;  // columns a warp
  extern __shared__ __align__(16) unsigned char blockSmem[];
  const int2 item = items[blockIdx.x];
  const BlockSystem s = systems[item.x];
  const int n = s.n, kd = s.kd, values = (kd + B) * B;
  const int W = ((maxKd + B - 1) / B + 1) * B;  // rows the window holds: kd before the block and the block
  const int warp = threadIdx.x / kWarp, lane = threadIdx.x % kWarp;
  const int r = lane % B, c = lane / B;
  const int col = item.y + warp * C + c;
  const bool live = col < s.nrhs;
  double* stages = reinterpret_cast<double*>(blockSmem);  // [stage][(maxKd + B) B]
  const int stageValues = (maxKd + B) * B;
  double* window = stages + kBlockStages * stageValues + warp * (W + B) * C;  // [row mod W][C]
  double* input = window + W * C;                                               // [B][C]
  double* x = (s.second ? second : first) + s.rhs + col;
  const long long nrhs = s.nrhs;

  auto stage = [&](const double* from, int slot) {
    double* to = stages + slot * stageValues;
    for (int e = threadIdx.x; e < values / 2; e += kBlockWarps * kWarp) {
      const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(to + 2 * e));
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(from + 2 * e) : "memory");
    }
  };
  auto commit = [] { asm volatile("cp.async.commit_group;\n" ::: "memory"); };

  for (int direction = 0; direction < 2; ++direction) {
    const bool forward = direction == 0;
    const double* coefficients = data + (forward ? s.forward : s.backward);
    auto blockOf = [&](int step) { return forward ? step : s.blocks - 1 - step; };
    __syncthreads();  // the stages' last use
    for (int q = 0; q < kBlockStages - 1; ++q) {
      if (q < s.blocks) stage(coefficients + static_cast<long long>(blockOf(q)) * values, q);
      commit();
    }
    for (int e = lane; e < W * C; e += kWarp) window[e] = 0.0;
    int row = blockOf(0) * B + r;
    double next = live && row < n ? x[row * nrhs] : 0.0;
    __syncwarp();
    for (int step = 0; step < s.blocks; ++step) {
      asm volatile("cp.async.wait_group %0;\n" ::"n"(kBlockStages - 2) : "memory");
      __syncthreads();
      const int ahead = step + kBlockStages - 1;
      if (ahead < s.blocks)
        stage(coefficients + static_cast<long long>(blockOf(ahead)) * values, ahead % kBlockStages);
      commit();
      const double* N = stages + (step % kBlockStages) * stageValues + r;
      const double* M = N + kd * B;
      const int j0 = blockOf(step) * B;
      row = j0 + r;
      input[r * C + c] = next;
      if (step + 1 < s.blocks) {
        const int later = blockOf(step + 1) * B + r;
        next = live && later < n ? x[later * nrhs] : 0.0;
      }
      __syncwarp();
      double sum = 0.0;
#pragma unroll
      for (int k = 0; k < B; ++k) sum = fma(M[k * B], input[k * C + c], sum);
      // row j0 - t (forward), j0 + B - 1 + t (backward) of the window
      int at = forward ? j0 % W : (j0 + B - 1) % W;
#pragma unroll 4
      for (int t = 0; t < kd; ++t) {
        at = forward ? (at == 0 ? W - 1 : at - 1) : (at == W - 1 ? 0 : at + 1);
        sum = fma(-N[t * B], window[at * C + c], sum);
      }
      __syncwarp();
      window[(row % W) * C + c] = sum;
      __syncwarp();
      if (live && row < n) x[row * nrhs] = !forward && s.scale >= 0 ? sum * scales[s.scale + row] : sum;
    }
  }
}

// The FP32 solves over row windows (the mixed form's corrections), the same
// recurrence: four columns a lane, so that a coefficient read from shared
// memory serves four products. FP32 chains are short; what bounded the
// row-by-row kernel was its instructions a row at a few warps an SM. A
// correction pass's solves: lmax 64 97 -> 28 us, lmax 128 157 -> 54 us. The
// coefficients are formed in FP64 and rounded once: forces on every row or on a
// lateral range's, degrees 2 to 100 of 40- to 80-element models, leave it off
// by 0.6e-7 to 8e-7 of the solution where the row form is by 0.9e-7 to 17e-7.
template <int B>
__global__ void __launch_bounds__(kBlockWarps* kWarp) BlockSolve32Kernel(const BlockSystem* systems, const int2* items,
                                                                        int firstCount, const float* data,
                                                                        float* first, float* second,
                                                                        const float* scales, const int2* windowsFirst,
                                                                        const int2* windowsSecond, int maxKd) {
  constexpr int C = kWarp / B;  // groups of four columns a warp
  extern __shared__ __align__(16) unsigned char block32Smem[];
  const int2 item = items[blockIdx.x];
  const BlockSystem s = systems[item.x];
  const int2 range = item.x < firstCount ? windowsFirst[item.x] : windowsSecond[item.x - firstCount];
  const int n = s.n, kd = s.kd, values = (kd + B) * B;
  const int lo = min(max(range.x, 0), n), hi = min(range.y, n - 1);
  const int b0 = lo / B, steps = s.blocks - b0;
  if (lo >= n) return;
  const int W = ((maxKd + B - 1) / B + 1) * B;
  const int warp = threadIdx.x / kWarp, lane = threadIdx.x % kWarp;
  const int r = lane % B, c = lane / B;
  const int col = item.y + (warp * C + c) * 4;
  const bool live0 = col < s.nrhs, live1 = col + 2 < s.nrhs;  // column pairs (nrhs is even)
  float* stages = reinterpret_cast<float*>(block32Smem);
  const int stageValues = (maxKd + B) * B;
  float4* window = reinterpret_cast<float4*>(stages + kBlockStages * stageValues) + warp * (W + B) * C;
  float4* input = window + W * C;
  float* x = (s.second ? second : first) + s.rhs + col;
  const long long nrhs = s.nrhs;
  const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);

  auto stage = [&](const float* from, int slot) {
    float* to = stages + slot * stageValues;
    for (int e = threadIdx.x; e < values / 4; e += kBlockWarps * kWarp) {
      const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(to + 4 * e));
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(from + 4 * e) : "memory");
    }
  };
  auto commit = [] { asm volatile("cp.async.commit_group;\n" ::: "memory"); };
  auto load = [&](int row) {
    float4 v = zero;
    if (live0) {
      const float2 p = *reinterpret_cast<const float2*>(x + row * nrhs);
      v.x = p.x;
      v.y = p.y;
    }
    if (live1) {
      const float2 p = *reinterpret_cast<const float2*>(x + row * nrhs + 2);
      v.z = p.x;
      v.w = p.y;
    }
    return v;
  };

  for (int direction = 0; direction < 2; ++direction) {
    const bool forward = direction == 0;
    const float* coefficients = data + (forward ? s.forward : s.backward);
    const int last = forward ? hi : n - 1;  // forward rows above hi are zero and not read
    auto blockOf = [&](int step) { return forward ? b0 + step : s.blocks - 1 - step; };
    __syncthreads();
    for (int q = 0; q < kBlockStages - 1; ++q) {
      if (q < steps) stage(coefficients + static_cast<long long>(blockOf(q)) * values, q);
      commit();
    }
    for (int e = lane; e < W * C; e += kWarp) window[e] = zero;
    int row = blockOf(0) * B + r;
    float4 next = row >= lo && row <= last ? load(row) : zero;
    __syncwarp();
    for (int step = 0; step < steps; ++step) {
      asm volatile("cp.async.wait_group %0;\n" ::"n"(kBlockStages - 2) : "memory");
      __syncthreads();
      const int ahead = step + kBlockStages - 1;
      if (ahead < steps) stage(coefficients + static_cast<long long>(blockOf(ahead)) * values, ahead % kBlockStages);
      commit();
      const float* N = stages + (step % kBlockStages) * stageValues + r;
      const float* M = N + kd * B;
      const int j0 = blockOf(step) * B;
      row = j0 + r;
      input[r * C + c] = next;
      if (step + 1 < steps) {
        const int later = blockOf(step + 1) * B + r;
        next = later >= lo && later <= last ? load(later) : zero;
      }
      __syncwarp();
      float4 sum = zero;
#pragma unroll
      for (int k = 0; k < B; ++k) {
        const float m = M[k * B];
        const float4 v = input[k * C + c];
        sum.x = fmaf(m, v.x, sum.x);
        sum.y = fmaf(m, v.y, sum.y);
        sum.z = fmaf(m, v.z, sum.z);
        sum.w = fmaf(m, v.w, sum.w);
      }
      int at = forward ? j0 % W : (j0 + B - 1) % W;
#pragma unroll 4
      for (int t = 0; t < kd; ++t) {
        at = forward ? (at == 0 ? W - 1 : at - 1) : (at == W - 1 ? 0 : at + 1);
        const float m = -N[t * B];
        const float4 v = window[at * C + c];
        sum.x = fmaf(m, v.x, sum.x);
        sum.y = fmaf(m, v.y, sum.y);
        sum.z = fmaf(m, v.z, sum.z);
        sum.w = fmaf(m, v.w, sum.w);
      }
      __syncwarp();
      window[(row % W) * C + c] = sum;
      __syncwarp();
      if (row >= lo && row < n) {
        const float f = !forward && s.scale >= 0 ? scales[s.scale + row] : 1.0f;
        if (live0) *reinterpret_cast<float2*>(x + row * nrhs) = make_float2(sum.x * f, sum.y * f);
        if (live1) *reinterpret_cast<float2*>(x + row * nrhs + 2) = make_float2(sum.z * f, sum.w * f);
      }
    }
  }
}

__global__ void RoundKernel(const double* in, long long n, float* out) {
  const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n; i += stride)
    out[i] = static_cast<float>(in[i]);
}

size_t BlockSmem32(int B, int kd) {
  const int W = ((kd + B - 1) / B + 1) * B, C = kWarp / B;
  return sizeof(float) * (static_cast<size_t>(kBlockStages) * (kd + B) * B + static_cast<size_t>(kBlockWarps) * (W + B) * C * 4);
}

size_t BlockSmem(int B, int kd) {
  const int W = ((kd + B - 1) / B + 1) * B, C = kWarp / B;
  return sizeof(double) * (static_cast<size_t>(kBlockStages) * (kd + B) * B + static_cast<size_t>(kBlockWarps) * (W + B) * C);
}

// A solve's time in cycles: the FP64 unit's (19 cycles an SM a warp
// instruction, 152 SMs) or the longest system's chain (64 cycles an
// instruction, and about 150 a block for its synchronisation), the larger.
struct SolveCost {
  double unit = 0.0, chain = 0.0;
  double Cycles() const { return std::max(unit * 19.0 / 152.0, chain); }
};
void AddRows(const sl3dgpu_band_system& s, SolveCost& c) {  // CholeskySolve64Kernel
  c.unit += 2.0 * s.n * (s.ku + 3) * ((s.nrhs + kWarp - 1) / kWarp);
  c.chain = std::max(c.chain, 2.0 * s.n * (s.ku + 3) * 64.0);
}
void AddBlocks(const sl3dgpu_band_system& s, int B, SolveCost& c) {
  const double blocks = (s.n + B - 1) / B, instructions = s.ku + B + 1;
  const int columns = kBlockWarps * kWarp / B;
  c.unit += 2.0 * blocks * instructions * kBlockWarps * ((s.nrhs + columns - 1) / columns);
  c.chain = std::max(c.chain, 2.0 * blocks * (64.0 * instructions + 150.0));
}

}  // namespace

int BuildBlockSolver(const std::vector<sl3dgpu_band_system>& first, const std::vector<sl3dgpu_band_system>& second,
                     const double* bands, const double* scales, bool fp32, BlockSolver& out, cudaStream_t stream) {
  out.block = 0;
  SolveCost rows[2], blocks8, blocks16;
  for (int which = 0; which < 2; ++which)
    for (const auto& s : which ? second : first) {
      AddRows(s, rows[which]);
      AddBlocks(s, 8, blocks8);
      AddBlocks(s, 16, blocks16);
    }
  // row by row the two lists are two launches
  const double byRows = rows[0].Cycles() + rows[1].Cycles();
  const int B = blocks16.Cycles() < blocks8.Cycles() ? 16 : 8;
  if (first.empty() || byRows <= std::min(blocks8.Cycles(), blocks16.Cycles())) return SL3DGPU_OK;
  std::vector<BlockSystem> systems;
  std::vector<sl3dgpu_band_system> bandSystems;
  std::vector<int2> items, items32;
  bool even = true;  // the FP32 form takes columns in pairs
  long long values = 0;
  int maxBlocks = 0;
  for (int which = 0; which < 2; ++which)
    for (const auto& s : which ? second : first) {
      BlockSystem b{};
      b.n = s.n;
      b.kd = s.ku;
      b.nrhs = s.nrhs;
      b.blocks = (s.n + B - 1) / B;
      const long long each = static_cast<long long>(b.blocks) * (b.kd + B) * B;
      b.forward = values;
      b.backward = values + each;
      values += 2 * each;
      b.rhs = s.rhs;
      b.scale = s.scale;
      b.second = which;
      for (int c = 0; c < s.nrhs; c += kBlockWarps * kWarp / B)
        items.push_back(make_int2(static_cast<int>(systems.size()), c));
      for (int c = 0; c < s.nrhs; c += 4 * kBlockWarps * kWarp / B)
        items32.push_back(make_int2(static_cast<int>(systems.size()), c));
      even = even && s.nrhs % 2 == 0 && s.rhs % 2 == 0;
      out.kd = std::max(out.kd, b.kd);
      maxBlocks = std::max(maxBlocks, b.blocks);
      systems.push_back(b);
      bandSystems.push_back(s);
    }
  if (BlockSmem(B, out.kd) > 200 * 1024) return SL3DGPU_OK;
  // the longest systems first
  auto longer = [&](const int2& a, const int2& b) {
    return systems[a.x].n * systems[a.x].kd > systems[b.x].n * systems[b.x].kd;
  };
  std::stable_sort(items.begin(), items.end(), longer);
  std::stable_sort(items32.begin(), items32.end(), longer);
  out.firstCount = static_cast<int>(first.size());
  out.itemCount = static_cast<int>(items.size());
  SL3D_CUDA(cudaMalloc(&out.systems, systems.size() * sizeof(BlockSystem)));
  SL3D_CUDA(cudaMalloc(&out.items, items.size() * sizeof(int2)));
  SL3D_CUDA(cudaMalloc(&out.data, values * sizeof(double)));
  SL3D_CUDA(CopyIn(out.systems, systems.data(), systems.size() * sizeof(BlockSystem)));
  SL3D_CUDA(CopyIn(out.items, items.data(), items.size() * sizeof(int2)));
  sl3dgpu_band_system* device = nullptr;
  SL3D_CUDA(cudaMalloc(&device, bandSystems.size() * sizeof(sl3dgpu_band_system)));
  cudaError_t e = CopyIn(device, bandSystems.data(), bandSystems.size() * sizeof(sl3dgpu_band_system));
  if (e == cudaSuccess) {
    prof::Scope scope(prof::kOther, stream);
    const dim3 grid(maxBlocks, static_cast<unsigned>(systems.size()));
    if (B == 8)
      BlockCoefficientsKernel<8><<<grid, kWarp, 0, stream>>>(out.systems, device, bands, scales, out.data);
    else
      BlockCoefficientsKernel<16><<<grid, kWarp, 0, stream>>>(out.systems, device, bands, scales, out.data);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
  }
  cudaFree(device);
  SL3D_CUDA(e);
  if (fp32 && even) {
    out.itemCount32 = static_cast<int>(items32.size());
    SL3D_CUDA(cudaMalloc(&out.items32, items32.size() * sizeof(int2)));
    SL3D_CUDA(cudaMalloc(&out.data32, values * sizeof(float)));
    SL3D_CUDA(CopyIn(out.items32, items32.data(), items32.size() * sizeof(int2)));
    RoundKernel<<<1216, 256, 0, stream>>>(out.data, values, out.data32);
    SL3D_CHECK_LAUNCH();
    SL3D_CUDA(cudaStreamSynchronize(stream));
  }
  out.block = B;
  return SL3DGPU_OK;
}

int RunBlockSolver(const BlockSolver& b, double* first, double* second, const double* scales, cudaStream_t stream) {
  const size_t smem = BlockSmem(b.block, b.kd);
  prof::Scope scope(prof::kBandSolve, stream);
  if (b.block == 8) {
    SL3D_CUDA(AllowDynamicSmem(BlockSolveKernel<8>));
    BlockSolveKernel<8><<<b.itemCount, kBlockWarps * kWarp, smem, stream>>>(b.systems, b.items, b.data, first, second,
                                                                            scales, b.kd);
  } else {
    SL3D_CUDA(AllowDynamicSmem(BlockSolveKernel<16>));
    BlockSolveKernel<16><<<b.itemCount, kBlockWarps * kWarp, smem, stream>>>(b.systems, b.items, b.data, first, second,
                                                                             scales, b.kd);
  }
  SL3D_CHECK_LAUNCH();
  return SL3DGPU_OK;
}

int RunBlockSolver32(const BlockSolver& b, float* first, float* second, const float* scales, const int2* windowsFirst,
                     const int2* windowsSecond, cudaStream_t stream) {
  const size_t smem = BlockSmem32(b.block, b.kd);
  prof::Scope scope(prof::kBandSolve32, stream);
  if (b.block == 8) {
    SL3D_CUDA(AllowDynamicSmem(BlockSolve32Kernel<8>));
    BlockSolve32Kernel<8><<<b.itemCount32, kBlockWarps * kWarp, smem, stream>>>(
        b.systems, b.items32, b.firstCount, b.data32, first, second, scales, windowsFirst, windowsSecond, b.kd);
  } else {
    SL3D_CUDA(AllowDynamicSmem(BlockSolve32Kernel<16>));
    BlockSolve32Kernel<16><<<b.itemCount32, kBlockWarps * kWarp, smem, stream>>>(
        b.systems, b.items32, b.firstCount, b.data32, first, second, scales, windowsFirst, windowsSecond, b.kd);
  }
  SL3D_CHECK_LAUNCH();
  return SL3DGPU_OK;
}

}  // namespace sl3dgpu
