// FP64-accumulating GEMM: schedule, split-K reduction, symmetric mirror and
// timing around the DMMA kernel of gemm_mma.cu.
//
//   C[M x N] = alpha * op(A)[M x K] * op(B)[K x N] (+ beta C)
//
// Every product and sum is FP64: this is the precision contract of the
// fitting path (results track the FP64 CPU reference to ~1e-12 rather than to
// FP32 rounding). Slices over K go to a scratch buffer and are summed in
// slice order, so results are bitwise deterministic run to run.
#include "gemm_mma.cuh"

#include <algorithm>
#include <utility>
#include <vector>

namespace fpls {

namespace {

// Element (row, col) of the sum of the slices, in slice order.
__device__ __forceinline__ double slice_sum(const double* __restrict__ slices, int splits, long at,
                                            long stride) {
  double v = slices[at];
  int z = 1;
  for (; z + 7 < splits; z += 8) {
    double x[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) x[u] = slices[at + (z + u) * stride];
#pragma unroll
    for (int u = 0; u < 8; ++u) v += x[u];
  }
  for (; z < splits; ++z) v += slices[at + z * stride];
  return v;
}

// C = alpha * (sum of `splits` contiguous M x N slices) - coff (+ beta C)
__global__ void sum_slices(const double* __restrict__ slices, int splits, int M, int N, double alpha,
                           double beta, double* C, long ldc, const double* __restrict__ coff,
                           int coff_parts) {
  const long total = (long)M * N;
  for (long idx = blockIdx.x * (long)blockDim.x + threadIdx.x; idx < total;
       idx += (long)gridDim.x * blockDim.x) {
    double v = alpha * slice_sum(slices, splits, idx, total);
    if (coff) v -= column_offset(coff, coff_parts, (int)(idx / M));
    double* dst = C + (idx % M) + (idx / M) * ldc;
    *dst = beta != 0.0 ? fma(beta, *dst, v) : v;
  }
}

// The same for many slices of a small result: 8 threads an element, thread q
// summing slices q, q + 8, ... and the 8 sums added in order, so that 144
// slices of a 9 x 9 Gram are 18 loads deep instead of 144 (61 us, 5 us so).
// Which of the two runs depends on the number of slices alone.
constexpr int kManySlices = 16;
__global__ void __launch_bounds__(256)
    sum_many_slices(const double* __restrict__ slices, int splits, int M, int N, double alpha,
                    double beta, double* C, long ldc, const double* __restrict__ coff, int coff_parts) {
  __shared__ double part[8][32];
  const long total = (long)M * N;
  const int x = threadIdx.x & 31, q = threadIdx.x >> 5;
  for (long base = blockIdx.x * 32L; base < total; base += gridDim.x * 32L) {
    const long idx = base + x;
    double v = 0.0;
    if (idx < total) {
#pragma unroll 6
      for (int z = q; z < splits; z += 8) v += slices[idx + z * total];
    }
    part[q][x] = v;
    __syncthreads();
    if (q == 0 && idx < total) {
#pragma unroll
      for (int u = 1; u < 8; ++u) v += part[u][x];
      v *= alpha;
      if (coff) v -= column_offset(coff, coff_parts, (int)(idx / M));
      double* dst = C + (idx % M) + (idx / M) * ldc;
      *dst = beta != 0.0 ? fma(beta, *dst, v) : v;
    }
    __syncthreads();
  }
}

// Symmetric result from its lower triangle: 32 x 32 tiles (bi >= bj) of the
// slice sum (splits 0: of C itself) times alpha, written to C and, through
// shared memory so that both stores are coalesced, mirrored above the
// diagonal. HBM-bound: one read of the lower triangle (per slice) and one
// write of the matrix.
constexpr int MIR = 32;
__global__ void __launch_bounds__(MIR * 8)
    mirror_lower(const double* __restrict__ slices, int splits, double alpha, double* C, int n, long ldc) {
  __shared__ double tile[MIR][MIR + 1];
  const int bi = blockIdx.x, bj = blockIdx.y;
  if (bi < bj) return;
  const int x = threadIdx.x & (MIR - 1);
  for (int y = threadIdx.x / MIR; y < MIR; y += 8) {
    const int r = bi * MIR + x, c = bj * MIR + y;
    if (r < n && c < n && r >= c) {
      double v;
      if (splits > 0) {
        v = alpha * slice_sum(slices, splits, r + (long)c * n, (long)n * n);
        C[r + (long)c * ldc] = v;
      } else {
        v = C[r + (long)c * ldc];
      }
      tile[y][x] = v;
    }
  }
  __syncthreads();
  for (int y = threadIdx.x / MIR; y < MIR; y += 8) {
    const int r = bj * MIR + x, c = bi * MIR + y;  // the mirrored element
    if (c < n && r < c) C[r + (long)c * ldc] = tile[x][y];
  }
}

void launch_mirror(const double* slices, int splits, double alpha, double* C, int n, long ldc,
                   cudaStream_t stream) {
  const unsigned t = ceil_div(n, MIR);
  mirror_lower<<<dim3(t, t), MIR * 8, 0, stream>>>(slices, splits, alpha, C, n, ldc);
  count_launch();
  FPLS_LAUNCH("mirror_lower");
}

// Live timing of GEMM launches (benchmark instrumentation): when enabled,
// every gemm_f64 call is bracketed by CUDA events on its own stream.
struct GemmTiming {
  bool enabled = false;
  std::vector<std::pair<cudaEvent_t, cudaEvent_t>> events;
  std::vector<double> flops;
};
GemmTiming& timing() {
  static GemmTiming t;
  return t;
}

}  // namespace

// Tile and K slices with the least modelled time. Per SM the DMMA pipe does
// 64 FMAs a clock (a 128 x 128 x 16 slab in 4096 clocks; 1.25 of that in
// practice), a slab takes no less than about 500 clocks of load latency
// through the 4-stage ring, a block about 4000 clocks to start, fill and
// store, and K slices cost a second kernel that reads them.
GemmPlan gemm_plan(int M, int N, int K, bool lower, int k_slice) {
  static const int tiles[5][2] = {{128, 128}, {128, 64}, {128, 32}, {128, 16}, {64, 64}};
  const double sms = num_sms();
  GemmPlan best;
  double best_cost = -1.0;
  for (const auto& t : tiles) {
    if (lower && t[0] != t[1]) continue;
    const long tm = ceil_div(M, t[0]), tn = ceil_div(N, t[1]);
    if (tm > 65535) continue;
    const double count = lower ? (double)tm * (tm + 1) / 2 : (double)tm * tn;
    const int occ = t[0] * t[1] >= 128 * 128 ? 1 : 2;
    const double slab_clk = t[0] * t[1] / 4.0 * 1.25;
    // slices are kept to 256 MB
    const double room = 256.0 * 1024 * 1024 / ((double)M * N * 8.0);
    const int most = (int)std::max(1.0, std::min(room, k_slice > 0 ? (double)ceil_div(std::max(K, 1), k_slice)
                                                                   : std::min(256.0, K / 64.0)));
    for (int s = k_slice > 0 ? most : 1; s <= most; s = s < 8 ? s + 1 : s + s / 8) {
      const double slabs = ceil_div(ceil_div(K, s), 16);
      const double per_sm = std::ceil(count * s / sms);
      const double waves = std::ceil(per_sm / occ);
      double cost = waves * 4000.0 + slabs * std::max(500.0 * waves, slab_clk * per_sm);
      if (s > 1) cost += 5000.0 + (double)M * N * 8.0 * (s + 1) / 2500.0;
      if (best_cost < 0.0 || cost < best_cost) {
        best_cost = cost;
        best.tm = t[0];
        best.tn = t[1];
        best.splits = s;
      }
    }
  }
  return best;
}

void gemm_profile_enable(bool on) { timing().enabled = on; }

void gemm_profile_read(double* ms, double* flops, unsigned long long* launches) {
  GemmTiming& t = timing();
  double total_ms = 0.0, total_flops = 0.0;
  for (size_t k = 0; k < t.events.size(); ++k) {
    float e = 0.f;
    cudaEventSynchronize(t.events[k].second);
    cudaEventElapsedTime(&e, t.events[k].first, t.events[k].second);
    total_ms += e;
    total_flops += t.flops[k];
    cudaEventDestroy(t.events[k].first);
    cudaEventDestroy(t.events[k].second);
  }
  if (ms) *ms = total_ms;
  if (flops) *flops = total_flops;
  if (launches) *launches = t.events.size();
  t.events.clear();
  t.flops.clear();
}

void gemm_f64(const GemmArgs& g, cudaStream_t stream) {
  require(g.M >= 0 && g.N >= 0 && g.K >= 0, "invalid GEMM dimensions");
  if (g.M == 0 || g.N == 0) return;
  require(!g.lower || (g.M == g.N && g.beta == 0.0 && !g.coff), "symmetric GEMM takes a square product");
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  if (timing().enabled) {
    FPLS_CHECK(cudaEventCreate(&ev0));
    FPLS_CHECK(cudaEventCreate(&ev1));
    FPLS_CHECK(cudaEventRecord(ev0, stream));
  }
  const GemmPlan plan = gemm_plan(g.M, g.N, g.K, g.lower, g.k_slice);
  if (plan.splits > 1) {
    const long total = (long)g.M * g.N;
    DeviceArray<double> slices((size_t)plan.splits * total, stream);
    gemm_mma_launch(g, plan, slices.get(), g.M, total, 1.0, 0.0, nullptr, stream);
    if (g.lower) {
      launch_mirror(slices.get(), plan.splits, g.alpha, g.C, g.M, g.ldc, stream);
    } else {
      if (plan.splits >= kManySlices)
        sum_many_slices<<<(unsigned)std::min<long>((total + 31) / 32, 32L * num_sms()), 256, 0, stream>>>(
            slices.get(), plan.splits, g.M, g.N, g.alpha, g.beta, g.C, g.ldc, g.coff, g.coff_parts);
      else
        sum_slices<<<(unsigned)std::min<long>((total + 127) / 128, 16L * num_sms()), 128, 0, stream>>>(
            slices.get(), plan.splits, g.M, g.N, g.alpha, g.beta, g.C, g.ldc, g.coff, g.coff_parts);
      count_launch();
      FPLS_LAUNCH("sum_slices");
    }
  } else {
    gemm_mma_launch(g, plan, g.C, g.ldc, 0, g.alpha, g.beta, g.coff, stream);
    if (g.lower) mirror_lower_triangle(g.C, g.M, g.ldc, stream);
  }
  if (ev0) {
    FPLS_CHECK(cudaEventRecord(ev1, stream));
    timing().events.emplace_back(ev0, ev1);
    // algorithmic FLOPs: a symmetric product needs only its lower triangle
    timing().flops.push_back(g.lower ? (double)g.M * (g.M + 1.0) * g.K
                                     : 2.0 * g.M * (double)g.N * g.K);
  }
}

void mirror_lower_triangle(double* C, int n, long ldc, cudaStream_t stream) {
  launch_mirror(nullptr, 0, 1.0, C, n, ldc, stream);
}

}  // namespace fpls
