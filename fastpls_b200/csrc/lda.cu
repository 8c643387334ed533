// Pooled-covariance LDA on latent scores (FP64 on the device).
//
// Reference: train_lda_prefixes / finalize_lda_prefixes
// (inst/include/fastpls/core/lda.hpp:88-223) and ResidentLda
// (src/cuda_resident_lda.cuh:41-121): class means, pooled within-class
// covariance (T^T T - sum_c n_c mu_c mu_c^T) / max(1, n - c), ridge
// rho * trace / k for rho in {1e-8, 1e-6, 1e-5, 1e-4, 1e-3, 1e-2} (first that
// factors), Cholesky solve, constants -0.5 mu^T Sigma^-1 mu + log prior.
// Moments come from two FP64 GEMMs (T^T T and onehot^T T); the per-prefix
// k x k factorisation runs in one block.
#include "lda.cuh"
#include "small.cuh"

#include <algorithm>
#include <cfloat>

namespace fpls {

namespace {

__global__ void one_hot_kernel(const int* __restrict__ labels, int n, int c,
                               double* oh) {
  const long total = (long)n * c;
  for (long idx = blockIdx.x * (long)blockDim.x + threadIdx.x; idx < total;
       idx += (long)gridDim.x * blockDim.x) {
    const int i = (int)(idx % n), k = (int)(idx / n);
    oh[idx] = labels[i] == k + 1 ? 1.0 : 0.0;
  }
}

// One block per prefix: pooled covariance for its first k components, ridge
// retries, linear (c x k) and constants (c). Latency-bound; the factor by the
// whole block and one class per thread in the solves, every prefix of a call
// in one launch (a serial thread per launch took 43 us a prefix at k <= 9, 10
// classes; 14 us for four prefixes so).
constexpr int kLdaBatch = 32;
struct LdaJobs {
  int k[kLdaBatch];
  double* linear[kLdaBatch];
  double* constants[kLdaBatch];
};
__global__ void lda_finalize(const double* __restrict__ gram, int a, const double* __restrict__ sums,
                             int c, const double* __restrict__ counts, int n, LdaJobs jobs, int* flag) {
  extern __shared__ double sm[];
  const int k = jobs.k[blockIdx.x];
  double* linear = jobs.linear[blockIdx.x];
  double* constants = jobs.constants[blockIdx.x];
  double* cov = sm;                 // k x k
  double* L = cov + k * k;          // k x k
  double* means = L + k * k;        // c x k (class-major)
  const int t = threadIdx.x;
  for (int idx = t; idx < c * k; idx += blockDim.x) {
    const int cls = idx / k, j = idx % k;
    means[cls * k + j] = sums[cls + (long)j * c] / counts[cls];
  }
  __syncthreads();
  const double denom = (double)max(1, n > c ? n - c : 1);
  for (int idx = t; idx < k * k; idx += blockDim.x) {
    const int i = idx % k, j = idx / k;
    double v = gram[i + (long)j * a];
    for (int cls = 0; cls < c; ++cls) v -= counts[cls] * means[cls * k + i] * means[cls * k + j];
    cov[i + j * k] = v / denom;
  }
  __syncthreads();
  double scale = 0.0;
  for (int i = 0; i < k; ++i) scale += cov[i + i * k];
  scale /= k;
  if (!isfinite(scale) || scale <= 0.0) scale = 1.0;
  const double grid[6] = {1e-8, 1e-6, 1e-5, 1e-4, 1e-3, 1e-2};
  bool solved = false;
  for (int g = 0; g < 6 && !solved; ++g) {
    __syncthreads();
    for (int idx = t; idx < k * k; idx += blockDim.x) L[idx] = cov[idx];
    if (!cholesky_block(L, k, grid[g] * scale)) continue;
    int ok = 1;
    for (int cls = t; cls < c; cls += blockDim.x) {
      for (int j = 0; j < k; ++j) linear[cls + (long)j * c] = means[cls * k + j];
      if (!cholesky_solve_strided(L, k, linear + cls, c)) ok = 0;
    }
    solved = __syncthreads_and(ok) != 0;
    if (solved && t == 0) constants[c] = grid[g] * scale;
  }
  if (!solved && t == 0) flag_error(flag, 5);
  for (int cls = t; cls < c; cls += blockDim.x) {
    double prod = 0.0;
    for (int j = 0; j < k; ++j) prod += means[cls * k + j] * linear[cls + (long)j * c];
    const double prior = counts[cls] / n;
    constants[cls] = -0.5 * prod + log(fmax(prior, DBL_MIN));
  }
}

}  // namespace

void LdaState::train(const double* scores, int n_, long lds, int a_,
                     const int* labels, int c_, const std::vector<int>& counts,
                     int* flag_, cudaStream_t stream) {
  n = n_;
  a = a_;
  c = c_;
  flag = flag_;
  std::vector<double> hc(c);
  for (int k = 0; k < c; ++k) {
    require(counts[k] > 0, "fastPLS LDA received an empty class");
    hc[k] = counts[k];
  }
  counts_dev.allocate(c, stream);
  FPLS_CHECK(cudaMemcpyAsync(counts_dev.get(), hc.data(), sizeof(double) * c,
                             cudaMemcpyHostToDevice, stream));
  gram.allocate((size_t)a * a, stream);
  sums.allocate((size_t)c * a, stream);
  DeviceArray<double> oh((size_t)n * c, stream);
  one_hot_kernel<<<std::min<unsigned>(ceil_div((size_t)n * c, 256), 8 * num_sms()), 256, 0, stream>>>(labels, n, c, oh.get());
  count_launch();
  FPLS_LAUNCH("one_hot");
  GemmArgs g;
  g.M = a;
  g.N = a;
  g.K = n;
  g.A = scores;
  g.lda = lds;
  g.trans_a = true;
  g.B = scores;
  g.ldb = lds;
  g.C = gram.get();
  g.ldc = a;
  gemm_f64(g, stream);
  GemmArgs h = g;
  h.M = c;
  h.N = a;
  h.A = oh.get();
  h.lda = n;
  h.C = sums.get();
  h.ldc = c;
  gemm_f64(h, stream);
  prefixes.clear();
}

void LdaState::finalize(const int* ks, int count, cudaStream_t stream) {
  // terms on their way: they join `prefixes` once the launch that computes them
  // is enqueued, so that a call that fails leaves none behind uncomputed
  std::vector<Prefix> pending;
  auto flush = [&] {
    if (pending.empty()) return;
    LdaJobs jobs;
    int kmax = 0;
    for (size_t j = 0; j < pending.size(); ++j) {
      jobs.k[j] = pending[j].k;
      jobs.linear[j] = pending[j].linear.get();
      jobs.constants[j] = pending[j].constants.get();
      kmax = std::max(kmax, pending[j].k);
    }
    const size_t smem = (2 * (size_t)kmax * kmax + (size_t)c * kmax) * sizeof(double);
    allow_shared_memory((const void*)lda_finalize);
    lda_finalize<<<(unsigned)pending.size(), 256, smem, stream>>>(gram.get(), a, sums.get(), c, counts_dev.get(), n,
                                                                  jobs, flag);
    count_launch();
    FPLS_LAUNCH("lda_finalize");
    for (Prefix& pr : pending) prefixes.push_back(std::move(pr));
    pending.clear();
  };
  for (int j = 0; j < count; ++j) {
    const int k = ks[j];
    require(k >= 1 && k <= a, "invalid LDA prefix");
    if (find(k)) continue;
    Prefix pr;
    pr.k = k;
    pr.linear.allocate((size_t)c * k, stream);
    pr.constants.allocate(c + 1, stream);
    pending.push_back(std::move(pr));
    if (pending.size() == kLdaBatch) flush();
  }
  flush();
}

const LdaState::Prefix* LdaState::find(int k) const {
  for (const auto& pr : prefixes)
    if (pr.k == k) return &pr;
  return nullptr;
}

void LdaState::discriminants(const double* scores, int rows, long lds, const int* ks, int count,
                             double* out, cudaStream_t stream) {
  finalize(ks, count, stream);
  apply_prefix_maps<double>(scores, rows, lds, c, maps(ks, count).data(), count, out, stream);
}

void LdaState::discriminants(const double* scores, int rows, long lds, const int* ks, int count,
                             float* out, cudaStream_t stream) {
  finalize(ks, count, stream);
  apply_prefix_maps<float>(scores, rows, lds, c, maps(ks, count).data(), count, out, stream);
}

std::vector<PrefixMap> LdaState::maps(const int* ks, int count) const {
  std::vector<PrefixMap> out(count);
  for (int j = 0; j < count; ++j) {
    const Prefix* pr = find(ks[j]);
    out[j] = {pr->k, pr->linear.get(), pr->constants.get(), c, 1};
  }
  return out;
}

}  // namespace fpls
