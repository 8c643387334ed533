// PLS-SVD on the device (FP64 arithmetic, raw X).
//
// Reference: assemble_plssvd_model (inst/include/fastpls/core/plssvd.hpp:57-166)
// and ResidentPlssvd::fit_loaded (src/cuda_resident_plssvd.cuh:82-154):
//   S = Xs^T Yc ; S = U D V^T (rank k) ; R = U_k ; T = Xs R ; G = T^T T ;
//   per prefix j: W_j = G_j^-1 diag(d_1..d_j) V_j^T, Yhat = ymean + T_j W_j.
// The reference's randomized SVD spans the whole response space whenever
// k + oversample >= m, so the SVD here is exact: the m x m Gram S^T S is
// diagonalised by Jacobi (one block) and U = S V D^-1 is formed with one small
// GEMM. One pass over X forms S, one more forms T.
#include "kernels.cuh"
#include "model.cuh"
#include "small.cuh"

#include <algorithm>

namespace fpls {

namespace {

// Eigen-decompose the packed Gram; emit sigma (k), Vk (m x k) and
// Z = Vk D^-1 (m x k) so that U = S Z.
__global__ void small_svd_kernel(const double* __restrict__ gpk, int m, int k,
                                 double* sigma, double* Vk, double* Z,
                                 int* flag) {
  extern __shared__ double sm[];
  double* A = sm;
  double* E = sm + m * m;
  int* order = reinterpret_cast<int*>(E + m * m);
  for (int c = threadIdx.x; c < m; c += blockDim.x)
    for (int d = 0; d <= c; ++d) {
      const double v = gpk[c * (c + 1) / 2 + d];
      A[c + d * m] = v;
      A[d + c * m] = v;
    }
  __syncthreads();
  jacobi_eigen(A, E, m);
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 0; i < m; ++i) order[i] = i;
    for (int i = 1; i < m; ++i) {  // insertion sort, descending eigenvalue
      const int key = order[i];
      int j = i - 1;
      while (j >= 0 && A[order[j] + order[j] * m] < A[key + key * m]) {
        order[j + 1] = order[j];
        --j;
      }
      order[j + 1] = key;
    }
    for (int c = 0; c < k; ++c) {
      const int src = order[c];
      const double lam = A[src + src * m];
      const double s = lam > 0.0 ? sqrt(lam) : 0.0;
      if (!(s > 0.0) || !isfinite(s)) flag_error(flag, 1);
      int arg = 0;
      for (int r = 1; r < m; ++r)
        if (fabs(E[r + src * m]) > fabs(E[arg + src * m])) arg = r;
      const double sgn = E[arg + src * m] < 0.0 ? -1.0 : 1.0;
      sigma[c] = s;
      for (int r = 0; r < m; ++r) {
        const double v = sgn * E[r + src * m];
        Vk[r + c * m] = v;
        Z[r + c * m] = s > 0.0 ? v / s : 0.0;
      }
    }
  }
}

// Block k - 1: the prefix-k weights W_k = G_k^-1 diag(sigma_1..k) V_k^T (k x m)
// from the Cholesky factor of the leading k x k block of the score Gram, one
// response column per thread. Latency-bound; one thread per prefix with a
// serial factor took 126 us at k = 9, 10 responses, 13 us so.
constexpr int kWeightThreads = 128;
__global__ void __launch_bounds__(kWeightThreads)
    plssvd_weights_kernel(const double* __restrict__ gram, int a, const double* __restrict__ sigma,
                          const double* __restrict__ Vk, int m, double* W, int* flag) {
  extern __shared__ double L[];  // k x k
  const int k = blockIdx.x + 1;
  for (int e = threadIdx.x; e < k * k; e += blockDim.x) L[e] = gram[e % k + (long)(e / k) * a];
  if (!cholesky_block(L, k, 0.0)) {
    if (threadIdx.x == 0) flag_error(flag, 6);
    return;
  }
  double* Wk = W + (size_t)(k - 1) * a * m;
  for (int r = threadIdx.x; r < m; r += blockDim.x) {
    for (int c = 0; c < k; ++c) Wk[c + (long)r * k] = sigma[c] * Vk[r + c * m];
    cholesky_solve_strided(L, k, Wk + (long)r * k, 1);
  }
}

}  // namespace

template <class T>
void fit_plssvd(const T* X, int n, int p, long ld, const double* Yc,
                const double* ycsum, int m, int components, int scaling,
                DeviceModel& model, Workspace& ws, cudaStream_t stream) {
  require(m >= 1 && m <= kMaxResponses, "PLS-SVD supports 1..112 responses or classes");
  require(components <= 128, "PLS-SVD supports at most 128 components");
  const int k = components;
  require(k <= std::min(p, m), "fastPLS PLS-SVD component count exceeds cross-covariance rank");
  if (model.classification && k >= m)
    throw std::invalid_argument("classification PLS-SVD components must be below class count");
  ws.ensure(n, p, m, k, stream);
  model.method = kPlssvd;
  model.n = n;
  model.p = p;
  model.feature_p = p;
  model.m = m;
  model.scaling = scaling;
  DeviceArray<double> S((size_t)p * m, stream);
  compute_crossprod<T>(X, n, p, ld, Yc, ycsum, m, scaling, model, S.get(), ws, stream);
  double* gpk = ws.small.get() + 8 + kMaxResponses;
  gram_of_columns(S.get(), p, m, gpk, ws, stream);
  model.sigma.allocate(k, stream);
  model.Q.allocate((size_t)m * k, stream);
  DeviceArray<double> Z((size_t)m * k, stream);
  const size_t smem = 2 * (size_t)m * m * sizeof(double) + m * sizeof(int) + 16;
  allow_shared_memory((const void*)small_svd_kernel);
  small_svd_kernel<<<1, jacobi_threads(m), smem, stream>>>(gpk, m, k, model.sigma.get(),
                                            model.Q.get(), Z.get(), ws.flag.get());
  count_launch();
  FPLS_LAUNCH("small_svd");
  // U = S Z  (p x k)
  model.R.allocate((size_t)p * k, stream);
  GemmArgs g;
  g.M = p;
  g.N = k;
  g.K = m;
  g.A = S.get();
  g.lda = p;
  g.B = Z.get();
  g.ldb = m;
  g.C = model.R.get();
  g.ldc = p;
  gemm_f64(g, stream);
  model.a = k;
  // T = Xs U  (n x k)
  model.T.allocate((size_t)n * k, stream);
  project_rows<T>(model, X, n, ld, k, model.T.get(), n, ws, stream);
  // G = T^T T (k x k)
  DeviceArray<double> gram((size_t)k * k, stream);
  GemmArgs h;
  h.M = k;
  h.N = k;
  h.K = n;
  h.A = model.T.get();
  h.lda = n;
  h.trans_a = true;
  h.B = model.T.get();
  h.ldb = n;
  h.C = gram.get();
  h.ldc = k;
  gemm_f64(h, stream);
  model.W.allocate((size_t)k * k * m, stream);
  const size_t smem_w = (size_t)k * k * sizeof(double);
  allow_shared_memory((const void*)plssvd_weights_kernel);
  plssvd_weights_kernel<<<k, kWeightThreads, smem_w, stream>>>(gram.get(), k, model.sigma.get(), model.Q.get(),
                                                               m, model.W.get(), ws.flag.get());
  count_launch();
  FPLS_LAUNCH("plssvd_weights");
}

template void fit_plssvd<float>(const float*, int, int, long, const double*,
                                const double*, int, int, int, DeviceModel&,
                                Workspace&, cudaStream_t);
template void fit_plssvd<double>(const double*, int, int, long, const double*,
                                 const double*, int, int, int, DeviceModel&,
                                 Workspace&, cudaStream_t);
template void fit_plssvd<bf16>(const bf16*, int, int, long, const double*,
                               const double*, int, int, int, DeviceModel&,
                               Workspace&, cudaStream_t);

}  // namespace fpls
