// Single-fit SIMPLS on the device (p-space, FP64 arithmetic, raw X).
//
// Reference algorithm: fit_simpls_preprocessed
// (inst/include/fastpls/core/simpls.hpp:479-763) and the resident CUDA
// component step (src/cuda_resident_component.cuh:94-130). Per component:
//   r = dominant left singular vector of the deflated cross-product S,
//   t = Xs r, r,t /= ||t||, p = Xs^T t, q = S0^T r,
//   v = p - V (V^T p), v /= ||v||, S -= v (v^T S).
//
// B200 design:
//  * X stays raw in HBM (FP32 or FP64). Centring and scaling are folded into
//    the two products, t = X (r / scale) - (mean . r / scale) and
//    p = (X^T t - mean * sum(t)) / scale, so X is never rewritten and each
//    component reads it exactly twice (stream.cu).
//  * The direction comes from the m x m Gram G = S^T S, recomputed from the
//    deflated S each component (no downdate drift) and diagonalised by
//    Jacobi in one block: r = S z / sqrt(lambda). The span of the
//    reference's randomized sketch equals the full response space in every
//    supported configuration, so this is the same dominant direction.
//  * Every p-length step is one kernel over 256-row blocks of S/V whose
//    cross-block sums finish in the last block to arrive (reduce.cuh):
//    deterministic, no atomics on data, no spin-waits.
#include "kernels.cuh"
#include "model.cuh"
#include "persistent.cuh"
#include "reduce.cuh"
#include "small.cuh"

#include <algorithm>
#include <memory>

namespace fpls {

namespace {

constexpr int TB = 256;
// Rows (predictors) per block of the p-vector kernels, whose TB threads share
// them: 157 blocks at p = 10000, where 256 rows a block left 108 SMs idle.
constexpr int PB = 64;
constexpr int kGemmCrossResponses = 5;

// One block per response: bound by the latency of its loads (1024 threads; 256
// took 83 us at 40003 rows, 12 classes, 29 now).
constexpr int kCenterThreads = 1024;
template <class T>
__global__ void __launch_bounds__(kCenterThreads) center_dense(const T* __restrict__ Y, int n, int m,
                             double* __restrict__ Yc, double* ymean,
                             double* ycsum, int* flag) {
  __shared__ double scratch[32];
  const int c = blockIdx.x;
  double s = 0.0;
#pragma unroll 4
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const double y = as_f64(Y[i + (long)c * n]);
    if (!isfinite(y)) flag_error(flag, 3);
    s += y;
  }
  const double mu = block_sum(s, scratch) / n;
  double r = 0.0;
#pragma unroll 4
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const double v = as_f64(Y[i + (long)c * n]) - mu;
    Yc[i + (long)c * n] = v;
    r += v;
  }
  r = block_sum(r, scratch);
  if (threadIdx.x == 0) {
    ymean[c] = mu;
    ycsum[c] = r;
  }
}

__global__ void __launch_bounds__(kCenterThreads) center_labels(const int* __restrict__ labels, int n, int m,
                              double* __restrict__ Yc, double* ymean,
                              double* ycsum, int* flag) {
  __shared__ double scratch[32];
  const int c = blockIdx.x;
  double cnt = 0.0;
#pragma unroll 4
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const int l = labels[i];
    if (l < 1 || l > m) flag_error(flag, 2);
    cnt += (l == c + 1) ? 1.0 : 0.0;
  }
  const double prior = block_sum(cnt, scratch) / n;
  double r = 0.0;
#pragma unroll 4
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const double v = (labels[i] == c + 1 ? 1.0 : 0.0) - prior;
    Yc[i + (long)c * n] = v;
    r += v;
  }
  r = block_sum(r, scratch);
  if (threadIdx.x == 0) {
    ymean[c] = prior;
    ycsum[c] = r;
  }
}

// mean / scale per column (supervised.hpp:53-90) and the scaled centred
// cross-product S = D^-1 (X^T Yc - mean * colsum(Yc)).
__global__ void finish_moments(const double* __restrict__ sum,
                               const double* __restrict__ sumsq,
                               const double* __restrict__ cross,
                               const double* __restrict__ ycsum, int n, int p,
                               int m, int scaling, double* mean, double* scale,
                               double* S, double* S0, int* flag) {
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < p;
       j += gridDim.x * blockDim.x) {
    const double mu = scaling != 3 ? sum[j] / n : 0.0;
    double sd = 1.0;
    if (scaling == 2) {
      const double cs = fmax(0.0, sumsq[j] - n * mu * mu);
      sd = sqrt(cs / (double)max(n - 1, 1));
      if (!isfinite(sd) || sd <= 0.0) sd = 1.0;
    }
    if (!isfinite(sum[j]) || !isfinite(sumsq[j])) flag_error(flag, 3);
    mean[j] = mu;
    scale[j] = sd;
    for (int c = 0; c < m; ++c) {
      const double s = (cross[j + (long)c * p] - mu * ycsum[c]) / sd;
      S[j + (long)c * p] = s;
      S0[j + (long)c * p] = s;
    }
  }
}

// Unpack the packed lower-triangular Gram, diagonalise, emit z / sqrt(lambda).
// The `count` dominant eigenpairs of the m x m right Gram (packed lower
// triangle), by decreasing eigenvalue (ties: lower index first):
// zs[k + j m] = z_j / sqrt(lambda_j), sign fixed so the largest-magnitude
// entry of z_j is positive; lambda_out = lambda_0.
// Whole block; sm: direction_smem(m) doubles.
__device__ void direction(const double* gpk, int m, double* zs, double* lambda_out, int* flag, int count,
                          double* sm) {
  double* A = sm;
  double* E = sm + m * m;
  for (int c = threadIdx.x; c < m; c += blockDim.x)
    for (int d = 0; d <= c; ++d) {
      const double v = __ldcg(gpk + c * (c + 1) / 2 + d);
      A[c + d * m] = v;
      A[d + c * m] = v;
    }
  __syncthreads();
  if (count == 1 && m <= kDominantMaxOrder) {
    // one direction: the dominant pair alone (repeated squaring)
    double* C = E + m * m;      // m^2 + 1
    double* v = C + m * m + 1;  // m + 1
    double lam = 0.0;
    const bool found = dominant_pair(A, E, C, v, m, lam);
    if (threadIdx.x == 0) {
      const bool ok = found && lam > 0.0 && isfinite(lam);
      if (!ok) flag_error(flag, 1);
      const double inv = ok ? 1.0 / sqrt(lam) : 0.0;
      int arg = 0;
      if (found)
        for (int k = 1; k < m; ++k)
          if (fabs(v[k]) > fabs(v[arg])) arg = k;
      const double sgn = found && v[arg] < 0.0 ? -1.0 : 1.0;
      for (int k = 0; k < m; ++k) zs[k] = found ? sgn * v[k] * inv : 0.0;
      if (lambda_out) *lambda_out = found ? lam : 0.0;
    }
    return;
  }
  jacobi_eigen(A, E, m);
  __syncthreads();
  if (threadIdx.x == 0) {
    double inv0 = 0.0;
    for (int j = 0; j < count; ++j) {
      int best = -1;
      for (int k = 0; k < m; ++k)
        if (best < 0 || A[k + k * m] > A[best + best * m]) best = k;
      const double lam = A[best + best * m];
      A[best + best * m] = -INFINITY;  // taken (A is scratch after the solve)
      const bool ok = lam > 0.0 && isfinite(lam);
      // The leading pair must exist (S not zero). A later candidate of a
      // block wider than the rank of S (a block of q classes, rank q - 1)
      // has a numerically zero eigenvalue: it takes the leading pair's scale
      // (R and T do not depend on the scale of r), as the reference's sketch
      // yields some unit direction there instead of failing.
      if (!ok && j == 0) flag_error(flag, 1);
      const double inv = ok ? 1.0 / sqrt(lam) : inv0;
      if (j == 0) inv0 = inv;
      // deterministic sign: largest-magnitude entry of z positive
      int arg = 0;
      for (int k = 1; k < m; ++k)
        if (fabs(E[k + best * m]) > fabs(E[arg + best * m])) arg = k;
      const double sgn = E[arg + best * m] < 0.0 ? -1.0 : 1.0;
      for (int k = 0; k < m; ++k) zs[k + j * m] = sgn * E[k + best * m] * inv;
      if (lambda_out && j == 0) *lambda_out = lam;
    }
  }
}

// A, B, C, v of the dominant pair (one direction), or A, E of the Jacobi sweeps
__host__ __device__ inline size_t direction_smem(int m) {
  return m <= kDominantMaxOrder ? 3 * (size_t)m * m + m + 2 : 2 * (size_t)m * m;
}

__global__ void direction_kernel(const double* __restrict__ gpk, int m,
                                 double* zs, double* lambda_out, int* flag, int count) {
  extern __shared__ double sm[];
  direction(gpk, m, zs, lambda_out, flag, count, sm);
}

// r = S zs ; rt = r / scale ; scal[0] = mean . rt
__global__ void rvec_kernel(const double* __restrict__ S, int p, int m,
                            const double* __restrict__ zs,
                            const double* __restrict__ mean,
                            const double* __restrict__ scale, double* r,
                            double* rt, double* partial, unsigned* counter,
                            double* scal) {
  __shared__ double scratch[32];
  __shared__ double vals[1];
  double acc = 0.0;
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j < p) {
    double v = 0.0;
    for (int c = 0; c < m; ++c) v = fma(S[j + (long)c * p], zs[c], v);
    const double w = v / scale[j];
    r[j] = v;
    rt[j] = w;
    acc = mean[j] * w;
  }
  const double s = block_sum(acc, scratch);
  if (threadIdx.x == 0) vals[0] = s;
  __syncthreads();
  last_block_reduce(vals, 1, partial, counter, scal);
}

// Dot products over the block's rows: out[k] = sum_{j in block} col_k[j] w[j]
// (w in shared memory), a warp per column, four columns of a warp at once so
// that their loads overlap.
__device__ inline void block_dots(const double* __restrict__ M, long ldm,
                                  int j0, int rows, const double* w, int count,
                                  double* out) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int W = TB / 32, U = 4;
  for (int kb = warp; kb < count; kb += U * W) {
    double acc[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      acc[u] = 0.0;
      const int k = kb + u * W;
      if (k < count)
#pragma unroll
        for (int j = 0; j < PB; j += 32)
          if (j + lane < rows) acc[u] = fma(M[j0 + j + lane + (long)k * ldm], w[j + lane], acc[u]);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const double s = warp_sum(acc[u]);
      if (lane == 0 && kb + u * W < count) out[kb + u * W] = s;
    }
  }
}

// p = (praw - mean * sum t) / (scale * ||t||) ; R[:,a] = r / ||t||
// out (last block): h = V^T p (a_cur), q = S0^T R[:,a] (m), also Q[:,a]
// When `loading` is given (cached-Gram route) p = loading / ||t|| directly.
// Latency-bound (p (a + m) doubles read once): 31 us at p = 10000, a + m = 35
// with 256-row blocks and serial partial sums, 16 us now.
__global__ void __launch_bounds__(TB)
    tail1_kernel(const double* __restrict__ praw,
                             const double* __restrict__ mean,
                             const double* __restrict__ scale,
                             const double* __restrict__ scal,
                             const double* __restrict__ r,
                             const double* __restrict__ S0,
                             const double* __restrict__ V, int p, int m,
                             int a_cur, double* pvec, double* Rcol,
                             double* partial, unsigned* counter, double* hq,
                             int* flag, double* Qcol, double* tnorm2,
                             const double* __restrict__ loading = nullptr) {
  extern __shared__ double sm[];
  double* ps = sm;            // PB
  double* rs = sm + PB;       // PB
  double* vals = sm + 2 * PB; // a_cur + m
  const int j0 = blockIdx.x * PB;
  const int rows = min(PB, p - j0);
  const double tn = sqrt(scal[1]);
  if (!(tn > 0.0) || !isfinite(tn)) {
    if (blockIdx.x == 0 && threadIdx.x == 0) flag_error(flag, 1);
  }
  const double inv = (tn > 0.0 && isfinite(tn)) ? 1.0 / tn : 0.0;
  const int t = threadIdx.x;
  if (t < rows) {
    const int j = j0 + t;
    const double pj = loading ? loading[j] * inv : (praw[j] - mean[j] * scal[2]) / scale[j] * inv;
    const double rj = r[j] * inv;
    pvec[j] = pj;
    Rcol[j] = rj;
    ps[t] = pj;
    rs[t] = rj;
  }
  __syncthreads();
  block_dots(V, p, j0, rows, ps, a_cur, vals);
  block_dots(S0, p, j0, rows, rs, m, vals + a_cur);
  __syncthreads();
  if (!last_block_reduce(vals, a_cur + m, partial, counter, hq)) return;
  // Q[:, a] and ||t||^2 (for the scaling of T after the last component)
  __syncthreads();
  for (int c = t; c < m; c += TB) Qcol[c] = hq[a_cur + c];
  if (t == 0) *tnorm2 = scal[1];
}

// v = p - V h ; out (last block): [v.v, S^T v (m)]. A row's sum over the
// components is shared by TB / PB threads. 24 us at p = 10000, a = 25 before,
// 12 us now.
__global__ void __launch_bounds__(TB)
    tail2_kernel(const double* __restrict__ pvec,
                             const double* __restrict__ V,
                             const double* __restrict__ hq,
                             const double* __restrict__ S, int p, int m,
                             int a_cur, double* v, double* partial,
                             unsigned* counter, double* vr) {
  extern __shared__ double sm[];
  double* vs = sm;             // PB
  double* vals = sm + PB;      // 1 + m
  __shared__ double scratch[32];
  __shared__ double part[TB];
  constexpr int G = TB / PB;
  const int j0 = blockIdx.x * PB;
  const int rows = min(PB, p - j0);
  const int t = threadIdx.x, row = t % PB, g = t / PB;
  double q = 0.0;
  if (row < rows) {
#pragma unroll 8
    for (int k = g; k < a_cur; k += G) q = fma(V[j0 + row + (long)k * p], hq[k], q);
  }
  part[t] = q;
  __syncthreads();
  double vj = 0.0;
  if (t < rows) {
    for (int u = 1; u < G; ++u) q += part[t + u * PB];
    vj = pvec[j0 + t] - q;
    v[j0 + t] = vj;
    vs[t] = vj;
  }
  __syncthreads();
  const double vv = block_sum(vj * vj, scratch);
  block_dots(S, p, j0, rows, vs, m, vals + 1);
  if (threadIdx.x == 0) vals[0] = vv;
  __syncthreads();
  last_block_reduce(vals, 1 + m, partial, counter, vr);
}

// V[:,a] = v / ||v|| ; S -= V[:,a] (row / ||v||) ; G partials of updated S
// (packed lower triangle) reduced by the last block into gpk.
// When `update` is false only the Gram of S is formed. With zs the last block
// goes on to the next direction (direction()), which was a launch of its own
// (15 us at 10 responses).
__global__ void __launch_bounds__(TB)
    tail3_kernel(const double* __restrict__ v,
                             const double* __restrict__ vr, double* S, int p,
                             int m, double* Vcol, bool update, double* partial,
                             unsigned* counter, double* gpk, int* flag, double* zs,
                             double* lambda_out) {
  extern __shared__ double sm[];
  double* ss = sm;                 // PB x m
  double* vals = sm + PB * m;      // m(m+1)/2
  const int j0 = blockIdx.x * PB;
  const int rows = min(PB, p - j0);
  const int t = threadIdx.x;
  double vn = 1.0;
  if (update) {
    vn = sqrt(vr[0]);
    if (!(vn > 0.0) || !isfinite(vn)) {
      if (blockIdx.x == 0 && t == 0) flag_error(flag, 1);
      vn = 0.0;
    }
  }
  const double inv = vn > 0.0 ? 1.0 / vn : 0.0;
  const int row = t % PB;
  if (row < rows) {
    const int j = j0 + row;
    const double vj = update ? v[j] * inv : 0.0;
    if (update && t < PB) Vcol[j] = vj;
#pragma unroll 4
    for (int c = t / PB; c < m; c += TB / PB) {
      double s = S[j + (long)c * p];
      if (update) {
        s = fma(-vj, vr[1 + c] * inv, s);
        S[j + (long)c * p] = s;
      }
      ss[row + c * PB] = s;
    }
  }
  __syncthreads();
  const int pairs = m * (m + 1) / 2;
  const int lane = t & 31, warp = t >> 5;
  for (int k = warp; k < pairs; k += TB / 32) {
    // k -> (c, d) with d <= c, k = c(c+1)/2 + d
    int c = (int)((sqrtf(8.0f * k + 1.0f) - 1.0f) * 0.5f);
    while (c * (c + 1) / 2 > k) --c;
    while ((c + 1) * (c + 2) / 2 <= k) ++c;
    const int d = k - c * (c + 1) / 2;
    double acc = 0.0;
#pragma unroll
    for (int j = 0; j < PB; j += 32)
      if (j + lane < rows) acc = fma(ss[j + lane + c * PB], ss[j + lane + d * PB], acc);
    acc = warp_sum(acc);
    if (lane == 0) vals[k] = acc;
  }
  __syncthreads();
  if (!last_block_reduce(vals, pairs, partial, counter, gpk) || !zs) return;
  __syncthreads();
  direction(gpk, m, zs, lambda_out, flag, 1, sm);
}

// T[:, a] /= ||t_a|| for every component, one pass after the last.
__global__ void scale_scores(double* T, int n, const double* __restrict__ tnorm2) {
  const double tn = sqrt(tnorm2[blockIdx.y]);
  const double inv = (tn > 0.0 && isfinite(tn)) ? 1.0 / tn : 0.0;
  double* col = T + (long)blockIdx.y * n;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) col[i] *= inv;
}

// Gs[j, k] = (G[j, k] - n mean_j mean_k) / (scale_j scale_k): the Gram of
// the standardised predictors from the raw X^T X.
__global__ void standardize_gram(double* G, int p, int n, const double* __restrict__ mean,
                                 const double* __restrict__ scale) {
  const long total = (long)p * p;
  for (long idx = blockIdx.x * (long)blockDim.x + threadIdx.x; idx < total;
       idx += (long)gridDim.x * blockDim.x) {
    const int j = (int)(idx % p), k = (int)(idx / p);
    G[idx] = (G[idx] - (double)n * mean[j] * mean[k]) / (scale[j] * scale[k]);
  }
}

// scal[1] = r . loading (= ||X_s r||^2), scal[2] = 0 (sum t unused on this route)
__global__ void gram_tstats(const double* __restrict__ r, const double* __restrict__ loading,
                            int p, double* partial, unsigned* counter, double* scal) {
  __shared__ double scratch[32];
  __shared__ double vals[2];
  double a = 0.0;
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < p; j += gridDim.x * blockDim.x)
    a = fma(r[j], loading[j], a);
  a = block_sum(a, scratch);
  if (threadIdx.x == 0) {
    vals[0] = a;
    vals[1] = 0.0;
  }
  __syncthreads();
  last_block_reduce(vals, 2, partial, counter, scal + 1);
}

void configure_small_kernels() {
  allow_shared_memory((const void*)tail3_kernel);
  allow_shared_memory((const void*)direction_kernel);
}

}  // namespace

void Workspace::ensure(int n, int p, int m, int a, cudaStream_t s) {
  const size_t blocks_p = ceil_div(std::max(p, 1), 64) + 8;
  const size_t width = std::max<size_t>(a + m + 2, (size_t)m * (m + 1) / 2 + 2);
  block_partial.reserve(blocks_p * width + 4096, s);
  if (!counters) {
    counters.allocate(64, s);
    counters.zero(s);
  }
  for (auto& v : vec_p) v.reserve(std::max(p, 1), s);
  for (auto& v : vec_n) v.reserve(std::max(n, 1), s);
  small.reserve(64 + 2 * (size_t)kMaxResponses * kMaxResponses + 4 * (size_t)std::max(a, 1) + m, s);
  if (!flag) {
    flag.allocate(1, s);
  }
}

void raise_on_flag(Workspace& ws, cudaStream_t stream, const char* message) {
  int bad = 0;
  FPLS_CHECK(cudaMemcpyAsync(&bad, ws.flag.get(), sizeof(int),
                             cudaMemcpyDeviceToHost, stream));
  FPLS_CHECK(cudaStreamSynchronize(stream));
  if (bad) throw std::runtime_error(message);
}

template <class T>
void prepare_responses(const T* Y, const int* labels, int n, int m, double* Yc,
                       double* ymean, double* ycsum, int* flag,
                       cudaStream_t stream) {
  const int threads = std::min(kCenterThreads, std::max(64, (n + 31) / 32 * 32));
  if (labels) center_labels<<<m, threads, 0, stream>>>(labels, n, m, Yc, ymean, ycsum, flag);
  else center_dense<T><<<m, threads, 0, stream>>>(Y, n, m, Yc, ymean, ycsum, flag);
  count_launch();
  FPLS_LAUNCH("prepare_responses");
}

__global__ void s_times_z(const double* __restrict__ S, int p, int m,
                          const double* __restrict__ zs, double* w) {
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < p; j += gridDim.x * blockDim.x) {
    double v = 0.0;
    for (int c = 0; c < m; ++c) v = fma(S[j + (long)c * p], zs[c], v);
    w[j] = v;
  }
}

void dominant_direction(const double* S, int p, int m, const double* gpk,
                        double* zs, double* w, Workspace& ws, cudaStream_t s) {
  const size_t smem_dir = direction_smem(m) * sizeof(double);
  configure_small_kernels();
  direction_kernel<<<1, jacobi_threads(m), smem_dir, s>>>(gpk, m, zs, nullptr, ws.flag.get(), 1);
  s_times_z<<<std::min<unsigned>(ceil_div(p, TB), 4 * num_sms()), TB, 0, s>>>(S, p, m, zs, w);
  count_launch(2);
  FPLS_LAUNCH("dominant_direction");
}

template <class T>
void compute_crossprod(const T* X, int n, int p, long ld, const double* Yc,
                       const double* ycsum, int m, int scaling,
                       DeviceModel& model, double* S, Workspace& ws,
                       cudaStream_t stream) {
  model.mean.allocate(p, stream);
  model.scale.allocate(p, stream);
  model.S0.allocate((size_t)p * m, stream);
  DeviceArray<double> moments((size_t)p * (2 + m), stream);
  double* sum = moments.get();
  double* sumsq = sum + p;
  double* cross = sumsq + p;
  if (model.label_view && m <= kClassMomentsMaxClasses)
    class_moments<T>(X, n, p, ld, model.label_view, m, model.ymean.get(), sum, sumsq, cross,
                     ws.stream_partial, stream);
  else if (m >= kGemmCrossResponses && (long)n * p >= (1L << 22)) {
    // several responses: the moments alone (one pass) and X^T Yc as a DMMA
    // product (a second one). With the responses in the moments pass the sums
    // and warp reductions of m columns bound it: 30011 x 10000 BF16, 10
    // responses 1.35 ms, 0.50 ms in two passes; 4513 x 10000 FP32, 3 responses 0.11
    // ms in one.
    column_moments<T>(X, n, p, ld, nullptr, 0, sum, sumsq, nullptr, ws.stream_partial, stream);
    GemmArgs g;
    g.M = p;
    g.N = m;
    g.K = n;
    g.A = X;
    g.lda = ld;
    g.a_type = gemm_type<T>::value;
    g.trans_a = true;
    g.B = Yc;
    g.ldb = n;
    g.C = cross;
    g.ldc = p;
    gemm_f64(g, stream);
  } else
    column_moments<T>(X, n, p, ld, Yc, m, sum, sumsq, cross, ws.stream_partial, stream);
  const unsigned gp = std::min<unsigned>(ceil_div(p, TB), 8 * num_sms());
  finish_moments<<<gp, TB, 0, stream>>>(sum, sumsq, cross, ycsum, n, p, m,
                                        scaling, model.mean.get(),
                                        model.scale.get(), S,
                                        model.S0.get(), ws.flag.get());
  count_launch();
  FPLS_LAUNCH("finish_moments");
}

void gram_of_columns(double* S, int p, int m, double* gpk, Workspace& ws,
                     cudaStream_t stream) {
  const unsigned g3 = ceil_div(p, PB);
  const size_t smem3 = ((size_t)PB * m + (size_t)m * (m + 1) / 2) * sizeof(double);
  configure_small_kernels();
  tail3_kernel<<<g3, TB, smem3, stream>>>(nullptr, nullptr, S, p, m, nullptr,
                                           false, ws.block_partial.get(),
                                           ws.counters.get() + 5, gpk,
                                           ws.flag.get(), nullptr, nullptr);
  count_launch();
  FPLS_LAUNCH("gram_of_columns");
}

template <class T>
void fit_simpls(const T* X, int n, int p, long ld, const double* Yc,
                const double* ycsum, int m, int components, int scaling,
                DeviceModel& model, Workspace& ws, cudaStream_t stream, int block,
                bool gram_route) {
  require(m >= 1 && m <= kMaxResponses, "SIMPLS supports 1..112 responses or classes");
  const int a_max = components;
  ws.ensure(n, p, m, a_max, stream);
  model.method = kSimpls;
  model.n = n;
  model.p = p;
  model.feature_p = p;
  model.m = m;
  model.scaling = scaling;
  model.R.allocate((size_t)p * a_max, stream);
  model.Q.allocate((size_t)m * a_max, stream);
  model.V.allocate((size_t)p * a_max, stream);
  model.T.allocate((size_t)n * a_max, stream);
  DeviceArray<double> S((size_t)p * m, stream);
  compute_crossprod<T>(X, n, p, ld, Yc, ycsum, m, scaling, model, S.get(), ws, stream);

  double* sm = ws.small.get();
  double* scal = sm;            // [c, sum t^2, sum t, lambda]
  double* zs = sm + 8;          // m
  double* gpk = zs + kMaxResponses;                // m(m+1)/2
  double* hq = gpk + kMaxResponses * kMaxResponses; // a + m
  double* vr = hq + a_max + m + 4;                  // 1 + m
  double* r = ws.vec_p[0].get();
  double* rt = ws.vec_p[1].get();
  double* pvec = ws.vec_p[2].get();
  double* v = ws.vec_p[3].get();
  double* praw = ws.vec_p[4].get();
  unsigned* ctr = ws.counters.get();
  double* part = ws.block_partial.get();

  const unsigned g3 = ceil_div(p, PB);
  const unsigned g1 = ceil_div(p, TB);
  const size_t smem_dir = direction_smem(m) * sizeof(double);
  configure_small_kernels();

  // cached-Gram route (FP32 / FP64 storage): Gs = X_s^T X_s once
  gram_route = gram_route && !std::is_same<T, bf16>::value;
  DeviceArray<double> Gs, loading;
  if (gram_route) {
    Gs.allocate((size_t)p * p, stream);
    loading.allocate(p, stream);
    GemmArgs g;
    g.M = p;
    g.N = p;
    g.K = n;
    g.A = X;
    g.lda = ld;
    g.trans_a = true;
    g.B = X;
    g.ldb = ld;
    g.a_type = g.b_type = gemm_type<T>::value;
    g.lower = true;
    g.C = Gs.get();
    g.ldc = p;
    gemm_f64(g, stream);
    const long total = (long)p * p;
    standardize_gram<<<(unsigned)std::min<long>((total + 255) / 256, 8L * num_sms()), 256, 0, stream>>>(
        Gs.get(), p, n, model.mean.get(), model.scale.get());
    count_launch();
    FPLS_LAUNCH("standardize_gram");
  }

  // one direction per component: the whole loop as one persistent launch
  // (or handed to the caller's batch when it collects plans)
  if (block <= 1 && !gram_route) {
    std::unique_ptr<PersistentPlan> plan(new PersistentPlan());
    const PersistentDeferral& defer = persistent_deferral();
    if (plan_simpls_persistent<T>(X, n, p, ld, m, a_max, model, S, gpk, ws, stream, *plan, defer.max_ctas)) {
      if (defer.sink) {
        *defer.sink = std::move(plan);
      } else {
        launch_persistent({plan.get()}, stream);
      }
      return;
    }
  }
  gram_of_columns(S.get(), p, m, gpk, ws, stream);

  // Candidate blocks (the reference's block refresh): the directions of
  // `use` consecutive components are the leading left singular vectors of S
  // at the start of the block, r_j = S_block z_j / sqrt(lambda_j), not
  // recomputed from the deflated S in between.
  block = std::max(1, std::min(block, std::min(a_max, std::min(p, m))));
  DeviceArray<double> zblk, Sblk;
  if (block > 1) {
    zblk.allocate((size_t)m * block, stream);
    Sblk.allocate((size_t)p * m, stream);
  }
  int use = 0, jb = 0;
  // with one direction a block (and where both fit its last block's shared
  // memory) the deflation of a component yields the next direction
  const bool chained = block == 1 && m <= kDominantMaxOrder;
  const size_t smem3 = std::max((size_t)PB * m + (size_t)m * (m + 1) / 2, chained ? direction_smem(m) : 0) *
                       sizeof(double);
  DeviceArray<double> tnorm2(a_max, stream);
  for (int a = 0; a < a_max; ++a) {
    if (jb == use) {
      use = std::min(block, a_max - a);
      jb = 0;
    }
    if (jb == 0 && !(chained && a > 0)) {
      direction_kernel<<<1, jacobi_threads(m), smem_dir, stream>>>(gpk, m, use > 1 ? zblk.get() : zs, scal + 3,
                                                    ws.flag.get(), use);
      count_launch();
      FPLS_LAUNCH("direction_kernel");
      if (use > 1)
        FPLS_CHECK(cudaMemcpyAsync(Sblk.get(), S.get(), sizeof(double) * p * m,
                                   cudaMemcpyDeviceToDevice, stream));
    }
    rvec_kernel<<<g1, TB, 0, stream>>>(use > 1 ? Sblk.get() : S.get(), p, m,
                                       use > 1 ? zblk.get() + (size_t)jb * m : zs,
                                       model.mean.get(), model.scale.get(), r, rt, part,
                                       ctr + 0, scal);
    ++jb;
    count_launch();
    FPLS_LAUNCH("rvec_kernel");
    double* tcol = model.T.get() + (size_t)a * n;
    if (gram_route) {
      // loading = Gs r (Gs symmetric: its columns dot r), ||t||^2 = r . loading
      xtv_product<double>(Gs.get(), p, p, p, r, p, 1, loading.get(), p, ws.stream_partial, stream);
      gram_tstats<<<std::min<unsigned>(ceil_div(p, TB), 2 * num_sms()), TB, 0, stream>>>(
          r, loading.get(), p, part, ctr + 1, scal);
      count_launch();
      FPLS_LAUNCH("gram_tstats");
    } else {
      const XrStats stats{part, ctr + 1, scal + 1};  // sum t^2, sum t
      xr_product<T>(X, n, p, ld, rt, p, 1, scal, 1, tcol, n, ws.stream_partial, stream, &stats, true);
      xtv_product<T>(X, n, p, ld, tcol, n, 1, praw, p, ws.stream_partial, stream, true);
    }
    tail1_kernel<<<g3, TB, (2 * PB + a + m) * sizeof(double), stream>>>(
        praw, model.mean.get(), model.scale.get(), scal, r, model.S0.get(),
        model.V.get(), p, m, a, pvec, model.R.get() + (size_t)a * p, part,
        ctr + 2, hq, ws.flag.get(), model.Q.get() + (size_t)a * m, tnorm2.get() + a,
        gram_route ? loading.get() : nullptr);
    tail2_kernel<<<g3, TB, (PB + 1 + m) * sizeof(double), stream>>>(
        pvec, model.V.get(), hq, S.get(), p, m, a, v, part, ctr + 3, vr);
    tail3_kernel<<<g3, TB, smem3, stream>>>(v, vr, S.get(), p, m,
                                             model.V.get() + (size_t)a * p,
                                             true, part, ctr + 4, gpk, ws.flag.get(),
                                             chained && a + 1 < a_max ? zs : nullptr, scal + 3);
    count_launch(3);
    FPLS_LAUNCH("simpls component");
  }
  model.a = a_max;
  if (gram_route) {
    // training scores T = X_s R (normalised: R holds r / ||t||), one pass
    project_rows<T>(model, X, n, ld, a_max, model.T.get(), n, ws, stream);
  } else {
    scale_scores<<<dim3(std::min<unsigned>(ceil_div(n, TB), 4 * num_sms()), a_max), TB, 0, stream>>>(
        model.T.get(), n, tnorm2.get());
    count_launch();
    FPLS_LAUNCH("scale_scores");
  }
}

template void prepare_responses<float>(const float*, const int*, int, int, double*,
                                       double*, double*, int*, cudaStream_t);
template void prepare_responses<double>(const double*, const int*, int, int, double*,
                                        double*, double*, int*, cudaStream_t);
#define FPLS_INSTANTIATE(T)                                                    \
  template void fit_simpls<T>(const T*, int, int, long, const double*,        \
                              const double*, int, int, int, DeviceModel&,     \
                              Workspace&, cudaStream_t, int, bool);           \
  template void compute_crossprod<T>(const T*, int, int, long, const double*, \
                                     const double*, int, int, DeviceModel&,   \
                                     double*, Workspace&, cudaStream_t);
FPLS_INSTANTIATE(float)
FPLS_INSTANTIATE(double)
FPLS_INSTANTIATE(bf16)
#undef FPLS_INSTANTIATE

}  // namespace fpls
