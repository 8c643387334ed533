// HBM-streaming kernels over the resident predictor matrix X (n x p,
// column-major, BF16, FP32 or FP64 storage, FP64 arithmetic).
//
// These are the GEMV-shaped steps of a single fit: the column moments
// (centre, scale, X^T Yc) in one pass, t = X r (scores) and p = X^T t
// (loadings). Each reads X exactly once per call with coalesced, unrolled
// loads (many independent loads in flight per warp) and reduces in a fixed
// order through per-chunk partials, so results are deterministic.
// Algorithmic bytes per call: n * p * sizeof(T) (+ O((n + p) * nb * 8)).
#include "common.cuh"
#include "kernels.cuh"
#include "reduce.cuh"

#include <algorithm>
#include <type_traits>

namespace fpls {

namespace {

constexpr int kThreads = 256;

// Two consecutive rows of one column in one load (bf16x2, float2, double2):
// 4-16 bytes per lane, 128-512 bytes per warp request. Used when the column
// stride is even and X is aligned to the pair size.
template <class T> struct Pair;
template <> struct Pair<float> {
  using type = float2;
  static __device__ __forceinline__ double lo(type v) { return v.x; }
  static __device__ __forceinline__ double hi(type v) { return v.y; }
  static __device__ __forceinline__ void finite(type v, double& lo, double& hi) {
    lo = finite_f64<float>::widen(v.x);
    hi = finite_f64<float>::widen(v.y);
  }
};
template <> struct Pair<double> {
  using type = double2;
  static __device__ __forceinline__ double lo(type v) { return v.x; }
  static __device__ __forceinline__ double hi(type v) { return v.y; }
  static __device__ __forceinline__ void finite(type v, double& lo, double& hi) {
    lo = v.x;
    hi = v.y;
  }
};
template <> struct Pair<bf16> {
  using type = __nv_bfloat162;
  static __device__ __forceinline__ double lo(type v) { return __low2float(v); }
  static __device__ __forceinline__ double hi(type v) { return __high2float(v); }
  static __device__ __forceinline__ void finite(type v, double& lo, double& hi) {
    finite_f64<bf16>::widen2(*reinterpret_cast<const unsigned*>(&v), lo, hi);
  }
};

template <class T>
bool pair_aligned(const T* X, long ld) {
  return ld % 2 == 0 && reinterpret_cast<uintptr_t>(X) % (2 * sizeof(T)) == 0;
}

// ---------------------------------------------------------------------------
// X^T V (and optionally column sums / sums of squares) -- CW columns per warp.
// Block = 8 warps over a tile of 32 columns and a chunk of `rc` rows whose
// V rows are staged in shared memory; each staged value is used for the CW
// columns a warp holds at once, whose loads are in flight together. partial
// layout: [chunk][j][slot] with slots = nb (+2 when MOMENTS: sum, sumsq at
// slots nb, nb+1). HBM-bound at one column of V; the once-per-fit moments with
// several responses are bound by the shared-memory reads of V (one column per
// warp: 180 MB of FP32 with 3 responses 107 us, 600 MB of BF16 with 10 1350 us;
// with a wider form, X^T Yc leaves for a DMMA product, fit.cu).
// ---------------------------------------------------------------------------
template <int MB>
constexpr int columns_per_warp() {
  return MB > 1 && MB <= 4 ? 4 : 1;
}

// PAIR: lane l takes rows 2 (l + 32 u) and 2 (l + 32 u) + 1 of the chunk in one
// load (rc and the column stride even), else rows l + 32 u.
// FINITE: the rows are known to be finite (finite_f64).
template <class T, int MB, bool MOMENTS, bool PAIR, bool FINITE>
__global__ void __launch_bounds__(kThreads)
    xtv_kernel(const T* __restrict__ X, int n, int p, long ld,
               const double* __restrict__ V, long ldv, int nb, int rc,
               double* __restrict__ partial) {
  constexpr int CW = columns_per_warp<MB>();
  constexpr int ROWS = PAIR ? 2 : 1;
  using P = Pair<T>;
  using L = typename std::conditional<PAIR, typename P::type, T>::type;
  extern __shared__ double vs[];  // rc x nb
  const int chunk = blockIdx.y;
  const int r0 = chunk * rc;
  const int rows = min(rc, n - r0);
  for (int idx = threadIdx.x; idx < rows * nb; idx += blockDim.x) {
    const int r = idx % rows, c = idx / rows;
    vs[r + c * rc] = V[(r0 + r) + (long)c * ldv] * (FINITE ? finite_f64<T>::weight : 1.0);
  }
  __syncthreads();
  const int slots = nb + (MOMENTS ? 2 : 0);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int steps = rows / ROWS;  // loads per column
  for (int jj = warp * CW; jj < 32; jj += kThreads / 32 * CW) {
    const int j0 = blockIdx.x * 32 + jj;
    if (j0 >= p) break;
    const int cw = min(CW, p - j0);
    const L* col[CW];
#pragma unroll
    for (int w = 0; w < CW; ++w)  // past the last column: the last one again, not stored
      col[w] = reinterpret_cast<const L*>(X + (long)(j0 + min(w, cw - 1)) * ld + r0);
    double acc[CW][MB > 0 ? MB : 1], s[CW], ss[CW];
#pragma unroll
    for (int w = 0; w < CW; ++w) {
      s[w] = ss[w] = 0.0;
#pragma unroll
      for (int c = 0; c < (MB > 0 ? MB : 1); ++c) acc[w][c] = 0.0;
    }
    auto add = [&](const L (&x)[CW], int q) {
      double lo[CW], hi[CW];
#pragma unroll
      for (int w = 0; w < CW; ++w) {
        if constexpr (PAIR && FINITE) {
          P::finite(x[w], lo[w], hi[w]);
        } else if constexpr (PAIR) {
          lo[w] = P::lo(x[w]);
          hi[w] = P::hi(x[w]);
        } else {
          lo[w] = FINITE ? finite_f64<T>::widen(x[w]) : as_f64(x[w]);
          hi[w] = 0.0;
        }
        if (MOMENTS) {
          s[w] += lo[w];
          ss[w] = fma(lo[w], lo[w], ss[w]);
          if (PAIR) {
            s[w] += hi[w];
            ss[w] = fma(hi[w], hi[w], ss[w]);
          }
        }
      }
#pragma unroll
      for (int c = 0; c < MB; ++c)
        if (c < nb) {
          if constexpr (PAIR) {
            const double2 v = *reinterpret_cast<const double2*>(vs + 2 * q + c * rc);
#pragma unroll
            for (int w = 0; w < CW; ++w) {
              acc[w][c] = fma(lo[w], v.x, acc[w][c]);
              acc[w][c] = fma(hi[w], v.y, acc[w][c]);
            }
          } else {
            const double v = vs[q + c * rc];
#pragma unroll
            for (int w = 0; w < CW; ++w) acc[w][c] = fma(lo[w], v, acc[w][c]);
          }
        }
    };
    int q = lane;
    for (; q + 96 < steps; q += 128) {
      L x[4][CW];
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int w = 0; w < CW; ++w) x[u][w] = col[w][q + 32 * u];
#pragma unroll
      for (int u = 0; u < 4; ++u) add(x[u], q + 32 * u);
    }
    for (; q < steps; q += 32) {
      L x[CW];
#pragma unroll
      for (int w = 0; w < CW; ++w) x[w] = col[w][q];
      add(x, q);
    }
    if (PAIR && (rows & 1) && lane == 0) {  // odd last row of the final chunk
      const int r = rows - 1;
#pragma unroll
      for (int w = 0; w < CW; ++w) {
        const T x = reinterpret_cast<const T*>(col[w])[r];
        const double a = FINITE ? finite_f64<T>::widen(x) : as_f64(x);
        if (MOMENTS) {
          s[w] += a;
          ss[w] = fma(a, a, ss[w]);
        }
#pragma unroll
        for (int c = 0; c < MB; ++c)
          if (c < nb) acc[w][c] = fma(a, vs[r + c * rc], acc[w][c]);
      }
    }
#pragma unroll
    for (int w = 0; w < CW; ++w) {
      double* out = partial + ((long)chunk * p + j0 + w) * slots;
      const bool mine = lane == 0 && w < cw;
#pragma unroll
      for (int c = 0; c < MB; ++c) {
        if (c < nb) {
          const double v = warp_sum(acc[w][c]);
          if (mine) out[c] = FINITE ? v * finite_f64<T>::result : v;
        }
      }
      if (MOMENTS) {
        const double a = warp_sum(s[w]), b = warp_sum(ss[w]);
        if (mine) {
          out[nb] = a;
          out[nb + 1] = b;
        }
      }
    }
  }
}

// Sum the per-chunk partials: out_c[j] (+ c*ldo) for each slot c < nb, and
// the moment slots into sum/sumsq.
__global__ void xtv_finish(const double* __restrict__ partial, int chunks,
                           int p, int nb, int slots, double* out, long ldo,
                           double* sum, double* sumsq) {
  const long total = (long)p * slots;
  for (long idx = blockIdx.x * (long)blockDim.x + threadIdx.x; idx < total;
       idx += (long)gridDim.x * blockDim.x) {
    const int j = (int)(idx / slots), c = (int)(idx % slots);
    double v = 0.0;
    int k = 0;
    for (; k + 7 < chunks; k += 8) {
      double x[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) x[u] = partial[(long)(k + u) * total + idx];
#pragma unroll
      for (int u = 0; u < 8; ++u) v += x[u];
    }
    for (; k < chunks; ++k) v += partial[(long)k * total + idx];
    if (c < nb) out[j + (long)c * ldo] = v;
    else if (c == nb) sum[j] = v;
    else sumsq[j] = v;
  }
}

constexpr int kXtvMaxColumns = 32;
// V rows of a chunk, before the chunk is rounded up to 128 rows (up to 76.8 KB then)
constexpr int kXtvStagedBytes = 64 * 1024;

template <class T, int MB, bool MOMENTS, bool FINITE>
void xtv_launch(const T* X, int n, int p, long ld, const double* V, long ldv,
                int nb, double* out, long ldo, double* sum, double* sumsq,
                DeviceArray<double>& scratch, cudaStream_t stream) {
  // rows per chunk: keep the staged V block near 64 KB and give the grid
  // enough blocks to cover every SM several times.
  int rc = 2048;
  if (nb > 0) rc = std::min(rc, std::max(128, kXtvStagedBytes / (int)sizeof(double) / nb / 64 * 64));
  const int col_tiles = (int)ceil_div(p, 32);
  int chunks = (int)ceil_div(n, rc);
  const int want = 6 * num_sms();
  if (col_tiles * chunks < want && n > 256) {
    const int target = std::min((int)ceil_div(n, 256), (int)ceil_div(want, col_tiles));
    if (target > chunks) {
      rc = std::max(256, (int)ceil_div(n, target));
      rc = (rc + 127) / 128 * 128;
      chunks = (int)ceil_div(n, rc);
    }
  }
  const int slots = nb + (MOMENTS ? 2 : 0);
  scratch.reserve((size_t)chunks * p * slots, stream);
  const size_t smem = (size_t)rc * std::max(nb, 1) * sizeof(double);
  require(nb <= kXtvMaxColumns, "X^T V takes up to 32 columns");
  auto run = [&](auto kernel) {
    allow_shared_memory((const void*)kernel);
    kernel<<<dim3(col_tiles, chunks), kThreads, smem, stream>>>(X, n, p, ld, V, ldv, nb, rc, scratch.get());
  };
  if (pair_aligned(X, ld)) run(xtv_kernel<T, MB, MOMENTS, true, FINITE>);
  else run(xtv_kernel<T, MB, MOMENTS, false, FINITE>);
  count_launch();
  FPLS_LAUNCH("xtv_kernel");
  const long total = (long)p * slots;
  const unsigned blocks = (unsigned)std::min<long>((total + 255) / 256, 8L * num_sms());
  xtv_finish<<<blocks, 256, 0, stream>>>(scratch.get(), chunks, p, nb, slots,
                                         out, ldo, sum, sumsq);
  count_launch();
  FPLS_LAUNCH("xtv_finish");
}

template <class T, bool MOMENTS, bool FINITE = false>
void xtv_dispatch(const T* X, int n, int p, long ld, const double* V, long ldv,
                  int nb, double* out, long ldo, double* sum, double* sumsq,
                  DeviceArray<double>& scratch, cudaStream_t stream) {
  if (nb == 0) xtv_launch<T, 0, MOMENTS, FINITE>(X, n, p, ld, V, ldv, nb, out, ldo, sum, sumsq, scratch, stream);
  else if (nb <= 1) xtv_launch<T, 1, MOMENTS, FINITE>(X, n, p, ld, V, ldv, nb, out, ldo, sum, sumsq, scratch, stream);
  else if (nb <= 4) xtv_launch<T, 4, MOMENTS, FINITE>(X, n, p, ld, V, ldv, nb, out, ldo, sum, sumsq, scratch, stream);
  else if (nb <= 8) xtv_launch<T, 8, MOMENTS, FINITE>(X, n, p, ld, V, ldv, nb, out, ldo, sum, sumsq, scratch, stream);
  else if (nb <= 16) xtv_launch<T, 16, MOMENTS, FINITE>(X, n, p, ld, V, ldv, nb, out, ldo, sum, sumsq, scratch, stream);
  else xtv_launch<T, 32, MOMENTS, FINITE>(X, n, p, ld, V, ldv, nb, out, ldo, sum, sumsq, scratch, stream);
}

// ---------------------------------------------------------------------------
// X R - offset: thread per row pair, block over 512 rows x a column chunk.
// partial layout: [chunk][c][row] (column-major per chunk, ld = n).
// ---------------------------------------------------------------------------
template <class T, int NB, bool FINITE>
__global__ void __launch_bounds__(kThreads)
    xr_kernel(const T* __restrict__ X, int n, int p, long ld,
              const double* __restrict__ R, long ldr, int nb, int cc,
              double* __restrict__ partial) {
  extern __shared__ double rs[];  // cc x NB
  auto wide = [](T v) { return FINITE ? finite_f64<T>::widen(v) : as_f64(v); };
  const int chunk = blockIdx.y;
  const int c0 = chunk * cc;
  const int cols = min(cc, p - c0);
  for (int idx = threadIdx.x; idx < cols * NB; idx += blockDim.x) {
    const int j = idx / NB, c = idx % NB;
    rs[idx] = c < nb ? R[(c0 + j) + (long)c * ldr] * (FINITE ? finite_f64<T>::weight : 1.0) : 0.0;
  }
  __syncthreads();
  const int i0 = blockIdx.x * (2 * kThreads) + threadIdx.x;
  const int i1 = i0 + kThreads;
  double a0[NB], a1[NB];
#pragma unroll
  for (int c = 0; c < NB; ++c) a0[c] = a1[c] = 0.0;
  const bool v0 = i0 < n, v1 = i1 < n;
  const T* base = X + (long)c0 * ld;
  int j = 0;
  for (; j + 3 < cols; j += 4) {
    double x0[4], x1[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      x0[u] = v0 ? wide(base[i0 + (long)(j + u) * ld]) : 0.0;
      x1[u] = v1 ? wide(base[i1 + (long)(j + u) * ld]) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int c = 0; c < NB; ++c) {
        const double r = rs[(j + u) * NB + c];
        a0[c] = fma(x0[u], r, a0[c]);
        a1[c] = fma(x1[u], r, a1[c]);
      }
  }
  for (; j < cols; ++j) {
    const double x0 = v0 ? wide(base[i0 + (long)j * ld]) : 0.0;
    const double x1 = v1 ? wide(base[i1 + (long)j * ld]) : 0.0;
#pragma unroll
    for (int c = 0; c < NB; ++c) {
      const double r = rs[j * NB + c];
      a0[c] = fma(x0, r, a0[c]);
      a1[c] = fma(x1, r, a1[c]);
    }
  }
  double* out = partial + (long)chunk * n * nb;
#pragma unroll
  for (int c = 0; c < NB; ++c) {
    if (c < nb) {
      const double f = FINITE ? finite_f64<T>::result : 1.0;
      if (v0) out[i0 + (long)c * n] = a0[c] * f;
      if (v1) out[i1 + (long)c * n] = a1[c] * f;
    }
  }
}

// X R with row vectors: thread t of a 256 x V row tile takes rows V t .. V t +
// V - 1 with one 16-byte load per column, 4 columns per step (4 FP32, 2 FP64
// rows), or 8-byte loads of 4 rows, 8 columns per step, for BF16: 8 rows a
// thread left 600 blocks at 30011 rows (213 us a pass of 600 MB, 153 us so and 128 with finite_f64).
// Needs a column stride that is a multiple of 8 elements and a 16-byte aligned
// X. Each row's sum runs over the chunk's columns in order, exactly as in
// xr_kernel.
template <class T>
struct RowVec {
  using type = typename std::conditional<sizeof(T) == 2, uint2, uint4>::type;
  static constexpr int V = sizeof(type) / sizeof(T);
  static constexpr int STEP = sizeof(T) == 2 ? 8 : 4;
  template <bool FINITE>
  static __device__ __forceinline__ void unpack(const type& raw, double (&x)[V]) {
    if constexpr (FINITE && sizeof(T) == 2) {
      finite_f64<bf16>::widen2(raw.x, x[0], x[1]);
      finite_f64<bf16>::widen2(raw.y, x[2], x[3]);
    } else {
      const T* v = reinterpret_cast<const T*>(&raw);
#pragma unroll
      for (int e = 0; e < V; ++e) x[e] = FINITE ? finite_f64<T>::widen(v[e]) : as_f64(v[e]);
    }
  }
};

template <class T, int NB, bool FINITE>
__global__ void __launch_bounds__(kThreads)
    xr_vec_kernel(const T* __restrict__ X, int n, int p, long ld,
                  const double* __restrict__ R, long ldr, int nb, int cc,
                  double* __restrict__ partial) {
  constexpr int V = RowVec<T>::V, STEP = RowVec<T>::STEP;
  using L = typename RowVec<T>::type;
  extern __shared__ double rs[];  // cc x NB
  const int chunk = blockIdx.y;
  const int c0 = chunk * cc;
  const int cols = min(cc, p - c0);
  for (int idx = threadIdx.x; idx < cols * NB; idx += blockDim.x) {
    const int j = idx / NB, c = idx % NB;
    rs[idx] = c < nb ? R[(c0 + j) + (long)c * ldr] * (FINITE ? finite_f64<T>::weight : 1.0) : 0.0;
  }
  __syncthreads();
  const int r0 = blockIdx.x * (kThreads * V) + threadIdx.x * V;
  if (r0 >= n) return;
  double acc[V][NB];
#pragma unroll
  for (int e = 0; e < V; ++e)
#pragma unroll
    for (int c = 0; c < NB; ++c) acc[e][c] = 0.0;
  const T* base = X + (long)c0 * ld + r0;
  if (r0 + V <= n) {
    int j = 0;
    for (; j + STEP - 1 < cols; j += STEP) {
      L raw[STEP];
#pragma unroll
      for (int u = 0; u < STEP; ++u)
        raw[u] = __ldcs(reinterpret_cast<const L*>(base + (long)(j + u) * ld));
#pragma unroll
      for (int u = 0; u < STEP; ++u) {
        double x[V];
        RowVec<T>::template unpack<FINITE>(raw[u], x);
#pragma unroll
        for (int c = 0; c < NB; ++c) {
          const double r = rs[(j + u) * NB + c];
#pragma unroll
          for (int e = 0; e < V; ++e) acc[e][c] = fma(x[e], r, acc[e][c]);
        }
      }
    }
    for (; j < cols; ++j) {
      double x[V];
      RowVec<T>::template unpack<FINITE>(__ldcs(reinterpret_cast<const L*>(base + (long)j * ld)), x);
#pragma unroll
      for (int c = 0; c < NB; ++c) {
        const double r = rs[j * NB + c];
#pragma unroll
        for (int e = 0; e < V; ++e) acc[e][c] = fma(x[e], r, acc[e][c]);
      }
    }
  } else {  // ragged last rows: element loads
    for (int j = 0; j < cols; ++j) {
#pragma unroll
      for (int e = 0; e < V; ++e) {
        if (r0 + e >= n) break;
        const T v = base[(long)j * ld + e];
        const double x = FINITE ? finite_f64<T>::widen(v) : as_f64(v);
#pragma unroll
        for (int c = 0; c < NB; ++c) acc[e][c] = fma(x, rs[j * NB + c], acc[e][c]);
      }
    }
  }
  double* out = partial + (long)chunk * n * nb;
#pragma unroll
  for (int c = 0; c < NB; ++c) {
    if (c < nb) {
#pragma unroll
      for (int e = 0; e < V; ++e)
        if (r0 + e < n) out[r0 + e + (long)c * n] = FINITE ? acc[e][c] * finite_f64<T>::result : acc[e][c];
    }
  }
}

// Sums of the column chunks in order (eight loads in flight), minus the
// offset; with stats also the sum of squares and the sum of the column (one
// column), which were a kernel of their own.
__global__ void __launch_bounds__(kReduceThreads)
    xr_finish(const double* __restrict__ partial, int chunks, int n, int nb, const double* offset,
              int offset_parts, double* out, long ldo, bool with_stats, XrStats stats) {
  __shared__ double scratch[32];
  __shared__ double vals[2];
  const long total = (long)n * nb;
  double s2 = 0.0, s1 = 0.0;
  for (long idx = blockIdx.x * (long)blockDim.x + threadIdx.x; idx < total;
       idx += (long)gridDim.x * blockDim.x) {
    const int i = (int)(idx % n), c = (int)(idx / n);
    double v = 0.0;
    int k = 0;
    for (; k + 7 < chunks; k += 8) {
      double x[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) x[u] = partial[(long)(k + u) * total + idx];
#pragma unroll
      for (int u = 0; u < 8; ++u) v += x[u];
    }
    for (; k < chunks; ++k) v += partial[(long)k * total + idx];
    if (offset) v -= column_offset(offset, offset_parts, c);
    out[i + (long)c * ldo] = v;
    s2 = fma(v, v, s2);
    s1 += v;
  }
  if (!with_stats) return;
  s2 = block_sum(s2, scratch);
  s1 = block_sum(s1, scratch);
  if (threadIdx.x == 0) {
    vals[0] = s2;
    vals[1] = s1;
  }
  __syncthreads();
  last_block_reduce(vals, 2, stats.partial, stats.counter, stats.out);
}

template <class T, int NB, bool FINITE = false>
void xr_launch(const T* X, int n, int p, long ld, const double* R, long ldr,
               int nb, const double* offset, int offset_parts, double* out, long ldo,
               DeviceArray<double>& scratch, cudaStream_t stream, const XrStats* stats) {
  static_assert(NB <= 2, "wider products run on the FP64 tensor path");
  // 16-byte row vectors where the column stride allows. The column chunks depend on n and p only (a nominal 1024-row tile), so every
  // storage type and both kernels sum each row in the same order.
  const bool vec = ld % 8 == 0 && reinterpret_cast<uintptr_t>(X) % 16 == 0;
  const int nominal_tiles = (int)ceil_div(n, 1024);
  const int want = 16 * num_sms();
  int chunks = std::max(1, std::min((int)ceil_div(want, nominal_tiles), (int)ceil_div(p, 64)));
  int cc = (int)ceil_div(p, chunks);
  cc = std::min(cc, (48 * 1024 / 8) / NB);
  chunks = (int)ceil_div(p, cc);
  scratch.reserve((size_t)chunks * n * nb, stream);
  const size_t smem = (size_t)cc * NB * sizeof(double);
  if (vec)
    xr_vec_kernel<T, NB, FINITE><<<dim3(ceil_div(n, kThreads * RowVec<T>::V), chunks), kThreads, smem,
                           stream>>>(X, n, p, ld, R, ldr, nb, cc, scratch.get());
  else
    xr_kernel<T, NB, FINITE><<<dim3(ceil_div(n, 2 * kThreads), chunks), kThreads, smem, stream>>>(
        X, n, p, ld, R, ldr, nb, cc, scratch.get());
  count_launch();
  FPLS_LAUNCH("xr_kernel");
  const long total = (long)n * nb;
  const unsigned blocks = (unsigned)std::min<long>((total + 255) / 256, std::min<long>(8L * num_sms(), kXrStatsPartial / 2));
  xr_finish<<<blocks, 256, 0, stream>>>(scratch.get(), chunks, n, nb, offset, offset_parts, out, ldo,
                                        stats != nullptr, stats ? *stats : XrStats{});
  count_launch();
  FPLS_LAUNCH("xr_finish");
}

__global__ void topk_kernel(const double* __restrict__ v, int rows, int classes,
                            int top, int* __restrict__ out, long ldo) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= rows) return;
  v += (long)blockIdx.y * rows * classes;  // prefix blockIdx.y
  out += (long)blockIdx.y * ldo * top;
  // repeated strict-'>' scans: the lowest index wins ties, ranks are distinct
  unsigned long long used_lo = 0ull;
  for (int k = 0; k < top; ++k) {
    int best = -1;
    double bv = 0.0;
    for (int c = 0; c < classes; ++c) {
      if (c < 64 && ((used_lo >> c) & 1ull)) continue;
      if (c >= 64) {
        bool taken = false;
        for (int q = 0; q < k; ++q)
          if (out[r + (long)q * ldo] == c + 1) taken = true;
        if (taken) continue;
      }
      const double x = v[r + (long)c * rows];
      if (best < 0 || x > bv) {
        best = c;
        bv = x;
      }
    }
    if (best < 64 && best >= 0) used_lo |= 1ull << best;
    out[r + (long)k * ldo] = best + 1;
  }
}

}  // namespace

template <class T>
void column_moments(const T* X, int n, int p, long ld, const double* Yc, int m,
                    double* sum, double* sumsq, double* cross,
                    DeviceArray<double>& scratch, cudaStream_t stream) {
  // the first pass carries the column sums and sums of squares with up to 32
  // response columns; further columns go in passes of 32 without them
  const int w0 = std::min(m, 32);
  xtv_dispatch<T, true>(X, n, p, ld, Yc, n, w0, cross, p, sum, sumsq, scratch,
                        stream);
  for (int c0 = 32; c0 < m; c0 += 32) {
    const int w = std::min(32, m - c0);
    xtv_dispatch<T, false>(X, n, p, ld, Yc + (long)c0 * n, n, w,
                           cross + (long)c0 * p, p, nullptr, nullptr, scratch,
                           stream);
  }
}

// ---------------------------------------------------------------------------
// Column moments with one-based class labels (classification): per column
// the sum, the sum of squares and the per-class sums, in one pass over X.
// Block = 8 warps over a 32-column tile and a chunk of rows whose labels are
// staged in shared memory; each lane keeps its own class accumulators in
// shared memory (acc[warp][class][lane]), so an element costs one add into
// its class's slot instead of m products with staged responses. partial
// layout: [chunk][j][slot], slots = classes, sum, sumsq.
template <class T>
__global__ void __launch_bounds__(kThreads)
    class_moments_kernel(const T* __restrict__ X, int n, int p, long ld,
                         const int* __restrict__ labels, int m, int rc,
                         double* __restrict__ partial) {
  extern __shared__ double csm[];
  int* lab = reinterpret_cast<int*>(csm);                  // rc labels
  double* acc = csm + (rc + 1) / 2;                        // 8 x m x 32
  const int chunk = blockIdx.y;
  const int r0 = chunk * rc;
  const int rows = min(rc, n - r0);
  for (int r = threadIdx.x; r < rows; r += blockDim.x) lab[r] = labels[r0 + r] - 1;
  __syncthreads();
  const int slots = m + 2;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double* my = acc + (long)warp * m * 32;
  for (int jj = warp; jj < 32; jj += kThreads / 32) {
    const int j = blockIdx.x * 32 + jj;
    if (j >= p) break;
    for (int c = 0; c < m; ++c) my[c * 32 + lane] = 0.0;
    __syncwarp();
    const T* col = X + (long)j * ld + r0;
    double s = 0.0, ss = 0.0;
    int r = lane;
    for (; r + 96 < rows; r += 128) {
      double x[4];
      int l[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        x[u] = as_f64(col[r + 32 * u]);
        l[u] = lab[r + 32 * u];
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        s += x[u];
        ss = fma(x[u], x[u], ss);
        if (l[u] >= 0 && l[u] < m) my[l[u] * 32 + lane] += x[u];
      }
    }
    for (; r < rows; r += 32) {
      const double x = as_f64(col[r]);
      const int l = lab[r];
      s += x;
      ss = fma(x, x, ss);
      if (l >= 0 && l < m) my[l * 32 + lane] += x;
    }
    __syncwarp();
    double* out = partial + ((long)chunk * p + j) * slots;
    for (int c = 0; c < m; ++c) {
      const double v = warp_sum(my[c * 32 + lane]);
      if (lane == 0) out[c] = v;
    }
    s = warp_sum(s);
    ss = warp_sum(ss);
    if (lane == 0) {
      out[m] = s;
      out[m + 1] = ss;
    }
    __syncwarp();
  }
}

// cross[j + c p] = classsum[j, c] - prior[c] * colsum[j] (= X^T (onehot -
// prior)), sum and sumsq, from the per-chunk partials.
__device__ __forceinline__ double chunk_sum(const double* __restrict__ at, int chunks, long stride) {
  double v = 0.0;
  int k = 0;
  for (; k + 7 < chunks; k += 8) {
    double x[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) x[u] = at[(k + u) * stride];
#pragma unroll
    for (int u = 0; u < 8; ++u) v += x[u];
  }
  for (; k < chunks; ++k) v += at[k * stride];
  return v;
}

// One thread per column and slot, each class thread summing its column's total
// beside its own (a thread per column took 89 us at 500 columns, 12 classes,
// 53 chunks: two blocks of serial loads; 18 us so).
__global__ void class_moments_finish(const double* __restrict__ partial, int chunks, int p,
                                     int m, const double* __restrict__ prior, double* sum,
                                     double* sumsq, double* cross) {
  const int slots = m + 2;
  const long total = (long)p * slots;
  for (long idx = blockIdx.x * (long)blockDim.x + threadIdx.x; idx < total;
       idx += (long)gridDim.x * blockDim.x) {
    const int j = (int)(idx / slots), c = (int)(idx % slots);
    const double v = chunk_sum(partial + idx, chunks, total);
    if (c == m) {
      sum[j] = v;
    } else if (c == m + 1) {
      sumsq[j] = v;
    } else {
      const double s = chunk_sum(partial + (long)j * slots + m, chunks, total);
      cross[j + (long)c * p] = v - prior[c] * s;
    }
  }
}

template <class T>
void class_moments(const T* X, int n, int p, long ld, const int* labels, int m,
                   const double* prior, double* sum, double* sumsq, double* cross,
                   DeviceArray<double>& scratch, cudaStream_t stream) {
  // rows per chunk: enough blocks to cover every SM several times
  const int col_tiles = (int)ceil_div(p, 32);
  int rc = 2048;
  int chunks = (int)ceil_div(n, rc);
  const int want = 6 * num_sms();
  if (col_tiles * chunks < want && n > 256) {
    const int target = std::min((int)ceil_div(n, 256), (int)ceil_div(want, col_tiles));
    if (target > chunks) {
      rc = std::max(256, (int)ceil_div(n, target));
      rc = (rc + 127) / 128 * 128;
      chunks = (int)ceil_div(n, rc);
    }
  }
  const int slots = m + 2;
  scratch.reserve((size_t)chunks * p * slots, stream);
  const size_t smem = (size_t)(rc + 1) / 2 * sizeof(double) + (size_t)8 * m * 32 * sizeof(double);
  allow_shared_memory((const void*)class_moments_kernel<T>);
  class_moments_kernel<T><<<dim3(col_tiles, chunks), kThreads, smem, stream>>>(
      X, n, p, ld, labels, m, rc, scratch.get());
  count_launch();
  FPLS_LAUNCH("class_moments_kernel");
  class_moments_finish<<<std::min<unsigned>(ceil_div((size_t)p * slots, 128), 16 * num_sms()), 128, 0, stream>>>(
      scratch.get(), chunks, p, m, prior, sum, sumsq, cross);
  count_launch();
  FPLS_LAUNCH("class_moments_finish");
}

template <class T>
void xtv_product(const T* X, int n, int p, long ld, const double* V, long ldv,
                 int nb, double* out, long ldo, DeviceArray<double>& scratch,
                 cudaStream_t stream, bool finite) {
  if (finite && nb == 1) {
    xtv_launch<T, 1, false, true>(X, n, p, ld, V, ldv, nb, out, ldo, nullptr, nullptr, scratch, stream);
    return;
  }
  for (int c0 = 0; c0 < nb; c0 += 32) {
    const int w = std::min(32, nb - c0);
    xtv_dispatch<T, false>(X, n, p, ld, V + (long)c0 * ldv, ldv, w,
                           out + (long)c0 * ldo, ldo, nullptr, nullptr,
                           scratch, stream);
  }
}

template <class T>
void xr_product(const T* X, int n, int p, long ld, const double* R, long ldr,
                int nb, const double* offset, int offset_parts, double* out, long ldo,
                DeviceArray<double>& scratch, cudaStream_t stream, const XrStats* stats, bool finite) {
  require(nb == 1 || (nb == 2 && !stats), "streamed X R takes one or two columns");
  if (nb == 1 && finite)
    xr_launch<T, 1, true>(X, n, p, ld, R, ldr, nb, offset, offset_parts, out, ldo, scratch, stream, stats);
  else if (nb == 1) xr_launch<T, 1>(X, n, p, ld, R, ldr, nb, offset, offset_parts, out, ldo, scratch, stream, stats);
  else xr_launch<T, 2>(X, n, p, ld, R, ldr, nb, offset, offset_parts, out, ldo, scratch, stream, nullptr);
}

void topk_rows(const double* values, int rows, int classes, int top, int count, int* out,
               long ldo, cudaStream_t stream) {
  if (rows <= 0 || count <= 0) return;
  topk_kernel<<<dim3(ceil_div(rows, 128), count), 128, 0, stream>>>(values, rows, classes, top, out, ldo);
  count_launch();
  FPLS_LAUNCH("topk_rows");
}

#define FPLS_INSTANTIATE(T)                                                   \
  template void class_moments<T>(const T*, int, int, long, const int*, int,  \
                                 const double*, double*, double*, double*,   \
                                 DeviceArray<double>&, cudaStream_t);        \
  template void column_moments<T>(const T*, int, int, long, const double*,    \
                                  int, double*, double*, double*,             \
                                  DeviceArray<double>&, cudaStream_t);        \
  template void xtv_product<T>(const T*, int, int, long, const double*, long, \
                               int, double*, long, DeviceArray<double>&,      \
                               cudaStream_t, bool);                           \
  template void xr_product<T>(const T*, int, int, long, const double*, long,  \
                              int, const double*, int, double*, long,         \
                              DeviceArray<double>&, cudaStream_t,             \
                              const XrStats*, bool);
FPLS_INSTANTIATE(float)
FPLS_INSTANTIATE(double)
FPLS_INSTANTIATE(bf16)
#undef FPLS_INSTANTIATE

}  // namespace fpls
