// Projection of new rows and predictions along a component path.
//
// Scores are one product X (R / scale) - mean . (R / scale) (xr_product); the
// responses of every prefix then come from one pass over the scores, written
// in the caller's result type. Per prefix this took a fill, a product on one
// 128 x 128 tile of a 3-response result, a conversion, a copy and a wait.
#include "kernels.cuh"
#include "model.cuh"

#include <algorithm>

namespace fpls {

namespace {

constexpr int TB = 256;
constexpr int kWeightCols = 1024;  // predictors per block of scaled_weights
constexpr int kMaxParts = 32;

// Rs = R / scale (p x k) and the partial sums of mean . Rs[:, c] over the
// block's predictors, roff[c * parts + block]. Latency-bound at the path's
// sizes (p k doubles); one block per column left 20 blocks on 148 SMs (38 us
// at 10000 x 20, 6 us over chunks of the predictors).
__global__ void scaled_weights(const double* __restrict__ R, int p, int k, int per,
                               const double* __restrict__ mean, const double* __restrict__ scale,
                               double* __restrict__ Rs, double* __restrict__ roff) {
  __shared__ double scratch[32];
  const int c = blockIdx.y;
  const int j0 = blockIdx.x * per, j1 = min(p, j0 + per);
  double acc = 0.0;
  for (int j = j0 + threadIdx.x; j < j1; j += blockDim.x) {
    const double w = R[j + (long)c * p] / scale[j];
    Rs[j + (long)c * p] = w;
    acc = fma(mean[j], w, acc);
  }
  acc = block_sum(acc, scratch);
  if (threadIdx.x == 0) roff[c * gridDim.x + blockIdx.x] = acc;
}

constexpr int kPrefixBatch = 64;
struct PrefixSet {
  int count;
  int k[kPrefixBatch];
};

// Thread (row, response): one running sum over the components, stored at each
// prefix. Reads the scores once per response (they stay in L2), writes every
// result once; bound by launch latency at the path's sizes.
template <class TO>
__global__ void predict_linear(const double* __restrict__ scores, int rows, long lds,
                               const double* __restrict__ Q, int m,
                               const double* __restrict__ ymean, PrefixSet ps, TO* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int r = blockIdx.y;
  if (i >= rows) return;
  const double base = ymean[r];
  double acc = 0.0;
  int c = 0;
  for (int j = 0; j < ps.count; ++j) {
    const int k = ps.k[j];
#pragma unroll 4
    for (; c < k; ++c) acc = fma(scores[i + (long)c * lds], Q[r + (long)c * m], acc);
    out[((long)j * m + r) * rows + i] = static_cast<TO>(acc + base);
  }
}

constexpr int kMapBatch = 32;
struct MapSet {
  PrefixMap map[kMapBatch];
};

template <class TO>
__global__ void predict_maps(const double* __restrict__ scores, int rows, long lds, int m, MapSet ms,
                             TO* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int r = blockIdx.y;
  if (i >= rows) return;
  const PrefixMap& mp = ms.map[blockIdx.z];
  const double* w = mp.w + (long)r * mp.stride_r;
  double acc = 0.0;
#pragma unroll 4
  for (int c = 0; c < mp.k; ++c) acc = fma(scores[i + (long)c * lds], w[(long)c * mp.stride_c], acc);
  out[((long)blockIdx.z * m + r) * rows + i] = static_cast<TO>(acc + mp.base[r]);
}

}  // namespace

template <class T>
void project_rows(const DeviceModel& model, const T* X, int rows, long ld,
                  int k, double* out, long ldo, Workspace& ws,
                  cudaStream_t stream) {
  require(k >= 1 && k <= model.a, "invalid projection prefix");
  const int p = model.p;
  const int parts = std::min<int>(kMaxParts, ceil_div(p, kWeightCols));
  DeviceArray<double> Rs((size_t)p * k + (size_t)k * parts, stream);
  double* roff = Rs.get() + (size_t)p * k;
  scaled_weights<<<dim3(parts, k), TB, 0, stream>>>(model.R.get(), p, k, ceil_div(p, parts), model.mean.get(),
                                                    model.scale.get(), Rs.get(), roff);
  count_launch();
  FPLS_LAUNCH("scaled_weights");
  // A large X: one or two columns stream it, 3..16 take it in one pass on
  // bulk-copy stages (both HBM-bound or near it). Otherwise a DMMA product
  // with X in its storage type and K in slices of 256 predictors, so that few
  // rows still fill the SMs and every sum has the same order at any number of
  // rows and columns (a prefix alone equals the same prefix in a path; the forms
  // for a large X depend on the number of columns). 451
  // new rows x 10000, 20 columns: 93 us in passes of 8, 8 and 4 columns
  // before, 37 us now; 4001 x 4000, 12 columns: 78 us, 46 us.
  const bool large = (long)rows * p >= (1L << 24);
  if (large && k <= 2) {
    xr_product<T>(X, rows, p, ld, Rs.get(), p, k, roff, parts, out, ldo, ws.stream_partial, stream);
    return;
  }
  if (large && xr_ring<T>(X, rows, p, ld, Rs.get(), p, k, roff, parts, out, ldo, ws.flag.get(), stream)) return;
  GemmArgs g;
  g.M = rows;
  g.N = k;
  g.K = p;
  g.A = X;
  g.lda = ld;
  g.a_type = gemm_type<T>::value;
  g.B = Rs.get();
  g.ldb = p;
  g.C = out;
  g.ldc = ldo;
  g.coff = roff;
  g.coff_parts = parts;
  g.k_slice = 256;
  gemm_f64(g, stream);
}

template <class TO>
void apply_prefix_maps(const double* scores, int rows, long lds, int m, const PrefixMap* maps,
                       int count, TO* out, cudaStream_t stream) {
  for (int j0 = 0; j0 < count; j0 += kMapBatch) {
    const int b = std::min(kMapBatch, count - j0);
    MapSet ms;
    std::copy(maps + j0, maps + j0 + b, ms.map);
    predict_maps<TO><<<dim3(ceil_div(rows, 128), m, b), 128, 0, stream>>>(
        scores, rows, lds, m, ms, out + (size_t)j0 * rows * m);
    count_launch();
    FPLS_LAUNCH("predict_maps");
  }
}

template <class TO>
void predict_prefixes(const DeviceModel& model, const double* scores, int rows, long lds,
                      const int* prefixes, int count, TO* out, cudaStream_t stream) {
  const int m = model.m, a = model.a;
  require(count >= 1 && prefixes[0] >= 1 && prefixes[count - 1] <= a, "invalid prediction prefix");
  if (model.method == kPlssvd) {
    // W block for prefix k: k x m at offset (k-1) * a * m in model.W
    std::vector<PrefixMap> maps(count);
    for (int j = 0; j < count; ++j)
      maps[j] = {prefixes[j], model.W.get() + (size_t)(prefixes[j] - 1) * a * m, model.ymean.get(), 1,
                 prefixes[j]};
    apply_prefix_maps<TO>(scores, rows, lds, m, maps.data(), count, out, stream);
    return;
  }
  for (int j0 = 0; j0 < count; j0 += kPrefixBatch) {
    PrefixSet ps;
    ps.count = std::min(kPrefixBatch, count - j0);
    std::copy(prefixes + j0, prefixes + j0 + ps.count, ps.k);
    predict_linear<TO><<<dim3(ceil_div(rows, 128), m), 128, 0, stream>>>(
        scores, rows, lds, model.Q.get(), m, model.ymean.get(), ps, out + (size_t)j0 * rows * m);
    count_launch();
    FPLS_LAUNCH("predict_linear");
  }
}

#define FPLS_INSTANTIATE(T)                                                     \
  template void project_rows<T>(const DeviceModel&, const T*, int, long, int,  \
                                double*, long, Workspace&, cudaStream_t);
FPLS_INSTANTIATE(float)
FPLS_INSTANTIATE(double)
FPLS_INSTANTIATE(bf16)
#undef FPLS_INSTANTIATE
#define FPLS_INSTANTIATE(TO)                                                             \
  template void predict_prefixes<TO>(const DeviceModel&, const double*, int, long,      \
                                     const int*, int, TO*, cudaStream_t);               \
  template void apply_prefix_maps<TO>(const double*, int, long, int, const PrefixMap*,  \
                                      int, TO*, cudaStream_t);
FPLS_INSTANTIATE(float)
FPLS_INSTANTIATE(double)
#undef FPLS_INSTANTIATE

}  // namespace fpls
