// Cross-validation drivers behind the reference's CV entry points
// (fastpls_resident_{simpls,plssvd}_cv_{regression,classification}).
//
// Behavioural contract: src/cuda_resident_api.cuh:538-1023 of the reference
// (validation and messages, fold status codes 1/2/4, metric assembly in long
// double, prediction and score output layouts). X and Y are uploaded once;
// each fold's training and held-out rows are split on the device and the
// fold model is fitted by the resident engine (fit.cu / plssvd.cu). Folds run
// in batches: the SIMPLS folds of a batch that take the persistent form run
// their component loops in one launch with the co-resident CTAs shared between
// them (a fold alone leaves most SMs idle: ten folds of 541 x 1500 FP64 were ten
// launches of 24 CTAs, 527 us each), the others' loops overlap on a few
// streams, the held-out predictions follow, and the call waits once per batch.
// The many-fold / many-permutation batched engine lives in batched.cu.
#include "upload.cuh"
#include "cv.cuh"
#include "cv_batches.hpp"
#include "handle.cuh"
#include "lda.cuh"
#include "persistent.cuh"

#include <algorithm>
#include <cmath>
#include <exception>
#include <limits>
#include <vector>

namespace fpls {

namespace {

// Block (response, prefix): squared errors and squares about the training mean.
__global__ void fold_sums_kernel(const double* __restrict__ pred,
                                 const double* __restrict__ y,
                                 const double* __restrict__ ymean, int n,
                                 int q, double* out) {
  __shared__ double scratch[32];
  const int c = blockIdx.x;
  pred += (long)blockIdx.y * n * q;
  out += (long)blockIdx.y * 2 * q;
  double sse = 0.0, st = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const double v = y[i + (long)c * n];
    const double e = v - pred[i + (long)c * n], d = v - ymean[c];
    sse = fma(e, e, sse);
    st = fma(d, d, st);
  }
  sse = block_sum(sse, scratch);
  st = block_sum(st, scratch);
  if (threadIdx.x == 0) {
    out[2 * c] = sse;
    out[2 * c + 1] = st;
  }
}

struct Folds {
  int count = 0;
  std::vector<std::vector<int>> test;
  int max_test = 0, max_train = 0;
};

Folds partition(const int* folds, int n) {
  Folds f;
  for (int i = 0; i < n; ++i) f.count = std::max(f.count, folds[i]);
  f.test.assign(f.count, {});
  for (int i = 0; i < n; ++i) f.test[folds[i] - 1].push_back(i);
  for (const auto& t : f.test) {
    f.max_test = std::max(f.max_test, (int)t.size());
    f.max_train = std::max(f.max_train, n - (int)t.size());
  }
  return f;
}

// Rows of X (n x p) and of Y (n x q, may be null) into the training and
// held-out matrices of one fold: pos[r] >= 0 is row r's training row, ~pos[r]
// its held-out row. Reads every element once, coalesced along the rows.
template <class T>
__global__ void split_rows_kernel(const T* __restrict__ X, const T* __restrict__ Y, int n, int p, int q,
                                  const int* __restrict__ pos, int ntr, int nte, T* __restrict__ Xtr,
                                  T* __restrict__ Xte, T* __restrict__ Ytr, double* __restrict__ Yte) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  const int at = pos[r];
  for (int c = blockIdx.y; c < p + q; c += gridDim.y) {
    if (c < p) {
      const T v = X[r + (long)c * n];
      if (at >= 0) Xtr[at + (long)c * ntr] = v;
      else Xte[~at + (long)c * nte] = v;
    } else {
      const T v = Y[r + (long)(c - p) * n];
      if (at >= 0) Ytr[at + (long)(c - p) * ntr] = v;
      else Yte[~at + (long)(c - p) * nte] = as_f64(v);
    }
  }
}

// One fold of a batch, its device state allocated on its stream.
template <class T>
struct Fold {
  int f = 0, ntr = 0, nte = 0, m = 0;  // fold, rows, responses or active classes
  cudaStream_t st = nullptr;
  Workspace ws;
  DeviceModel model;
  std::unique_ptr<PersistentPlan> plan;
  DeviceArray<T> Xtr, Xte, Ytr;
  DeviceArray<double> Yte, Yc, ycsum, scores, pred, sums;
  const int *pos = nullptr, *lab = nullptr;  // into the batch's arrays
  std::unique_ptr<LdaState> lda;
  std::vector<int> active;
  std::vector<double> host_pred;
  size_t at_sums = 0, at_pred = 0, at_labels = 0, at_flag = 0;  // into the batch's Results
};

// What the host reads of a batch, in one device buffer and one copy: a copy to
// pageable memory waits for its stream, 15 us each, and three per fold were 460
// of the 3500 us of a 10-fold call (601 x 1500). Allocated and freed on `main`.
struct Results {
  size_t bytes = 0;
  DeviceArray<unsigned char> dev;
  std::vector<unsigned char> host;
  size_t take(size_t b) {
    const size_t at = bytes;
    bytes += (b + 255) / 256 * 256;
    return at;
  }
  template <class V>
  V* on_device(size_t at) { return reinterpret_cast<V*>(dev.get() + at); }
  template <class V>
  const V* on_host(size_t at) const { return reinterpret_cast<const V*>(host.data() + at); }
};

// Lanes of the call's folds (cv_batches.hpp).
int call_lanes(int method, int folds, int n, int p, int m, int a, bool classification, int elem) {
  if (method == kPlssvd || (long)n * p > kPersistMaxElements) return 0;
  const bool persistent = persistent_enabled() && persistent_supported(m, a) && persistent_ctas(n, p) > 0 &&
                          persistent_capacity(elem) > 0 && !simpls_gram_route(n, p, a, classification) &&
                          simpls_block_size(n, p, m, a, classification, elem == 4) <= 1;
  return fold_lanes(folds, !persistent);
}

// The streams of one call: `main` (uploads, shared launches) and the lanes
// that prepare and finish the folds, if any.
struct Lanes {
  cudaStream_t main = nullptr, lane[kLanes] = {};
  cudaEvent_t ev = nullptr;
  const int count;
  explicit Lanes(int lanes) : count(lanes) {
    FPLS_CHECK(cudaStreamCreateWithFlags(&main, cudaStreamNonBlocking));
    FPLS_CHECK(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
    for (int k = 0; k < count; ++k) FPLS_CHECK(cudaStreamCreateWithFlags(&lane[k], cudaStreamNonBlocking));
  }
  // the stream of the k-th fold of a batch
  cudaStream_t of(size_t k) const { return count > 0 ? lane[k % count] : main; }
  ~Lanes() {
    for (cudaStream_t s : lane)
      if (s) {
        cudaStreamSynchronize(s);
        cudaStreamDestroy(s);
      }
    if (main) {
      cudaStreamSynchronize(main);
      cudaStreamDestroy(main);
    }
    if (ev) cudaEventDestroy(ev);
  }
  Lanes(const Lanes&) = delete;
  Lanes& operator=(const Lanes&) = delete;
  void after(cudaStream_t later, cudaStream_t earlier) {
    FPLS_CHECK(cudaEventRecord(ev, earlier));
    FPLS_CHECK(cudaStreamWaitEvent(later, ev, 0));
  }
  void lanes_after_main() {
    FPLS_CHECK(cudaEventRecord(ev, main));
    for (cudaStream_t s : lane)
      if (s) FPLS_CHECK(cudaStreamWaitEvent(s, ev, 0));
  }
  void main_after_lanes() {
    for (cudaStream_t s : lane)
      if (s) after(main, s);
  }
  void sync() {
    for (cudaStream_t s : lane)
      if (s) FPLS_CHECK(cudaStreamSynchronize(s));
    FPLS_CHECK(cudaStreamSynchronize(main));
  }
};

// Declared after what the lanes use: nothing is freed while they run, on an
// error too.
struct Settle {
  Lanes& lanes;
  ~Settle() {
    for (cudaStream_t s : lanes.lane)
      if (s) cudaStreamSynchronize(s);
    cudaStreamSynchronize(lanes.main);
  }
};

// The grouping of the call's folds (cv_batches.hpp).
template <class T>
CvBatches batch_shape(int method, const Folds& fp, int n, int p, int m, int a, size_t pred_bytes) {
  const double one = (double)n * p * sizeof(T) + 8.0 * ((double)p * (2.0 * a + 4.0 * m + 16.0) +
                                                      (double)n * (2.0 * a + 3.0 * m + 8.0)) +
                     (double)pred_bytes + 64.0 * 1024 * 1024;
  const bool simpls = method != kPlssvd;
  return cv_batches(
      fp.count, one, device_memory(), simpls ? persistent_capacity((int)sizeof(T)) : -1,
      simpls && (long)fp.max_train * p > kPersistMaxElements,
      [&](int share) { return persistent_ctas(fp.max_train, p, share); },
      [] {
        size_t free_b = 0, total_b = 0;
        FPLS_CHECK(cudaMemGetInfo(&free_b, &total_b));
        return (double)free_b;
      });
}

// run(f0, f1) for all folds in batches. A batch that does not find its memory
// leaves no result behind (run writes them last) and is taken again in halves,
// down to one fold. run returns the error of a fold, if any, after the results
// of the folds before it.
template <class F>
void in_batches(int folds, int per_batch, F&& run) {
  for (int f0 = 0; f0 < folds;) {
    const int f1 = std::min(folds, f0 + per_batch);
    try {
      if (std::exception_ptr failed = run(f0, f1)) std::rethrow_exception(failed);
      f0 = f1;
    } catch (const OutOfMemory&) {
      if (f1 - f0 <= 1) throw;
      per_batch = (f1 - f0) / 2;
    }
  }
}

// The fit of a prepared fold on its stream; a SIMPLS fold that takes the
// persistent form leaves its plan for the batch's launch.
template <class T>
void fit_fold(int method, Fold<T>& d, int p, int a, int scaling, int max_ctas) {
  const int n = d.ntr, m = d.m;
  if (method == kPlssvd) {
    fit_plssvd<T>(d.Xtr.get(), n, p, n, d.Yc.get(), d.ycsum.get(), m, a, scaling, d.model, d.ws, d.st);
    return;
  }
  struct Sink {
    explicit Sink(std::unique_ptr<PersistentPlan>* plan, int ctas) { persistent_deferral() = {plan, ctas}; }
    ~Sink() { persistent_deferral() = {}; }
  } sink(&d.plan, max_ctas);
  fit_simpls<T>(d.Xtr.get(), n, p, n, d.Yc.get(), d.ycsum.get(), m, a, scaling, d.model, d.ws, d.st,
                simpls_block_size(n, p, m, a, d.model.classification, std::is_same<T, float>::value),
                simpls_gram_route(n, p, a, d.model.classification));
}

// The component loops of the batch's deferred folds, as many per launch as
// are co-resident.
template <class T>
void launch_plans(std::vector<std::unique_ptr<Fold<T>>>& batch, Lanes& lanes) {
  std::vector<PersistentPlan*> plans;
  int ctas = 0;
  const int cap = persistent_capacity((int)sizeof(T));
  bool any = false;
  for (auto& d : batch) any = any || d->plan;
  if (!any) return;
  lanes.main_after_lanes();
  for (auto& d : batch) {
    if (!d->plan) continue;
    if (ctas + d->plan->fit.C > cap) {
      launch_persistent(plans, lanes.main);
      plans.clear();
      ctas = 0;
    }
    plans.push_back(d->plan.get());
    ctas += d->plan->fit.C;
  }
  launch_persistent(plans, lanes.main);
  lanes.lanes_after_main();
}

// The flags of the batch's fits beside its results, then one copy of all of it
// after every lane.
template <class T>
void collect(std::vector<std::unique_ptr<Fold<T>>>& batch, Results& out, Lanes& lanes) {
  if (batch.empty()) return;
  for (auto& d : batch)
    FPLS_CHECK(cudaMemcpyAsync(out.on_device<int>(d->at_flag), d->ws.flag.get(), sizeof(int),
                               cudaMemcpyDeviceToDevice, d->st));
  out.host.resize(out.bytes);
  lanes.main_after_lanes();
  FPLS_CHECK(cudaMemcpyAsync(out.host.data(), out.dev.get(), out.bytes, cudaMemcpyDeviceToHost, lanes.main));
}

// Position of every row in the training (k) or held-out (~k) matrix of the
// fold that holds out `held`, into pos (n).
void fold_positions(const std::vector<int>& held, int n, int* pos) {
  std::fill(pos, pos + n, 0);
  for (size_t k = 0; k < held.size(); ++k) pos[held[k]] = ~(int)k;
  int at = 0;
  for (int i = 0; i < n; ++i)
    if (pos[i] >= 0) pos[i] = at++;
}

template <class T>
void split_fold(Fold<T>& d, const T* X, const T* Y, int n, int p, int q) {
  d.Xtr.allocate((size_t)d.ntr * p, d.st);
  d.Xte.allocate((size_t)d.nte * p, d.st);
  if (Y) {
    d.Ytr.allocate((size_t)d.ntr * q, d.st);
    d.Yte.allocate((size_t)d.nte * q, d.st);
  }
  const int cols = p + (Y ? q : 0);
  const unsigned gx = ceil_div(n, 256);
  const unsigned gy = (unsigned)std::max(1L, std::min<long>(cols, std::min<long>(65535, 16L * num_sms() / gx)));
  split_rows_kernel<T><<<dim3(gx, gy), 256, 0, d.st>>>(X, Y, n, p, Y ? q : 0, d.pos, d.ntr, d.nte,
                                                       d.Xtr.get(), d.Xte.get(), d.Ytr.get(), d.Yte.get());
  count_launch();
  FPLS_LAUNCH("split_rows");
}

}  // namespace

template <class T>
void cv_regression(int method, const T* predictors, const T* responses,
                   const int* folds, int n, int p, int q, const int* prefixes,
                   int prefix_count, int scaling, int metric,
                   bool store_predictions, double* prediction_output,
                   int* status, double* metrics, double* q2_values,
                   double* rmsd_values, double* observed_r2_values) {
  if (!predictors || !responses || !folds || !prefixes || !status || !metrics ||
      n < 2 || p < 1 || q < 1 || prefix_count < 1 || scaling < 1 ||
      scaling > 3 || metric < 2 || metric > 4)
    throw std::invalid_argument("invalid resident CUDA regression CV input");
  int maximum_prefix = 0;
  for (int j = 0; j < prefix_count; ++j) {
    if (prefixes[j] <= maximum_prefix)
      throw std::invalid_argument("CUDA CV component path must be strictly increasing");
    maximum_prefix = prefixes[j];
  }
  for (int i = 0; i < n; ++i)
    if (folds[i] < 1) throw std::invalid_argument("invalid CUDA CV fold");
  if (maximum_prefix > std::min(n - 1, p) || (store_predictions && !prediction_output))
    throw std::invalid_argument("invalid CUDA regression CV output or rank");
  Folds fp = partition(folds, n);
  if (fp.max_test < 1 || fp.max_train < 2)
    throw std::invalid_argument("CUDA CV contains an empty train or test fold");

  long double total_ss = 0.0L;
  for (int c = 0; c < q; ++c) {
    long double s = 0.0L, ss = 0.0L;
    for (int i = 0; i < n; ++i) {
      const long double v = responses[(size_t)c * n + i];
      s += v;
      ss += v * v;
    }
    total_ss += ss - s * s / n;
  }

  Lanes lanes(call_lanes(method, fp.count, fp.max_train, p, q, maximum_prefix, false, (int)sizeof(T)));
  {
    DeviceArray<T> X((size_t)n * p, lanes.main), Y((size_t)n * q, lanes.main);
    upload_h2d(X.get(), predictors, sizeof(T) * n * p, lanes.main);
    FPLS_CHECK(cudaMemcpyAsync(Y.get(), responses, sizeof(T) * n * q, cudaMemcpyHostToDevice, lanes.main));
    lanes.lanes_after_main();
    const size_t block = (size_t)fp.max_test * q;
    const int step = prefixes_at_once(block * sizeof(double), prefix_count);
    const CvBatches shape = batch_shape<T>(method, fp, n, p, q, maximum_prefix, block * step * sizeof(double));
    std::fill(metrics, metrics + prefix_count, 0.0);
    std::vector<double> counts(prefix_count, 0.0), fold_ss(prefix_count, 0.0);
    in_batches(fp.count, shape.per_batch, [&](int f0, int f1) {
      std::exception_ptr failed;
      // row positions of the batch's folds: one copy (a copy from pageable
      // memory waits for its stream)
      std::vector<int> host_pos((size_t)(f1 - f0) * n);
      for (int f = f0; f < f1; ++f) fold_positions(fp.test[f], n, host_pos.data() + (size_t)(f - f0) * n);
      DeviceArray<int> pos(host_pos.size(), lanes.main);
      FPLS_CHECK(cudaMemcpyAsync(pos.get(), host_pos.data(), sizeof(int) * host_pos.size(),
                                 cudaMemcpyHostToDevice, lanes.main));
      lanes.lanes_after_main();
      std::vector<std::unique_ptr<Fold<T>>> batch;
      Results out;
      Settle settle{lanes};
      try {
        for (int f = f0; f < f1; ++f) {
          const auto& held = fp.test[f];
          if (held.empty()) {
            status[f] = 2;
            continue;
          }
          if (maximum_prefix > std::min(n - (int)held.size() - 1, p))
            throw std::invalid_argument("CUDA CV component count exceeds a fold rank");
          std::unique_ptr<Fold<T>> fold(new Fold<T>());
          Fold<T>& d = *fold;
          d.f = f;
          d.m = q;
          d.st = lanes.of(batch.size());
          d.nte = (int)held.size();
          d.ntr = n - d.nte;
          d.pos = pos.get() + (size_t)(f - f0) * n;
          split_fold(d, X.get(), Y.get(), n, p, q);
          d.ws.ensure(d.ntr, p, q, maximum_prefix, d.st);
          FPLS_CHECK(cudaMemsetAsync(d.ws.flag.get(), 0, sizeof(int), d.st));
          d.Yc.allocate((size_t)d.ntr * q, d.st);
          d.ycsum.allocate(q, d.st);
          d.model.ymean.allocate(q, d.st);
          prepare_responses<T>(d.Ytr.get(), nullptr, d.ntr, q, d.Yc.get(), d.model.ymean.get(), d.ycsum.get(),
                               d.ws.flag.get(), d.st);
          fit_fold<T>(method, d, p, maximum_prefix, scaling, shape.max_ctas);
          batch.push_back(std::move(fold));
        }
      } catch (const OutOfMemory&) {
        throw;
      } catch (...) {
        failed = std::current_exception();  // after the folds before it
      }
      const bool copy_pred = store_predictions && step == prefix_count;
      for (auto& fold : batch) {
        Fold<T>& d = *fold;
        d.at_sums = out.take(sizeof(double) * 2 * q * prefix_count);
        if (copy_pred) d.at_pred = out.take(sizeof(double) * d.nte * q * prefix_count);
        d.at_flag = out.take(sizeof(int));
      }
      out.dev.allocate(out.bytes, lanes.main);
      launch_plans(batch, lanes);
      lanes.lanes_after_main();
      for (auto& fold : batch) {
        Fold<T>& d = *fold;
        d.scores.allocate((size_t)d.nte * maximum_prefix, d.st);
        if (!copy_pred) d.pred.allocate((size_t)d.nte * q * step, d.st);
        double* pred = copy_pred ? out.on_device<double>(d.at_pred) : d.pred.get();
        double* sums = out.on_device<double>(d.at_sums);
        if (store_predictions && !copy_pred) d.host_pred.resize((size_t)d.nte * q * prefix_count);
        project_rows<T>(d.model, d.Xte.get(), d.nte, d.nte, maximum_prefix, d.scores.get(), d.nte, d.ws, d.st);
        for (int j = 0; j < prefix_count; j += step) {
          const int w = std::min(step, prefix_count - j);
          predict_prefixes<double>(d.model, d.scores.get(), d.nte, d.nte, prefixes + j, w, pred, d.st);
          fold_sums_kernel<<<dim3(q, w), 256, 0, d.st>>>(pred, d.Yte.get(), d.model.ymean.get(), d.nte,
                                                         q, sums + (size_t)2 * q * j);
          count_launch();
          FPLS_LAUNCH("fold_sums");
          if (store_predictions && step < prefix_count)
            FPLS_CHECK(cudaMemcpyAsync(d.host_pred.data() + (size_t)j * d.nte * q, pred,
                                       sizeof(double) * d.nte * q * w, cudaMemcpyDeviceToHost, d.st));
        }
      }
      collect(batch, out, lanes);
      lanes.sync();
      for (auto& fold : batch) {
        Fold<T>& d = *fold;
        if (*out.on_host<int>(d.at_flag))
          throw std::runtime_error(method == kPlssvd
              ? "resident PLS-SVD failed: invalid labels, decomposition or score Gram"
              : "resident SIMPLS failed: invalid labels, decomposition or component norm");
        const auto& held = fp.test[d.f];
        const double* sums = out.on_host<double>(d.at_sums);
        const double* pred = copy_pred ? out.on_host<double>(d.at_pred) : d.host_pred.data();
        for (int j = 0; j < prefix_count; ++j) {
          long double sse = 0.0L, tss = 0.0L;
          for (int c = 0; c < q; ++c) {
            sse += sums[(size_t)2 * q * j + 2 * c];
            tss += sums[(size_t)2 * q * j + 2 * c + 1];
          }
          metrics[j] += (double)sse;
          fold_ss[j] += (double)tss;
          counts[j] += (double)d.nte * q;
          if (store_predictions)
            for (int c = 0; c < q; ++c)
              for (int i = 0; i < d.nte; ++i)
                prediction_output[(size_t)j * n * q + (size_t)c * n + held[i]] =
                    pred[((size_t)j * q + c) * d.nte + i];
        }
        status[d.f] = 1;
      }
      return failed;
    });
    const double nan = std::numeric_limits<double>::quiet_NaN();
    for (int j = 0; j < prefix_count; ++j) {
      const double sse = metrics[j];
      const double rmsd = counts[j] > 0.0 ? std::sqrt(sse / counts[j]) : nan;
      const double q2 = fold_ss[j] > 0.0 ? 1.0 - sse / fold_ss[j] : nan;
      const double r2 = total_ss > 0.0L ? 1.0 - sse / (double)total_ss : nan;
      if (rmsd_values) rmsd_values[j] = rmsd;
      if (q2_values) q2_values[j] = q2;
      if (observed_r2_values) observed_r2_values[j] = r2;
      metrics[j] = metric == 4 ? rmsd : metric == 3 ? q2 : r2;
    }
  }
}

template <class T>
void cv_classification(int method, const T* predictors, const int* labels,
                       const int* folds, int n, int p, int classes,
                       const int* prefixes, int prefix_count, int scaling,
                       bool use_lda, bool store_predictions, bool store_scores,
                       int* prediction_output, T* score_output, int* status,
                       double* metrics) {
  if (!predictors || !labels || !folds || !prefixes || !status || !metrics ||
      n < 2 || p < 1 || classes < 2 || prefix_count < 1 || scaling < 1 || scaling > 3)
    throw std::invalid_argument("invalid resident CUDA CV input");
  int maximum_prefix = 0;
  for (int j = 0; j < prefix_count; ++j) {
    if (prefixes[j] <= maximum_prefix)
      throw std::invalid_argument("CUDA CV component path must be strictly increasing");
    maximum_prefix = prefixes[j];
  }
  for (int i = 0; i < n; ++i)
    if (labels[i] < 1 || labels[i] > classes || folds[i] < 1)
      throw std::invalid_argument("invalid CUDA CV label or fold");
  if (maximum_prefix > std::min(n - 1, p))
    throw std::invalid_argument("CUDA CV component count exceeds rank");
  if (store_predictions && !prediction_output)
    throw std::invalid_argument("null CUDA CV prediction output");
  if (store_scores && !score_output)
    throw std::invalid_argument("null CUDA CV score output");
  Folds fp = partition(folds, n);
  if (fp.max_test < 1 || fp.max_train < 2)
    throw std::invalid_argument("CUDA CV contains an empty train or test fold");

  Lanes lanes(call_lanes(method, fp.count, fp.max_train, p, classes, maximum_prefix, true, (int)sizeof(T)));
  {
    DeviceArray<T> X((size_t)n * p, lanes.main);
    upload_h2d(X.get(), predictors, sizeof(T) * n * p, lanes.main);
    lanes.lanes_after_main();
    const size_t block = (size_t)fp.max_test * classes;
    const int step = prefixes_at_once(block * sizeof(double), prefix_count);
    const CvBatches shape = batch_shape<T>(method, fp, n, p, classes, maximum_prefix, 2 * block * step * sizeof(double));
    std::fill(metrics, metrics + prefix_count, 0.0);
    std::vector<double> counts(prefix_count, 0.0);
    if (store_scores) std::fill(score_output, score_output + (size_t)n * classes * prefix_count, T(0));
    in_batches(fp.count, shape.per_batch, [&](int f0, int f1) {
      std::exception_ptr failed;
      // row positions and compacted training labels of the batch's folds: one
      // copy each (a copy from pageable memory waits for its stream)
      std::vector<int> host_pos((size_t)(f1 - f0) * n), host_lab(host_pos.size(), 1);
      std::vector<std::vector<int>> counts_of(f1 - f0, std::vector<int>(classes, 0));
      for (int f = f0; f < f1; ++f) {
        int* at = host_pos.data() + (size_t)(f - f0) * n;
        int* lab = host_lab.data() + (size_t)(f - f0) * n;
        std::vector<int>& cnt = counts_of[f - f0];
        fold_positions(fp.test[f], n, at);
        for (int i = 0; i < n; ++i)
          if (at[i] >= 0) ++cnt[labels[i] - 1];
        std::vector<int> map(classes, 0);
        int next = 0;
        for (int c = 0; c < classes; ++c)
          if (cnt[c] > 0) map[c] = ++next;
        for (int i = 0; i < n; ++i)
          if (at[i] >= 0) lab[at[i]] = map[labels[i] - 1];
      }
      DeviceArray<int> pos(host_pos.size(), lanes.main), lab(host_lab.size(), lanes.main);
      FPLS_CHECK(cudaMemcpyAsync(pos.get(), host_pos.data(), sizeof(int) * host_pos.size(),
                                 cudaMemcpyHostToDevice, lanes.main));
      FPLS_CHECK(cudaMemcpyAsync(lab.get(), host_lab.data(), sizeof(int) * host_lab.size(),
                                 cudaMemcpyHostToDevice, lanes.main));
      lanes.lanes_after_main();
      std::vector<std::pair<int, int>> single;  // folds left with one class to learn, and that class
      std::vector<std::unique_ptr<Fold<T>>> batch;
      Results out;
      Settle settle{lanes};
      try {
        for (int f = f0; f < f1; ++f) {
          const auto& held = fp.test[f];
          if (held.empty()) {
            status[f] = 2;
            continue;
          }
          const std::vector<int>& cnt = counts_of[f - f0];
          std::vector<int> active;
          for (int c = 0; c < classes; ++c)
            if (cnt[c] > 0) active.push_back(c + 1);
          if (active.size() <= 1) {
            single.push_back({f, active.empty() ? 1 : active.front()});
            continue;
          }
          if (maximum_prefix > std::min(n - (int)held.size() - 1, p))
            throw std::invalid_argument("CUDA CV component count exceeds a fold rank");
          std::unique_ptr<Fold<T>> fold(new Fold<T>());
          Fold<T>& d = *fold;
          d.f = f;
          d.m = (int)active.size();
          d.active = active;
          d.st = lanes.of(batch.size());
          d.nte = (int)held.size();
          d.ntr = n - d.nte;
          d.pos = pos.get() + (size_t)(f - f0) * n;
          d.lab = lab.get() + (size_t)(f - f0) * n;
          split_fold(d, X.get(), static_cast<const T*>(nullptr), n, p, 0);
          d.ws.ensure(d.ntr, p, d.m, maximum_prefix, d.st);
          FPLS_CHECK(cudaMemsetAsync(d.ws.flag.get(), 0, sizeof(int), d.st));
          d.Yc.allocate((size_t)d.ntr * d.m, d.st);
          d.ycsum.allocate(d.m, d.st);
          d.model.classification = true;
          d.model.label_view = d.lab;
          for (int c : active) d.model.class_counts.push_back(cnt[c - 1]);
          d.model.ymean.allocate(d.m, d.st);
          prepare_responses<T>(nullptr, d.lab, d.ntr, d.m, d.Yc.get(), d.model.ymean.get(),
                               d.ycsum.get(), d.ws.flag.get(), d.st);
          fit_fold<T>(method, d, p, maximum_prefix, scaling, shape.max_ctas);
          batch.push_back(std::move(fold));
        }
      } catch (const OutOfMemory&) {
        throw;
      } catch (...) {
        failed = std::current_exception();  // after the folds before it
      }
      for (auto& fold : batch) {
        fold->at_labels = out.take(sizeof(int) * (size_t)fold->nte * prefix_count);
        fold->at_flag = out.take(sizeof(int));
      }
      out.dev.allocate(out.bytes, lanes.main);
      launch_plans(batch, lanes);
      lanes.lanes_after_main();
      std::vector<std::vector<double>> host_scores(batch.size());
      for (size_t b = 0; b < batch.size(); ++b) {
        Fold<T>& d = *batch[b];
        const int c = d.m;
        d.scores.allocate((size_t)d.nte * maximum_prefix, d.st);
        d.pred.allocate((size_t)d.nte * c * step, d.st);
        if (use_lda && store_scores) d.sums.allocate((size_t)d.nte * c * step, d.st);
        int* top = out.on_device<int>(d.at_labels);
        project_rows<T>(d.model, d.Xte.get(), d.nte, d.nte, maximum_prefix, d.scores.get(), d.nte, d.ws, d.st);
        if (use_lda) {
          d.lda.reset(new LdaState());
          d.lda->train(d.model.T.get(), d.ntr, d.ntr, maximum_prefix, d.lab, c, d.model.class_counts,
                       d.ws.flag.get(), d.st);
        }
        if (store_scores) host_scores[b].resize((size_t)d.nte * c * prefix_count);
        for (int j = 0; j < prefix_count; j += step) {
          const int w = std::min(step, prefix_count - j);
          // class indicators (stored, or decoded by the argmax head) and the
          // LDA discriminants
          double* resp = use_lda ? d.sums.get() : d.pred.get();
          if (store_scores || !use_lda)
            predict_prefixes<double>(d.model, d.scores.get(), d.nte, d.nte, prefixes + j, w, resp, d.st);
          if (use_lda) d.lda->discriminants(d.scores.get(), d.nte, d.nte, prefixes + j, w, d.pred.get(), d.st);
          topk_rows(d.pred.get(), d.nte, c, 1, w, top + (size_t)j * d.nte, d.nte, d.st);
          if (store_scores && step < prefix_count)
            FPLS_CHECK(cudaMemcpyAsync(host_scores[b].data() + (size_t)j * d.nte * c, resp,
                                       sizeof(double) * d.nte * c * w, cudaMemcpyDeviceToHost, d.st));
        }
      }
      // copies to pageable memory wait for their stream: after every fold is enqueued
      if (store_scores && step == prefix_count)
        for (size_t b = 0; b < batch.size(); ++b) {
          Fold<T>& d = *batch[b];
          FPLS_CHECK(cudaMemcpyAsync(host_scores[b].data(), use_lda ? d.sums.get() : d.pred.get(),
                                     sizeof(double) * host_scores[b].size(), cudaMemcpyDeviceToHost, d.st));
        }
      collect(batch, out, lanes);
      lanes.sync();
      for (const auto& [f, fallback] : single) {
        for (int j = 0; j < prefix_count; ++j)
          for (int r : fp.test[f]) {
            if (store_predictions) prediction_output[(size_t)j * n + r] = fallback;
            metrics[j] += labels[r] == fallback ? 1.0 : 0.0;
            counts[j] += 1.0;
          }
        status[f] = 4;
      }
      for (size_t b = 0; b < batch.size(); ++b) {
        Fold<T>& d = *batch[b];
        const int c = d.m;
        const auto& held = fp.test[d.f];
        const int* labels_of = out.on_host<int>(d.at_labels);
        if (*out.on_host<int>(d.at_flag))
          throw std::runtime_error(method == kPlssvd
              ? "resident PLS-SVD failed: invalid labels, decomposition or score Gram"
              : "resident SIMPLS failed: invalid labels, decomposition or component norm");
        for (int j = 0; j < prefix_count; ++j) {
          for (int i = 0; i < d.nte; ++i) {
            const int predicted = d.active[labels_of[(size_t)j * d.nte + i] - 1];
            const int row = held[i];
            if (store_predictions) prediction_output[(size_t)j * n + row] = predicted;
            metrics[j] += predicted == labels[row] ? 1.0 : 0.0;
            counts[j] += 1.0;
          }
          if (store_scores)
            for (int ai = 0; ai < c; ++ai) {
              const int dest = d.active[ai] - 1;
              for (int i = 0; i < d.nte; ++i)
                score_output[(size_t)j * n * classes + (size_t)dest * n + held[i]] =
                    static_cast<T>(host_scores[b][((size_t)j * c + ai) * d.nte + i]);
            }
        }
        status[d.f] = 1;
      }
      return failed;
    });
    for (int j = 0; j < prefix_count; ++j)
      metrics[j] = counts[j] > 0.0 ? metrics[j] / counts[j]
                                   : std::numeric_limits<double>::quiet_NaN();
  }
}

#define FPLS_INSTANTIATE(T)                                                     \
  template void cv_regression<T>(int, const T*, const T*, const int*, int, int, \
                                 int, const int*, int, int, int, bool, double*, \
                                 int*, double*, double*, double*, double*);     \
  template void cv_classification<T>(int, const T*, const int*, const int*,     \
                                     int, int, int, const int*, int, int, bool, \
                                     bool, bool, int*, T*, int*, double*);
FPLS_INSTANTIATE(float)
FPLS_INSTANTIATE(double)
#undef FPLS_INSTANTIATE

}  // namespace fpls
