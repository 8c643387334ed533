// How the folds of a cross-validation are grouped (no CUDA here, so that the
// rule can be tested on the host).
#pragma once

#include <algorithm>

namespace fpls {

constexpr int kLanes = 4;

// Streams beside the main one that the folds of a batch are spread over (0:
// everything on the main one). Folds whose component loop is a chain of small
// kernels overlap on lanes; the others have no chain to hide, and lanes cost
// them: an allocation that takes a block last used on another stream is about
// 10 us instead of 0.6, some 30 a fold, and a stream about 0.14 ms to make and
// destroy. us a call with no lane / four lanes (one fold after another before
// the batches): 246 x 62, 5 folds 640 / 1620 (1090); PLS-SVD 288 x 7, 60 folds
// 7000 / 26300 (12800); 601 x 1500, 10 folds 2080 / 3120 (9380). With the loop as
// kernels: 60 x 40, 40 responses, 6 components, 10 folds 9950 / 4580 (22900);
// 3000 x 200 in 12 classes, 10 components, 10 folds 9900 / 6980 (30200).
inline int fold_lanes(int folds, bool kernel_loops) { return kernel_loops ? std::min(folds, kLanes) : 0; }

struct CvBatches {
  int per_batch = 1;  // folds resident at a time
  int max_ctas = 0;   // persistent CTAs of each (0: no shared launch)
};

// folds: their number; fold_bytes: device memory of one; device_bytes: of the
// device; capacity: co-resident persistent CTAs; alone: a fold takes a launch of
// its own; ctas(share): CTAs a fold takes out of a share; free_bytes(): asked
// only when the folds take more than a 32nd of the device, since the query is
// a call into the driver that other processes' calls hold up (66 to 220 us at
// the median, 2 ms at the 90th percentile and 30 to 60 at the 99th on a shared
// host, where a small cross-validation takes 0.5 ms).
//
// The CTA share decides how a fold's sums are split, so it follows from the
// shape, the number of folds and the device alone: as many folds as 8 GB and
// the co-resident CTAs hold, in batches of equal size. Free memory (a quarter
// of it, at least one fold) only lowers how many of them are resident at a time.
template <class Ctas, class Free>
CvBatches cv_batches(int folds, double fold_bytes, double device_bytes, int capacity, bool alone, Ctas&& ctas,
                     Free&& free_bytes) {
  CvBatches out;
  int most = alone ? 1 : (int)std::max(1.0, std::min((double)folds, 8e9 / fold_bytes));
  if (capacity >= 0) {
    while (most > 1 && most * ctas(capacity / most) > capacity) --most;
    if (capacity > 0) out.max_ctas = capacity / most;
  }
  const int batches = (folds + most - 1) / most;
  out.per_batch = (folds + batches - 1) / batches;
  if (out.per_batch * fold_bytes > device_bytes / 32)
    out.per_batch = std::min(out.per_batch, (int)std::max(1.0, std::min((double)folds, 0.25 * free_bytes() / fold_bytes)));
  return out;
}

}  // namespace fpls
