// How the folds of a cross-validation are grouped (no CUDA here, so that the
// rule can be tested on the host).
#pragma once

#include <algorithm>

namespace fpls {

struct CvBatches {
  int per_batch = 1;  // folds resident at a time
  int max_ctas = 0;   // persistent CTAs of each (0: no shared launch)
};

// folds: their number; fold_bytes: device memory of one; device_bytes: of the
// device; capacity: co-resident persistent CTAs; alone: a fold takes a launch of
// its own; ctas(share): CTAs a fold takes out of a share; free_bytes(): asked
// only when the folds take more than a 64th of the device, since the query is
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
  if (out.per_batch * fold_bytes > device_bytes / 64)
    out.per_batch = std::min(out.per_batch, (int)std::max(1.0, std::min((double)folds, 0.25 * free_bytes() / fold_bytes)));
  return out;
}

}  // namespace fpls
