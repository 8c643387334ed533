// Deterministic grid-wide reductions without spin-waiting: every block
// publishes its partial sums, the last block to arrive (ticket counter) adds
// all partials in block-index order and writes the result.
#pragma once

#include "common.cuh"

namespace fpls {

// vals: k block-level sums in shared memory (valid in every thread).
// partial: gridDim.x * k doubles of global scratch; counter: zero-initialised
// unsigned in global memory (reset to 0 by the last block). out: k doubles.
// Returns true in the block that wrote `out`. Blocks of at most
// kReduceThreads threads. The last block's threads share each value's
// partials: Q of them per value sum blocks q, q + Q, ... (eight loads in
// flight), then those sums are added in order; one thread per value with its
// loads one after another was most of a p-vector kernel's time (60 values of
// 40 blocks: 28 of 31 us).
constexpr int kReduceThreads = 256;
__device__ inline bool last_block_reduce(const double* vals, int k,
                                         double* partial, unsigned* counter,
                                         double* out) {
  __shared__ bool am_last;
  __shared__ double part[kReduceThreads];
  for (int i = threadIdx.x; i < k; i += blockDim.x)
    partial[(long)blockIdx.x * k + i] = vals[i];
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned ticket = atomicAdd(counter, 1u);
    am_last = (ticket == gridDim.x - 1);
  }
  __syncthreads();
  if (!am_last) return false;
  __threadfence();
  const int blocks = (int)gridDim.x;
  for (int base = 0; base < k; base += blockDim.x) {
    const int w = min(k - base, (int)blockDim.x);
    const int Q = min((int)blockDim.x / w, (blocks + 7) / 8);
    const int i = threadIdx.x % w, q = threadIdx.x / w;
    if (q < Q) {
      double s = 0.0;
#pragma unroll 8
      for (int b = q; b < blocks; b += Q) s += __ldcg(&partial[(long)b * k + base + i]);
      part[threadIdx.x] = s;
    }
    __syncthreads();
    if (threadIdx.x < w) {
      double s = part[threadIdx.x];
      for (int u = 1; u < Q; ++u) s += part[u * w + threadIdx.x];
      out[base + threadIdx.x] = s;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) *counter = 0u;
  return true;
}

}  // namespace fpls
