// Kernel launchers of the fitting library (declarations).
#pragma once

#include "common.cuh"

namespace fpls {

// ---------------------------------------------------------------- gemm.cu
// A and B of one type (FP64 or FP32, any transposes), or A FP32 / BF16 and B
// FP64 (B not transposed).
enum class GemmType { kF64, kF32, kBf16 };
template <class T> struct gemm_type;
template <> struct gemm_type<double> { static constexpr GemmType value = GemmType::kF64; };
template <> struct gemm_type<float> { static constexpr GemmType value = GemmType::kF32; };
template <> struct gemm_type<bf16> { static constexpr GemmType value = GemmType::kBf16; };
struct GemmArgs {
  int M = 0, N = 0, K = 0;
  const void* A = nullptr;
  long lda = 0;
  const void* B = nullptr;
  long ldb = 0;
  GemmType a_type = GemmType::kF64, b_type = GemmType::kF64;
  bool trans_a = false, trans_b = false;
  double alpha = 1.0, beta = 0.0;
  double* C = nullptr;
  long ldc = 0;
  bool lower = false;  // symmetric result: compute the lower tiles, mirror
  // K per slice when the sums' order must not depend on M and N (0: planned);
  // only a result past 256 MB of slices takes longer ones
  int k_slice = 0;
  // subtracted from every row of the product: column c's value is the sum, in
  // order, of coff[c * coff_parts ..] (coff_parts values); null: nothing
  const double* coff = nullptr;
  int coff_parts = 1;
};
__device__ __forceinline__ double column_offset(const double* coff, int parts, int c) {
  double s = coff[(long)c * parts];
  for (int k = 1; k < parts; ++k) s += coff[(long)c * parts + k];
  return s;
}
void gemm_f64(const GemmArgs& g, cudaStream_t stream);
void gemm_profile_enable(bool on);
void mirror_lower_triangle(double* C, int n, long ldc, cudaStream_t stream);
void gemm_profile_read(double* ms, double* flops, unsigned long long* launches);

// Stream that the batched entry points run on when the caller set one
// (fastpls_b200_set_stream); nullptr means "create a private stream".
cudaStream_t& caller_stream();

// Measured FP64 FMA throughput of the device (TFLOP/s), probe.cu.
double fp64_fma_tflops();

// -------------------------------------------------------------- stream.cu
// Column moments of X (n x p, column-major, leading dimension ld):
// sum[j], sumsq[j] and cross[j + c*p] = sum_i X[i,j] * Yc[i,c] (FP64),
// Yc an n x m FP64 column-major block (m may be 0). One pass over X.
template <class T>
void column_moments(const T* X, int n, int p, long ld, const double* Yc, int m,
                    double* sum, double* sumsq, double* cross,
                    DeviceArray<double>& scratch, cudaStream_t stream);

// Classification: sum[j], sumsq[j] and cross[j + c*p] = X^T (onehot - prior)
// from one-based labels (n), classes m <= kClassMomentsMaxClasses, in one
// pass over X (per-class column sums minus prior * column sum).
constexpr int kClassMomentsMaxClasses = 32;
template <class T>
void class_moments(const T* X, int n, int p, long ld, const int* labels, int m,
                   const double* prior, double* sum, double* sumsq, double* cross,
                   DeviceArray<double>& scratch, cudaStream_t stream);

// Sum of squares and sum of the (one) column xr_product writes, into out[0]
// and out[1]; partial: scratch of kXrStatsPartial doubles, counter: a
// last_block_reduce ticket.
constexpr int kXrStatsPartial = 4096;
struct XrStats {
  double* partial;
  unsigned* counter;
  double* out;
};

// out[i + c*n] = sum_j X[i,j] * R[j + c*ldr] - offset_c   (c < nb)
// (scores of a scaled/centred X folded into R and offset); offset_c is the sum
// of offset[c * offset_parts ..] (offset null: 0). FP64 result, nb = 1 or 2
// (HBM-bound); wider products are FP64-bound and run as GEMMs. finite: X holds
// no infinity or NaN (finite_f64; one column).
template <class T>
void xr_product(const T* X, int n, int p, long ld, const double* R, long ldr,
                int nb, const double* offset, int offset_parts, double* out, long ldo,
                DeviceArray<double>& scratch, cudaStream_t stream, const XrStats* stats = nullptr,
                bool finite = false);

// The one-pass form of xr_product for 3 <= nb <= 16 columns (persistent.cu):
// X streamed once through the single fit's bulk-copy stages, each stage also
// carrying its rows of R. flag is set to 5 if a stage never arrives (a bounded
// wait ran out). Returns false (nothing enqueued) for shapes it does not take.
template <class T>
bool xr_ring(const T* X, int n, int p, long ld, const double* R, long ldr, int nb,
             const double* offset, int offset_parts, double* out, long ldo, int* flag,
             cudaStream_t stream);

// out[j + c*p] = sum_i X[i,j] * V[i + c*ldv]   (c < nb, FP64). finite: X holds
// no infinity or NaN (finite_f64; used at one column).
template <class T>
void xtv_product(const T* X, int n, int p, long ld, const double* V, long ldv,
                 int nb, double* out, long ldo, DeviceArray<double>& scratch,
                 cudaStream_t stream, bool finite = false);

// ---------------------------------------------------------------- misc
// One-based top-k per row of `count` consecutive column-major (rows x classes)
// FP64 matrices (out: ldo x top each); the lower class index wins ties
// (strict '>' scan). count <= 65535.
void topk_rows(const double* values, int rows, int classes, int top, int count, int* out,
               long ldo, cudaStream_t stream);

}  // namespace fpls
