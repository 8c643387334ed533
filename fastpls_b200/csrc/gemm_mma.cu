// FP64 GEMM on the FP64 tensor-core path (DMMA, mma.sync m16n8k8 f64).
//
//   C[M x N] = alpha * op(A)[M x K] * op(B)[K x N] (+ beta C), column-major;
//   op(X) = X or X^T, A and B both FP64 or both FP32, or (A predictors, B
//   not transposed) A FP32 or BF16 and B FP64; narrow types are widened
//   exactly as the fragments are loaded, every product and sum is FP64.
//
// B200 has no tcgen05 kind for FP64; its FP64 tensor path is the warp-level
// DMMA instruction (36.8 to 37.0 TFLOP/s measured for every shape from m8n8k4
// to m16n8k16, the rate of DFMA, but one instruction does 1024 FMAs from
// register fragments, so shared-memory and issue bandwidth stop being the
// limit of a SIMT register-tiled kernel).
//
// Block tile TM x TN x 16, 8 warps. Operand slabs stream through a 4-stage
// cp.async ring: 16-byte copies when the operand's base and column stride
// are 16-byte multiples, one element per copy otherwise (odd row counts,
// which a SIMT kernel took before), zero-filled outside the matrix either
// way. Shared layouts are padded so that fragment loads are conflict-free:
// k-major [16][T + pad] for operands contiguous along M or N (row stride
// 4 mod 16 doubles or 8 mod 32 floats), row-major [T][20] ([T][24]
// for BF16) for operands contiguous along K. `lower` restricts the grid to the lower triangle of
// square block tiles (symmetric products such as the Gram X X^T).
//
// The tile and the K splits come from gemm_plan (gemm.cu): most products of
// this library are far from square -- a sketch of 41 columns, a 41 x 41 Gram
// over 3000 rows, a 500 x 500 Gram over 40000 -- so narrow tiles and slices
// over K are what fill the SMs. 128 x 128 alone and whole K left a 41 x 41
// Gram over 3001 rows on one SM.
#include "common.cuh"
#include "gemm_mma.cuh"
#include "kernels.cuh"

#include <algorithm>

namespace fpls {

namespace {

constexpr int TK = 16, STAGES = 4, NT = 256;

// Elements per row of a k-major slab [TK][row] / of a row-major slab [T][TK + 4].
template <class T>
constexpr int row_pad(int t) {
  return t + (sizeof(T) == 8 ? 4 : 8);
}
template <class T>
constexpr int row_stride() {  // 16-byte multiples, conflict-free
  return TK + (sizeof(T) == 2 ? 8 : 4);
}

template <class T>
constexpr int slab_elems(bool kcontig, int t) {
  return kcontig ? t * row_stride<T>() : TK * row_pad<T>(t);
}

// Copies of 16 bytes (or one element) with the bytes past `bytes` zero-filled.
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, int bytes) {
  const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(bytes));
}
__device__ __forceinline__ void cp_async1(double* smem, const double* gmem, bool ok) {
  const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s), "l"(gmem), "r"(ok ? 8 : 0));
}
__device__ __forceinline__ void cp_async1(float* smem, const float* gmem, bool ok) {
  const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(s), "l"(gmem), "r"(ok ? 4 : 0));
}
__device__ __forceinline__ void cp_async1(bf16* smem, const bf16* gmem, bool ok) {
  // cp.async copies no less than 4 bytes: a plain store, ordered by the
  // barrier that ends the stage's wait
  *smem = ok ? *gmem : __ushort_as_bfloat16((unsigned short)0);
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

// D += A B: A 16 x 8 (a[i]: row g + 8 (i & 1), k tg + 4 (i >> 1)), B 8 x 8
// (b[i]: k tg + 4 i, column g), C rows g, g + 8 and columns 2 tg, 2 tg + 1.
__device__ __forceinline__ void dmma(double (&c)[4], const double (&a)[4], const double (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}

// One slab (TR rows of op(X) by TK of k) into shared memory. Element (r, k)
// is X[k + r ld] when KCONTIG, X[r + k ld] otherwise.
template <class T, bool KCONTIG, int TR>
__device__ __forceinline__ void load_slab(T* s, const T* __restrict__ X, long ld, int rows, int kend,
                                          int r0, int k0, bool vec) {
  constexpr int V = 16 / (int)sizeof(T);
  const int tid = threadIdx.x;
  if (vec) {
    constexpr int CH = TR * TK / V;
#pragma unroll
    for (int it = 0; it < (CH + NT - 1) / NT; ++it) {
      const int c = tid + it * NT;
      if (CH % NT != 0 && c >= CH) break;
      if (KCONTIG) {
        const int r = c / (TK / V), k = (c % (TK / V)) * V;
        const int left = r0 + r < rows ? min(V, max(0, kend - (k0 + k))) : 0;
        cp_async16(s + r * row_stride<T>() + k, left ? X + (k0 + k) + (long)(r0 + r) * ld : X, left * (int)sizeof(T));
      } else {
        const int k = c / (TR / V), r = (c % (TR / V)) * V;
        const int left = k0 + k < kend ? min(V, max(0, rows - (r0 + r))) : 0;
        cp_async16(s + k * row_pad<T>(TR) + r, left ? X + (r0 + r) + (long)(k0 + k) * ld : X,
                   left * (int)sizeof(T));
      }
    }
  } else {
    constexpr int CH = TR * TK;
    static_assert(CH % NT == 0, "whole passes of element copies");
#pragma unroll
    for (int it = 0; it < CH / NT; ++it) {
      const int c = tid + it * NT;
      if (KCONTIG) {
        const int r = c / TK, k = c % TK;
        const bool ok = r0 + r < rows && k0 + k < kend;
        cp_async1(s + r * row_stride<T>() + k, ok ? X + (k0 + k) + (long)(r0 + r) * ld : X, ok);
      } else {
        const int k = c / TR, r = c % TR;
        const bool ok = r0 + r < rows && k0 + k < kend;
        cp_async1(s + k * row_pad<T>(TR) + r, ok ? X + (r0 + r) + (long)(k0 + k) * ld : X, ok);
      }
    }
  }
}

template <class T, bool KCONTIG, int TR>
__device__ __forceinline__ double slab_at(const T* s, int r, int k) {
  return as_f64(KCONTIG ? s[r * row_stride<T>() + k] : s[k * row_pad<T>(TR) + r]);
}

// A_T: A stored K x M (contiguous along K); B_T: B stored N x K (contiguous
// along N).
template <class TA, class TB, bool A_T, bool B_T, int TM, int TN>
__global__ void __launch_bounds__(NT, TM * TN >= 128 * 128 ? 1 : 2)
    dgemm_mma(int M, int N, int K, const TA* __restrict__ A, long lda, const TB* __restrict__ B,
              long ldb, double alpha, double beta, double* __restrict__ C, long ldc,
              long split_stride, int k_per_split, int lower, int vec,
              const double* __restrict__ coff, int coff_parts) {
  constexpr int WARPS_N = TN == 128 ? 4 : TN == 64 ? 2 : 1;
  constexpr int WARPS_M = 8 / WARPS_N;
  constexpr int WM = TM / WARPS_M, WN = TN / WARPS_N;
  constexpr int MT = WM / 16, NTL = WN / 8;
  static_assert(WM % 16 == 0 && WN % 8 == 0, "whole DMMA tiles per warp");
  constexpr int SA = slab_elems<TA>(A_T, TM), SB = slab_elems<TB>(!B_T, TN);
  static_assert(STAGES * SA * sizeof(TA) % 16 == 0, "B slabs stay 16-byte aligned");
  extern __shared__ __align__(16) unsigned char gemm_smem[];
  TA* As = reinterpret_cast<TA*>(gemm_smem);  // STAGES slabs of A, then of B
  TB* Bs = reinterpret_cast<TB*>(As + STAGES * SA);

  int bm, bn;
  if (lower) {
    // blockIdx.x enumerates lower-triangular tile pairs (bm >= bn)
    const int t = blockIdx.x;
    bm = (int)((sqrt(8.0 * t + 1.0) - 1.0) * 0.5);
    while (bm * (bm + 1) / 2 > t) --bm;
    while ((bm + 1) * (bm + 2) / 2 <= t) ++bm;
    bn = t - bm * (bm + 1) / 2;
  } else {
    bn = blockIdx.x;
    bm = blockIdx.y;
  }
  const int m0 = bm * TM, n0 = bn * TN;
  const int kbeg = min(K, (int)blockIdx.z * k_per_split);
  const int kend = min(K, kbeg + k_per_split);
  const int ktiles = (kend - kbeg + TK - 1) / TK;
  double* Cz = C + (long)blockIdx.z * split_stride;

  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int wm = (warp / WARPS_N) * WM, wn = (warp % WARPS_N) * WN;

  auto load_stage = [&](int stage, int kt) {
    load_slab<TA, A_T, TM>(As + stage * SA, A, lda, M, kend, m0, kbeg + kt * TK, vec & 1);
    load_slab<TB, !B_T, TN>(Bs + stage * SB, B, ldb, N, kend, n0, kbeg + kt * TK, vec & 2);
  };

  double acc[MT][NTL][4];
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int j = 0; j < NTL; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.0;

#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < ktiles) load_stage(s, s);
    cp_commit();
  }
  const int g = lane >> 2, tg = lane & 3;
  for (int kt = 0; kt < ktiles; ++kt) {
    cp_wait<STAGES - 2>();
    __syncthreads();
    const int pre = kt + STAGES - 1;
    if (pre < ktiles) load_stage(pre % STAGES, pre);
    cp_commit();
    const TA* as = As + (kt % STAGES) * SA;
    const TB* bs = Bs + (kt % STAGES) * SB;
#pragma unroll
    for (int kk = 0; kk < TK; kk += 8) {
      double af[MT][4], bf[NTL][2];
#pragma unroll
      for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          af[i][e] = slab_at<TA, A_T, TM>(as, wm + i * 16 + g + 8 * (e & 1), kk + tg + 4 * (e >> 1));
#pragma unroll
      for (int j = 0; j < NTL; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) bf[j][e] = slab_at<TB, !B_T, TN>(bs, wn + j * 8 + g, kk + tg + 4 * e);
#pragma unroll
      for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NTL; ++j) dmma(acc[i][j], af[i], bf[j]);
    }
  }
  cp_wait<0>();

#pragma unroll
  for (int j = 0; j < NTL; ++j)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int col = n0 + wn + j * 8 + tg * 2 + h;
      if (col >= N) continue;
      const double off = coff ? column_offset(coff, coff_parts, col) : 0.0;
#pragma unroll
      for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int row = m0 + wm + i * 16 + g + 8 * e;
          if (row < M) {
            double* dst = Cz + row + (long)col * ldc;
            const double v = alpha * acc[i][j][2 * e + h] - off;
            *dst = beta != 0.0 ? fma(beta, *dst, v) : v;
          }
        }
    }
}

bool aligned16(const void* p, long ld, size_t es) {
  return (reinterpret_cast<uintptr_t>(p) & 15u) == 0 && (ld * (long)es) % 16 == 0;
}

// Where the result goes: C, or the slices over K.
struct Target {
  double* C;
  long ldc, stride;
  double alpha, beta;
  const double* coff;
};

template <class TA, class TB, bool A_T, bool B_T, int TM, int TN>
void launch(const GemmArgs& g, const GemmPlan& plan, const Target& t, cudaStream_t stream) {
  constexpr size_t smem = (size_t)STAGES * (slab_elems<TA>(A_T, TM) * sizeof(TA) +
                                            slab_elems<TB>(!B_T, TN) * sizeof(TB));
  allow_shared_memory((const void*)dgemm_mma<TA, TB, A_T, B_T, TM, TN>);
  const int kps = ((g.K + plan.splits - 1) / plan.splits + TK - 1) / TK * TK;
  const unsigned tm = ceil_div(g.M, TM), tn = ceil_div(g.N, TN);
  const dim3 grid = g.lower ? dim3(tm * (tm + 1) / 2, 1, plan.splits) : dim3(tn, tm, plan.splits);
  const int vec = (aligned16(g.A, g.lda, sizeof(TA)) ? 1 : 0) | (aligned16(g.B, g.ldb, sizeof(TB)) ? 2 : 0);
  dgemm_mma<TA, TB, A_T, B_T, TM, TN><<<grid, NT, smem, stream>>>(
      g.M, g.N, g.K, static_cast<const TA*>(g.A), g.lda, static_cast<const TB*>(g.B), g.ldb, t.alpha,
      t.beta, t.C, t.ldc, t.stride, kps, g.lower ? 1 : 0, vec, t.coff, g.coff_parts);
  count_launch();
  FPLS_LAUNCH("dgemm_mma");
}

template <class TA, class TB, bool A_T, bool B_T>
void by_tile(const GemmArgs& g, const GemmPlan& pl, const Target& t, cudaStream_t s) {
  if (pl.tm == 64) launch<TA, TB, A_T, B_T, 64, 64>(g, pl, t, s);
  else if (pl.tn == 128) launch<TA, TB, A_T, B_T, 128, 128>(g, pl, t, s);
  else if (pl.tn == 64) launch<TA, TB, A_T, B_T, 128, 64>(g, pl, t, s);
  else if (pl.tn == 32) launch<TA, TB, A_T, B_T, 128, 32>(g, pl, t, s);
  else launch<TA, TB, A_T, B_T, 128, 16>(g, pl, t, s);
}

template <class T>
void by_layout(const GemmArgs& g, const GemmPlan& pl, const Target& t, cudaStream_t s) {
  if (g.trans_a) {
    if (g.trans_b) by_tile<T, T, true, true>(g, pl, t, s);
    else by_tile<T, T, true, false>(g, pl, t, s);
  } else {
    if (g.trans_b) by_tile<T, T, false, true>(g, pl, t, s);
    else by_tile<T, T, false, false>(g, pl, t, s);
  }
}

}  // namespace

void gemm_mma_launch(const GemmArgs& g, const GemmPlan& plan, double* C, long ldc, long split_stride,
                     double alpha, double beta, const double* coff, cudaStream_t stream) {
  const Target t{C, ldc, split_stride, alpha, beta, coff};
  if (g.a_type == g.b_type) {
    require(g.a_type != GemmType::kBf16, "FP64 GEMM: unsupported operand types");
    if (g.a_type == GemmType::kF32) by_layout<float>(g, plan, t, stream);
    else by_layout<double>(g, plan, t, stream);
    return;
  }
  require(g.b_type == GemmType::kF64 && !g.trans_b, "FP64 GEMM: unsupported operand types");
  if (g.a_type == GemmType::kF32) {
    if (g.trans_a) by_tile<float, double, true, false>(g, plan, t, stream);
    else by_tile<float, double, false, false>(g, plan, t, stream);
  } else {
    if (g.trans_a) by_tile<bf16, double, true, false>(g, plan, t, stream);
    else by_tile<bf16, double, false, false>(g, plan, t, stream);
  }
}

}  // namespace fpls
