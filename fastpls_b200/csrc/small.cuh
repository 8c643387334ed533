// Small dense FP64 linear algebra executed inside one block (device code).
#pragma once

#include "common.cuh"

namespace fpls {

// Jacobi eigen-decomposition of a symmetric m x m matrix (m <= 128) held in
// shared memory (column-major A[i + j*m]); eigenvectors accumulate in E.
// Parallel ordering (Brent-Luk round robin): each sweep runs m - 1 (m even)
// or m (m odd) rounds of up to m / 2 disjoint rotations. All threads of the
// block cooperate (every thread must call it, with the same arguments): the
// rotations of a round are computed one per thread into shared memory, then
// applied together: every pair of rotations (k1, k2) owns the 2 x 2 block of A
// in rows p1, q1 and columns p2, q2, takes both its sides at once in registers
// and stores the block and its mirror image, beside the column rotations of E.
// Rotations of one round touch disjoint rows and columns, so a rotation's own
// 2 x 2 block is unchanged by the others of its round; its off-diagonal pair
// is annihilated (tangent of the smaller root of t^2 + 2 theta t = 1, theta =
// (a_qq - a_pp) / (2 a_pq)). Latency-bound: two barriers and one rotation's
// chain of two reciprocal square roots per round.
// Columns of A and E and then rows of A, a barrier between them and all of A
// twice, took 498 us at m = 41 (fastsvd's Gram) against 364 us now.
// Stops at off <= 1e-30 diag (sums of squares) or at the rounding floor.
// Returns the number of sweeps used (<= max_sweeps). Matrices of order
// m <= warp_limit run in the first warp alone.
constexpr int kJacobiMaxRotations = 64;
// its static arrays: rotations and the block sum's scratch
constexpr int kJacobiStaticBytes = kJacobiMaxRotations * 2 * (int)(sizeof(int) + sizeof(double)) + 32 * 8;

// threads for a block that runs jacobi_eigen on an m x m matrix
inline unsigned jacobi_threads(int m) { return m > 32 ? 512u : m > 16 ? 256u : 64u; }

__device__ inline int jacobi_eigen(double* A, double* E, int m, int max_sweeps = 40, int warp_limit = 8) {
  __shared__ int rot_p[kJacobiMaxRotations], rot_q[kJacobiMaxRotations];
  __shared__ double rot_c[kJacobiMaxRotations], rot_s[kJacobiMaxRotations];
  __shared__ double red[32];
  if (m > 2 * kJacobiMaxRotations) return 0;  // callers keep m <= 128
  // small matrices (m <= warp_limit): the first warp alone (warp barriers
  // are cheaper than block barriers on the latency-bound path); the other
  // threads wait at the final barrier
  const bool warp_only = m <= warp_limit;
  if (warp_only && threadIdx.x >= 32) {
    __syncthreads();
    return 0;
  }
  const int tid = threadIdx.x, nt = warp_only ? 32 : (int)blockDim.x;
  auto sync = [&]() {
    if (warp_only) __syncwarp();
    else __syncthreads();
  };
  auto total = [&](double v) { return warp_only ? warp_sum(v) : block_sum(v, red); };
  for (int k = tid; k < m * m; k += nt) E[k] = (k % m == k / m) ? 1.0 : 0.0;
  sync();
  const int players = m + (m & 1);  // odd m: one index sits a round out
  const int half = players / 2;     // rotations per round (<= 64)
  const int wrap = players - 1;
  // pairs of rotations: (k, k + d mod half) for d = 0 .. half / 2, the last
  // distance of an even half once only
  const int dmax = half / 2;
  const int pairs = half * dmax + (half & 1 ? half : half / 2);
  const int work = half * m;  // column rotations of E: (rotation, row)
  // this thread's first items and the steps between them: pair (k, k + d), and
  // (from the other end of the block, which has fewer pairs) E's (k, i)
  const int pk0 = tid % half, pd0 = tid / half, pdk = nt % half, pdd = nt / half;
  const int et = nt - 1 - tid;
  const int ek0 = et / m, ei0 = et % m, edk = nt / m, edi = nt % m;
  int sweep = 0;
  double prev = 0.0;
  int shift = 0;  // A is held times 2^-shift
  auto masses = [&](double& off, double& diag) {
    off = diag = 0.0;
    for (int k = tid; k < m * m; k += nt) {
      const int i = k % m, j = k / m;
      if (i != j) off += A[k] * A[k];
      else diag += A[k] * A[k];
    }
    off = total(off);
    diag = total(diag);
  };
  for (; sweep < max_sweeps && m > 1; ++sweep) {
    double off, diag;
    masses(off, diag);
    if (sweep == 0 && !(diag > 0x1p-800 && diag < 0x1p800)) {
      // entries whose squares vanish or pass the range (data of about 1e-60 or
      // 1e60 and beyond): the stopping rule would see nothing to do
      double top = 0.0;
      for (int k = 0; k < m * m; ++k) top = fmax(top, fabs(A[k]));
      sync();
      if (top > 0.0 && isfinite(top)) {
        shift = ilogb(top);
        for (int k = tid; k < m * m; k += nt) A[k] = scalbn(A[k], -shift);
        sync();
        masses(off, diag);
      }
    }
    if (off <= 1e-30 * diag || off == 0.0) break;
    // at the rounding floor (large m) the off-diagonal mass stops shrinking
    if (sweep > 0 && off <= 1e-24 * diag && off > 0.25 * prev) break;
    prev = off;
    for (int round = 0; round < wrap; ++round) {
      for (int slot = tid; slot < half; slot += nt) {
        // circle method: player players-1 fixed, the others rotate
        int a = slot == 0 ? wrap : round + slot;
        if (slot != 0 && a >= wrap) a -= wrap;
        int b = round - slot;
        if (b < 0) b += wrap;
        if (a > b) {
          const int t = a;
          a = b;
          b = t;
        }
        double c = 1.0, s = 0.0;
        if (b < m) {
          const double apq = A[a + b * m];
          if (apq != 0.0) {
            // theta = d / e, d = a_qq - a_pp, e = 2 a_pq; with h = sqrt(d^2
            // + e^2) the half-angle forms c^2 = (1 + |d| / h) / 2 and
            // s = sgn(d) e / (2 c h): two reciprocal square roots on the
            // dependent path
            double d = A[b + b * m] - A[a + a * m], e = 2.0 * apq;
            double h2 = fma(d, d, e * e);
            // h^2 outside [2^-900, 2^901): the squares lose bits, vanish or
            // pass the range. The angle does not depend on a common factor,
            // so both legs are brought near 1 by a power of two (the test
            // costs 7 of 314 us at m = 41).
            if ((unsigned)(__double2hiint(h2) - (123 << 20)) >= (1801u << 20)) {
              const double f = h2 < 1.0 ? 0x1p600 : 0x1p-600;
              d *= f;
              e *= f;
              h2 = fma(d, d, e * e);
            }
            const double rh = rsqrt(h2);
            const double c2 = fma(0.5 * fabs(d), rh, 0.5);
            const double rc = rsqrt(c2);
            c = c2 * rc;
            s = (d >= 0 ? 0.5 : -0.5) * e * rh * rc;
          }
        } else {
          b = -1;  // index a sits out
        }
        rot_p[slot] = a;
        rot_q[slot] = b;
        rot_c[slot] = c;
        rot_s[slot] = s;
      }
      sync();
      for (int w = tid, pk = pk0, pd = pd0; w < pairs; w += nt) {
        const int k1 = pk;
        int k2 = k1 + pd;
        if (k2 >= half) k2 -= half;
        pk += pdk;
        pd += pdd;
        if (pk >= half) {
          pk -= half;
          ++pd;
        }
        const int p1 = rot_p[k1], q1 = rot_q[k1], p2 = rot_p[k2], q2 = rot_q[k2];
        const double c1 = rot_c[k1], s1 = rot_s[k1], c2 = rot_c[k2], s2 = rot_s[k2];
        if (s1 == 0.0 && s2 == 0.0) continue;
        const bool two1 = q1 >= 0, two2 = q2 >= 0;
        const double app = A[p1 + p2 * m];
        const double apq = two2 ? A[p1 + q2 * m] : 0.0;
        const double aqp = two1 ? A[q1 + p2 * m] : 0.0;
        const double aqq = two1 && two2 ? A[q1 + q2 * m] : 0.0;
        // columns (J2), then rows (J1)
        const double xpp = c2 * app - s2 * apq, xpq = s2 * app + c2 * apq;
        const double xqp = c2 * aqp - s2 * aqq, xqq = s2 * aqp + c2 * aqq;
        const double ypp = c1 * xpp - s1 * xqp, yqp = s1 * xpp + c1 * xqp;
        const double ypq = c1 * xpq - s1 * xqq, yqq = s1 * xpq + c1 * xqq;
        if (k1 == k2) {
          A[p1 + p1 * m] = ypp;
          A[q1 + q1 * m] = yqq;
          A[p1 + q1 * m] = 0.0;
          A[q1 + p1 * m] = 0.0;
        } else {
          A[p1 + p2 * m] = ypp;
          A[p2 + p1 * m] = ypp;
          if (two2) {
            A[p1 + q2 * m] = ypq;
            A[q2 + p1 * m] = ypq;
          }
          if (two1) {
            A[q1 + p2 * m] = yqp;
            A[p2 + q1 * m] = yqp;
          }
          if (two1 && two2) {
            A[q1 + q2 * m] = yqq;
            A[q2 + q1 * m] = yqq;
          }
        }
      }
      for (int w = et, ek = ek0, ei = ei0; w < work; w += nt) {
        const int k = ek, i = ei;
        ek += edk;
        ei += edi;
        if (ei >= m) {
          ei -= m;
          ++ek;
        }
        const double sk = rot_s[k];
        if (sk != 0.0) {
          const int pk = rot_p[k], qk = rot_q[k];
          const double ck = rot_c[k];
          const double ekp = E[i + pk * m], ekq = E[i + qk * m];
          E[i + pk * m] = ck * ekp - sk * ekq;
          E[i + qk * m] = sk * ekp + ck * ekq;
        }
      }
      sync();
    }
  }
  if (shift != 0) {
    sync();
    for (int i = tid; i < m; i += nt) A[i + i * m] = scalbn(A[i + i * m], shift);
  }
  __syncthreads();
  return sweep;
}

// Dominant eigenpair of a symmetric positive semidefinite m x m matrix A
// (shared, column-major), whole block. Repeated squaring: B = A / tr(A),
// then B <- B^2 / tr(B^2). For B of trace one, tr(B^2) is the sum of its
// squared eigenvalues, 1 exactly when B has rank one; each squaring raises
// the eigenvalue ratios to the power two, so once tr(B^2) >= 1 - 1e-12 two
// more squarings leave the non-dominant part below rounding. Then v = the
// column of B with the largest diagonal entry, normalised (B = v v^T up to
// rounding), and lam = v^T A v. On random SPD matrices up to 32 x 32
// (clustered, rank one, condition 1e12) the residual |A v - lam v| / |A|
// stays below 1e-15 in about 13 squarings (at most 64; an exactly repeated
// leading eigenvalue yields a vector of its eigenspace). B and C are m x m
// shared scratch (C with one extra slot), v (m + 1 slots) the shared
// output; lam is returned in every thread. Returns false when tr(A) is not
// positive and finite.
// dominant_pair for order M <= 4 in one thread's registers: the same
// operations in the same order as the shared-memory form below (so the same
// bits), without its barriers. A is read from shared memory; v (M + 1) and
// C[M] receive the result as in that form.
template <int M>
__device__ inline void dominant_pair_regs(const double* A, double* C, double* v, int max_squarings) {
  double a[M * M], b[M * M], c[M * M];
#pragma unroll
  for (int k = 0; k < M * M; ++k) a[k] = A[k];
  double tr = 0.0;
#pragma unroll
  for (int i = 0; i < M; ++i) tr += a[i * (M + 1)];
  if (!(tr > 0.0) || !isfinite(tr)) {
    v[M] = 0.0;
    C[M] = 0.0;
    return;
  }
  const double inv_tr = 1.0 / tr;
#pragma unroll
  for (int k = 0; k < M * M; ++k) b[k] = a[k] * inv_tr;
  int left = -1;
  for (int it = 0; it < max_squarings; ++it) {
#pragma unroll
    for (int k = 0; k < M * M; ++k) {
      const int i = k % M, j = k / M;
      double acc = 0.0;
#pragma unroll
      for (int l = 0; l < M; ++l) acc = fma(b[i + l * M], b[l + j * M], acc);
      c[k] = acc;
    }
    double s = 0.0;
#pragma unroll
    for (int i = 0; i < M; ++i) s += c[i * (M + 1)];
    if (left < 0 && 1.0 - s <= 1e-12) left = 2;
    if (left == 0) break;
    const double inv_s = 1.0 / s;
#pragma unroll
    for (int k = 0; k < M * M; ++k) b[k] = c[k] * inv_s;
    if (left > 0) --left;
  }
  int j = 0;
  double bjj = b[0];
#pragma unroll
  for (int i = 1; i < M; ++i)
    if (b[i * (M + 1)] > bjj) {
      bjj = b[i * (M + 1)];
      j = i;
    }
  double col[M];
#pragma unroll
  for (int i = 0; i < M; ++i) {
    double bij = b[i];
#pragma unroll
    for (int jj = 1; jj < M; ++jj)
      if (jj == j) bij = b[i + jj * M];
    col[i] = bij;
  }
  double n2 = 0.0;
#pragma unroll
  for (int i = 0; i < M; ++i) n2 = fma(col[i], col[i], n2);
  const double inv_n = 1.0 / sqrt(n2);
  double vv[M];
#pragma unroll
  for (int i = 0; i < M; ++i) vv[i] = col[i] * inv_n;
  double lam = 0.0;
#pragma unroll
  for (int i = 0; i < M; ++i) {
    double acc = 0.0;
#pragma unroll
    for (int l = 0; l < M; ++l) acc = fma(a[i + l * M], vv[l], acc);
    lam = fma(vv[i], acc, lam);
  }
#pragma unroll
  for (int i = 0; i < M; ++i) v[i] = vv[i];
  v[M] = 1.0;
  C[M] = lam;
}

constexpr int kDominantMaxOrder = 64;  // callers size 3 m^2 + m + 2 shared doubles up to this order
__device__ inline bool dominant_pair(const double* A, double* B, double* C, double* v, int m,
                                     double& lam, int max_squarings = 64) {
  // orders up to 8: the first warp alone with warp barriers (the squarings
  // are a few FMAs per lane; block barriers would dominate); the other
  // warps wait at the final barrier and read lam from the shared v slot
  if (m <= 4) {
    // one thread, registers only
    if (threadIdx.x == 0) {
      if (m == 1) dominant_pair_regs<1>(A, C, v, max_squarings);
      else if (m == 2) dominant_pair_regs<2>(A, C, v, max_squarings);
      else if (m == 3) dominant_pair_regs<3>(A, C, v, max_squarings);
      else dominant_pair_regs<4>(A, C, v, max_squarings);
    }
    __syncthreads();
    const bool found = v[m] != 0.0;
    lam = C[m];
    __syncthreads();
    return found;
  }
  const bool one_warp = m <= 8;
  if (one_warp && threadIdx.x >= 32) {
    __syncthreads();
    const bool found = v[m] != 0.0;
    lam = C[m];
    __syncthreads();
    return found;
  }
  const int tid = threadIdx.x, nt = one_warp ? 32 : blockDim.x, mm = m * m;
  auto sync = [&] {
    if (one_warp) __syncwarp();
    else __syncthreads();
  };
  // the result for the other warps (one_warp): v[m] = found, C[m] = lam
  auto finish = [&](bool found, double l) {
    if (one_warp) {
      if (tid == 0) {
        v[m] = found ? 1.0 : 0.0;
        C[m] = l;
      }
      __syncwarp();
      __syncthreads();
      __syncthreads();
    }
    return found;
  };
  double tr = 0.0;
  for (int i = 0; i < m; ++i) tr += A[i * (m + 1)];
  if (!(tr > 0.0) || !isfinite(tr)) {
    lam = 0.0;
    return finish(false, 0.0);
  }
  const double inv_tr = 1.0 / tr;
  for (int k = tid; k < mm; k += nt) B[k] = A[k] * inv_tr;
  sync();
  int left = -1;  // squarings still to run once converged
  for (int it = 0; it < max_squarings; ++it) {
    for (int k = tid; k < mm; k += nt) {
      const int i = k % m, j = k / m;
      double acc = 0.0;
      for (int l = 0; l < m; ++l) acc = fma(B[i + l * m], B[l + j * m], acc);
      C[k] = acc;
    }
    sync();
    double s = 0.0;  // tr(B^2), the same in every thread
    for (int i = 0; i < m; ++i) s += C[i * (m + 1)];
    if (left < 0 && 1.0 - s <= 1e-12) left = 2;
    if (left == 0) break;
    const double inv_s = 1.0 / s;
    for (int k = tid; k < mm; k += nt) B[k] = C[k] * inv_s;
    sync();
    if (left > 0) --left;
  }
  int j = 0;
  for (int i = 1; i < m; ++i)
    if (B[i * (m + 1)] > B[j * (m + 1)]) j = i;
  double n2 = 0.0;
  for (int i = 0; i < m; ++i) n2 = fma(B[i + j * m], B[i + j * m], n2);
  const double inv_n = 1.0 / sqrt(n2);
  sync();  // every thread has read B
  for (int i = tid; i < m; i += nt) v[i] = B[i + j * m] * inv_n;
  sync();
  for (int i = tid; i < m; i += nt) {
    double acc = 0.0;
    for (int l = 0; l < m; ++l) acc = fma(A[i + l * m], v[l], acc);
    C[i] = acc;
  }
  sync();
  lam = 0.0;
  for (int i = 0; i < m; ++i) lam = fma(v[i], C[i], lam);
  sync();
  return finish(true, lam);
}

// In-place Cholesky (lower) of an SPD k x k matrix A (+ ridge on the
// diagonal), one thread. Returns false on a non-positive or non-finite pivot.
__device__ inline bool cholesky_serial(double* A, int k, double ridge) {
  for (int i = 0; i < k; ++i) {
    for (int j = 0; j <= i; ++j) {
      double v = A[i + j * k] + (i == j ? ridge : 0.0);
      for (int q = 0; q < j; ++q) v -= A[i + q * k] * A[j + q * k];
      if (i == j) {
        if (!(v > 0.0) || !isfinite(v)) return false;
        A[i + i * k] = sqrt(v);
      } else {
        A[i + j * k] = v / A[j + j * k];
      }
    }
  }
  return true;
}

// The same factorisation by the whole block (A in shared memory; every thread
// calls it and receives the result): right-looking, the trailing columns
// updated element by element after each pivot.
__device__ inline bool cholesky_block(double* A, int k, double ridge) {
  __syncthreads();
  for (int i = threadIdx.x; i < k; i += blockDim.x) A[i + i * k] += ridge;
  __syncthreads();
  for (int j = 0; j < k; ++j) {
    const double piv = A[j + j * k];
    if (!(piv > 0.0) || !isfinite(piv)) return false;  // the same value in every thread
    const double d = sqrt(piv);
    __syncthreads();
    for (int i = j + threadIdx.x; i < k; i += blockDim.x) A[i + j * k] = i == j ? d : A[i + j * k] / d;
    __syncthreads();
    const int left = k - 1 - j;
    for (int e = threadIdx.x; e < left * left; e += blockDim.x) {
      const int i = j + 1 + e % left, c = j + 1 + e / left;
      if (i >= c) A[i + c * k] = fma(-A[i + j * k], A[c + j * k], A[i + c * k]);
    }
    __syncthreads();
  }
  return true;
}

// Solve L L^T x = b in place for b[i * stride] (L lower, k x k,
// column-major), one thread.
__device__ inline bool cholesky_solve_strided(const double* L, int k, double* b, long stride) {
  for (int i = 0; i < k; ++i) {
    double v = b[i * stride];
    for (int q = 0; q < i; ++q) v -= L[i + q * k] * b[q * stride];
    b[i * stride] = v / L[i + i * k];
  }
  bool ok = true;
  for (int i = k - 1; i >= 0; --i) {
    double v = b[i * stride];
    for (int q = i + 1; q < k; ++q) v -= L[q + i * k] * b[q * stride];
    v /= L[i + i * k];
    b[i * stride] = v;
    ok = ok && isfinite(v);
  }
  return ok;
}

// Solve L L^T x = b in place (L lower, k x k, column-major), one thread.
__device__ inline bool cholesky_solve_serial(const double* L, int k, double* b) {
  for (int i = 0; i < k; ++i) {
    double v = b[i];
    for (int q = 0; q < i; ++q) v -= L[i + q * k] * b[q];
    b[i] = v / L[i + i * k];
  }
  for (int i = k - 1; i >= 0; --i) {
    double v = b[i];
    for (int q = i + 1; q < k; ++q) v -= L[q + i * k] * b[q];
    b[i] = v / L[i + i * k];
    if (!isfinite(b[i])) return false;
  }
  return true;
}

}  // namespace fpls
