// CTA-level FP64 dense routines for the l x l (and 2l x 2l) steps of the iSVD
// stages: symmetric eigendecomposition (the reference calls LAPACK dsyev /
// dgesvd there, include/mcnla/core/la/dense/driver/syev.hpp:150-160,
// gesvd.hpp:159-193), matrix inversion (dgetrf + dgetri,
// include/mcnla/core/la/dense/driver/getrfi.hpp:117-124) and small products.
//
// One thread block owns one small problem.  The eigensolver is the cyclic
// two-sided Jacobi method with a round-robin (tournament) ordering, so the
// n/2 rotations of a round touch disjoint row/column pairs and run in
// parallel (Golub & Van Loan, Matrix Computations, 4th ed., sec. 8.5:
// Algorithm 8.5.2 for the 2 x 2 rotation, sec. 8.5.5 for the parallel
// ordering).  The inverse is Gauss-Jordan elimination with partial pivoting,
// on registers.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

namespace mb {
namespace small {

// Round-robin pairing of P (even) players over P-1 rounds: pair 0 is
// (r, P-1); pair k >= 1 is ((r+k) mod (P-1), (r-k) mod (P-1)).  Every pair of
// distinct players meets exactly once per sweep.
__device__ __forceinline__ void rr_pair(int P, int r, int k, int& p, int& q) {
  if (k == 0) { p = r; q = P - 1; }
  else {                        // 0 <= r < P - 1 and 1 <= k < P / 2: one wrap at most
    p = r + k;
    if (p >= P - 1) p -= P - 1;
    q = r - k;
    if (q < 0) q += P - 1;
  }
  if (p > q) { int t = p; p = q; q = t; }
}

struct JacobiScratch {
  double2* cs;  // npairs: (cos, sin) of each pair's rotation
  int2* pq;     // npairs: the pair's indices (p < q)
  double* t;    // npairs (tangent, for the exact diagonal update)
  double* apq;  // npairs
  double* app;  // npairs
  double* aqq;  // npairs
  int* count;   // 1 (rotations applied this round)
  double* red;  // 32
};

// Frobenius norm^2 of the n x n matrix a (lda), all threads return it.
__device__ inline double cta_frob2(const double* a, int lda, int n, double* red) {
  double s = 0.0;
  for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
    double v = a[(e / n) * lda + (e % n)];
    s += v * v;
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  double tot = 0.0;
  const int nw = (blockDim.x + 31) >> 5;
  for (int w = 0; w < nw; ++w) tot += red[w];
  __syncthreads();
  return tot;
}

// Eigendecomposition of the symmetric n x n matrix a (row stride lda, any
// memory space; shared memory is fastest).  On return diag(a) holds the
// eigenvalues (unsorted) and the ROWS of v (row stride ldv) the eigenvectors:
// v[k * ldv + i] is component i of eigenvector k (the transpose of the usual
// V, so that a rotation of two eigenvectors touches two contiguous rows, which
// matters when v lives in global memory).  When init_v is false, v must hold
// an orthogonal starting basis (rows) in which a is expressed (warm start);
// otherwise v is set to I.  Returns the number of sweeps.
//
// A round has two phases and two barriers: the angles (one thread per pair),
// then one update phase.  The rotations of a round act on disjoint index
// pairs, so a <- J' a J splits into 2 x 2 blocks (rows of pair K1, columns of
// pair K2) that depend only on their own four entries and the two pairs'
// rotations: each (K1, K2) block is one item (rows rotated first, then
// columns; the diagonal blocks are written exactly, J' B J = diag(app - t apq,
// aqq + t apq)).  The eigenvector rows of each pair are items of the same
// phase.  The rounds are latency-bound: launch it with many warps (1024
// threads) rather than give a thread several items' loads at once.
__device__ inline int cta_jacobi_eig(double* a, int lda, double* v, int ldv, int n, bool init_v,
                                     const JacobiScratch& js, int max_sweeps) {
  const int tid = threadIdx.x, nt = blockDim.x;
  if (init_v) {
    for (int e = tid; e < n * n; e += nt) v[(e / n) * ldv + (e % n)] = ((e / n) == (e % n)) ? 1.0 : 0.0;
  }
  __syncthreads();
  if (n <= 1) return 0;
  const int P = (n + 1) & ~1;
  const int npairs = P / 2;
  const double fro2 = cta_frob2(a, lda, n, js.red);
  // An off-diagonal entry is left alone when it is below eps * sqrt(|app aqq|)
  // (relative test) or below eps * ||A||_F (absolute floor: LAPACK's
  // eigensolvers are normwise accurate to that level, and below it rounding
  // in the rotations regenerates off-diagonal noise faster than a sweep
  // removes it).  Both tests compare squares.
  const double eps = 2.220446049250313e-16;
  const double eps2 = eps * eps;
  const double abs_floor = eps2 * fro2;
  // block items (K1, K2), K2 fastest, and eigenvector items (pair k, component i), i fastest:
  // thread tid takes e = tid, tid + nt, ..., walked with fixed increments
  const int b1_start = tid / npairs, b2_start = tid - b1_start * npairs;
  const int b1_step = nt / npairs, b2_step = nt - b1_step * npairs;
  const int k_start = tid / n, i_start = tid - k_start * n;
  const int k_step = nt / n, i_step = nt - k_step * n;
  int sweep = 0;
  for (; sweep < max_sweeps; ++sweep) {
    int rotated = 0;
    for (int r = 0; r < P - 1; ++r) {
      // 1. angles, one thread per pair
      int mine = 0;
      for (int k = tid; k < npairs; k += nt) {
        int p, q;
        rr_pair(P, r, k, p, q);
        double c = 1.0, s = 0.0, t = 0.0, apq = 0.0, app = 0.0, aqq = 0.0;
        if (q < n) {
          apq = a[p * lda + q];
          app = a[p * lda + p];
          aqq = a[q * lda + q];
          const double apq2 = apq * apq;
          if (apq2 > eps2 * fabs(app * aqq) && apq2 > abs_floor) {
            // t = sgn(theta) / (|theta| + sqrt(1 + theta^2)), theta = d / g (d = aqq - app,
            // g = 2 apq), written as sgn(d) g / (|d| + sqrt(d^2 + g^2)): one division, one
            // square root and one reciprocal square root on the round's critical path.  t is
            // invariant under scaling d and g together, so entries far from 1 are scaled by
            // 2^-600 or 2^600 (exactly) before d^2 + g^2 could overflow or lose precision.
            double d = aqq - app, g = 2.0 * apq;
            const double mx = fmax(fabs(d), fabs(g));
            if (mx > 1e150) { d *= 0x1p-600; g *= 0x1p-600; }
            else if (mx < 1e-150) { d *= 0x1p600; g *= 0x1p600; }
            t = (d >= 0.0 ? g : -g) / (fabs(d) + sqrt(fma(d, d, g * g)));
            c = rsqrt(fma(t, t, 1.0));
            s = t * c;
            ++mine;
          } else {
            apq = 0.0;
          }
        }
        js.cs[k] = make_double2(c, s);
        js.pq[k] = make_int2(p, q);
        js.t[k] = t; js.apq[k] = apq; js.app[k] = app; js.aqq[k] = aqq;
      }
      // the barrier also counts the threads that set up a rotation
      const int cnt = __syncthreads_count(mine);
      if (cnt == 0) continue;
      rotated += cnt;
      // 2a. a <- J' a J by 2 x 2 blocks
      for (int k1 = b1_start, k2 = b2_start; k1 < npairs;) {
        const double2 cs1 = js.cs[k1], cs2 = js.cs[k2];
        const double s1 = cs1.y, s2 = cs2.y;
        if (s1 != 0.0 || s2 != 0.0) {
          const int2 pq1 = js.pq[k1], pq2 = js.pq[k2];
          const int p1 = pq1.x, q1 = pq1.y, p2 = pq2.x, q2 = pq2.y;
          if (k1 == k2) {
            const double ta = js.t[k1] * js.apq[k1];
            a[p1 * lda + p1] = js.app[k1] - ta;
            a[q1 * lda + q1] = js.aqq[k1] + ta;
            a[p1 * lda + q1] = 0.0;
            a[q1 * lda + p1] = 0.0;
          } else {
            // q1 / q2 is the padding index n of an odd n only in a pair that does not rotate
            const bool h1 = q1 < n, h2 = q2 < n;
            double xpp = a[p1 * lda + p2];
            double xpq = h2 ? a[p1 * lda + q2] : 0.0;
            double xqp = h1 ? a[q1 * lda + p2] : 0.0;
            double xqq = (h1 && h2) ? a[q1 * lda + q2] : 0.0;
            if (s1 != 0.0) {
              const double c1 = cs1.x;
              const double rpp = c1 * xpp - s1 * xqp, rqp = s1 * xpp + c1 * xqp;
              const double rpq = c1 * xpq - s1 * xqq, rqq = s1 * xpq + c1 * xqq;
              xpp = rpp; xqp = rqp; xpq = rpq; xqq = rqq;
            }
            if (s2 != 0.0) {
              const double c2 = cs2.x;
              const double ypp = c2 * xpp - s2 * xpq, ypq = s2 * xpp + c2 * xpq;
              const double yqp = c2 * xqp - s2 * xqq, yqq = s2 * xqp + c2 * xqq;
              xpp = ypp; xpq = ypq; xqp = yqp; xqq = yqq;
            }
            a[p1 * lda + p2] = xpp;
            if (h2) a[p1 * lda + q2] = xpq;
            if (h1) a[q1 * lda + p2] = xqp;
            if (h1 && h2) a[q1 * lda + q2] = xqq;
          }
        }
        k1 += b1_step;
        k2 += b2_step;
        if (k2 >= npairs) { k2 -= npairs; ++k1; }
      }
      // 2b. rows p, q of v
      for (int k = k_start, i = i_start; k < npairs;) {
        const double2 cs = js.cs[k];
        if (cs.y != 0.0) {
          const int2 pq = js.pq[k];
          const double vx = v[pq.x * ldv + i], vy = v[pq.y * ldv + i];
          v[pq.x * ldv + i] = cs.x * vx - cs.y * vy;
          v[pq.y * ldv + i] = cs.y * vx + cs.x * vy;
        }
        k += k_step;
        i += i_step;
        if (i >= n) { i -= n; ++k; }
      }
      __syncthreads();
    }
    if (rotated == 0) break;
  }
  return sweep;
}

// Gauss-Jordan inverse with the matrix in registers (below).
constexpr int kGjWarps = 16;
constexpr int kGjThreads = 32 * kGjWarps;
struct GjPivot {
  double inv;    // 1 / pivot
  int row;       // the pivot's row
  int pos;       // its position in the interchanged order
  int zero;      // 1: the pivot is exactly zero
};
template <int RA>
struct GjShared {
  double col[2][32 * RA];   // the pivot column, double-buffered across steps
  GjPivot piv[2];
  int at[32 * RA];          // the row at each position, after the last step
};

// The pivot of step k: the first position of the largest |v| among the rows at positions >= k (as
// idamax; NaN never wins, and a column of NaN takes position k).  v[a] is the entry of row
// lane + 32 a of column k, pos[a] that row's position.  One warp calls it; the column and the
// pivot go to shared memory.
template <int RA>
__device__ __forceinline__ void gj_pick(const double (&v)[RA], const int (&pos)[RA], int k, double* col, GjPivot* piv) {
  const int lane = threadIdx.x & 31;
  unsigned long long key = 0;
  int bp = 0x7fffffff, br = 0;
  double bv = 0.0;
#pragma unroll
  for (int a = 0; a < RA; ++a) {
    col[lane + 32 * a] = v[a];
    // |v|'s bits order as |v| does; 0 is left for NaN, so that zero beats it
    const double av = fabs(v[a]);
    const unsigned long long ka = isnan(av) ? 0ull : (unsigned long long)__double_as_longlong(av) + 1ull;
    const bool ok = pos[a] >= k;   // a row already used has a smaller position
    if (ok && (bp == 0x7fffffff || ka > key || (ka == key && pos[a] < bp))) {
      key = ka;
      bp = pos[a];
      br = lane + 32 * a;
      bv = v[a];
    }
  }
  const unsigned hi = bp == 0x7fffffff ? 0u : unsigned(key >> 32);
  const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
  const unsigned lo = (bp != 0x7fffffff && hi == mh) ? unsigned(key) : 0u;
  const unsigned ml = __reduce_max_sync(0xffffffffu, lo);
  const unsigned cand = (bp != 0x7fffffff && hi == mh && unsigned(key) == ml) ? unsigned(bp) : 0xffffffffu;
  const unsigned mp = __reduce_min_sync(0xffffffffu, cand);
  if (cand == mp && mp != 0xffffffffu) {   // positions are distinct: one lane
    piv->inv = 1.0 / bv;
    piv->row = br;
    piv->pos = int(mp);
    piv->zero = bv == 0.0;
  }
}

// Inverse of an n x n matrix (n <= 32 RA) by Gauss-Jordan elimination with partial pivoting, in
// place in registers: thread (warp w, lane) of the kGjThreads holds x[a][b] = entry (lane + 32 a,
// w + 16 b), zero outside the matrix.  The operations, pivots and rounding are those of the
// row-interchange form (pivot row scaled, every other row eliminated), but rows stay where they
// are and pos[a] tracks the position of row lane + 32 a.  On return entry (i, j) of the inverse is
// at row position i, that is: the thread holding row r, column j has the inverse's element
// (pos(r), sh.at[j]).  Returns 0, or k + 1 when the k-th pivot is exactly zero (the same on all
// threads).
//
// What bounds it: the chain of n steps.  A warp holds whole columns, so the pivot row reaches a
// column's other rows by a shuffle and a step needs one block barrier: every warp applies step k
// to its columns, the owner of column k + 1 first, which then picks the next pivot (three warp
// reductions and the division) while the others still eliminate.  The matrix in shared memory
// instead took two barriers a step and ~40 instructions an entry.  One inverse, before and now, the
// same bits: n = 64: 212 and 74 us, n = 128: 733 and 186 us, n = 160: 1223 and 411 us.
template <int RA>
__device__ int gj_inverse_regs(double (&x)[RA][2 * RA], int (&pos)[RA], int n, GjShared<RA>& sh) {
  constexpr int CB = 2 * RA;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int a = 0; a < RA; ++a) pos[a] = lane + 32 * a < n ? lane + 32 * a : -1;   // -1: never a pivot
  if (wid == 0) {
    double v[RA];
#pragma unroll
    for (int a = 0; a < RA; ++a) v[a] = x[a][0];
    gj_pick<RA>(v, pos, 0, sh.col[0], &sh.piv[0]);
  }
  __syncthreads();
#pragma unroll
  for (int s = 0; s < CB; ++s) {
#pragma unroll 1
    for (int w = 0; w < kGjWarps; ++w) {
      const int k = s * kGjWarps + w;
      if (k >= n) break;
      const GjPivot pv = sh.piv[k & 1];
      if (pv.zero) return k + 1;
      const int ap = pv.row >> 5, lp = pv.row & 31;
      double f[RA];
      bool isp[RA];
#pragma unroll
      for (int a = 0; a < RA; ++a) {
        f[a] = sh.col[k & 1][lane + 32 * a];
        isp[a] = lane == lp && a == ap;
        if (isp[a]) pos[a] = k;
        else if (pos[a] == k) pos[a] = pv.pos;
      }
      const bool next_here = k + 1 < n && wid == ((w + 1) & (kGjWarps - 1));
#pragma unroll
      for (int bb = 0; bb < CB; ++bb) {
        const int b = (s + bb) % CB;           // column k's slot first, then column k + 1's when w = 15
        double xp = x[0][b];
#pragma unroll
        for (int a = 1; a < RA; ++a) xp = a == ap ? x[a][b] : xp;
        xp = __shfl_sync(0xffffffffu, xp, lp);
        if (bb == 0 && wid == w) {             // column k itself
#pragma unroll
          for (int a = 0; a < RA; ++a) x[a][b] = isp[a] ? pv.inv : -f[a] * pv.inv;
        } else {
          const double pj = xp * pv.inv;
#pragma unroll
          for (int a = 0; a < RA; ++a) x[a][b] = isp[a] ? pj : fma(-f[a], pj, x[a][b]);
        }
        if (next_here && bb == (w == kGjWarps - 1 ? 1 : 0)) {
          double v[RA];
#pragma unroll
          for (int a = 0; a < RA; ++a) v[a] = x[a][b];
          gj_pick<RA>(v, pos, k + 1, sh.col[(k + 1) & 1], &sh.piv[(k + 1) & 1]);
        }
      }
      __syncthreads();
    }
  }
  if (wid == 0) {
#pragma unroll
    for (int a = 0; a < RA; ++a)
      if (pos[a] >= 0) sh.at[pos[a]] = lane + 32 * a;
  }
  __syncthreads();
  return 0;
}

// C := alpha * op(A) * op(B) + beta * C for small matrices (any memory space),
// all threads of the block cooperating; op(X) = X or X' (tA / tB).  C must not
// alias A or B.  Ends with a block barrier.
__device__ inline void cta_mm(int M, int N, int K, double alpha, const double* A, int lda, bool tA, const double* B,
                              int ldb, bool tB, double beta, double* C, int ldc) {
  for (int e = threadIdx.x; e < M * N; e += blockDim.x) {
    const int i = e / N, j = e % N;
    double s = 0.0;
    for (int k = 0; k < K; ++k) {
      const double x = tA ? A[k * lda + i] : A[i * lda + k];
      const double y = tB ? B[j * ldb + k] : B[k * ldb + j];
      s = fma(x, y, s);
    }
    C[i * ldc + j] = (beta == 0.0) ? alpha * s : alpha * s + beta * C[i * ldc + j];
  }
  __syncthreads();
}

// Block-wide sum of one value per thread; every thread gets the total.
__device__ inline double cta_sum(double v, double* red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double tot = 0.0;
  const int nw = (blockDim.x + 31) >> 5;
  for (int w = 0; w < nw; ++w) tot += red[w];
  __syncthreads();
  return tot;
}

}  // namespace small
}  // namespace mb
