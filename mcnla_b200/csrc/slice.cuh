// FP64 products of a fixed large matrix with a few columns, on the int8 tensor cores (tcgen05 kind::i8).
//
//   C (M x l) := alpha A (M x K) B (K x l)
//
// The iteration loops multiply the same A (Bs, Qs) by a new l-column B in every iteration; in FP64 that is bound by
// the DMMA rate.  Row i of A and column j of B are scaled by powers of two to 55-bit integers and cut into
// kSlices signed bytes (balanced base-256 digits); the products of slices s and t with s + t = d share one exact
// 32-bit accumulator, d = 0 .. kSlices, and the eight sums are put together in FP64.  (Ozaki, Ogita, Oishi and Rump,
// "Error-free transformations of matrix multiplication", Numer. Algorithms 59, 2012.)  A is cut once (7 bytes an
// element, less than its FP64 form).
//
// Error: the integers' rounding, about 2^-56 (max|a_i| |b_j| + |a_i| max|b_j|), and what is left out (d > kSlices),
// about 2^-64 sqrt(K) max|a_i| max|b_j|: for any row and column at most about 2^-55 |a_i| |b_j|, and for rows and columns
// without dominating entries below that by the square root of K.  (Without the order d = kSlices, 2^-56 sqrt(K) max|a_i|
// max|b_j| was left out: 4e-15 |a_i| |b_j| where one entry dominates at K = 16384, and 12 iterations on such bases were
// off by 6e-13 in the Frobenius norm, where they are by 3e-14 now and with the DMMA GEMM.)  That is normwise by rows and
// columns, as the bases themselves are known (an orthogonalizer's sums leave 1e-16 of a row's norm in its every entry),
// so small entries beside large ones have no rule of their own; one that kept rows with dominating entries on the
// DMMA GEMM, as the residue products do, took every Bs with directions the sketches do not share (rows near the unit
// vectors), for the same results.
// Any finite magnitude of a row or column is taken; NaN or an infinity in it makes its results NaN.
#pragma once
#include "common.cuh"

namespace mb {

constexpr int kSlices = 7;

struct SlicePlan {
  bool use = false;
  int64_t M = 0, K = 0;
  int l = 0;
  int nb = 0;             // columns of a group: 32 or 64
  int groups = 0;
  int splits = 0;         // K is cut into this many parts, added in order
  int64_t kt_per = 0;     // k-tiles of a part
  size_t a_bytes = 0;     // A's slices and scales
  size_t w_bytes = 0;     // B's slices and scales, and the parts' sums
};

// The plan, or use = false where the DMMA GEMM is the faster one.  c may be null (an estimate).
SlicePlan plan_slices(const Context* c, int64_t M, int64_t K, int l);
// Whether a KN loop with Qs and Qs' cuts Qs at all: by the problem alone, so that a solve gives the same bits in a
// server's worker as alone.
inline bool use_qs_slices(int maxit) { return maxit >= 8; }
// Cuts A (unit stride along K or along M) into aw (plan.a_bytes).
int slice_a(Context* c, const SlicePlan& p, CMat A, void* aw);
// C := alpha A B (B with unit stride along its columns' direction l, C row-major), with A's slices in aw; ww:
// plan.w_bytes of scratch.  Honours the context's iteration guard; nothing but launches.
int slice_mul(Context* c, const SlicePlan& p, const void* aw, CMat B, double alpha, DMat C, void* ww);

}  // namespace mb
