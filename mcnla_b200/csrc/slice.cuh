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
// about 2^-64 sqrt(K) max|a_i| max|b_j|: for any row and column at most about the 2^-55 |a_i| |b_j| of a running FP64
// sum, and for rows and columns without dominating entries below it by the square root of K.  (Without the order
// d = kSlices, 2^-56 sqrt(K) max|a_i| max|b_j| was left out: 4e-15 |a_i| |b_j| where one entry dominates at K = 16384.)
// A sum over few large terms loses less than that bound in FP64, so where a row of A has few entries near its largest
// (2-norm^2 below K / 256 times the largest entry^2, the residue products' rule), or NaN or infinities, slice_a says
// so and the caller keeps the DMMA GEMM.  Any finite magnitude of a row or column is taken; NaN or an infinity in a
// column of B makes that column of C NaN.
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
// Cuts A (unit stride along K or along M) into aw (plan.a_bytes), and sets `bit` in the device scalar slice_few when a
// row is not for the slices.  slice_bits reads that scalar and waits for it.
int slice_a(Context* c, const SlicePlan& p, CMat A, void* aw, int bit);
int slice_bits(Context* c, int* bits);
// C := alpha A B (B with unit stride along its columns' direction l, C row-major), with A's slices in aw; ww:
// plan.w_bytes of scratch.  Honours the context's iteration guard; nothing but launches.
int slice_mul(Context* c, const SlicePlan& p, const void* aw, CMat B, double alpha, DMat C, void* ww);

}  // namespace mb
