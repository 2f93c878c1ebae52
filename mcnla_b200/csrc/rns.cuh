// FP64 products on the int8 tensor cores (tcgen05 kind::i8) by residue arithmetic.
//
//   C (M x N) := A (M x K) B (K x N), FP64 in and out
//
// Row i of A is scaled by a power of two and rounded to integers a' of at most ~2^57 in 2-norm, column
// j of B likewise to b' (~2^58), so the integer dot product stays below P / 4 for the product P of
// kRnsModuli coprime moduli <= 256 (Cauchy-Schwarz).  Its residue modulo each modulus is an int8 GEMM
// with exact 32-bit accumulation, and the Chinese remainder theorem gives the integer back, scaled to
// FP64 with one rounding.  (Ozaki, Uchino and Imamura, "Ozaki Scheme II: A GEMM-oriented emulation of
// floating-point matrix multiplication using an integer modular technique", 2025.)  The only
// errors are the rounding of a' and b' (about 2^-57 of the row's and the column's 2-norm, against the
// ~2^-54 |a| |b| that the running sum of a DGEMM loses) and the final rounding.
//
// Rows and columns for which that bound says too little are flagged: those with NaN, infinities, magnitudes outside
// 2^+-400, or few large entries (2-norm^2 below K / 256 times the largest entry^2; a running sum of such a row rounds
// less often).  A 128 x 256 tile of C with a flagged row or column goes to the DMMA GEMM as a whole.  (Element by
// element both paths ran over nearly everything where the flagged rows are spread out.)  Which way a tile goes
// depends on its rows of A and its columns of B alone, and integer sums have no order, so the result does not depend
// on how the rows are cut into blocks of whole tiles.
#pragma once
#include "dgemm.cuh"

namespace mb {

constexpr int kRnsModuli = 15;
constexpr int kRnsRowAlign = kFlagRows;

struct RnsPlan {
  bool use = false;       // this product runs on the int8 path
  bool streamed = false;  // row blocks will come one call each
  bool same = false;      // A' = B (a Gramian Q' Q, lower triangle): one set of residues
  int64_t M = 0, N = 0, K = 0;
  int64_t kc = 0;         // K per chunk (chunks are added in FP64)
  int chunks = 0;
  int64_t mb = 0;         // rows of A per block
  size_t bytes = 0;       // workspace
};

// The int8 plan for a product of this shape, or use = false where the DMMA GEMM is the faster one.
// max_rows: the most rows a call will pass (a streamed product's row blocks, which start on multiples of kRnsRowAlign);
// the decision itself depends on M, N and K only.  c may be null (an estimate of the workspace).
RnsPlan plan_rns(const Context* c, int64_t M, int64_t N, int64_t K, bool same, int64_t max_rows = 0);

// C := A B for `rows` rows of the planned product.  ws: plan.bytes; dws: the DMMA path's split-K
// workspace (for the flagged tiles), splits its split count.  reuse_b: B's
// residues are still in ws from the previous call (one chunk only; otherwise they are made again).
int rns_gemm(Context* c, const RnsPlan& plan, int64_t rows, CMat A, CMat B, DMat C, void* ws, double* dws, int splits,
             bool reuse_b);

}  // namespace mb
