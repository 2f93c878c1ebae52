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
// A sum over few large terms, or one whose large a meet small b, loses less than that in FP64: its error goes with
// |a|.|b| = sum |a_k| |b_k| (2.4e-17 |a| |b| for dense normal rows, 2.6e-18 where |a|.|b| is a sixteenth of |a| |b|; the
// residue product's is 2e-18 to 3.8e-18 |a| |b| throughout).  So the DMMA GEMM takes
//   * rows and columns with NaN, infinities, magnitudes outside 2^+-400, or a 1-norm below sqrt(K) / 8 times the 2-norm
//     (dense normal entries: 0.8; a share p of them, the rest zero: 0.8 sqrt(p)), and
//   * where B is a caller's or another product (RnsKind::Given), elements with |a|.|b| below |a| |b| / 16, by one more
//     int8 product, of the magnitudes in units of a sixteenth of a row's or column's root mean square.  A B of
//     independent normal numbers, as the library draws Omega (RnsKind::Drawn), has 0.8 times the row's ratio above.
// A 128 x 256 tile of C with such a row, column or element goes to the DMMA GEMM as a whole.  (Element by element both
// paths ran over nearly everything where such rows are spread out.)  Which way a tile goes depends on its rows of A and
// its columns of B alone, and integer sums have no order, so the result does not depend on how the rows are cut into
// blocks of whole tiles.  A Gramian of orthonormal columns is held to the columns' norms (RnsKind::Gramian).
#pragma once
#include "dgemm.cuh"

namespace mb {

constexpr int kRnsModuli = 15;
constexpr int kRnsRowAlign = kFlagRows;

enum class RnsKind {
  Drawn,      // B: independent normal numbers
  Given,      // B: anything
  Gramian,    // A' = B (Q' Q, lower triangle): one set of residues
};

struct RnsPlan {
  bool use = false;       // this product runs on the int8 path
  bool streamed = false;  // row blocks will come one call each
  bool same = false;      // RnsKind::Gramian
  int planes = 0;         // of residues, and with RnsKind::Given one of magnitudes
  int64_t M = 0, N = 0, K = 0;
  int64_t kc = 0;         // K per chunk (chunks are added in FP64)
  int chunks = 0;
  int64_t mb = 0;         // rows of A per block
  size_t bytes = 0;       // workspace
};

// The int8 plan for a product of this shape, or use = false where the DMMA GEMM is the faster one.
// max_rows: the most rows a call will pass (a streamed product's row blocks, which start on multiples of kRnsRowAlign);
// the decision itself depends on M, N, K and Gramian or not.  c may be null (an estimate of the workspace).
RnsPlan plan_rns(const Context* c, int64_t M, int64_t N, int64_t K, RnsKind kind, int64_t max_rows = 0);

// C := A B for `rows` rows of the planned product.  ws: plan.bytes; dws: the DMMA path's split-K
// workspace (for the flagged tiles), splits its split count.  reuse_b: B's
// residues are still in ws from the previous call (one chunk only; otherwise they are made again).
int rns_gemm(Context* c, const RnsPlan& plan, int64_t rows, CMat A, CMat B, DMat C, void* ws, double* dws, int splits,
             bool reuse_b);

}  // namespace mb
