// Batched symmetric eigendecomposition of l x l matrices (the reference's dgesvd / dsyev of the Gram
// matrices, include/mcnla/core/la/dense/driver/gesvd.hpp:159-193, syev.hpp:150-160).
//
// The cyclic two-sided Jacobi method in round-robin order (small.cuh), in two kernels.  What bounds it is the
// chain of (n - 1) x ~9 rounds, whose angles depend on the round before; the eigenvectors do not feed back.  So
// k_jacobi_rotations, one CTA per matrix, carries the matrix alone through the rounds and writes down
// the rotations, and k_jacobi_vectors applies them to V, cut by components over many CTAs.
//   * The next round's angles are part of the update phase: the block of two pairs that holds a pivot of the
//     next round is updated by that pair's own thread, which then has the pivot and both diagonal entries
//     (they follow from this round's angles) and computes the angle: one barrier a round.
//   * Of the symmetric matrix each entry is kept once, by the difference of its two players: in round r pair k is
//     (r + k, r - k) modulo R = P - 1 (pair 0: r and the fixed player R), so the differences within a block are
//     the same in every round and an entry's place moves by one column a round.  Half the memory of a
//     square, no index work, and no bank conflicts with lanes along a diagonal of blocks.
// Measured against one kernel doing both with two barriers a round on a square (V in global memory for n > 112):
// us a call, before and now: n = 12 (8 matrices) 93, 70; 20 (16) 182, 151; 32 (16) 335, 268; 64 (64) 1208, 878;
// 80 (32) 2241, 1315; 96 (8) 3379, 1549; 128 (16) 8435, 3120; 160 (16) 16771, 5773.  At n = 160 the rotations'
// kernel is at 86 % of the shared-memory pipe (every entry read and written once a round).
#include "kernels.cuh"
#include "small.cuh"

#include <algorithm>

namespace mb {
namespace {

constexpr int kJacThreads = 1024;
constexpr int kJacSweeps = 30;
constexpr int kJacItems = 4;        // blocks a thread updates in a round, n <= 160
constexpr int kVecCols = 16;        // components of V per CTA of k_jacobi_vectors
constexpr int kVecGroups = 16;      // half-warps of k_jacobi_vectors, each with a component a lane
constexpr int kVecThreads = kVecCols * kVecGroups;
constexpr int kFusedMax = 32;       // up to this n the matrix' own CTA carries V along
constexpr int kVecPairs = 5;        // pairs a half-warp rotates in a round, n <= 160

struct JacWork {                    // per matrix, in global memory
  double2* log;                     // [round][pair]: (c, s)
  int* rank;                        // [n]
  int* count;                       // rounds up to the last that rotates
};

__host__ __device__ constexpr int jac_pairs(int n) { return (n + 1) / 2; }
__host__ __device__ constexpr int jac_rounds(int n) { return 2 * jac_pairs(n) - 1; }
__host__ __device__ constexpr size_t jac_log_rounds(int n) { return size_t(kJacSweeps) * jac_rounds(n) + 1; }
__host__ __device__ constexpr size_t jac_align(size_t b) { return (b + 255) & ~size_t(255); }
__host__ __device__ constexpr size_t jac_log_bytes(int n) {
  return jac_align(jac_log_rounds(n) * jac_pairs(n) * sizeof(double2));
}
size_t jac_bytes(int n) { return jac_log_bytes(n) + jac_align((size_t(n) + 1) * sizeof(int)); }   // per matrix
__device__ JacWork jac_work(char* base, size_t per, int n, int i) {
  char* p = base + per * i;
  JacWork w;
  w.log = reinterpret_cast<double2*>(p);
  w.rank = reinterpret_cast<int*>(p + jac_log_bytes(n));
  w.count = w.rank + n;
  return w;
}

struct Rotation { double c, s, tap; };   // tap: tangent times a(p, q), what the diagonal entries move by

// The rotation that zeroes apq, or none where it is below eps sqrt(|app aqq|) or the absolute floor (LAPACK's
// eigensolvers are normwise accurate to that level; below it rounding in the rotations makes off-diagonal noise
// faster than a sweep removes it).  Both tests compare squares.
__device__ __forceinline__ Rotation rotation_of(double app, double aqq, double apq, double abs_floor) {
  const double eps2 = 2.220446049250313e-16 * 2.220446049250313e-16;
  Rotation r{1.0, 0.0, 0.0};
  const double apq2 = apq * apq;
  if (apq2 > eps2 * fabs(app * aqq) && apq2 > abs_floor) {
    // d = aqq - app, g = 2 apq: cos 2x = |d| / sqrt(d^2 + g^2), c = sqrt((1 + cos 2x) / 2) and
    // s = sgn(d) sin 2x / (2 c) by two reciprocal square roots (the round's critical path), |x| <= pi / 4.  The matrix
    // is scaled to entries of at most 1 and g is above the floor, so nothing overflows or underflows.
    const double d = aqq - app, g = 2.0 * apq;
    const double h = rsqrt(fma(d, d, g * g));
    const double c2 = fma(0.5 * fabs(d), h, 0.5);
    const double ic = rsqrt(c2);                     // 1 / c
    double c = c2 * ic, sn = (d >= 0.0 ? 0.5 : -0.5) * g * h * ic;
    // one step towards c^2 + s^2 = 1 (the rotations' rounding adds up over V)
    const double f = 0.5 * fma(-sn, sn, fma(-c, c, 1.0));
    r.c = fma(c, f, c);
    r.s = fma(sn, f, sn);
    r.tap = sn * ic * apq;
  }
  return r;
}

// An entry's place: row (a difference) times the pitch in the upper half, the column it has in round 0 in the lower.
using Place = unsigned;
static_assert(80 * 159 <= 65535, "a place's row fits 16 bits");
__device__ __forceinline__ Place make_place(int row, int col) { return unsigned(row) << 16 | unsigned(col); }

// The entry of two players given by their offsets from r (kFixed: the fixed player), as place.
constexpr int kFixed = 1 << 20;
__device__ __forceinline__ Place place_of(int x, int y, int np) {
  const int R = 2 * np - 1;
  if (x == kFixed || y == kFixed) {
    const int z = x == kFixed ? y : x;
    return make_place(0, z < 0 ? z + R : z);
  }
  int d = y - x;
  if (d < 0) d += R;                       // from x to y, in [1, R)
  const bool from_x = d < np;
  const int c = from_x ? x : y;
  return make_place((from_x ? d : R - d) * R, c < 0 ? c + R : c);
}

// Column of a place in round r: (col + r) mod R.
__device__ __forceinline__ int at(Place p, int r, int R) {
  const unsigned c = (p & 0xffffu) + unsigned(r);
  return int((p >> 16) + min(c, c - unsigned(R)));
}

// The block of pairs k1 < k2 (plus players +k, minus players -k): (p1, p2), (m1, m2), (m1, p2), (p1, m2).
struct Block { double pp, mm, mp, pm; };
struct BlockPlaces { Place pp, mm, mp, pm; };
__device__ __forceinline__ BlockPlaces block_places(int k1, int k2, int np) {
  const int m1 = k1 == 0 ? kFixed : -k1;
  return BlockPlaces{place_of(k1, k2, np), place_of(m1, -k2, np), place_of(m1, k2, np), place_of(k1, -k2, np)};
}

// rows p' = c p - s m, m' = s p + c m of pair 1, then the columns of pair 2
__device__ __forceinline__ Block rotate_block(const Block& b, double2 r1, double2 r2) {
  const double pp = r1.x * b.pp - r1.y * b.mp, mp = r1.y * b.pp + r1.x * b.mp;
  const double pm = r1.x * b.pm - r1.y * b.mm, mm = r1.y * b.pm + r1.x * b.mm;
  return Block{r2.x * pp - r2.y * pm, r2.y * mp + r2.x * mm, r2.x * mp - r2.y * mm, r2.y * pp + r2.x * pm};
}

// WITH_V: the other warps rotate V (in shared memory) as well, and nothing is logged.
template <bool WITH_V>
__global__ void __launch_bounds__(kJacThreads) k_jacobi_rotations(int n, const double* A, int64_t lda, int64_t a_bs,
                                                                 double* W, double* V, int order, char* work,
                                                                 size_t per, const int* only_if) {
  extern __shared__ __align__(16) double jac_smem[];
  if (only_if && *only_if == 0) return;
  __shared__ double red[32];
  __shared__ int ex_s, rank_s[WITH_V ? kFusedMax : 1];
  const int np = jac_pairs(n), P = 2 * np, R = P - 1;      // an odd n gets a zero row and column
  const int tid = threadIdx.x, nt = blockDim.x;
  double2* cs = reinterpret_cast<double2*>(jac_smem);      // [2][np]: a round's (c, s), double-buffered
  double2* dd = cs + 2 * np;                               // [2][np]: the pair's diagonal entries after its rotation
  double* a = reinterpret_cast<double*>(dd + 2 * np);      // [difference][column]: np x R
  double* vs = a + np * R;                                 // WITH_V: P eigenvectors of n components
  const JacWork w = WITH_V ? JacWork{nullptr, nullptr, nullptr} : jac_work(work, per, n, blockIdx.x);
  const double* Ab = A + blockIdx.x * a_bs;
  if (WITH_V)
    for (int e = tid; e < P * n; e += nt) vs[e] = e / n == e % n ? 1.0 : 0.0;
  // scaled by a power of two to a largest entry in [1/2, 1) (left alone where it is zero or not finite)
  double mx = 0.0;
  for (int e = tid; e < n * n; e += nt) {
    const int i = e / n, j = e - i * n;
    if (j >= i) mx = fmax(mx, fabs(Ab[i * lda + j]));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((tid & 31) == 0) red[tid >> 5] = mx;
  __syncthreads();
  for (int i = 0; i < nt / 32; ++i) mx = fmax(mx, red[i]);
  __syncthreads();
  int ex = 0;
  if (mx > 0.0 && mx <= 1.7976931348623157e308) frexp(mx, &ex);
  if (tid == 0) ex_s = ex;
  const double s1 = scalbn(1.0, -ex / 2), s2 = scalbn(1.0, -ex - (-ex / 2));   // 2^-ex as two factors
  double part = 0.0;
  for (int e = tid; e < P * P; e += nt) {
    const int i = e / P, j = e - i * P;
    if (j < i) continue;
    const double x = j < n ? Ab[i * lda + j] * s1 * s2 : 0.0;
    if (j > i) {
      a[at(place_of(i == R ? kFixed : i, j == R ? kFixed : j, np), 0, R)] = x;
    }
    part = fma(i == j ? x : 2.0 * x, x, part);
  }
  const double fro2 = small::cta_sum(part, red);
  const double abs_floor = 2.220446049250313e-16 * 2.220446049250313e-16 * fro2;

  // Thread k < np: the block with the pivot of the next round's pair k.  Pair k of round r + 1 is (r + 1 + k,
  // r + 1 - k): players of pairs k + 1 and k - 1 of round r, except at the ends.
  const int k = tid;
  int k1 = 0, k2 = 1;
  if (k > 0 && k < np - 1) { k1 = k - 1; k2 = k + 1; }
  else if (k > 0) { k1 = np - 2; k2 = np - 1; }
  // which entry is the pivot, and which of the two pairs' diagonal entries are its players'
  const bool last = k == np - 1 && np > 2;                       // (m2, m1)
  const bool second = k == 1 && np > 2;                          // (p2, p1)
  // the other blocks: threads past those warps; diagonals of blocks (k2 - k1 = D) folded in twos, lanes along k1
  const int t0 = (np + 31) & ~31;
  int items[kJacItems];
#pragma unroll
  for (int u = 0; u < kJacItems; ++u) {
    items[u] = -1;
    const int t = tid - t0 + u * (nt - t0);
    if (tid < t0 || np < 3) continue;
    const int f = t / np, j = t - f * np;   // diagonals f + 1 (np - 1 - f blocks) and np - 1 - f (f + 1)
    int D = f + 1, i = j;
    if (j >= np - 1 - f) {
      D = np - 1 - f;
      i = j - (np - 1 - f);
      if (D == f + 1) continue;                                  // the middle diagonal has no partner
    }
    if (f + 1 > np - 1 - f) continue;
    if (D == 2 || (D == 1 && (i == 0 || i == np - 2))) continue; // a pivot's
    items[u] = i << 8 | (i + D);
  }
  BlockPlaces places[kJacItems];
#pragma unroll
  for (int u = 0; u < kJacItems; ++u) {
    const int x = items[u] < 0 ? 0 : items[u] >> 8, y = items[u] < 0 ? 1 : items[u] & 255;
    places[u] = block_places(x, y, np);
  }
  if (tid < np && np > 1) places[0] = block_places(k1, k2, np);
  const Place own = place_of(k, k == 0 ? kFixed : -k, np);       // this round's pivot of pair k

  int count = 0, quiet = 0, r = 0, b = 0, mine = 0;
  int row = k;                                                   // this pair's entry in the log, of the round to come
  const int most = kJacSweeps * R;
  double dp = 0.0, dm = 0.0, sn = 0.0;                           // pair k's diagonal before its rotation; its sine
  if (tid < np) {
    const int p = k, m = k == 0 ? R : R - k;
    dp = p < n ? Ab[p * lda + p] * s1 * s2 : 0.0;
    dm = m < n ? Ab[m * lda + m] * s1 * s2 : 0.0;
  }
  __syncthreads();
  if (tid < np) {
    const Rotation ro = rotation_of(dp, dm, a[at(own, 0, R)], abs_floor);
    cs[k] = make_double2(ro.c, ro.s);
    dd[k] = make_double2(dp - ro.tap, dm + ro.tap);
    if (!WITH_V) w.log[row] = make_double2(ro.c, ro.s);
    sn = ro.s;
    mine = ro.s != 0.0;
  }
  // the barrier also counts the rotations that the round about to run has
  int cnt = __syncthreads_count(mine);
  for (int round = 0;; ++round) {
    quiet = cnt == 0 ? quiet + 1 : 0;
    if (quiet >= R || round >= most) break;                      // every pair was left alone, one after the other
    if (cnt > 0) count = round + 1;
    row += np;
    const double2* c0 = cs + b * np;
    const double2* d0 = dd + b * np;
    const int rn = r + 1 == R ? 0 : r + 1;
    mine = 0;
    if (tid < np) {
      if (np == 1) {                                             // one pair: the rotation leaves a zero
        const double2 d = d0[0];
        dp = d.x;
        dm = d.y;
        sn = 0.0;
        cs[b ^ 1] = make_double2(1.0, 0.0);
        if (!WITH_V) w.log[row] = make_double2(1.0, 0.0);
        dd[b ^ 1] = d;
      } else if (np > 2 || k == 0) {
        const double2 r1 = c0[k1], r2 = c0[k2], e1 = d0[k1], e2 = d0[k2];
        const BlockPlaces& pl = places[0];
        const int ipp = at(pl.pp, r, R), imm = at(pl.mm, r, R), imp = at(pl.mp, r, R), ipm = at(pl.pm, r, R);
        Block bl{a[ipp], a[imm], a[imp], a[ipm]};
        bl = rotate_block(bl, r1, r2);                           // exact where neither pair rotates
        if (cnt > 0) {
          a[ipp] = bl.pp;
          a[imm] = bl.mm;
          a[imp] = bl.mp;
          a[ipm] = bl.pm;
        }
        if (sn != 0.0) a[at(own, r, R)] = 0.0;                   // this round's pivot, in no block of the round
        const double piv = last ? bl.mm : (second ? bl.pp : bl.mp);
        dp = last ? e2.y : e2.x;
        dm = second ? e1.x : e1.y;
        const Rotation ro = rotation_of(dp, dm, piv, abs_floor);
        cs[(b ^ 1) * np + k] = make_double2(ro.c, ro.s);
        dd[(b ^ 1) * np + k] = make_double2(dp - ro.tap, dm + ro.tap);
        if (!WITH_V) w.log[row] = make_double2(ro.c, ro.s);
        sn = ro.s;
        mine = ro.s != 0.0;
        if (np == 2) {
          // two pairs: their one block also holds the next pivot of pair 1, (m2, p1); its own one is zeroed here
          if (c0[1].y != 0.0) a[at(place_of(1, -1, 2), r, R)] = 0.0;
          const Rotation r3 = rotation_of(e2.y, e1.x, bl.pm, abs_floor);
          cs[(b ^ 1) * np + 1] = make_double2(r3.c, r3.s);
          dd[(b ^ 1) * np + 1] = make_double2(e2.y - r3.tap, e1.x + r3.tap);
          if (!WITH_V) w.log[row + 1] = make_double2(r3.c, r3.s);
          mine |= r3.s != 0.0;
        }
      }
    } else if (cnt > 0) {
#pragma unroll
      for (int u = 0; u < kJacItems; ++u) {
        if (items[u] < 0) continue;
        const double2 r1 = c0[items[u] >> 8], r2 = c0[items[u] & 255];
        if (r1.y == 0.0 && r2.y == 0.0) continue;
        const int ipp = at(places[u].pp, r, R), imm = at(places[u].mm, r, R), imp = at(places[u].mp, r, R),
                  ipm = at(places[u].pm, r, R);
        const Block bl = rotate_block(Block{a[ipp], a[imm], a[imp], a[ipm]}, r1, r2);
        a[ipp] = bl.pp;
        a[imm] = bl.mm;
        a[imp] = bl.mp;
        a[ipm] = bl.pm;
      }
    }
    if (WITH_V && cnt > 0 && tid >= t0) {
      const int lane = tid & 31;                                 // a warp per pair, a lane per component
      for (int q = (tid - t0) >> 5; q < np; q += (nt - t0) >> 5) {
        const double2 x = c0[q];
        if (x.y == 0.0 || lane >= n) continue;
        int p = r + q, m = r - q;
        if (p >= R) p -= R;
        if (m < 0) m += R;
        if (q == 0) m = R;
        double *vp = vs + p * n + lane, *vm = vs + m * n + lane;
        const double y = *vp, z = *vm;
        *vp = x.x * y - x.y * z;
        *vm = x.y * y + x.x * z;
      }
    }
    cnt = __syncthreads_count(mine);
    r = rn;
    b ^= 1;
  }
  // eigenvalues (the pairs' diagonal entries before the rotations that are not applied), ranked
  double* d = reinterpret_cast<double*>(dd);                     // 4 np doubles each
  double* dn = reinterpret_cast<double*>(cs);
  double2 fin = make_double2(dp, dm);
  int pi = k + r, mi = r - k;
  if (pi >= R) pi -= R;
  if (mi < 0) mi += R;
  if (k == 0) mi = R;
  if (np == 2 && tid == 1) {
    // pair 1's entries are carried by thread 0; dd has them, as nothing rotates in the last round
    fin = dd[b * np + 1];
  }
  __syncthreads();
  if (tid < np) {
    d[pi] = fin.x;
    d[mi] = fin.y;
  }
  __syncthreads();
  // (NaN last: the ranks are a permutation whatever the values)
  auto key = [&](double x) {
    if (isnan(x)) return order ? -1.0 : __longlong_as_double(0x7ff0000000000000LL);
    return order ? fabs(x) : x;
  };
  for (int j = tid; j < n; j += nt) {
    const double dj = key(d[j]);
    int rk = 0;
    for (int i = 0; i < n; ++i) {
      const double di = key(d[i]);
      rk += order ? (di > dj || (di == dj && i < j)) : (di < dj || (di == dj && i < j));
    }
    if (WITH_V) rank_s[j] = rk;
    else w.rank[j] = rk;
    dn[rk] = scalbn(order ? fabs(d[j]) : d[j], ex_s);
  }
  __syncthreads();
  double* Wb = W + size_t(blockIdx.x) * n;
  for (int j = tid; j < n; j += nt) Wb[j] = dn[j];
  if (!WITH_V && tid == 0) *w.count = count;
  if (WITH_V) {
    double* Vb = V + size_t(blockIdx.x) * n * n;
    for (int e = tid; e < n * n; e += nt) Vb[(e % n) * n + rank_s[e / n]] = vs[e];
  }
}

// V := the product of the logged rotations, columns ranked.  A CTA carries kVecCols components of every
// eigenvector (32 components took 1545 instead of 1105 us on 16 matrices of n = 160); a half-warp applies a pair's
// rotation to them, and the half-warps of a round meet at a barrier.  Bound by that chain of barriers and
// shared-memory round trips; the rounds' rotations come through a ring of kVecRing rounds in shared memory.
constexpr int kVecRing = 8;
__global__ void __launch_bounds__(kVecThreads) k_jacobi_vectors(int n, double* V, char* work, size_t per,
                                                                const int* only_if) {
  extern __shared__ __align__(16) double vec_smem[];
  if (only_if && *only_if == 0) return;
  const int np = jac_pairs(n), P = 2 * np, R = P - 1;
  const int lane = threadIdx.x % kVecCols, h = threadIdx.x / kVecCols;
  constexpr int H = kVecGroups;
  static_assert(kVecPairs * H >= 80, "a round's pairs for n <= 160");
  const int c0 = blockIdx.x * kVecCols;
  const JacWork w = jac_work(work, per, n, blockIdx.y);
  double2* ring = reinterpret_cast<double2*>(vec_smem);          // [kVecRing][np]
  double* v = vec_smem + 2 * kVecRing * np;                // [eigenvector][component]
  for (int j = h; j < P; j += H) v[j * kVecCols + lane] = j == c0 + lane ? 1.0 : 0.0;
  const int count = *w.count;
  auto fetch = [&](int s) {                                      // one commit group a round, empty past the log
    if (s < count && int(threadIdx.x) < np) {
      const unsigned dst = unsigned(__cvta_generic_to_shared(ring + (s % kVecRing) * np + threadIdx.x));
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(w.log + size_t(s) * np + threadIdx.x));
    }
    asm volatile("cp.async.commit_group;");
  };
  for (int s = 0; s < kVecRing - 1; ++s) fetch(s);
  int r = 0;
  for (int s = 0; s < count; ++s) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kVecRing - 2));
    __syncthreads();                                             // round s has landed, round s - 1 is applied
    fetch(s + kVecRing - 1);                                     // into round s - 1's place
    const double2* cs = ring + (s % kVecRing) * np;
    // all loads before the stores: the pairs of a round share no eigenvector
    double2 x[kVecPairs];
    double *vp[kVecPairs], *vm[kVecPairs], y[kVecPairs], z[kVecPairs];
#pragma unroll
    for (int u = 0; u < kVecPairs; ++u) {
      const int k = h + u * H;
      x[u] = k < np ? cs[k] : make_double2(1.0, 0.0);
      int p = r + k, m = r - k;
      if (p >= R) p -= R;
      if (m < 0) m += R;
      if (k == 0) m = R;
      vp[u] = v + p * kVecCols + lane;
      vm[u] = v + m * kVecCols + lane;
    }
#pragma unroll
    for (int u = 0; u < kVecPairs; ++u)
      if (x[u].y != 0.0) {
        y[u] = *vp[u];
        z[u] = *vm[u];
      }
#pragma unroll
    for (int u = 0; u < kVecPairs; ++u)
      if (x[u].y != 0.0) {
        *vp[u] = x[u].x * y[u] - x[u].y * z[u];
        *vm[u] = x[u].y * y[u] + x[u].x * z[u];
      }
    r = r + 1 == R ? 0 : r + 1;
  }
  asm volatile("cp.async.wait_all;");
  __syncthreads();
  const int i = c0 + lane;
  if (i < n) {
    double* Vb = V + size_t(blockIdx.y) * n * n;
    for (int j = h; j < n; j += H) Vb[i * n + w.rank[j]] = v[j * kVecCols + lane];
  }
}

size_t jac_smem_bytes(int n) {
  const size_t np = size_t(jac_pairs(n));
  return (8 * np + np * (2 * np - 1) + (n <= kFusedMax ? 2 * np * size_t(n) : 0)) * sizeof(double);
}
size_t jac_vec_smem_bytes(int n) {
  const size_t np = size_t(jac_pairs(n));
  return (2 * kVecRing * np + 2 * np * kVecCols) * sizeof(double);
}

// One thread per pivot block and, in warps of their own, one per other block up to 1024: a barrier of fewer
// warps is cheaper, and past 1024 the blocks of a thread follow one another.
int jac_threads(int n) {
  const int np = jac_pairs(n), t0 = (np + 31) & ~31;
  const int others = std::max((np * np / 2 + 31) & ~31, n <= kFusedMax ? 32 * std::min(np, 8) : 0);
  return std::min(kJacThreads, t0 + others);
}

constexpr size_t kJacGroupBytes = size_t(512) << 20;   // rotation logs of the matrices of one launch

int jac_group(int n, int batch) {
  const size_t most = std::min<size_t>(32768, std::max<size_t>(1, kJacGroupBytes / jac_bytes(n)));
  return int(std::min<size_t>(size_t(batch), most));
}

}  // namespace

size_t syev_work_bytes(int n, int batch) { return n <= kFusedMax ? 0 : jac_bytes(n) * jac_group(n, batch); }

int launch_syev(Context* c, int n, int batch, const double* A, int64_t lda, int64_t a_bs, double* W, double* V,
                int order, void* work, const int* only_if) {
  if (n < 1 || n > MCNLA_B200_MAX_DIM_SKETCH || batch < 1) return MCNLA_B200_ERR_UNSUPPORTED;
  const size_t smem = jac_smem_bytes(n);
  if (smem > c->smem_optin) return MCNLA_B200_ERR_UNSUPPORTED;
  if (n <= kFusedMax) {
    // V in the same CTA: n = 12 (8 matrices) 56 us against 53 + 18 in two kernels, n = 32 (16) 256 against 188 + 69,
    // n = 64 (64) 919 against 497 + 318
    MB_CHECK(set_smem(c, reinterpret_cast<const void*>(k_jacobi_rotations<true>), smem));
    k_jacobi_rotations<true><<<batch, jac_threads(n), smem, c->stream>>>(n, A, lda, a_bs, W, V, order, nullptr, 0,
                                                                        only_if);
    MB_CHECK_CUDA(cudaGetLastError());
    c->kernels_launched++;
    return MCNLA_B200_OK;
  }
  if (!work) return MCNLA_B200_ERR_WORKSPACE;
  const size_t vsmem = jac_vec_smem_bytes(n);
  MB_CHECK(set_smem(c, reinterpret_cast<const void*>(k_jacobi_rotations<false>), smem));
  const int group = jac_group(n, batch);
  const size_t per = jac_bytes(n);
  for (int b0 = 0; b0 < batch; b0 += group) {
    const int m = std::min(group, batch - b0);
    k_jacobi_rotations<false><<<m, jac_threads(n), smem, c->stream>>>(
        n, A + b0 * a_bs, lda, a_bs, W + size_t(b0) * n, V, order, static_cast<char*>(work), per, only_if);
    MB_CHECK_CUDA(cudaGetLastError());
    k_jacobi_vectors<<<dim3(unsigned(cdiv(n, kVecCols)), unsigned(m)), kVecThreads, vsmem, c->stream>>>(
        n, V + size_t(b0) * n * n, static_cast<char*>(work), per, only_if);
    MB_CHECK_CUDA(cudaGetLastError());
    c->kernels_launched += 2;
  }
  return MCNLA_B200_OK;
}

}  // namespace mb
