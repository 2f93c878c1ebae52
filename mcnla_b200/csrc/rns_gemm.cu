// FP64 products through int8 tensor-core residue products (see rns.cuh).
//
// The scales of A's rows and of B's columns, which also say which tiles of C the DMMA GEMM takes; then for the other
// tiles the residues (K-contiguous int8 planes, one per modulus), the int8 GEMMs of all moduli in one persistent
// launch (tcgen05 kind::i8), and the CRT back to FP64; then the DMMA GEMM on the flagged tiles.  With a B that is not
// drawn, the same kernel forms the products of the magnitudes first, which flag tiles too.
#include "rns.cuh"
#include "rns_math.cuh"
#include "tma.cuh"

#include <algorithm>
#include <atomic>
#include <cmath>

namespace mb {
namespace {

static_assert(rns::kNum == kRnsModuli, "one plane per modulus");
__constant__ rns::Tables kT = rns::make_tables();

constexpr int kKTile = 128;                 // K of a shared-memory tile: one 128-byte swizzle row
constexpr int64_t kMaxChunk = 131071;       // 32-bit sums of products of two signed bytes
constexpr int kTileM = 128, kTileN = 256;    // output tile of a CTA
static_assert(kTileM == kFlagRows && kTileN == kFlagCols, "the DMMA GEMM takes whole tiles");
constexpr double kMaxScale = 0x1p800, kMinScale = 0x1p-800;   // squares: entries within 2^+-400

__device__ __forceinline__ double pow2(int e) {   // |e| < 1023
  return __longlong_as_double((long long)(e + 1023) << 52);
}

// The scale of a row or column from its squared 2-norm and 1-norm: exponent s such that the 2-norm
// times 2^s is at most 2^target.  bad: the DMMA path takes it.
__device__ __forceinline__ int scale_of(double norm2, double norm1, int64_t K, int target, bool* bad) {
  if (norm1 == 0.0 && norm2 == 0.0) { *bad = false; return 0; }
  *bad = !(norm2 <= kMaxScale) || !(norm2 >= kMinScale) || norm1 * norm1 * 64.0 < double(K) * norm2;
  if (*bad) return 0;
  const int e = int((__double_as_longlong(norm2) >> 52) & 0x7ff) - 1022;   // norm2 < 2^e
  return target - ((e + 1) >> 1);
}

// Magnitudes in units of a sixteenth of the root mean square, at most 127, from the upper words of the integers (as the
// residues are; the FP64 conversions cost the residue kernels another 15 %).
constexpr double kLevel = 16.0;
__device__ __forceinline__ float level_of(double norm2, int e, int64_t K) {   // e: the scale's exponent
  return float(kLevel * sqrt(double(K) / (norm2 * pow2(e) * pow2(e))) * 0x1p32);
}
__device__ __forceinline__ uint32_t magnitude(uint64_t u, float level) {
  const int h = int(uint32_t(u >> 32)) - int(rns::kOffset >> 32);
  return uint32_t(min(127, __float2int_rn(fabsf(float(h)) * level)));
}
__device__ __forceinline__ uint32_t pack4_magnitude(const uint64_t (&u)[4], float level) {
  return magnitude(u[0], level) | magnitude(u[1], level) << 8 | magnitude(u[2], level) << 16 | magnitude(u[3], level) << 24;
}

// Four consecutive residue bytes of plane i; u: the elements times their scale, rounded, plus the offset.
__device__ __forceinline__ uint32_t pack4(const uint64_t (&u)[4], const rns::Bytes& w, int i) {
  const uint32_t r0 = rns::residue(u[0], w, kT, i), r1 = rns::residue(u[1], w, kT, i);
  const uint32_t r2 = rns::residue(u[2], w, kT, i), r3 = rns::residue(u[3], w, kT, i);
  return __byte_perm(__byte_perm(r0, r1, 0x0040), __byte_perm(r2, r3, 0x0040), 0x5410);
}

__device__ __forceinline__ uint64_t to_int(double x, double s1, double s2) {
  return uint64_t(__double2ll_rn(x * s1 * s2) + (long long)rns::kOffset);
}

// s = s1 s2: a scale of up to 2^+-460 as two factors, so that no intermediate product leaves the range
__device__ __forceinline__ void split_scale(int s, double* s1, double* s2) {
  const int h = s / 2;
  *s1 = pow2(h);
  *s2 = pow2(s - h);
}

struct Out {
  uint8_t* planes;        // [modulus][row][kp], then the magnitudes
  int64_t rows_pad;       // rows per plane
  int64_t kp;             // bytes per row: K rounded up to kKTile, zero past K
  const uint8_t* live;    // per 1 << live_shift rows: 0 when every tile of theirs is the DMMA path's
  int live_shift;
  const float* level;     // per row: of the magnitudes; null: there are none
};

// Per row: the scale, what undoes it, and whether the DMMA path takes the row's tiles (never cleared here).
struct Scales {
  int* scale;             // exponent; kFlagged
  double* unscale;        // 2^-scale
  uint8_t* flag;
  float* level;           // of the magnitudes; 0: a zero row
};
constexpr int kFlagged = INT32_MIN;

__device__ __forceinline__ void put_scale(const Scales& o, int64_t row, double norm2, double norm1, int64_t K, int target) {
  bool bad;
  const int e = scale_of(norm2, norm1, K, target, &bad);
  o.scale[row] = bad ? kFlagged : e;
  o.unscale[row] = pow2(-e);
  o.level[row] = bad || norm2 == 0.0 ? 0.0f : level_of(norm2, e, K);
  if (bad) o.flag[row] = 1;
}

constexpr int kRowThreads = 256;
template <bool VEC>
__device__ __forceinline__ void load_quad(const double* a, int64_t q, int64_t K, double (&x)[4]) {
  const int64_t k = 4 * q;
  if (VEC && k + 4 <= K) {
    const double2 p0 = *reinterpret_cast<const double2*>(a + k), p1 = *reinterpret_cast<const double2*>(a + k + 2);
    x[0] = p0.x; x[1] = p0.y; x[2] = p1.x; x[3] = p1.y;
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) x[j] = k + j < K ? a[k + j] : 0.0;
  }
}

// Scales of the rows of a K-contiguous matrix, one CTA per row.  A pass of its own, so that which tiles are the
// DMMA path's is known before any row is converted: with a norm and a conversion in one kernel, a matrix with a sparse
// row in every 64 took 1.3 times as long as by the DMMA GEMM alone.  HBM-bound.
template <bool VEC>
__global__ void __launch_bounds__(kRowThreads) k_rns_rowscale(const double* __restrict__ A, int64_t lda, int64_t K,
                                                              int target, Scales o) {
  __shared__ double red_s[kRowThreads / 32], red_m[kRowThreads / 32];
  const int64_t row = blockIdx.x;
  const double* a = A + row * lda;
  const int tid = threadIdx.x;
  double s = 0.0, n1 = 0.0;
  const int64_t quads = (K + 3) / 4;
#pragma unroll 2
  for (int64_t q = tid; q < quads; q += kRowThreads) {
    double x[4];
    load_quad<VEC>(a, q, K, x);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      s = fma(x[j], x[j], s);      // NaN and infinities reach the sum
      n1 += fabs(x[j]);
    }
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    s += __shfl_xor_sync(0xffffffffu, s, d);
    n1 += __shfl_xor_sync(0xffffffffu, n1, d);
  }
  if ((tid & 31) == 0) { red_s[tid >> 5] = s; red_m[tid >> 5] = n1; }
  __syncthreads();
  if (tid == 0) {
    for (int w = 1; w < kRowThreads / 32; ++w) { s += red_s[w]; n1 += red_m[w]; }
    put_scale(o, row, s, n1, K, target);
  }
}

// Residues of the rows of a K-contiguous matrix, one CTA per row.  Bound by the integer pipe: ~100 instructions an
// element (15 residues of a 64-bit integer, two dp4a and a division by rounding each) against 8 bytes read and 15
// written.
template <bool VEC, bool IS_B>
__global__ void __launch_bounds__(kRowThreads) k_rns_rows(const double* __restrict__ A, int64_t lda, int64_t K,
                                                          const int* __restrict__ scale, Out o) {
  const int64_t row = blockIdx.x;
  if (o.live && !o.live[row >> o.live_shift]) return;
  const int e = scale[row];
  if (e == kFlagged) return;       // its planes' bytes are not used
  const double* a = A + row * lda;
  const int64_t quads = (K + 3) / 4;
  double s1, s2;
  split_scale(e, &s1, &s2);
  const int64_t plane = o.rows_pad * o.kp;
  for (int64_t q = threadIdx.x; q < o.kp / 4; q += kRowThreads) {
    uint32_t* w = reinterpret_cast<uint32_t*>(o.planes + row * o.kp) + q;
    if (q >= quads) {
#pragma unroll
      for (int i = 0; i < kRnsModuli; ++i) *reinterpret_cast<uint32_t*>(reinterpret_cast<uint8_t*>(w) + i * plane) = 0u;
      if (o.level) *reinterpret_cast<uint32_t*>(reinterpret_cast<uint8_t*>(w) + kRnsModuli * plane) = 0u;
      continue;
    }
    double x[4];
    load_quad<VEC>(a, q, K, x);
    uint64_t u[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) u[j] = to_int(x[j], s1, s2);   // past K: zero, whose residues are zero
#pragma unroll
    for (int i = 0; i < kRnsModuli; ++i)
      *reinterpret_cast<uint32_t*>(reinterpret_cast<uint8_t*>(w) + i * plane) = pack4(u, IS_B ? kT.b : kT.a, i);
    if (o.level)
      *reinterpret_cast<uint32_t*>(reinterpret_cast<uint8_t*>(w) + kRnsModuli * plane) = pack4_magnitude(u, o.level[row]);
  }
}

// The same for a matrix whose rows run along the other dimension (element (row r, k) at p[k ld + r]): squared
// norms and 1-norms per chunk of kStatK rows of k, combined in order; then tiles through shared memory.
constexpr int kStatK = 256;
__global__ void __launch_bounds__(256) k_rns_colstats(const double* __restrict__ B, int64_t ld, int64_t R, int64_t K,
                                                      double* part) {
  __shared__ double ss[8][33], sm[8][33];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t r = int64_t(blockIdx.x) * 32 + lane;
  const int64_t k0 = int64_t(blockIdx.y) * kStatK, k1 = min(K, k0 + kStatK);
  double s = 0.0, n1 = 0.0;
  if (r < R) {
#pragma unroll 4
    for (int64_t k = k0 + w; k < k1; k += 8) {
      const double x = B[k * ld + r];
      s = fma(x, x, s);
      n1 += fabs(x);
    }
  }
  ss[w][lane] = s;
  sm[w][lane] = n1;
  __syncthreads();
  if (w == 0 && r < R) {
    for (int i = 1; i < 8; ++i) { s += ss[i][lane]; n1 += sm[i][lane]; }
    part[(2 * int64_t(blockIdx.y)) * R + r] = s;
    part[(2 * int64_t(blockIdx.y) + 1) * R + r] = n1;
  }
}

__global__ void k_rns_colscale(const double* part, int64_t R, int64_t K, int chunks, int target, Scales o) {
  const int64_t r = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (r >= R) return;
  double s = 0.0, n1 = 0.0;
  for (int c = 0; c < chunks; ++c) {
    s += part[2 * int64_t(c) * R + r];
    n1 += part[(2 * int64_t(c) + 1) * R + r];
  }
  put_scale(o, r, s, n1, K, target);
}

// The tiles that the DMMA path takes: those with a flagged row or column (added to what an earlier chunk of K flagged),
// whole, since a tile costs either path the same whatever it holds.  One CTA per panel of kTileM rows; live[panel]: a
// tile is left to the int8 path, any_live: to any panel.  lower: tiles above the diagonal count for nothing.
__global__ void __launch_bounds__(kTileN) k_rns_tiles(const uint8_t* __restrict__ row_flag,
                                                      const uint8_t* __restrict__ col_flag, int64_t M, int64_t N,
                                                      int lower, uint8_t* tile, uint8_t* live, uint8_t* any_live,
                                                      int* any) {
  const int64_t panel = blockIdx.x, r = panel * kTileM + threadIdx.x;
  const int nt = int((N + kTileN - 1) / kTileN);
  const int row_bad = __syncthreads_or(threadIdx.x < kTileM && r < M && row_flag[r]);
  bool alive = false, bad = false;
  for (int t = 0; t < nt; ++t) {
    const int64_t c = int64_t(t) * kTileN + threadIdx.x;
    const int col_bad = __syncthreads_or(c < N && col_flag[c]);
    uint8_t* p = tile + panel * nt + t;
    const bool dmma = row_bad || col_bad || *p;
    __syncthreads();
    if (threadIdx.x == 0 && dmma) *p = 1;
    if (lower && int64_t(t) * kTileN >= (panel + 1) * kTileM) continue;
    alive |= !dmma;
    bad |= dmma;
  }
  if (threadIdx.x != 0) return;
  live[panel] = alive;
  if (alive) *any_live = 1;
  if (bad) *any = 1;
}

// The tiles in which the magnitudes' product flagged an element, to the others.
__global__ void k_rns_low_tiles(const uint8_t* __restrict__ low, int64_t count, uint8_t* tile, int* any) {
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= count || !low[i]) return;
  tile[i] = 1;
  *any = 1;
}

constexpr int kColTile = 32;
template <bool IS_B>
__global__ void __launch_bounds__(256) k_rns_cols(const double* __restrict__ B, int64_t ld, int64_t R, int64_t K,
                                                  const int* scale, Out o) {
  __shared__ double tile[kColTile][kKTile + 2];   // [row][k]
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t r0 = int64_t(blockIdx.y) * kColTile, k0 = int64_t(blockIdx.x) * kKTile;
  if (o.live && !o.live[r0 >> o.live_shift]) return;
  const int64_t r = r0 + lane;
  for (int k = w; k < kKTile; k += 8) tile[lane][k] = (r < R && k0 + k < K) ? B[(k0 + k) * ld + r] : 0.0;
  __syncthreads();
  const int64_t plane = o.rows_pad * o.kp;
  for (int i = w; i < kColTile; i += 8) {          // a warp writes one row's 128 bytes of a plane
    const int64_t row = r0 + i;
    if (row >= R) break;
    const int e = scale[row];
    if (e == kFlagged) continue;
    double s1, s2;
    split_scale(e, &s1, &s2);
    uint64_t u[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) u[j] = to_int(tile[i][4 * lane + j], s1, s2);
    uint8_t* dst = o.planes + row * o.kp + k0 + 4 * lane;
#pragma unroll
    for (int m = 0; m < kRnsModuli; ++m)
      *reinterpret_cast<uint32_t*>(dst + m * plane) = pack4(u, IS_B ? kT.b : kT.a, m);
    if (o.level) *reinterpret_cast<uint32_t*>(dst + kRnsModuli * plane) = pack4_magnitude(u, o.level[row]);
  }
}

// ---------------------------------------------------------------------------
// int8 GEMM of every modulus: D_p = A_p B_p' modulo m_p, as CRT digits
// ---------------------------------------------------------------------------
struct GemmArgs {
  int64_t a_rows_pad, b_rows_pad;   // rows per plane of the operand maps
  int a_row0;                       // first row of A's planes (a block of a Gramian)
  int mt, nt;                       // tiles
  int kt;                           // k-tiles
  int lower;                        // 1: only tiles with a_row0 + m0 + kTileM > n0
  int64_t jobs;
  uint8_t* y;                       // [modulus][y_rows][ldy] digits
  int64_t y_rows, ldy;
  const uint8_t* tile;              // [mt][nt]: tiles that the DMMA path takes
  // the magnitudes' product
  const float *row_level, *col_level;    // 0: a zero row or column
  int M, N;                         // valid rows and columns
  int low_sum;                      // below it an element is flagged
  uint8_t* low;                     // [mt][nt]
  int* status;
};

constexpr int kStages = 4;
constexpr int kABytes = kTileM * kKTile, kBBytes = kTileN * kKTile, kStageBytes = kABytes + kBBytes;
constexpr size_t kGemmSmem = size_t(kStages) * kStageBytes + 1024;
// instruction descriptor, kind::i8: D s32, A and B signed 8-bit, K-major, M = 128, N = 256
constexpr uint32_t kIdesc = (2u << 4) | (1u << 7) | (1u << 10) | (uint32_t(kTileN >> 3) << 17) |
                            (uint32_t(kTileM >> 4) << 24);
constexpr uint32_t kTmemCols = 512;         // two 256-column accumulators
constexpr int kEpiWarps = 8;                // two per TMEM lane quarter, 128 columns each
constexpr int kGemmThreads = 128 + 32 * kEpiWarps;

// Job -> modulus and tile (false: a tile above the diagonal).  Rows of tiles run fastest, so concurrent CTAs share
// B's tiles.
struct Job { int p, m, n; };
// The planes of a launch: the residues', the magnitudes' behind them, or all.
enum : int { kResidues = 0, kMagnitudes = 1, kAllPlanes = 2 };
template <int PLANES>
__device__ __forceinline__ bool job_of(const GemmArgs& g, int64_t j, Job* out) {
  const int64_t per = int64_t(g.mt) * g.nt;
  out->p = PLANES == kMagnitudes ? kRnsModuli : int(j / per);
  const int64_t t = j % per;
  out->n = int(t / g.mt);
  out->m = int(t % g.mt);
  return !(g.lower && int64_t(out->n) * kTileN >= g.a_row0 + int64_t(out->m + 1) * kTileM);
}

// Whether the DMMA path takes a tile (the same on all threads).
__device__ __forceinline__ bool tile_unused(const GemmArgs& g, const Job& jb) {
  return g.tile[int64_t(jb.m) * g.nt + jb.n] != 0;
}

// A CTA computes 128 x 256 tiles of every plane's product.  Warp 0: TMA into the ring of 48 KB stages; warp 1: MMA
// issue (M = 128, N = 256, K = 32); warps 4-11: the finished accumulator to CRT digits while the next tile
// accumulates in the other TMEM half.  Every wait is bounded.  What bounds it on long K is power: 2.6 POP/s at the
// 1000 W limit on 2048 x 4096 x 20000 blocks (CTA pairs with cta_group::2, which read a third less from L2, ran
// at the same rate; and pairs launched from several streams at once did not get past their start).
// The magnitudes' plane gives instead of digits whether an element's sum is low.
template <int PLANES>
__global__ void __launch_bounds__(kGemmThreads, 1)
    rns_gemm_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b, GemmArgs g) {
  extern __shared__ uint8_t smem_dyn[];
  __shared__ __align__(8) uint64_t full_bar[kStages];    // the stage's copies have landed
  __shared__ __align__(8) uint64_t empty_bar[kStages];   // the MMAs have read the stage
  __shared__ __align__(8) uint64_t acc_full[2];          // accumulator b is complete
  __shared__ __align__(8) uint64_t acc_empty[2];         // accumulator b has been read
  __shared__ __align__(8) uint64_t mma_done;             // every issued MMA has completed
  __shared__ uint32_t tmem_base_s;
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)),
                 "r"(kTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], kEpiWarps);
    }
    mbar_init(&mma_done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = tmem_base_s;

  if (warp == 0) {
    // ---- producer (the whole warp walks the jobs; one lane copies)
    int64_t it = 0, issued = 0;
    bool ok = true;
    for (int64_t j = blockIdx.x; j < g.jobs && ok; j += gridDim.x) {
      Job jb;
      if (!job_of<PLANES>(g, j, &jb) || tile_unused(g, jb)) continue;
      if (lane == 0) {
        const int ya = int(int64_t(jb.p) * g.a_rows_pad) + g.a_row0 + jb.m * kTileM;
        const int yb = int(int64_t(jb.p) * g.b_rows_pad) + jb.n * kTileN;
        for (int kt = 0; kt < g.kt; ++kt) {
          const int64_t i = it + kt;
          const int s = int(i % kStages);
          if (i >= kStages && !mbar_wait(&empty_bar[s], uint32_t(((i / kStages) & 1) ^ 1))) {
            ok = false;
            break;
          }
          mbar_expect_tx(&full_bar[s], kStageBytes);
          uint8_t* sa = smem + s * kStageBytes;
          tma_load_2d(sa, &tm_a, &full_bar[s], kt * kKTile, ya);
          tma_load_2d(sa + kABytes, &tm_b, &full_bar[s], kt * kKTile, yb);
          ++issued;
        }
      }
      it += g.kt;
      ok = __all_sync(0xffffffffu, ok);
    }
    if (lane == 0) {
      if (!ok) atomicExch(g.status, MCNLA_B200_ERR_DEVICE_TIMEOUT);
      // the copies in flight land before the CTA's shared memory goes away, whoever gave up
      for (int64_t f = issued > kStages ? issued - kStages : 0; f < issued; ++f)
        mbar_wait(&full_bar[f % kStages], uint32_t((f / kStages) & 1));
    }
  } else if (warp == 1) {
    // ---- MMA issuer
    int64_t it = 0, done = 0;
    bool ok = true;
    for (int64_t j = blockIdx.x; j < g.jobs && ok; j += gridDim.x) {
      Job jb;
      if (!job_of<PLANES>(g, j, &jb) || tile_unused(g, jb)) continue;
      if (lane == 0) {
        const int b = int(done & 1);
        if (done >= 2 && !mbar_wait(&acc_empty[b], uint32_t(((done >> 1) - 1) & 1))) ok = false;
        fence_after();
        for (int kt = 0; kt < g.kt && ok; ++kt) {
          const int64_t i = it + kt;
          const int s = int(i % kStages);
          if (!mbar_wait(&full_bar[s], uint32_t((i / kStages) & 1))) { ok = false; break; }
          fence_after();
          const uint32_t sa = smem_u32(smem + s * kStageBytes);
          const uint32_t sb = sa + kABytes;
#pragma unroll
          for (int k = 0; k < kKTile / 32; ++k)
            umma_i8(tmem + uint32_t(b * kTileN), sw128_desc(sa + k * 32), sw128_desc(sb + k * 32), kIdesc,
                    (kt | k) ? 1u : 0u);
          umma_commit(&empty_bar[s]);
        }
        if (ok) umma_commit(&acc_full[b]);
        else atomicExch(g.status, MCNLA_B200_ERR_DEVICE_TIMEOUT);
      }
      it += g.kt;
      ++done;
      ok = __all_sync(0xffffffffu, ok);
    }
    if (lane == 0) {
      umma_commit(&mma_done);      // every MMA issued above completes before TMEM goes back, whatever was given up
      mbar_wait(&mma_done, 0);
    }
  } else if (warp >= 4) {
    // ---- epilogue: residue sums -> digits
    const int q = warp & 3;
    const int c0 = ((warp - 4) >> 2) * (kTileN / 2);
    const bool with_inverse = g.lower != 0;       // a Gramian's one set of residues has no factor
    int64_t done = 0;
    for (int64_t j = blockIdx.x; j < g.jobs; j += gridDim.x) {
      Job jb;
      if (!job_of<PLANES>(g, j, &jb) || tile_unused(g, jb)) continue;
      const int b = int(done & 1);
      // warp-uniform outcome: the TMEM loads below are .sync.aligned
      const bool ok = __all_sync(0xffffffffu, mbar_wait(&acc_full[b], uint32_t((done >> 1) & 1)));
      fence_after();
      if (!ok) {
        if (lane == 0) atomicExch(g.status, MCNLA_B200_ERR_DEVICE_TIMEOUT);
        break;
      }
      if (PLANES == kMagnitudes || (PLANES == kAllPlanes && jb.p == kRnsModuli)) {
        const int row = jb.m * kTileM + q * 32 + lane;
        const bool row_ok = row < g.M && g.row_level[row < g.M ? row : 0] != 0.0f;
        bool low = false;
#pragma unroll 1
        for (int c = 0; c < kTileN / 64; ++c) {
          const int col = jb.n * kTileN + c0 + c * 32 + lane;
          const unsigned cols = __ballot_sync(0xffffffffu, col < g.N && g.col_level[col < g.N ? col : 0] != 0.0f);
          uint32_t r[32];
          tmem_ld32(tmem + (uint32_t(q * 32) << 16) + uint32_t(b * kTileN + c0 + c * 32), r);
#pragma unroll
          for (int e = 0; e < 32; ++e) low |= ((cols >> e) & 1u) && int32_t(r[e]) < g.low_sum;
        }
        if (__any_sync(0xffffffffu, low && row_ok) && lane == 0) g.low[int64_t(jb.m) * g.nt + jb.n] = 1;
        fence_before();
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&acc_empty[b])) : "memory");
        ++done;
        continue;
      }
      uint8_t* dst = g.y + (int64_t(jb.p) * g.y_rows + int64_t(jb.m) * kTileM + q * 32 + lane) * g.ldy +
                     int64_t(jb.n) * kTileN + c0;
#pragma unroll 1
      for (int c = 0; c < kTileN / 64; ++c) {
        uint32_t r[32];
        tmem_ld32(tmem + (uint32_t(q * 32) << 16) + uint32_t(b * kTileN + c0 + c * 32), r);
        uint32_t w[8];
#pragma unroll
        for (int e = 0; e < 32; ++e) r[e] = rns::digit(int32_t(r[e]), kT, jb.p, with_inverse);
#pragma unroll
        for (int e = 0; e < 8; ++e)
          w[e] = __byte_perm(__byte_perm(r[4 * e], r[4 * e + 1], 0x0040),
                             __byte_perm(r[4 * e + 2], r[4 * e + 3], 0x0040), 0x5410);
        uint4* d = reinterpret_cast<uint4*>(dst + c * 32);
        d[0] = make_uint4(w[0], w[1], w[2], w[3]);
        d[1] = make_uint4(w[4], w[5], w[6], w[7]);
      }
      fence_before();
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&acc_empty[b])) : "memory");
      ++done;
    }
  }
  __syncwarp();
  fence_before();
  __syncthreads();
  if (warp == 2) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols));
  }
}

// CRT: the digits of every modulus to FP64 (adding to C when add).  A thread takes four columns, a warp reads
// 128 bytes of each plane.
__global__ void __launch_bounds__(256) k_rns_crt(const uint8_t* __restrict__ y, int64_t y_rows, int64_t ldy, int64_t M,
                                                 int64_t N, const double* __restrict__ ua,
                                                 const double* __restrict__ ub, double* C, int64_t ldc, int add,
                                                 int64_t lower_row0, const uint8_t* __restrict__ tile, int nt) {
  const int64_t row = blockIdx.y;
  const int64_t q = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  const int64_t col = 4 * q;
  if (col >= N || (lower_row0 >= 0 && col > lower_row0 + row) || tile[row / kTileM * nt + col / kTileN]) return;
  const uint8_t* src = y + row * ldy + col;
  const int64_t plane = y_rows * ldy;
  rns::Crt acc[4];
#pragma unroll
  for (int i = 0; i < rns::kGroups; ++i) {
    uint32_t w[3];
#pragma unroll
    for (int h = 0; h < 3; ++h) w[h] = *reinterpret_cast<const uint32_t*>(src + (3 * i + h) * plane);
#pragma unroll
    for (int j = 0; j < 4; ++j)
      acc[j].add((w[0] >> (8 * j)) & 255u, (w[1] >> (8 * j)) & 255u, (w[2] >> (8 * j)) & 255u, kT, i);
  }
  const double sa = ua[row];
  double* dst = C + row * ldc + col;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    if (col + j >= N) break;
    const double v = acc[j].value(kT) * sa * ub[col + j];
    dst[j] = add ? dst[j] + v : v;
  }
}

// ---- host
struct Work {   // workspace layout
  uint8_t *pa, *pb, *y, *row_flag, *col_flag, *tile, *live, *any_live, *low;
  double *ua, *ub, *part;
  float *la, *lb;
  int *scale, *any;
  int64_t a_pad, b_pad, kp, y_rows, ldy, nt;
  size_t block_flags, flags;   // bytes from `any` on: of a call's rows, and with the columns'
  size_t bytes;
};

size_t up(size_t b) { return (b + 1023) & ~size_t(1023); }

Work layout(const RnsPlan& p, void* ws) {
  Work w;
  w.kp = cdiv(p.kc, kKTile) * kKTile;
  w.a_pad = cdiv(p.mb, kTileM) * kTileM;
  w.b_pad = cdiv(p.N, kTileN) * kTileN;
  w.nt = cdiv(p.N, kTileN);
  w.y_rows = w.a_pad;
  w.ldy = w.b_pad;
  char* base = static_cast<char*>(ws);
  size_t off = 0;
  auto take = [&](size_t b) { char* q = base + off; off += up(b); return q; };
  w.pb = reinterpret_cast<uint8_t*>(take(size_t(p.planes) * w.b_pad * w.kp));
  w.pa = p.same ? w.pb : reinterpret_cast<uint8_t*>(take(size_t(p.planes) * w.a_pad * w.kp));
  w.y = reinterpret_cast<uint8_t*>(take(size_t(kRnsModuli) * w.y_rows * w.ldy));
  const int64_t most = std::max(p.M, p.N);
  w.part = reinterpret_cast<double*>(take(size_t(2 * cdiv(p.kc, kStatK)) * most * 8));   // of strided operands
  w.scale = reinterpret_cast<int*>(take(size_t(p.N + p.M) * 4));                          // B's, then A's
  w.ub = reinterpret_cast<double*>(take(size_t(p.N) * 8));
  w.ua = p.same ? w.ub : reinterpret_cast<double*>(take(size_t(p.M) * 8));
  w.lb = reinterpret_cast<float*>(take(size_t(p.N) * 4));
  w.la = p.same ? w.lb : reinterpret_cast<float*>(take(size_t(p.M) * 4));
  w.live = reinterpret_cast<uint8_t*>(take(size_t(cdiv(p.M, kTileM))));
  // cleared together, the columns' flags only where B is new
  const size_t off0 = off;
  w.any = reinterpret_cast<int*>(take(2 * sizeof(int)));
  w.any_live = reinterpret_cast<uint8_t*>(w.any + 1);
  w.tile = reinterpret_cast<uint8_t*>(take(size_t(cdiv(p.M, kTileM) * w.nt)));
  w.low = reinterpret_cast<uint8_t*>(take(size_t(cdiv(p.M, kTileM) * w.nt)));
  if (!p.same) w.row_flag = reinterpret_cast<uint8_t*>(take(size_t(p.M)));
  w.block_flags = off - off0;
  w.col_flag = reinterpret_cast<uint8_t*>(take(size_t(w.b_pad)));
  if (p.same) w.row_flag = w.col_flag;
  w.flags = off - off0;
  w.bytes = off;
  return w;
}

// Scales of R rows (element (r, k) at x.p[r x.rs + k x.cs]).
int scales(Context* c, CMat x, int64_t R, int64_t K, bool is_b, double* part, const Scales& o) {
  const int target = is_b ? rns::kTB : rns::kTA;
  if (x.cs == 1) {
    const bool vec = (reinterpret_cast<uintptr_t>(x.p) & 15) == 0 && x.rs % 2 == 0;
    auto kern = vec ? k_rns_rowscale<true> : k_rns_rowscale<false>;
    kern<<<unsigned(R), kRowThreads, 0, c->stream>>>(x.p, x.rs, K, target, o);
    c->kernels_launched++;
  } else {
    const int chunks = int(cdiv(K, kStatK));
    k_rns_colstats<<<dim3(unsigned(cdiv(R, 32)), unsigned(chunks)), 256, 0, c->stream>>>(x.p, x.cs, R, K, part);
    k_rns_colscale<<<unsigned(cdiv(R, 256)), 256, 0, c->stream>>>(part, R, K, chunks, target, o);
    c->kernels_launched += 2;
  }
  MB_CHECK_CUDA(cudaGetLastError());
  return MCNLA_B200_OK;
}

// Residues of R rows with their scales.  is_b: B's, which carry the CRT's factors.
int residues(Context* c, CMat x, int64_t R, int64_t K, bool is_b, const int* scale, const Out& o) {
  if (x.cs == 1) {
    const bool vec = (reinterpret_cast<uintptr_t>(x.p) & 15) == 0 && x.rs % 2 == 0;
    auto kern = vec ? (is_b ? k_rns_rows<true, true> : k_rns_rows<true, false>)
                    : (is_b ? k_rns_rows<false, true> : k_rns_rows<false, false>);
    kern<<<unsigned(R), kRowThreads, 0, c->stream>>>(x.p, x.rs, K, scale, o);
  } else {
    auto kern = is_b ? k_rns_cols<true> : k_rns_cols<false>;
    kern<<<dim3(unsigned(o.kp / kKTile), unsigned(cdiv(R, kColTile))), 256, 0, c->stream>>>(x.p, x.cs, R, K, scale, o);
  }
  c->kernels_launched++;
  MB_CHECK_CUDA(cudaGetLastError());
  return MCNLA_B200_OK;
}

}  // namespace

// Where the line lies: estimated microseconds of both paths.  The DMMA GEMM runs at ~31 TFLOP/s on tiles
// of 128 columns; the int8 path costs 8.5 ps an element of A (15 residues), 10 ps of B, 12 ps an element of C (digits and
// CRT), waves of 128 x 256 tiles of 15 int8 products at 0.48 us a k-tile (below K = 1024 the epilogue bounds a tile) and
// ~40 us of launches.  Measured, DMMA and int8 (with the magnitudes) in us for M x K by N columns:
//   2048 x 1024:  768: 194, 178   1536: 325, 208     700 x 8192: 512: 257, 272   768: 419, 295
//   4096 x 4096:  192: 422, 319    768: 997, 428    1536: 1850, 646
//   8192 x 2048:  192: 382, 321    256: 391, 321     512: 718, 376
//   16384 x 1024: 192: 406, 354    512: 665, 459    1536: 1744, 802
// A Gramian's triangle halves the products of both.
RnsPlan plan_rns(const Context* c, int64_t M, int64_t N, int64_t K, RnsKind kind, int64_t max_rows) {
  RnsPlan p;
  const bool same = kind == RnsKind::Gramian;
  const int most_planes = same ? kRnsModuli : kRnsModuli + 1;
  p.planes = kind == RnsKind::Given ? kRnsModuli + 1 : kRnsModuli;
  p.M = M; p.N = N; p.K = K; p.same = same;
  p.streamed = max_rows > 0;
  if (M < 1 || N < 1 || K < 1) return p;
  const double m = double(M), n = double(N), k = double(K), half = same ? 0.5 : 1.0;
  const double n128 = double(cdiv(N, 128)) * 128.0;
  const double tiles = double(cdiv(M, kTileM)) * double(cdiv(N, kTileN));
  // a triangle's tiles on the diagonal are whole
  const double computed = same ? 0.5 * (tiles + 2.0 * double(cdiv(N, kTileM))) : tiles;
  const double dmma = half * 2.0 * m * n128 * k / 31e6;
  const double int8 = 40.0 + (same ? 0.0 : 8.5e-6 * m * k) + 10e-6 * n * k + half * 12e-6 * m * n +
                      std::ceil(kRnsModuli * computed / double(c ? c->num_sms : 148)) * 0.48 * std::max(k, 1024.0) / kKTile;
  if (int8 >= dmma) return p;
  if (c && (!c->int8 || c->smem_optin < kGemmSmem)) return p;
  // B's planes within ~1.3 GB (a Gramian's, beside the integrator's state, 0.5 GB): K in chunks of equal size
  const int64_t b_pad = cdiv(N, kTileN) * kTileN;
  const int64_t b_most = int64_t(same ? 512 : 1300) << 20;
  const int64_t most = std::min<int64_t>(kMaxChunk, std::max<int64_t>(4096, b_most / (most_planes * b_pad)));
  p.chunks = int(cdiv(K, most));
  p.kc = p.chunks == 1 ? K : cdiv(cdiv(K, p.chunks), kKTile) * kKTile;
  p.chunks = int(cdiv(K, p.kc));
  // A's planes and the digits of a block of rows within twice C's size, 320 MB at least and 0.7 GB at most; among
  // those, the block whose tiles fill the SMs' waves best (a k-tile takes ~0.48 us, a block's launches ~10 us)
  const int64_t kp = cdiv(p.kc, kKTile) * kKTile;
  const int64_t rows = max_rows > 0 ? std::min(max_rows, M) : M;
  const int64_t cap = std::min<int64_t>(int64_t(700) << 20, std::max<int64_t>(int64_t(320) << 20, 16 * M * N));
  const int64_t row_bytes = p.planes * (same ? 0 : kp) + kRnsModuli * b_pad;
  const int64_t panels = cdiv(rows, kTileM), most_panels = std::max<int64_t>(1, cap / row_bytes / kTileM);
  const int64_t sms = c ? c->num_sms : 148, per_panel = p.planes * cdiv(N, kTileN);
  double best = 0.0;
  for (int64_t q = 1; q <= std::min(panels, most_panels); ++q) {
    const double us = double(cdiv(panels, q)) * (double(cdiv(q * per_panel, sms)) * 0.48 * double(kp / kKTile) + 10.0);
    if (p.mb == 0 || us <= best) {
      best = us;
      p.mb = std::min(rows, q * kTileM);
    }
  }
  // a plane's row index is a 32-bit tensor coordinate, a grid dimension at most 65535
  if (p.planes * b_pad > INT32_MAX / 2 || cdiv(N, kColTile) > 65535 || p.mb > 65535 || cdiv(K, kStatK) > 65535)
    return p;
  p.bytes = layout(p, nullptr).bytes + 1024;
  p.use = true;
  return p;
}

int rns_gemm(Context* c, const RnsPlan& plan, int64_t rows, CMat A, CMat B, DMat C, void* ws, double* dws, int splits,
             bool reuse_b) {
  if (!plan.use || !ws) return MCNLA_B200_ERR_ARG;
  if (C.cs != 1) return MCNLA_B200_ERR_LAYOUT;
  if ((A.cs != 1 && A.rs != 1) || (B.cs != 1 && B.rs != 1)) return MCNLA_B200_ERR_LAYOUT;
  if (rows < 1 || rows > plan.M || (plan.same && rows != plan.N)) return MCNLA_B200_ERR_SHAPE;
  const Work w = layout(plan, reinterpret_cast<void*>((reinterpret_cast<uintptr_t>(ws) + 1023) & ~uintptr_t(1023)));
  const bool magnitudes = plan.planes > kRnsModuli;
  const bool keep_b = reuse_b && plan.chunks == 1 && !plan.same;
  // the flags collect over chunks and blocks; a kept B keeps its own
  MB_CHECK_CUDA(cudaMemsetAsync(w.any, 0, keep_b ? w.block_flags : w.flags, c->stream));
  static std::atomic<uint64_t> attr_set{0};   // the shared-memory opt-in: one bit per device
  const uint64_t bit = uint64_t(1) << (c->device & 63);
  if (!(attr_set.load(std::memory_order_acquire) & bit)) {
    for (auto kern : {rns_gemm_kernel<kResidues>, rns_gemm_kernel<kMagnitudes>, rns_gemm_kernel<kAllPlanes>})
      MB_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kGemmSmem)));
    attr_set.fetch_or(bit, std::memory_order_acq_rel);
  }
  for (int ch = 0; ch < plan.chunks; ++ch) {
    const int64_t k0 = ch * plan.kc, kn = std::min(plan.kc, plan.K - k0);
    const int64_t kp = cdiv(kn, kKTile) * kKTile;
    const CMat ak = cm(A.p + k0 * A.cs, A.rs, A.cs);
    const CMat bk = cm(B.p + k0 * B.rs, B.cs, B.rs);
    int* const sb = w.scale;
    int* const sa = plan.same ? sb : w.scale + plan.N;
    if (!keep_b) MB_CHECK(scales(c, bk, plan.N, kn, !plan.same, w.part, Scales{sb, w.ub, w.col_flag, w.lb}));
    if (!plan.same) MB_CHECK(scales(c, ak, rows, kn, false, w.part, Scales{sa, w.ua, w.row_flag, w.la}));
    k_rns_tiles<<<unsigned(cdiv(rows, kTileM)), kTileN, 0, c->stream>>>(
        w.row_flag, w.col_flag, rows, plan.N, plan.same ? 1 : 0, w.tile, w.live, w.any_live, w.any);
    MB_CHECK_CUDA(cudaGetLastError());
    c->kernels_launched++;
    // a B that later blocks of rows will keep is converted whatever this block needs
    if (!keep_b)
      MB_CHECK(residues(c, bk, plan.N, kn, !plan.same, sb,
                        Out{w.pb, w.b_pad, kp, plan.streamed ? nullptr : w.any_live, 31, magnitudes ? w.lb : nullptr}));
    CUtensorMap tb;
    MB_CHECK(make_map_u8(&tb, w.pb, plan.planes * w.b_pad, kp, kp, kKTile, kTileN));
    for (int64_t r0 = 0; r0 < rows; r0 += plan.mb) {
      const int64_t rn = std::min(plan.mb, rows - r0);
      CUtensorMap ta;
      if (!plan.same) {
        static_assert(kTileM == 1 << 7, "a panel's rows");
        MB_CHECK(residues(c, cm(ak.p + r0 * A.rs, A.rs, A.cs), rn, kn, false, sa + r0,
                          Out{w.pa, w.a_pad, kp, w.live + r0 / kTileM, 7, magnitudes ? w.la + r0 : nullptr}));
        MB_CHECK(make_map_u8(&ta, w.pa, plan.planes * w.a_pad, kp, kp, kKTile, kTileM));
      } else {
        MB_CHECK(make_map_u8(&ta, w.pb, plan.planes * w.b_pad, kp, kp, kKTile, kTileM));
      }
      GemmArgs g;
      g.a_rows_pad = plan.same ? w.b_pad : w.a_pad;
      g.b_rows_pad = w.b_pad;
      g.a_row0 = plan.same ? int(r0) : 0;
      g.mt = int(cdiv(rn, kTileM));
      g.nt = int(cdiv(plan.N, kTileN));
      g.kt = int(kp / kKTile);
      g.lower = plan.same ? 1 : 0;
      g.y = w.y;
      g.y_rows = w.y_rows;
      g.ldy = w.ldy;
      g.tile = w.tile + r0 / kTileM * w.nt;
      g.status = &c->scal->wait_status;
      g.row_level = w.la + r0;
      g.col_level = w.lb;
      g.M = int(rn);
      g.N = int(plan.N);
      g.low_sum = int(double(kn) * kLevel * kLevel / 16.0);
      g.low = w.low + r0 / kTileM * w.nt;
      const int64_t tiles = int64_t(g.mt) * g.nt;
      auto gemm = [&](auto kern, int64_t jobs) -> int {
        g.jobs = jobs;
        kern<<<unsigned(std::min<int64_t>(jobs, c->num_sms)), kGemmThreads, kGemmSmem, c->stream>>>(ta, tb, g);
        MB_CHECK_CUDA(cudaGetLastError());
        c->kernels_launched++;
        return MCNLA_B200_OK;
      };
      if (!magnitudes) {
        MB_CHECK(gemm(rns_gemm_kernel<kResidues>, kRnsModuli * tiles));
      } else {
        // in a launch of their own first, so that the residues' skips the tiles they flag, where that costs at most a
        // twenty-fifth of the waves; else in the same launch
        const int64_t apart = cdiv(tiles, c->num_sms) + cdiv(kRnsModuli * tiles, c->num_sms);
        const int64_t together = cdiv((kRnsModuli + 1) * tiles, c->num_sms);
        const bool first = 25 * (apart - together) <= together;
        if (first) MB_CHECK(gemm(rns_gemm_kernel<kMagnitudes>, tiles));
        else MB_CHECK(gemm(rns_gemm_kernel<kAllPlanes>, (kRnsModuli + 1) * tiles));
        k_rns_low_tiles<<<unsigned(cdiv(tiles, 256)), 256, 0, c->stream>>>(g.low, tiles, w.tile + r0 / kTileM * w.nt,
                                                                          w.any);
        MB_CHECK_CUDA(cudaGetLastError());
        c->kernels_launched++;
        if (first) MB_CHECK(gemm(rns_gemm_kernel<kResidues>, kRnsModuli * tiles));
      }
      k_rns_crt<<<dim3(unsigned(cdiv(plan.N, 1024)), unsigned(rn)), 256, 0, c->stream>>>(
          w.y, w.y_rows, w.ldy, rn, plan.N, w.ua + r0, w.ub, C.p + r0 * C.rs, C.rs, ch > 0,
          plan.same ? r0 : -1, g.tile, g.nt);
      MB_CHECK_CUDA(cudaGetLastError());
      c->kernels_launched++;
    }
  }
  c->waits_pending = true;
  // what was flagged, over the whole K
  GemmFlags fl;
  fl.tile = w.tile;
  fl.nt = w.nt;
  fl.any = w.any;
  return dgemm(c, rows, plan.N, plan.K, 1.0, A, B, 0.0, C, GemmBatch(), dws, splits, plan.same, &fl);
}

}  // namespace mb
