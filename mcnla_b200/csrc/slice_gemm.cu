// FP64 products of a fixed matrix with few columns on the int8 tensor cores (see slice.cuh).
#include "slice.cuh"
#include "tma.cuh"

#include <algorithm>
#include <atomic>
#include <cooperative_groups.h>
#include <utility>

namespace mb {
namespace {

namespace cg = cooperative_groups;

constexpr int kKTile = 128;                // bytes of K in a shared-memory tile: one 128-byte swizzle row
constexpr int kTileM = 128;
constexpr int kSums = 8;                   // orders d = s + t kept
constexpr int64_t kMaxK = 18000;           // of a part: 7 K 2^14 < 2^31
constexpr int kStatK = 256;
constexpr unsigned long long kBias = 0x80808080808080ull;   // seven digits of 128: digit = byte ^ 0x80, signed

__device__ __forceinline__ double pow2(int e) {   // |e| < 1023
  return __longlong_as_double((long long)(e + 1023) << 52);
}

constexpr int kNotFinite = INT32_MIN;

// Exponent s with max |x| 2^s below 0.99 2^55 (the largest seven digits hold), and what undoes it per slice base:
// 2^*unscale = 2^(48 - s).  Any finite maximum, subnormal ones included; not finite: kNotFinite.
__device__ __forceinline__ int scale_of(double mx, int* unscale) {
  *unscale = 0;
  if (mx == 0.0) return 0;
  if (!(mx <= 1.7976931348623157e308)) {
    *unscale = kNotFinite;
    return 0;
  }
  int e;
  const double f = frexp(mx, &e);                                       // mx = f 2^e, f in [1/2, 1)
  if (f >= 0.99) ++e;
  *unscale = e - 7;
  return 55 - e;
}

// v 2^e for the sum of two such exponents (below 2^-1120 everything here is zero)
__device__ __forceinline__ double times_pow2(double v, int e) {
  const int c = max(e, -1120), h = c / 2;
  return v * pow2(h) * pow2(c - h);
}

__device__ __forceinline__ unsigned long long digits(double y) {   // y: the scaled entry
  return (unsigned long long)(__double2ll_rn(y) + (long long)kBias);
}

// Slices in tiles of `tile` rows by 128 bytes of K, a tile's seven slices one after the other, tiles along K, then
// along the rows: what a CTA reads is contiguous (128-byte pieces of rows of K bytes apart ran at 2.6 TB/s).
struct Sliced {
  uint8_t* base;
  int* unscale;         // [row]: exponents
  int64_t kt;           // k-tiles
  int64_t tile;         // rows of a tile
  __device__ __forceinline__ uint8_t* at(int64_t row, int64_t k) const {   // slice 0 (the highest digit)
    return base + (((row / tile) * kt + k / kKTile) * kSlices * tile + row % tile) * kKTile + k % kKTile;
  }
  __device__ __forceinline__ int64_t plane() const { return tile * kKTile; }
};

// Four digits of consecutive k, one word a plane.
__device__ __forceinline__ void store4(const unsigned long long (&u)[4], uint8_t* dst, int64_t plane) {
#pragma unroll
  for (int s = 0; s < kSlices; ++s) {
    const int sh = 8 * (kSlices - 1 - s);
    const uint32_t w = uint32_t((u[0] >> sh) & 255u) | uint32_t((u[1] >> sh) & 255u) << 8 |
                       uint32_t((u[2] >> sh) & 255u) << 16 | uint32_t((u[3] >> sh) & 255u) << 24;
    *reinterpret_cast<uint32_t*>(dst + s * plane) = w ^ 0x80808080u;
  }
}

// Rows with K contiguous, one CTA a row.
__global__ void __launch_bounds__(256) k_slice_rows(const double* __restrict__ A, int64_t lda, int64_t K, Sliced o) {
  __shared__ double red[8];
  const int64_t row = blockIdx.x;
  const double* a = A + row * lda;
  double mx = 0.0;
  bool nan = false;
  for (int64_t k = threadIdx.x; k < K; k += 256) {
    const double x = fabs(a[k]);
    nan |= x != x;
    mx = fmax(mx, x);
  }
  if (nan) mx = __longlong_as_double(0x7ff0000000000000LL);    // fmax drops NaN
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, d));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
  __syncthreads();
  for (int w = 0; w < 8; ++w) mx = fmax(mx, red[w]);
  int un;
  const int e = scale_of(mx, &un);
  if (threadIdx.x == 0) o.unscale[row] = un;
  const int h = e / 2;
  const double s1 = pow2(h), s2 = pow2(e - h);
  const bool ok = un != kNotFinite;
  for (int64_t q = threadIdx.x; q < o.kt * (kKTile / 4); q += 256) {
    unsigned long long u[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int64_t k = 4 * q + j;
      u[j] = digits(ok && k < K ? a[k] * s1 * s2 : 0.0);
    }
    store4(u, o.at(row, 4 * q), o.plane());
  }
}

// Rows along the other dimension (element (r, k) at p[k ld + r]): the maxima of chunks of kStatK, then tiles
// through shared memory; each CTA of the second kernel combines its rows' maxima itself.
__global__ void __launch_bounds__(256) k_slice_max(const double* __restrict__ B, int64_t ld, int64_t R, int64_t K,
                                                   double* part) {
  __shared__ double sm[8][33];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t r = int64_t(blockIdx.x) * 32 + lane;
  const int64_t k0 = int64_t(blockIdx.y) * kStatK, k1 = min(K, k0 + kStatK);
  double mx = 0.0;
  bool nan = false;
  if (r < R) {
#pragma unroll 8
    for (int64_t k = k0 + w; k < k1; k += 8) {
      const double x = fabs(B[k * ld + r]);
      nan |= x != x;
      mx = fmax(mx, x);
    }
  }
  sm[w][lane] = nan ? __longlong_as_double(0x7ff0000000000000LL) : mx;
  __syncthreads();
  if (w == 0 && r < R) {
    for (int i = 0; i < 8; ++i) mx = fmax(mx, sm[i][lane]);
    part[int64_t(blockIdx.y) * R + r] = mx;
  }
}

__global__ void __launch_bounds__(256) k_slice_cols(const double* __restrict__ B, int64_t ld, int64_t R, int64_t K,
                                                    const double* __restrict__ part, int chunks, Sliced o) {
  __shared__ double tile[32][kKTile + 2];
  __shared__ double sm[8][33];
  __shared__ int se[32];
  __shared__ int sok[32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t r0 = int64_t(blockIdx.y) * 32, k0 = int64_t(blockIdx.x) * kKTile;
  const int64_t r = r0 + lane;
  double mx = 0.0;
  if (r < R)
    for (int c = w; c < chunks; c += 8) mx = fmax(mx, part[int64_t(c) * R + r]);
  sm[w][lane] = mx;
  for (int k = w; k < kKTile; k += 8) tile[lane][k] = (r < R && k0 + k < K) ? B[(k0 + k) * ld + r] : 0.0;
  __syncthreads();
  if (w == 0) {
    for (int i = 1; i < 8; ++i) mx = fmax(mx, sm[i][lane]);
    int un;
    se[lane] = scale_of(mx, &un);
    sok[lane] = un != kNotFinite;
    if (r < R && blockIdx.x == 0) o.unscale[r] = un;
  }
  __syncthreads();
  for (int i = w; i < 32; i += 8) {
    if (r0 + i >= R) break;
    const int e = se[i], h = e / 2;
    const double s1 = pow2(h), s2 = pow2(e - h);
    unsigned long long u[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) u[j] = digits(sok[i] ? tile[i][4 * lane + j] * s1 * s2 : 0.0);
    store4(u, o.at(r0 + i, k0 + 4 * lane), o.plane());
  }
}

// The l columns of B (element (k, j) at p[k ld + j]) in one launch: four columns a cluster, K cut over its CTAs, which
// exchange their maxima through shared memory and read their part again (from cache) into slices.  A warp reads
// eight 32-byte pieces of rows and writes 32 bytes a column and slice.  Latency-bound: one CTA of 1024 threads per
// four columns took 11.6 us for 64 columns of 4096, the clusters 5.2.
constexpr int kFewThreads = 256, kFewCtas = 8;
__global__ void __cluster_dims__(kFewCtas, 1, 1) __launch_bounds__(kFewThreads)
    k_slice_few(const double* __restrict__ B, int64_t ld, int l, int64_t K, Sliced o, const int* guard_stop,
                int guard_it) {
  if (guard_stop && *guard_stop < guard_it) return;
  __shared__ double red[kFewThreads / 32][4];
  __shared__ double cmax[kFewCtas][4];
  auto cluster = cg::this_cluster();
  // a CTA's shared memory may be written from outside only once the CTA runs; the read of B hides the wait
  auto started = cluster.barrier_arrive();
  const int rank = int(cluster.block_rank());
  const int c = threadIdx.x & 3, col = int(blockIdx.x / kFewCtas) * 4 + c;
  const double* b = B + col;
  const int64_t k0 = o.kt * rank / kFewCtas * kKTile, k1 = o.kt * (rank + 1) / kFewCtas * kKTile;
  double mx = 0.0;
  bool nan = false;
  if (col < l) {
#pragma unroll 8
    for (int64_t k = k0 + (threadIdx.x >> 2); k < min(k1, K); k += kFewThreads / 4) {
      const double x = fabs(b[k * ld]);
      nan |= x != x;
      mx = fmax(mx, x);
    }
  }
  if (nan) mx = __longlong_as_double(0x7ff0000000000000LL);
#pragma unroll
  for (int d = 16; d >= 4; d >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, d));
  if ((threadIdx.x & 31) < 4) red[threadIdx.x >> 5][c] = mx;
  __syncthreads();
  cluster.barrier_wait(std::move(started));
  if (threadIdx.x < 4 * kFewCtas) {        // this CTA's maxima to CTA threadIdx.x / 4
    for (int w = 0; w < kFewThreads / 32; ++w) mx = fmax(mx, red[w][c]);
    *cluster.map_shared_rank(&cmax[rank][c], threadIdx.x >> 2) = mx;
  }
  cluster.sync();
#pragma unroll
  for (int w = 0; w < kFewCtas; ++w) mx = fmax(mx, cmax[w][c]);
  int un;
  const int e = scale_of(mx, &un), h = e / 2;
  const double s1 = pow2(h), s2 = pow2(e - h);
  const bool ok = un != kNotFinite && col < l;
  if (rank == 0 && threadIdx.x < 4) o.unscale[col] = un;
  for (int64_t k = k0 + 4 * (threadIdx.x >> 2); k < k1; k += kFewThreads) {
    unsigned long long u[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) u[j] = ok && k + j < K ? digits(b[(k + j) * ld] * s1 * s2) : kBias;
    store4(u, o.at(col, k), o.plane());
  }
}

struct SArgs {
  int b_rows;               // rows of B's tiles (columns, padded to the groups)
  int M, l;
  int kt, kt_per;           // k-tiles in all and of a part
  const int *ua, *ub;       // exponents of the rows and the columns
  double* out;              // [part][M][l]
  int* status;
  const int* guard_stop;
  int guard_it;
};

constexpr int kARing = 6;
constexpr int kATile = kTileM * kKTile;
template <int NB>
struct SCfg {
  static constexpr int BTILE = NB * kKTile;                      // one slice of a group
  static constexpr int BBYTES = kSlices * BTILE;
  static constexpr size_t SMEM = size_t(kARing) * kATile + 2 * size_t(BBYTES) + 1024;
  static constexpr uint32_t TMEM = kSums * NB;
  static_assert(TMEM == 256 || TMEM == 512, "a power of two, the whole of an SM's at most");
};
constexpr uint32_t slice_idesc(int n) {   // kind::i8: D s32, A and B signed 8-bit, K-major, M = 128
  return (2u << 4) | (1u << 7) | (1u << 10) | (uint32_t(n >> 3) << 17) | (uint32_t(kTileM >> 4) << 24);
}

// A CTA: 128 rows of A, one column group, one part of K.  For every k-tile the group's seven slices of B are loaded
// once and the seven slices of A stream past them: slice s of A times the stacked slices of B up to order
// s + t = 7 accumulates into the sums d = s .. 7, which lie side by side in TMEM (NB columns each, all of an SM's TMEM
// for NB = 64).  Warp 0: TMA; warp 1: MMA issue; warps 4-7: the sums to FP64.  Bound by reading A's slices (7 bytes an
// element) and, about as much, by the 34 int8 products.  Every wait is bounded.
template <int NB>
__global__ void __launch_bounds__(256, 1)
    slice_gemm_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b, SArgs g) {
  using T = SCfg<NB>;
  if (g.guard_stop && *g.guard_stop < g.guard_it) return;
  extern __shared__ uint8_t smem_dyn[];
  __shared__ __align__(8) uint64_t full_a[kARing], empty_a[kARing], full_b[2], empty_b[2], acc_full, mma_done;
  __shared__ uint32_t tmem_base_s;
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
  uint8_t* smem_b = smem + kARing * kATile;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = blockIdx.x * kTileM, grp = blockIdx.y, part = blockIdx.z;
  const int kt0 = part * g.kt_per, nkt = min(g.kt - kt0, g.kt_per);

  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)),
                 "r"(T::TMEM));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < kARing; ++s) {
      mbar_init(&full_a[s], 1);
      mbar_init(&empty_a[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&full_b[b], 1);
      mbar_init(&empty_b[b], 1);
    }
    mbar_init(&acc_full, 1);
    mbar_init(&mma_done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = tmem_base_s;

  if (warp == 0 && lane == 0) {
    // ---- producer
    bool ok = true;
    int issued_a = 0, issued_b = 0;
    for (int kt = 0; kt < nkt && ok; ++kt) {
      const int b = kt & 1;
      if (kt >= 2 && !mbar_wait(&empty_b[b], uint32_t(((kt >> 1) & 1) ^ 1))) { ok = false; break; }
      mbar_expect_tx(&full_b[b], T::BBYTES);
      for (int s = 0; s < kSlices; ++s)
        tma_load_2d(smem_b + b * T::BBYTES + s * T::BTILE, &tm_b, &full_b[b], 0,
                    ((kt0 + kt) * kSlices + s) * g.b_rows + grp * NB);
      ++issued_b;
      for (int s = 0; s < kSlices; ++s) {
        const int i = kt * kSlices + s, slot = i % kARing;
        if (i >= kARing && !mbar_wait(&empty_a[slot], uint32_t(((i / kARing) & 1) ^ 1))) { ok = false; break; }
        mbar_expect_tx(&full_a[slot], kATile);
        tma_load_2d(smem + slot * kATile, &tm_a, &full_a[slot], 0,
                    ((int(blockIdx.x) * g.kt + kt0 + kt) * kSlices + s) * kTileM);
        ++issued_a;
      }
    }
    if (!ok) atomicExch(g.status, MCNLA_B200_ERR_DEVICE_TIMEOUT);
    // the copies in flight land before the CTA's shared memory goes away, whoever gave up
    for (int i = max(0, issued_a - kARing); i < issued_a; ++i)
      mbar_wait(&full_a[i % kARing], uint32_t((i / kARing) & 1));
    for (int i = max(0, issued_b - 2); i < issued_b; ++i) mbar_wait(&full_b[i & 1], uint32_t((i >> 1) & 1));
  } else if (warp == 1 && lane == 0) {
    // ---- MMA issuer
    bool ok = true;
    for (int kt = 0; kt < nkt && ok; ++kt) {
      const int b = kt & 1;
      if (!mbar_wait(&full_b[b], uint32_t((kt >> 1) & 1))) { ok = false; break; }
      fence_after();
      const uint32_t sb = smem_u32(smem_b + b * T::BBYTES);
#pragma unroll
      for (int s = 0; s < kSlices; ++s) {
        const int i = kt * kSlices + s, slot = i % kARing;
        if (ok && !mbar_wait(&full_a[slot], uint32_t((i / kARing) & 1))) ok = false;
        if (!ok) break;
        fence_after();
        const uint32_t sa = smem_u32(smem + slot * kATile);
        constexpr int kMaxN = 256;
        const int n = NB * (s == 0 ? kSlices : kSums - s);      // slice s reaches the orders s .. 7 (0: to 6)
        // order 7 starts with slice 1, whose last NB columns are an instruction of their own in the first k-step
        const int cut = s == 1 ? n - NB : n;
#pragma unroll
        for (int k = 0; k < kKTile / 32; ++k) {
          auto mma = [&](int c0, int cols, uint32_t accumulate) {
            umma_i8(tmem + uint32_t(s * NB + c0), sw128_desc(sa + k * 32), sw128_desc(sb + c0 * kKTile + k * 32),
                    slice_idesc(cols), accumulate);
          };
          const bool first = kt == 0 && k == 0;
          const uint32_t more = first && s == 0 ? 0u : 1u;
          mma(0, cut < kMaxN ? cut : kMaxN, more);
          if (cut > kMaxN) mma(kMaxN, cut - kMaxN, more);
          if (cut < n) mma(cut, n - cut, first ? 0u : 1u);
        }
        umma_commit(&empty_a[slot]);
      }
      if (ok) umma_commit(&empty_b[b]);
    }
    if (ok) umma_commit(&acc_full);
    else atomicExch(g.status, MCNLA_B200_ERR_DEVICE_TIMEOUT);
    umma_commit(&mma_done);      // every MMA issued above completes before TMEM goes back, whatever was given up
    mbar_wait(&mma_done, 0);
  } else if (warp >= 4) {
    // ---- the sums to FP64: D_0 + 2^-8 (D_1 + 2^-8 (...))
    const int q = warp & 3;
    const bool ok = __all_sync(0xffffffffu, mbar_wait(&acc_full, 0));
    fence_after();
    if (!ok) {
      if (lane == 0) atomicExch(g.status, MCNLA_B200_ERR_DEVICE_TIMEOUT);
    } else {
      const int row = m0 + q * 32 + lane;
      const int ua = row < g.M ? g.ua[row] : 0;
      // every MMA has completed, so the ring is idle: 32 x 32 blocks go through it and out a row at a time
      double* stg = reinterpret_cast<double*>(smem) + q * 32 * 33;
#pragma unroll 1
      for (int c = 0; c < NB; c += 32) {
        double acc[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) acc[j] = 0.0;
#pragma unroll 1
        for (int d = kSums - 1; d >= 0; --d) {
          uint32_t r[32];
          tmem_ld32(tmem + (uint32_t(q * 32) << 16) + uint32_t(d * NB + c), r);
#pragma unroll
          for (int j = 0; j < 32; ++j) acc[j] = fma(acc[j], 0x1p-8, double(int(r[j])));
        }
#pragma unroll
        for (int j = 0; j < 32; ++j) stg[lane * 33 + j] = acc[j];
        __syncwarp();
        const int col = grp * NB + c + lane;
        const int ub = col < g.l ? g.ub[col] : 0;
#pragma unroll 4
        for (int i = 0; i < 32; ++i) {
          const int ui = __shfl_sync(0xffffffffu, ua, i);
          if (m0 + q * 32 + i < g.M && col < g.l)
            g.out[(int64_t(part) * g.M + m0 + q * 32 + i) * g.l + col] =
                ui == kNotFinite || ub == kNotFinite ? __longlong_as_double(0x7ff8000000000000LL)
                                                     : times_pow2(stg[i * 33 + lane], ui + ub);
        }
        __syncwarp();
      }
    }
  }
  __syncwarp();
  fence_before();
  __syncthreads();
  if (warp == 2) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(T::TMEM));
  }
}

// C := alpha times the sum of the parts, in order.
__global__ void k_slice_sum(const double* __restrict__ P, int parts, int64_t M, int l, double alpha, double* C,
                            int64_t ldc, const int* guard_stop, int guard_it) {
  if (guard_stop && *guard_stop < guard_it) return;
  const int64_t total = M * l;
  for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < total; e += int64_t(gridDim.x) * blockDim.x) {
    double v = 0.0;
    for (int z = 0; z < parts; ++z) v += P[z * total + e];
    C[(e / l) * ldc + e % l] = alpha * v;
  }
}

size_t up(size_t b) { return (b + 1023) & ~size_t(1023); }

struct ALayout { Sliced o; double* part; int64_t rows; size_t bytes; };
ALayout a_layout(const SlicePlan& p, void* w) {
  ALayout a;
  a.o.kt = cdiv(p.K, kKTile);
  a.o.tile = kTileM;
  a.rows = cdiv(p.M, kTileM) * a.o.kt * kSlices * kTileM;       // of 128 bytes
  char* base = reinterpret_cast<char*>(up(reinterpret_cast<uintptr_t>(w)));
  a.o.base = reinterpret_cast<uint8_t*>(base);
  size_t off = up(size_t(a.rows) * kKTile);
  a.o.unscale = reinterpret_cast<int*>(base + off);
  off += up(size_t(p.M) * 4);
  a.part = reinterpret_cast<double*>(base + off);
  off += up(size_t(cdiv(p.K, kStatK)) * p.M * 8);
  a.bytes = off + 1024;
  return a;
}

struct WLayout { Sliced o; double* sums; int64_t rows; size_t bytes; };
WLayout w_layout(const SlicePlan& p, void* w) {
  WLayout b;
  b.o.kt = cdiv(p.K, kKTile);
  b.o.tile = int64_t(p.groups) * p.nb;
  b.rows = b.o.kt * kSlices * b.o.tile;
  char* base = reinterpret_cast<char*>(up(reinterpret_cast<uintptr_t>(w)));
  b.o.base = reinterpret_cast<uint8_t*>(base);
  size_t off = up(size_t(b.rows) * kKTile);
  b.o.unscale = reinterpret_cast<int*>(base + off);
  off += up(size_t(b.o.tile) * 4);
  b.sums = reinterpret_cast<double*>(base + off);
  off += up(size_t(p.splits) * p.M * p.l * 8);
  b.bytes = off + 1024;
  return b;
}

template <int NB>
int launch_slices(Context* c, const SlicePlan& p, const CUtensorMap& ta, const CUtensorMap& tb, const SArgs& g) {
  static std::atomic<uint64_t> attr_set{0};   // the shared-memory opt-in: one bit per device
  const uint64_t bit = uint64_t(1) << (c->device & 63);
  if (!(attr_set.load(std::memory_order_acquire) & bit)) {
    MB_CHECK_CUDA(cudaFuncSetAttribute(slice_gemm_kernel<NB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       int(SCfg<NB>::SMEM)));
    attr_set.fetch_or(bit, std::memory_order_acq_rel);
  }
  const dim3 grid(unsigned(cdiv(p.M, kTileM)), unsigned(p.groups), unsigned(p.splits));
  slice_gemm_kernel<NB><<<grid, 256, SCfg<NB>::SMEM, c->stream>>>(ta, tb, g);
  MB_CHECK_CUDA(cudaGetLastError());
  return MCNLA_B200_OK;
}

}  // namespace

// Where the line lies: three launches and the summing of the parts against the DMMA GEMM's m K l products.  One
// iteration of the row-block integrator (Qs B and Qs' X, 48 iterations), us, DMMA -> slices:
//     l   L     m       M K     us                   l   L     m       M K     us
//    64   512   8000   4.1e6   107 -> 116           32  1536   8000   1.2e7   137 -> 119
//    64   512  16000   8.2e6   159 -> 154           32  1536  16000   2.5e7   200 -> 152
//    64  2048   4000   8.2e6   171 -> 129           12   768  16000   1.2e7   132 -> 120
//    64  2048  16000   3.3e7   409 -> 217           12   768  32000   2.5e7   200 -> 169
//    32   512  16000   8.2e6   101 -> 117           96   768  16000   1.2e7   304 -> 216
//    32   512  32000   1.6e7   159 -> 160          160  1280   8000   1.0e7   391 -> 285
// so from 8e6 elements of A on, and where K or M is short (its slices leave most of a wave idle in one of the two
// products) only with l enough for 6e8 products.
SlicePlan plan_slices(const Context* c, int64_t M, int64_t K, int l) {
  SlicePlan p;
  p.M = M; p.K = K; p.l = l;
  const double mk = double(M) * double(K);
  if (l < 1 || M < 256 || K < 512 || mk < 8e6) return p;
  if (std::min(M, K) < 768 && mk * l < 6e8) return p;
  p.nb = l <= 32 ? 32 : 64;
  p.groups = int(cdiv(l, p.nb));
  const int64_t sms = c ? c->num_sms : 148;
  if (c && (!c->int8 || c->smem_optin < (p.nb == 32 ? SCfg<32>::SMEM : SCfg<64>::SMEM))) return p;
  const int64_t kt = cdiv(K, kKTile), tiles = cdiv(M, kTileM) * p.groups;
  // parts of K until the CTAs fill the SMs, at least four k-tiles each, and short enough for the 32-bit sums
  int64_t splits = std::max<int64_t>(cdiv(K, kMaxK), std::min<int64_t>(kt / 4, sms / std::max<int64_t>(1, tiles)));
  splits = std::max<int64_t>(1, splits);
  p.kt_per = cdiv(kt, splits);
  p.splits = int(cdiv(kt, p.kt_per));
  // row indices of the slices are 32-bit tensor coordinates, grid dimensions at most 65535
  if (cdiv(M, kTileM) * kt * kSlices * kTileM > INT32_MAX / 2 || kt * kSlices * p.groups * p.nb > INT32_MAX / 2 ||
      cdiv(M, 32) > 65535 || cdiv(K, kStatK) > 65535 || p.splits > 65535)
    return p;
  p.a_bytes = a_layout(p, nullptr).bytes;
  p.w_bytes = w_layout(p, nullptr).bytes;
  p.use = true;
  return p;
}

int slice_a(Context* c, const SlicePlan& p, CMat A, void* aw) {
  if (!p.use || !aw) return MCNLA_B200_ERR_ARG;
  const ALayout a = a_layout(p, aw);
  if (A.cs == 1) {
    k_slice_rows<<<unsigned(p.M), 256, 0, c->stream>>>(A.p, A.rs, p.K, a.o);
    c->kernels_launched++;
  } else if (A.rs == 1) {
    const int chunks = int(cdiv(p.K, kStatK));
    k_slice_max<<<dim3(unsigned(cdiv(p.M, 32)), unsigned(chunks)), 256, 0, c->stream>>>(A.p, A.cs, p.M, p.K, a.part);
    k_slice_cols<<<dim3(unsigned(a.o.kt), unsigned(cdiv(p.M, 32))), 256, 0, c->stream>>>(A.p, A.cs, p.M, p.K, a.part,
                                                                                       chunks, a.o);
    c->kernels_launched += 2;
  } else {
    return MCNLA_B200_ERR_LAYOUT;
  }
  MB_CHECK_CUDA(cudaGetLastError());
  return MCNLA_B200_OK;
}

int slice_mul(Context* c, const SlicePlan& p, const void* aw, CMat B, double alpha, DMat C, void* ww) {
  if (!p.use || !aw || !ww) return MCNLA_B200_ERR_ARG;
  if (B.cs != 1 || C.cs != 1) return MCNLA_B200_ERR_LAYOUT;
  const ALayout a = a_layout(p, const_cast<void*>(aw));
  const WLayout b = w_layout(p, ww);
  k_slice_few<<<unsigned(b.o.tile / 4 * kFewCtas), kFewThreads, 0, c->stream>>>(B.p, B.rs, p.l, p.K, b.o, c->guard_stop,
                                                                               c->guard_it);
  MB_CHECK_CUDA(cudaGetLastError());
  CUtensorMap ta, tb;
  MB_CHECK(make_map_u8(&ta, a.o.base, a.rows, kKTile, kKTile, kKTile, kTileM));
  MB_CHECK(make_map_u8(&tb, b.o.base, b.rows, kKTile, kKTile, kKTile, p.nb));
  SArgs g;
  g.b_rows = int(b.o.tile);
  g.M = int(p.M);
  g.l = p.l;
  g.kt = int(a.o.kt);
  g.kt_per = int(p.kt_per);
  g.ua = a.o.unscale;
  g.ub = b.o.unscale;
  g.out = b.sums;
  g.status = &c->scal->wait_status;
  g.guard_stop = c->guard_stop;
  g.guard_it = c->guard_it;
  if (p.nb == 32) MB_CHECK(launch_slices<32>(c, p, ta, tb, g));
  else MB_CHECK(launch_slices<64>(c, p, ta, tb, g));
  const int blocks = int(std::min<int64_t>(cdiv(p.M * p.l, 256), int64_t(c->num_sms) * 8));
  k_slice_sum<<<blocks, 256, 0, c->stream>>>(b.sums, p.splits, p.M, p.l, alpha, C.p, C.rs, c->guard_stop, c->guard_it);
  MB_CHECK_CUDA(cudaGetLastError());
  c->kernels_launched += 3;
  c->waits_pending = true;
  return MCNLA_B200_OK;
}

}  // namespace mb
