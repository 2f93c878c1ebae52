// Kolmogorov-Nagumo step by power series: device building blocks shared by
// the stand-alone step kernel (kn_series.cu) and the persistent row-block
// Gramian integrator (gkn_persistent.cu).
//
// The step needs C = f(Z) and inv(C) for f(x) = sqrt(1/2 + sqrt(1/4 - x)),
// which the reference forms from an eigendecomposition of the symmetric Z
// (row_block_kolmogorov_nagumo_integrator.hpp:159-180,
// kolmogorov_nagumo_integrator.hpp:146-164).  With c(x) the generating
// function of the Catalan numbers, c(x) = (1 - sqrt(1 - 4x)) / (2x), one has
// (1 + sqrt(1 - 4x)) / 2 = 1 / c(x), so
//     f(x) = c(x)^(-1/2),   1 / f(x) = c(x)^(1/2),
// and the powers of c have the closed-form series (Lagrange inversion)
//     c(x)^r = sum_n  r / (2n + r) * binom(2n + r, n) * x^n,   |x| < 1/4.
// Both series have |a_{n+1}| / |a_n| < 4, so for z = ||Z||_F (>= ||Z||_2)
// the tail after degree d is below |a_{d+1}| z^(d+1) / (1 - 4z).  The step
// picks the smallest d with a tail under 1e-17 and evaluates both
// polynomials by Paterson-Stockmeyer (Z^2 .. Z^s, then Horner in Z^s) on the
// FP64 MMA.  Near convergence Z is tiny (4 ||Z|| ~ 1e-4 .. 1e-2: degree 3 to
// 10); when 4 ||Z||_F > 1/2 (the first iterations) the step declines and the
// caller runs the matrix-function / eigendecomposition form instead.
//
// Work split: CTA b < ceil(l/8) owns rows [8b, 8b + 8) of every l x l
// matrix.  A product X Y with Y = Z or Z^s (read-only, in global memory)
// only needs the CTA's own rows of X, so the powers and the Horner steps run
// without exchange; grid barriers (cooperative launch, bounded waits)
// separate the phases that read whole matrices written by other CTAs: Z,
// Z^s, inv(C) and Fc.  Every CTA of the grid takes part in the barriers.
#pragma once
#include "kernels.cuh"

namespace mb {
namespace {

constexpr int kSerThreads = 256;        // of the CTAs that take the step: a warp a row of the CTA's eight
constexpr int kSerCoefs = 320;          // series coefficients kept in constant memory
constexpr int kSerMaxDegree = 300;      // degree search limit
constexpr int kSerMaxS = 18;            // most power slabs Z^1 .. Z^s on chip (fewer when they do not fit)
constexpr int kSerDirectMax = 12;       // degree up to which plain powers replace Paterson-Stockmeyer
constexpr int kSerZsMax = 112;          // l up to which Z is staged in shared memory for its products
constexpr double kSerMaxRho = 0.9;      // 4 ||Z|| above this: the step declines
constexpr double kSerTail = 1e-17;
constexpr long long kBarrierCycles = 4000000000LL;   // about 2 s at the boost clock

// Series coefficients a_n(r) = r / (2n + r) * binom(2n + r, n) of c(x)^r
// for r = -1/2 (C) and r = +1/2 (inv(C)), from the ratio
// binom(2n + r + 2, n + 1) / binom(2n + r, n) = (2n + r + 2)(2n + r + 1) / ((n + 1)(n + r + 1)),
// evaluated at compile time (IEEE double arithmetic, the same on host and device).
struct SeriesCoefs {
  double f[kSerCoefs];
  double g[kSerCoefs];
};

constexpr SeriesCoefs make_series_coefs() {
  SeriesCoefs t{};
  double bF = 1.0, bG = 1.0;
  for (int n = 0; n < kSerCoefs; ++n) {
    t.f[n] = -0.5 / (2.0 * n - 0.5) * bF;
    t.g[n] = 0.5 / (2.0 * n + 0.5) * bG;
    bF *= (2.0 * n + 1.5) * (2.0 * n + 0.5) / ((n + 1.0) * (n + 0.5));
    bG *= (2.0 * n + 2.5) * (2.0 * n + 1.5) / ((n + 1.0) * (n + 1.5));
  }
  return t;
}

__constant__ SeriesCoefs c_series = make_series_coefs();
__device__ const SeriesCoefs g_series = make_series_coefs();   // for lanes that read different n

// Operands of one step (all l x l blocks row-major with row stride l).
struct SeriesArgs {
  int l;
  const double* z_in;     // plain: Z (l x l), upper triangle read
  const double* dd;       // row block: [Dc | Dgc] (l x 2l)
  double inv_n;
  double* out;            // [C; inv(C)] or [Fc; inv(C)]  (2l x l)
  double* outn;           // [Fc; inv(C)/N] (optional)
  const double* ff;       // F~c (optional, l x l)
  double* ffn;            // F~c Fc
  double* zg;             // scratch: Z (l x l)
  double* zsg;            // scratch: Z^s (l x l)
  double* partials;       // scratch: 3 * ceil(l/8)
  DevScalars* scal;
  int smax;               // power slabs on chip (kn_series_smax)
};

// Shared memory of the step: smax + 4 slabs of 8 rows, reduction space and,
// for l <= kSerZsMax, an l x l operand padded to whole tiles (the slab row stride).
__host__ __device__ constexpr size_t kn_series_smem_doubles(int l, int smax) {
  return size_t(smax + 4) * 8 * (((l + 7) & ~7) + 4) + 32 +
         (l <= kSerZsMax ? size_t((l + 7) & ~7) * (((l + 7) & ~7) + 4) : 0);
}

// Most power slabs (<= kSerMaxS) whose step fits `optin` bytes of shared
// memory next to `extra` doubles of the calling kernel (0 when even 5 do not).
inline int kn_series_smax(int l, size_t optin, size_t extra) {
  for (int smax = kSerMaxS; smax >= 5; --smax)
    if ((kn_series_smem_doubles(l, smax) + extra) * sizeof(double) + 1024 <= optin) return smax;
  return 0;
}

__device__ __forceinline__ void dmma(double& c0, double& c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

// Barrier over the whole (co-resident) grid.  scal->bar_count only grows: at
// a launch it is a multiple of the grid size (zeroed with the scalars at the
// start of a stage; every CTA passes the same number of barriers), so an
// arriving CTA whose atomic returns `old` waits until the count reaches the
// next multiple of gridDim.x.  One release (fence + relaxed add) per CTA and
// acquire polls: no reset on the critical path.  Returns false when the wait
// gave up (MCNLA_B200_ERR_DEVICE_TIMEOUT is recorded); the kernel returns.
__device__ __noinline__ bool grid_sync(DevScalars* scal, volatile int* flag) {
  __syncthreads();
  if (gridDim.x == 1) return true;
  if (threadIdx.x == 0) {
    unsigned* cnt = &scal->bar_count;
    unsigned old;
    asm volatile("fence.acq_rel.gpu;" ::: "memory");
    asm volatile("atom.add.relaxed.gpu.global.u32 %0, [%1], 1;" : "=r"(old) : "l"(cnt) : "memory");
    const unsigned target = (old / gridDim.x + 1) * gridDim.x;
    int ok = 1;
    const long long t0 = clock64();
    while (true) {
      unsigned cur;
      asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(cur) : "l"(cnt) : "memory");
      if (int(cur - target) >= 0) break;
      if (clock64() - t0 > kBarrierCycles) {
        ok = 0;
        atomicExch(&scal->status, MCNLA_B200_ERR_DEVICE_TIMEOUT);
        break;
      }
    }
    asm volatile("fence.acq_rel.gpu;" ::: "memory");
    *flag = ok;
  }
  __syncthreads();
  return *flag != 0;
}

__device__ double block_sum(double v, double* red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x == 0)
    for (int w = 0; w < int(blockDim.x >> 5); ++w) s += red[w];
  return s;                       // valid in thread 0
}

// Fragment loop of one 8 x 8 output tile: c += sum_{k in [kb, ke)} A(g, k) B(k, g')
// with the m8n8k4 FP64 MMA, where lane (g, t4) supplies fa(k) = A(row g, k)
// and fb(k) = B(k, column g) for k = k0 + t4 (both return 0 outside the
// operands; k < ke is checked here).  The loads of kU consecutive k-steps are
// issued before their MMAs so that kU L2 round trips overlap; two
// accumulation chains.  c0, c1: the lane's two accumulator elements.
constexpr int kU = 8;

template <class FA, class FB>
__device__ __forceinline__ void tile_acc(FA fa, FB fb, int kb, int ke, double& c0, double& c1) {
  const int t4 = threadIdx.x & 3;
  double e0 = 0.0, e1 = 0.0;
  for (int k = kb; k < ke; k += 4 * kU) {
    double a[kU], b[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const int kk = k + 4 * u + t4;
      const bool kv = kk < ke;
      a[u] = kv ? fa(kk) : 0.0;
      b[u] = kv ? fb(kk) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < kU; u += 2) {
      dmma(c0, c1, a[u], b[u]);
      dmma(e0, e1, a[u + 1], b[u + 1]);
    }
  }
  c0 += e0;
  c1 += e1;
}

// Two tiles with the same B fragments: c += A1 B, d += A2 B.
template <class FA1, class FA2, class FB>
__device__ __forceinline__ void tile_acc2(FA1 fa1, FA2 fa2, FB fb, int kb, int ke, double& c0, double& c1, double& d0,
                                          double& d1) {
  const int t4 = threadIdx.x & 3;
  for (int k = kb; k < ke; k += 4 * kU) {
    double a1[kU], a2[kU], b[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const int kk = k + 4 * u + t4;
      const bool kv = kk < ke;
      a1[u] = kv ? fa1(kk) : 0.0;
      a2[u] = kv ? fa2(kk) : 0.0;
      b[u] = kv ? fb(kk) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      dmma(c0, c1, a1[u], b[u]);
      dmma(d0, d1, a2[u], b[u]);
    }
  }
}

// C1 = A1 Y (and C2 = A2 Y): A 8 x l slabs in shared memory (row stride ld,
// zero beyond column l), Y l x l in global memory (row stride ldy; or in
// shared memory for SMEM_Y), C slabs in shared memory.  One warp per 8-column
// tile; the two products share the Y fragments.  Ends with a block barrier.
template <bool TRANS_Y = false, bool SMEM_Y = false>
__device__ void slab_mm(const double* A1, const double* A2, int ld, const double* Y, int ldy, int l, double* C1,
                        double* C2) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int g = lane >> 2, t4 = lane & 3;
  const int ntiles = (l + 7) >> 3;
  for (int t = warp; t < ntiles; t += nw) {
    const int n = t * 8 + g;
    const bool nv = n < l;
    // Y(k, n), or Y(n, k) for TRANS_Y
    auto fy = [&](int k) {
      const double* y = TRANS_Y ? Y + size_t(n) * ldy + k : Y + size_t(k) * ldy + n;
      return nv ? (SMEM_Y ? *y : __ldcg(y)) : 0.0;
    };
    double c0 = 0.0, c1 = 0.0;
    double* o1 = C1 + g * ld + t * 8 + 2 * t4;
    if (A2) {
      double d0 = 0.0, d1 = 0.0;
      tile_acc2([&](int k) { return A1[g * ld + k]; }, [&](int k) { return A2[g * ld + k]; }, fy, 0, l, c0, c1, d0,
                d1);
      double* o2 = C2 + g * ld + t * 8 + 2 * t4;
      o2[0] = d0;
      o2[1] = d1;
    } else {
      tile_acc([&](int k) { return A1[g * ld + k]; }, fy, 0, l, c0, c1);
    }
    o1[0] = c0;
    o1[1] = c1;
  }
  __syncthreads();
}

// Step operands with the scratch carved out of `work` (kn_series_work_doubles(l)).
inline SeriesArgs series_args(Context* c, int l, const double* z, const double* dd, double inv_n, double* out,
                       double* outn, const double* ff, double* ffn, double* work, int smax) {
  SeriesArgs a;
  a.l = l;
  a.z_in = z;
  a.dd = dd;
  a.inv_n = inv_n;
  a.out = out;
  a.outn = outn;
  a.ff = ff;
  a.ffn = ffn;
  a.zg = work;
  a.zsg = work + size_t(l) * l;
  a.partials = work + 2 * size_t(l) * l;
  a.scal = c->scal;
  a.smax = smax;
  return a;
}

enum : int { kStepTimeout = -1, kStepDeclined = 0, kStepDone = 1 };

// An l x l matrix (row stride lds) into shared memory (row stride ld, zero up to
// whole tiles): a warp per row, asynchronous 16-byte copies where rows start on
// 16 bytes (l even).  Complete after copies_landed() and a block barrier.
__device__ __noinline__ void load_square(double* dst, int ld, const double* src, int lds, int l) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5, lp8 = (l + 7) & ~7;
#pragma unroll 1
  for (int i = warp; i < lp8; i += nw) {
    double* d = dst + i * ld;
    const double* s = src + size_t(i) * lds;
    const int n = i < l ? l : 0;
    if ((l & 1) == 0) {
#pragma unroll 1
      for (int j = 2 * lane; j < n; j += 64)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(unsigned(__cvta_generic_to_shared(d + j))),
                     "l"(s + j)
                     : "memory");
    } else {
#pragma unroll 1
      for (int j = lane; j < n; j += 32) d[j] = __ldcg(s + j);
    }
#pragma unroll 1
    for (int j = n + lane; j < lp8; j += 32) d[j] = 0.0;
  }
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}
__device__ __forceinline__ void copies_landed() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// Sums that a product's owner lanes update with its elements: F += f C1, G += g C1, D += h C2 (F, G, D slabs).
struct SlabSums {
  double *F, *G, *D;
  double f, g, h;
};

// C1 = A1 Y (and C2 = A2 Y where A2 is given): 8 x l slabs (row stride ld, zero up to whole tiles) in shared memory,
// Y(k, n) = Y[k ys + n yn] in shared or global memory.  A warp per 8-column tile, two accumulation chains: the two
// products', or one's even and odd k-steps.  The precision form's BF16 loop turns other roundings here into 1e-9 of
// its result, so the order of the sums is part of the step.
// One copy of this code for every product of the step (see kn_series_step).  No barrier at the end.
__device__ __noinline__ void slab_product(const double* A1, const double* A2, int ld, const double* Y, int ys, int yn,
                                          int l, double* C1, double* C2, SlabSums sum) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
  const int lp8 = (l + 7) & ~7;
#pragma unroll 1
  for (int t = warp; t * 8 < lp8; t += kSerThreads / 32) {
    const int n = t * 8 + g;
    const double* y = Y + (n < l ? n * yn : 0);
    const int kn = n < l ? l : 0;
    double c0 = 0.0, c1 = 0.0, e0 = 0.0, e1 = 0.0, d0 = 0.0, d1 = 0.0;
    const int o = g * ld + t4;
#pragma unroll 4
    for (int k = 0; k < lp8; k += 8) {
      const double y0 = k + t4 < kn ? y[(k + t4) * ys] : 0.0, y1 = k + 4 + t4 < kn ? y[(k + 4 + t4) * ys] : 0.0;
      if (A2) {
        dmma(c0, c1, A1[o + k], y0);
        dmma(d0, d1, A2[o + k], y0);
        dmma(c0, c1, A1[o + k + 4], y1);
        dmma(d0, d1, A2[o + k + 4], y1);
      } else {
        dmma(c0, c1, A1[o + k], y0);
        dmma(e0, e1, A1[o + k + 4], y1);
      }
    }
    c0 += e0; c1 += e1;
    const int q = g * ld + t * 8 + 2 * t4;
    C1[q] = c0; C1[q + 1] = c1;
    if (A2) { C2[q] = d0; C2[q + 1] = d1; }
    if (sum.F) { sum.F[q] += sum.f * c0; sum.F[q + 1] += sum.f * c1; }
    if (sum.G) { sum.G[q] += sum.g * c0; sum.G[q + 1] += sum.g * c1; }
    if (sum.D) { sum.D[q] += sum.h * d0; sum.D[q + 1] += sum.h * d1; }
  }
}

// One KN step (see the file comment).  Every CTA of the grid calls it
// (kSerThreads threads); CTAs [0, ceil(l/8)) do the work.  Returns kStepDone (C / Fc / inv(C) / F~+ in
// global memory, *norm = ||C - I||_F and *degree in every thread),
// kStepDeclined (4 min(||Z||_F, ||Z||_inf) > 0.9 or not finite; nothing
// written but Z) or
// kStepTimeout.  end_barrier: end with a grid barrier after [Fc; inv(C)] are
// written (when other CTAs read them next); F~+ is written after it.
//
// Latency-bound: a few barriers (1.4 us each) and a chain of small products, and bound by the fetching of its own
// instructions when each of a dozen products is inlined (the stand-alone kernel's code was 155 KB, the persistent
// kernel's 231 KB, run through once an iteration; now 54 and 80): all products are one function, and loops are not
// unrolled but where loads have to be in flight together.  The l x l operands come in by asynchronous copies; the
// plain powers' sums belong to the lanes that form the products, so a power is one call and one block barrier; row
// sums and the degree search are a warp's work without block reductions.  The stand-alone step went from 27 to 20 us
// at l = 64 and from 14.5 to 10.8 at l = 20, an iteration of the persistent kernel from 24.6 to 20.9 us (l = 12,
// N l = 96), 37.4 to 31 (48, 384) and 69 to 61 (96, 768).  16 warps a CTA were slower (registers: 21.2 and 12.8 us).
__device__ int kn_series_step(const SeriesArgs& a, double* sm, volatile int* flag, bool end_barrier, double* norm,
                              int* degree) {
  __shared__ int s_d, s_s;
  __shared__ double s_norm;
  const int l = a.l, tid = threadIdx.x, nt = blockDim.x;
  const int warp = tid >> 5, lane = tid & 31;
  const int gkn = (l + 7) >> 3;
  const bool mine = int(blockIdx.x) < gkn;
  const int lp8 = (l + 7) & ~7, ld = lp8 + 4;
  const int r0 = blockIdx.x * 8;
  const int slab = 8 * ld;
  double* P = sm;                                   // P + (j-1) slab: rows of Z^j, j = 1 .. s
  const int smax = a.smax;
  double* accF = P + smax * slab;
  double* accG = accF + slab;
  double* tF = accG + slab;
  double* tG = tF + slab;
  double* red = tG + slab;
  double* DW = P + 4 * slab;                        // the plain powers: rows of sum g_j Dc Z^j
  double* zs = red + 32;                            // an l x l operand: Dc, then Z, then Fc
  const double* coefF = c_series.f;                 // c^(-1/2): C
  const double* coefG = c_series.g;                 // c^(1/2):  inv(C)
  const int ldd = 2 * l;
  const bool rb = a.dd != nullptr;
  const bool zs_smem = l <= kSerZsMax;
  double* sq = a.partials;                          // per row: squares, absolute values; then ||C - I||_F^2's parts
  double* ab = sq + lp8;
  double* np = ab + lp8;
  if (mine) {
    // ---- Z rows [r0, r0 + 8), a warp per row
    const int i = r0 + warp;
    if (rb) {
      // Z := Dgc - Dc Dc'   (row_block_kolmogorov_nagumo_integrator.hpp:150-156): Dc rows in tF, Dgc's in P
      if (zs_smem) load_square(zs, ld, a.dd, ldd, l);
#pragma unroll 1
      for (int j = lane; j < lp8; j += 32) {
        const bool in = i < l && j < l;
        const double* row = a.dd + size_t(in ? i : 0) * ldd + (in ? j : 0);
        const double x = __ldcg(row), y = __ldcg(row + l);
        tF[warp * ld + j] = in ? x : 0.0;
        P[warp * ld + j] = in ? y : 0.0;
      }
      copies_landed();
      __syncthreads();
      slab_product(tF, nullptr, ld, zs_smem ? zs : a.dd, 1, zs_smem ? ld : ldd, l, tG, nullptr, SlabSums{});
      __syncthreads();
    }
    double ss = 0.0, rs = 0.0;
#pragma unroll 1
    for (int j = lane; j < lp8; j += 32) {
      const bool in = i < l && j < l;
      const int o = warp * ld + j;
      double z;
      // plain: the upper triangle mirrored (the reference's symmetric eigensolver reads one triangle)
      if (rb) z = P[o] - tG[o];
      else z = in ? __ldcg(a.z_in + size_t(min(i, j)) * l + max(i, j)) : 0.0;
      P[o] = z;
      if (in) a.zg[size_t(i) * l + j] = z;
      ss += z * z;
      rs += fabs(z);
      // the plain powers' first terms
      const double id = i == j ? 1.0 : 0.0;
      accF[o] = coefF[0] * id + coefF[1] * z;
      accG[o] = coefG[0] * id + coefG[1] * z;
      if (rb) DW[o] = coefG[0] * tF[o];
    }
    for (int o = 16; o > 0; o >>= 1) {
      ss += __shfl_xor_sync(0xffffffffu, ss, o);
      rs += __shfl_xor_sync(0xffffffffu, rs, o);
    }
    if (lane == 0) {
      sq[i] = ss;
      ab[i] = rs;
    }
  }
  if (!grid_sync(a.scal, flag)) return kStepTimeout;

  // Z for the products below: a shared-memory copy when it fits, in flight behind the degree search
  if (mine && zs_smem) load_square(zs, ld, a.zg, l, l);
  // ---- degree from z = min(||Z||_F, ||Z||_inf) >= ||Z||_2 (the same arithmetic in every CTA): lane n - 1 tests n
  if (warp == 0) {
    double cn = fmax(fabs(__ldg(g_series.f + lane + 1)), fabs(__ldg(g_series.g + lane + 1)));
    double s2 = 0.0, zi = 0.0;
#pragma unroll 1
    for (int b = lane; b < lp8; b += 32) {
      s2 += __ldcg(sq + b);
      zi = fmax(zi, __ldcg(ab + b));
    }
    for (int o = 16; o > 0; o >>= 1) {
      s2 += __shfl_xor_sync(0xffffffffu, s2, o);
      zi = fmax(zi, __shfl_xor_sync(0xffffffffu, zi, o));
    }
    const double z = fmin(sqrt(s2), zi);
    int d = -1;
    if (4.0 * z <= kSerMaxRho) {                    // false for NaN; the same in every lane
      const double scale = 1.0 / (1.0 - 4.0 * z);
      double zn = 1.0, base = z;                    // zn = z^(lane + 1)
#pragma unroll
      for (int e = 0; e < 6; ++e) {
        if (((lane + 1) >> e) & 1) zn *= base;
        base *= base;
      }
      const double z32 = __shfl_sync(0xffffffffu, zn, 31);
#pragma unroll 1
      for (int n0 = 0; n0 <= kSerMaxDegree; n0 += 32) {
        const int n = n0 + lane + 1;
        const unsigned hit = __ballot_sync(0xffffffffu, n <= kSerMaxDegree + 1 && cn * zn * scale <= kSerTail);
        if (hit) {
          d = n0 + __ffs(int(hit)) - 1;             // n - 1
          break;
        }
        zn *= z32;
        const int nn = min(n + 32, kSerCoefs - 1);
        cn = fmax(fabs(__ldg(g_series.f + nn)), fabs(__ldg(g_series.g + nn)));
      }
      if (d == 0) d = 1;
    }
    int s = 1;
#pragma unroll 1
    while (d >= 0 && s * s < d + 1) ++s;
    if (lane == 0) {
      s_d = d;
      s_s = min(s, smax);
    }
  }
  copies_landed();
  __syncthreads();
  const int d = s_d;
  if (d < 0) return kStepDeclined;                  // uniform over the grid
  const int s = s_s;
  const int nq = (d + s) / s;                       // blocks of s coefficients: degree nq*s - 1 >= d
  double* cinv = a.out + size_t(l) * l;
  const double* zy = zs_smem ? zs : a.zg;
  const int zys = zs_smem ? ld : l;
  // C1 = A1 Z, C2 = A2 Z
  auto mm_z = [&](const double* A1, const double* A2, double* C1, double* C2, SlabSums sum) {
    slab_product(A1, A2, ld, zy, zys, 1, l, C1, C2, sum);
    __syncthreads();
  };
  // ||C - I||_F from the rows' parts, by warp 0 (read by all threads after the next block barrier)
  auto norm_of = [&]() {
    if (warp == 0) {
      double s2 = 0.0;
#pragma unroll 1
      for (int b = lane; b < lp8; b += 32) s2 += __ldcg(np + b);
      for (int o = 16; o > 0; o >>= 1) s2 += __shfl_xor_sync(0xffffffffu, s2, o);
      if (lane == 0) s_norm = sqrt(s2);
    }
  };
  // F~+ := F~c Fc   (row_block_gramian_kolmogorov_nagumo_integrator.hpp:197), after the barrier behind Fc
  auto ff_rows = [&]() {
    if (zs_smem) load_square(zs, ld, a.out, l, l);
#pragma unroll 1
    for (int j = lane; j < lp8; j += 32)
      tF[warp * ld + j] = (r0 + warp < l && j < l) ? __ldcg(a.ff + size_t(r0 + warp) * l + j) : 0.0;
    copies_landed();
    __syncthreads();
    slab_product(tF, nullptr, ld, zs_smem ? zs : a.out, zs_smem ? ld : l, 1, l, tG, nullptr, SlabSums{});
    __syncthreads();
#pragma unroll 1
    for (int j = lane; j < l; j += 32)
      if (r0 + warp < l) a.ffn[size_t(r0 + warp) * l + j] = tG[warp * ld + j];
  };
  // The CTA's rows of the results from C in F, inv(C) in G and Dc inv(C) in W (row block), with ||C - I||_F^2's part
  auto put_rows = [&](const double* F, const double* G, const double* W) {
    const int i = r0 + warp;
    double part = 0.0;
    if (i < l) {
#pragma unroll 1
      for (int j = lane; j < l; j += 32) {
        const int o = warp * ld + j;
        const size_t e = size_t(i) * l + j;
        const double c = F[o], ci = G[o], dlt = c - (i == j ? 1.0 : 0.0);
        part += dlt * dlt;
        cinv[e] = ci;
        // Fc := C - Dc inv(C)   (row_block_kolmogorov_nagumo_integrator.hpp:186)
        const double fc = rb ? c - W[o] : c;
        a.out[e] = fc;
        if (rb && a.outn) {
          a.outn[e] = fc;
          a.outn[size_t(l) * l + e] = ci * a.inv_n;
        }
      }
    }
    for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
    if (lane == 0) np[i] = part;
  };

  if (d <= kSerDirectMax) {
    // ---- plain powers: C = sum f_j Z^j, inv(C) = sum g_j Z^j and, for the
    // row-block step, Dc inv(C) = sum g_j (Dc Z^j), all accumulated from the
    // CTA's rows of Z^j and Dc Z^j (products with the full Z only), so Fc
    // = C - Dc inv(C) needs no exchange of C or inv(C).
    if (mine) {
      const double* pc = P;                          // rows of Z^(j-1)
      const double* wc = P + 2 * slab;               // rows of Dc Z^(j-1)
      if (rb) mm_z(tF, nullptr, P + 2 * slab, nullptr, SlabSums{DW, nullptr, nullptr, coefG[1], 0.0, 0.0});
#pragma unroll 1
      for (int j = 2; j <= d; ++j) {
        double* pn = P + (j & 1 ? 0 : 1) * slab;
        double* wn = P + (j & 1 ? 2 : 3) * slab;
        mm_z(pc, rb ? wc : nullptr, pn, wn, SlabSums{accF, accG, rb ? DW : nullptr, coefF[j], coefG[j], coefG[j]});
        pc = pn;
        wc = wn;
      }
      put_rows(accF, accG, DW);
    }
    if (!grid_sync(a.scal, flag)) return kStepTimeout;
    norm_of();
    if (rb && a.ff && a.ffn && mine) ff_rows();
    __syncthreads();
    *norm = s_norm;
    *degree = d;
    return kStepDone;
  }

  // ---- rows of Z^2 .. Z^s (Z^s only when a Horner step needs it)
  if (mine) {
    const int top = nq > 1 ? s : s - 1;
#pragma unroll 1
    for (int j = 2; j <= top; ++j) mm_z(P + (j - 2) * slab, nullptr, P + (j - 1) * slab, nullptr, SlabSums{});
    if (nq > 1) {
#pragma unroll 1
      for (int e = tid; e < 8 * l; e += nt) {
        const int rr = e / l, j = e % l, i = r0 + rr;
        if (i < l) a.zsg[size_t(i) * l + j] = P[(s - 1) * slab + rr * ld + j];
      }
    }
  }
  if (nq > 1 && !grid_sync(a.scal, flag)) return kStepTimeout;

  if (mine) {
    // ---- Horner in Z^s:  acc = B_{nq-1};  acc = acc Z^s + B_q,  B_q = sum_j a_{qs+j} Z^j
    auto add_block = [&](int q, double* dF, double* dG, bool accumulate) {
#pragma unroll 1
      for (int e = tid; e < 8 * lp8; e += nt) {
        const int rr = e / lp8, j = e % lp8, i = r0 + rr;
        double vF = 0.0, vG = 0.0;
        if (i < l && j < l) {
          if (i == j) {
            vF = coefF[q * s];
            vG = coefG[q * s];
          }
#pragma unroll 1
          for (int p = 1; p < s; ++p) {
            const double x = P[(p - 1) * slab + rr * ld + j];
            vF = fma(coefF[q * s + p], x, vF);
            vG = fma(coefG[q * s + p], x, vG);
          }
        }
        const int o = rr * ld + j;
        if (accumulate) {
          dF[o] += vF;
          dG[o] += vG;
        } else {
          dF[o] = vF;
          dG[o] = vG;
        }
      }
      __syncthreads();
    };
    add_block(nq - 1, accF, accG, false);
#pragma unroll 1
    for (int q = nq - 2; q >= 0; --q) {
      slab_product(accF, accG, ld, a.zsg, l, 1, l, tF, tG, SlabSums{});
      __syncthreads();
      add_block(q, tF, tG, true);
      double* x = accF; accF = tF; tF = x;
      x = accG; accG = tG; tG = x;
    }
    // ---- C in accF, inv(C) in accG;  ||e - 1||_2 = ||C - I||_F
    if (rb) {
      // inv(C) for the other CTAs' Dc inv(C)
#pragma unroll 1
      for (int j = lane; j < l; j += 32)
        if (r0 + warp < l) cinv[size_t(r0 + warp) * l + j] = accG[warp * ld + j];
    } else {
      put_rows(accF, accG, nullptr);
    }
  }
  if (!grid_sync(a.scal, flag)) return kStepTimeout;

  if (rb) {
    if (mine) {
      if (zs_smem) load_square(zs, ld, cinv, l, l);
#pragma unroll 1
      for (int j = lane; j < lp8; j += 32)
        tF[warp * ld + j] = (r0 + warp < l && j < l) ? __ldcg(a.dd + size_t(r0 + warp) * ldd + j) : 0.0;
      copies_landed();
      __syncthreads();
      slab_product(tF, nullptr, ld, zs_smem ? zs : cinv, zs_smem ? ld : l, 1, l, tG, nullptr, SlabSums{});
      __syncthreads();
      put_rows(accF, accG, tG);
    }
    // the parts of ||C - I||_F, and Fc for the next product
    if (!grid_sync(a.scal, flag)) return kStepTimeout;
    norm_of();
    if (a.ff && a.ffn && mine) ff_rows();
  } else {
    norm_of();
    if (end_barrier && !grid_sync(a.scal, flag)) return kStepTimeout;
  }
  __syncthreads();
  *norm = s_norm;
  *degree = d;
  return kStepDone;
}

}  // namespace
}  // namespace mb
