// Persistent row-block Gramian Kolmogorov-Nagumo integrator
// (row_block_gramian_kolmogorov_nagumo_integrator.hpp:137-214): one
// cooperative kernel runs the iterations back to back with every operand in
// L2 / HBM and no host round trip, instead of five to seven launches per
// iteration.
//
// State (the same buffers and parity as the launch-per-product loop):
// EB[i & 1] = [E~c | Bc | Bgc] (L x 3l), FF[i & 1] = F~c (l x l); Bs (L x L).
// Iteration i (the products over 16 x 16 tiles spread over the grid, each
// element the same fold of K chunks whatever the grid size; grid_tiles):
//   P1  Bgc := 1/N Bs Bc                                              (:152)
//   --- grid barrier
//   P2  [Dc | Dgc] := 1/N Bc' [Bc | Bgc]                              (:155-158)
//   --- grid barrier
//   P3  the KN step by power series on CTAs [0, ceil(l/8)) (kn_series.cuh):
//       Z, C, inv(C), Fc, ||C - I||_F                                 (:164-214)
//   P4  E~+ := [E~c Bc] [Fc; inv(C)/N],  B+ := [Bc Bgc] [Fc; inv(C)],
//       F~+ := F~c Fc                                                 (:194-204)
//   --- grid barrier; stop when !(||C - I||_F >= tol) (after P4, like the
//       reference's loop condition) or at maxit.
// When the series declines an iteration (4 ||Z||_F > 1/2, usually the first
// one or two), the kernel records it in scal->resume_it and returns; the host
// runs that iteration on the launch-per-product path with the
// matrix-function / eigendecomposition step and starts the kernel again at
// the next one.
#include "kn_series.cuh"

namespace mb {
namespace {

constexpr int kGknThreads = kSerThreads;
constexpr int kGknChunks = 8;            // K chunks of a product's element
static_assert(kGknThreads == 256 && kGknChunks * 32 == 256, "a warp a chunk, a thread an element of a 16 x 16 tile");
constexpr int64_t kGknMaxL = 1536;

struct GknArgs {
  int l, L;
  double inv_n, tol;
  int it0, maxit;
  const double* bs;         // L x L
  double* eb0;              // L x 3l: [E~ | Bc | Bgc], even iterations
  double* eb1;              //   odd iterations
  double* ff0;              // l x l
  double* ff1;
  double* dd;               // l x 2l
  double* fc;               // [Fc; inv(C)]     (2l x l)
  double* fcn;              // [Fc; inv(C)/N]
  double* work;             // series scratch (kn_series_work_doubles(l))
  DevScalars* scal;
  int smax;                 // power slabs of the series step
};

// C (M x N, row stride ldc) := scale A B with A(i, k) = A[i sa + k] (transposed: A[k sa + i]), B(k, j) = B[k ldb + j].
struct Prod {
  const double* A;
  const double* B;
  double* C;
  int sa, ldb, ldc, M, N, K, tiles;
  double scale;
};

__device__ Prod make_prod(const double* A, int sa, const double* B, int ldb, double* C, int ldc, int M, int N, int K,
                          double scale) {
  return Prod{A, B, C, sa, ldb, ldc, M, N, K, ((M + 15) >> 4) * ((N + 15) >> 4), scale};
}

// Sum over k in [kb, ke) of one 16 x 16 tile with the m8n8k4 FP64 MMA: 2 x 2 register blocking, the loads of kU
// k-steps issued before their MMAs, two chains (even and odd k-steps) added at the end.  a: A(row of the lane, t4)
// (AT: the same, K across rows); b: B(t4, column of the lane).  LDG_A: A does not change while the kernel runs (read
// through L1; everything else from L2).  Latency-bound: two doubles a load (by reordering k and the columns) left
// the time as it was.
template <bool AT, bool LDG_A>
__device__ __forceinline__ void tile_chunk(const Prod& p, const double* a, const double* b, bool iv0, bool iv1,
                                           bool jv0, bool jv1, int kb, int ke, double (&s)[2][2][2]) {
  const int t4 = threadIdx.x & 3;
  double c[2][2][2], e[2][2][2];
  auto ld = [](const double* x) { return LDG_A ? __ldg(x) : __ldcg(x); };
#pragma unroll
  for (int q = 0; q < 8; ++q) (&c[0][0][0])[q] = (&e[0][0][0])[q] = 0.0;
#pragma unroll 1
  for (int k = kb; k < ke; k += 4 * kU) {
    double a0[kU], a1[kU], b0[kU], b1[kU];
    const double* ak = a + (AT ? int64_t(k) * p.sa : int64_t(k));
    const double* bk = b + int64_t(k) * p.ldb;
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const bool kv = k + 4 * u + t4 < ke;
      const double* x = ak + (AT ? 4 * u * p.sa : 4 * u);
      const double* y = bk + 4 * u * p.ldb;
      a0[u] = kv && iv0 ? ld(x) : 0.0;
      a1[u] = kv && iv1 ? ld(x + (AT ? 8 : 8 * p.sa)) : 0.0;
      b0[u] = kv && jv0 ? __ldcg(y) : 0.0;
      b1[u] = kv && jv1 ? __ldcg(y + 8) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < kU; u += 2) {
      dmma(c[0][0][0], c[0][0][1], a0[u], b0[u]);
      dmma(c[0][1][0], c[0][1][1], a0[u], b1[u]);
      dmma(c[1][0][0], c[1][0][1], a1[u], b0[u]);
      dmma(c[1][1][0], c[1][1][1], a1[u], b1[u]);
      dmma(e[0][0][0], e[0][0][1], a0[u + 1], b0[u + 1]);
      dmma(e[0][1][0], e[0][1][1], a0[u + 1], b1[u + 1]);
      dmma(e[1][0][0], e[1][0][1], a1[u + 1], b0[u + 1]);
      dmma(e[1][1][0], e[1][1][1], a1[u + 1], b1[u + 1]);
    }
  }
#pragma unroll
  for (int q = 0; q < 8; ++q) (&s[0][0][0])[q] = (&c[0][0][0])[q] + (&e[0][0][0])[q];
}

// The 16 x 16 tiles of `count` products, one after another, spread round-robin over the grid.  Every element is the
// same fold: K is cut into kGknChunks chunks (a function of K alone), each chunk summed by
// tile_chunk, and the chunk sums added in chunk order starting from zero.
// Two ways to compute it, chosen per launch (the bits do not change):
//  * fewer tiles than the grid has warps: a CTA takes one tile at a time,
//    warp w sums chunk w, and the chunk sums are folded in warp order through
//    shared memory (red: 8 x 256 doubles, two block barriers);
//  * otherwise a warp takes whole tiles and folds their chunks itself (no
//    shared memory, no barrier) — on a small share of the SMs (a server
//    worker's) the reduction and its barriers dominated.
// Not inlined: the kernel runs through all of its code once an iteration, from the instruction cache or slowly.
template <bool AT, bool LDG_A>
__device__ __noinline__ void grid_tiles(const Prod* prods, int count, double* red) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t4 = lane & 3;
  int ntiles = 0;
#pragma unroll 1
  for (int q = 0; q < count; ++q) ntiles += prods[q].tiles;
  const int nwarps = int(gridDim.x) * kGknChunks;
  const bool whole = ntiles >= nwarps;
  const int first = whole ? int(blockIdx.x) * kGknChunks + warp : int(blockIdx.x);
  const int step = whole ? nwarps : int(gridDim.x);
#pragma unroll 1
  for (int t = first; t < ntiles; t += step) {
    int lt = t;
    const Prod* pp = prods;
    while (lt >= pp->tiles) lt -= (pp++)->tiles;
    const Prod p = *pp;
    const int ntl = (p.N + 15) >> 4;
    const int ti = (lt / ntl) * 16, tj = (lt % ntl) * 16;
    const int chunk = ((p.K + kGknChunks - 1) / kGknChunks + 3) & ~3;
    const int i0 = ti + g, j0 = tj + g;
    const double* a = AT ? p.A + int64_t(t4) * p.sa + i0 : p.A + int64_t(i0) * p.sa + t4;
    const double* b = p.B + int64_t(t4) * p.ldb + j0;
    double acc[2][2][2];
#pragma unroll
    for (int q = 0; q < 8; ++q) (&acc[0][0][0])[q] = 0.0;
    const int w0 = whole ? 0 : warp, w1 = whole ? kGknChunks : warp + 1;
#pragma unroll 1
    for (int w = w0; w < w1; ++w) {
      const int kb = min(p.K, w * chunk), ke = min(p.K, kb + chunk);
      double cs[2][2][2];
      tile_chunk<AT, LDG_A>(p, a, b, i0 < p.M, i0 + 8 < p.M, j0 < p.N, j0 + 8 < p.N, kb, ke, cs);
#pragma unroll
      for (int q = 0; q < 8; ++q) (&acc[0][0][0])[q] += (&cs[0][0][0])[q];
    }
    if (whole) {
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int i = ti + 8 * (q >> 2) + g, j = tj + 8 * ((q >> 1) & 1) + 2 * t4 + (q & 1);
        if (i < p.M && j < p.N) p.C[int64_t(i) * p.ldc + j] = p.scale * (&acc[0][0][0])[q];
      }
      continue;
    }
#pragma unroll
    for (int q = 0; q < 8; ++q)
      red[warp * 256 + (8 * (q >> 2) + g) * 16 + 8 * ((q >> 1) & 1) + 2 * t4 + (q & 1)] = (&acc[0][0][0])[q];
    __syncthreads();
    {
      const int e = threadIdx.x, r = e >> 4, cc = e & 15;
      double v = 0.0;
#pragma unroll
      for (int w = 0; w < kGknChunks; ++w) v += red[w * 256 + e];
      if (ti + r < p.M && tj + cc < p.N) p.C[int64_t(ti + r) * p.ldc + tj + cc] = p.scale * v;
    }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(kGknThreads, 1) k_gkn_persistent(GknArgs a) {
  extern __shared__ __align__(16) double sm[];
  __shared__ int s_flag;
  const int l = a.l, L = a.L, l3 = 3 * l;
  // the products' reduction space (8 x 256 doubles) aliases the series step's
  // shared memory: the step writes what it reads there and ends on a grid barrier
  double* red = sm;
  // the iterations' products, for even and odd iterations: P1, P2, and P4's three
  __shared__ Prod s_prod[2][5];
  if (threadIdx.x < 2) {
    const int cur = threadIdx.x;
    double* E = cur ? a.eb1 : a.eb0;                   // [E~c | Bc | Bgc]
    double* En = cur ? a.eb0 : a.eb1;
    const double* F = cur ? a.ff1 : a.ff0;
    double* Fn = cur ? a.ff0 : a.ff1;
    Prod* p = s_prod[cur];
    p[0] = make_prod(a.bs, L, E + l, l3, E + 2 * l, l3, L, l, L, a.inv_n);
    p[1] = make_prod(E + l, l3, E + l, l3, a.dd, 2 * l, l, 2 * l, L, a.inv_n);
    p[2] = make_prod(E, l3, a.fcn, l, En, l3, L, l, 2 * l, 1.0);
    p[3] = make_prod(E + l, l3, a.fc, l, En + l, l3, L, l, 2 * l, 1.0);
    p[4] = make_prod(F, l, a.fc, l, Fn, l, l, l, l, 1.0);
  }
  __syncthreads();
#pragma unroll 1
  for (int it = a.it0; it < a.maxit; ++it) {
    const Prod* prod = s_prod[it & 1];
    // P1: Bgc := 1/N Bs Bc
    grid_tiles<false, true>(prod, 1, red);
    if (!grid_sync(a.scal, &s_flag)) return;
    // P2: [Dc | Dgc] := 1/N Bc' [Bc | Bgc]
    grid_tiles<true, false>(prod + 1, 1, red);
    if (!grid_sync(a.scal, &s_flag)) return;
    // P3: KN step (C, inv(C), Fc) by power series
    SeriesArgs s;
    s.l = l;
    s.z_in = nullptr;
    s.dd = a.dd;
    s.inv_n = a.inv_n;
    s.out = a.fc;
    s.outn = a.fcn;
    s.ff = nullptr;                                  // F~+ is one of P4's products
    s.ffn = nullptr;
    s.zg = a.work;
    s.zsg = a.work + size_t(l) * l;
    s.partials = a.work + 2 * size_t(l) * l;
    s.scal = a.scal;
    s.smax = a.smax;
    double norm = 0.0;
    int degree = 0;
    const int r = kn_series_step(s, sm, &s_flag, true, &norm, &degree);
    if (r == kStepTimeout) return;
    if (r == kStepDeclined) {
      if (blockIdx.x == 0 && threadIdx.x == 0) a.scal->resume_it = it;
      return;
    }
    // P4: E~+ := [E~c Bc] [Fc; inv(C)/N];  B+ := [Bc Bgc] [Fc; inv(C)];  F~+ := F~c Fc.  One run of tiles: taken one
    // after the other the products left half the grid without a tile at the smallest sizes.
    grid_tiles<false, false>(prod + 2, 3, red);
    const bool converged = !(norm >= a.tol);
    if (converged) {
      if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.scal->norm = norm;
        a.scal->sweeps = 1000 + degree;
        a.scal->stop_it = it;
      }
      return;
    }
    if (!grid_sync(a.scal, &s_flag)) return;
  }
}

}  // namespace

// Grid: enough CTAs for two 8 x 8 tiles of Bs Bc each, at most one per SM
// or the context's share of the SMs, and at least the ceil(l/8) CTAs of the
// KN step.
int gkn_persistent_grid(const Context* c, int l, int64_t L) {
  const int64_t tiles = ((L + 7) / 8) * ((l + 7) / 8);
  int64_t cap = c->num_sms;
  if (c->coop_cta_limit > 0) cap = std::min<int64_t>(cap, c->coop_cta_limit);
  return int(std::max<int64_t>(std::min<int64_t>(cap, (tiles + 1) / 2), (l + 7) / 8));
}

bool gkn_persistent_fits(const Context* c, int l, int64_t L) {
  // Bs Bc here reads its operands straight from L2; past L ~ 1536 the
  // smem-pipelined GEMM of the launch-per-product loop is faster
  if (l < 1 || l > MCNLA_B200_MAX_DIM_SKETCH || L > kGknMaxL) return false;
  return kn_series_smax(l, c->smem_optin, 0) > 0 && (l + 7) / 8 <= c->num_sms;
}

int launch_gkn_persistent(Context* c, int l, int64_t L, int N, double tol, int it0, int maxit, const double* Bs,
                          double* const EB[2], double* const FF[2], double* DD, double* FC, double* FCN,
                          double* work) {
  if (!gkn_persistent_fits(c, l, L)) return MCNLA_B200_ERR_UNSUPPORTED;
  const int smax = kn_series_smax(l, c->smem_optin, 0);
  const size_t smem =
      std::max<size_t>(kn_series_smem_doubles(l, smax), kGknChunks * 256) * sizeof(double);
  MB_CHECK(set_smem(c, reinterpret_cast<const void*>(k_gkn_persistent), smem));
  GknArgs a;
  a.l = l;
  a.L = int(L);
  a.inv_n = 1.0 / N;
  a.tol = tol;
  a.it0 = it0;
  a.maxit = maxit;
  const int G = gkn_persistent_grid(c, l, L);
  a.bs = Bs;
  a.eb0 = EB[0];
  a.eb1 = EB[1];
  a.ff0 = FF[0];
  a.ff1 = FF[1];
  a.dd = DD;
  a.fc = FC;
  a.fcn = FCN;
  a.work = work;
  a.scal = c->scal;
  a.smax = smax;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(G));
  cfg.blockDim = dim3(kGknThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = c->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  MB_CHECK_CUDA(cudaLaunchKernelEx(&cfg, k_gkn_persistent, a));
  c->kernels_launched++;
  return MCNLA_B200_OK;
}

}  // namespace mb
