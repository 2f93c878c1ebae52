// A context whose int8 products are off, as a stage runs again when their workspace does not fit on the device: the
// sketch and the integrators give the int8 results to rounding, and the same iteration count.
#include <cmath>
#include <cstdio>
#include <vector>

#include "../../mcnla_b200/csrc/common.cuh"

static int fails = 0;
static void ok(int status, const char* what) {
  if (status != MCNLA_B200_OK) {
    std::printf("%s: status %d (%s)\n", what, status, mcnla_b200_last_error());
    ++fails;
  }
}

static double difference(const double* x, const double* y, size_t n) {   // relative, in the Frobenius norm
  std::vector<double> a(n), b(n);
  cudaMemcpy(a.data(), x, n * 8, cudaMemcpyDeviceToHost);
  cudaMemcpy(b.data(), y, n * 8, cudaMemcpyDeviceToHost);
  double d = 0.0, s = 0.0;
  for (size_t i = 0; i < n; ++i) {
    d += (a[i] - b[i]) * (a[i] - b[i]);
    s += a[i] * a[i];
  }
  return std::sqrt(d / s);
}

int main() {
  const int64_t m = 8200, n = 900, l = 64, N = 16, L = l * N;
  const mcnla_b200_params p{m, n, 48, 16, int(N)};
  mcnla_b200_ctx* ctx = nullptr;
  if (mcnla_b200_create(&ctx, 0, nullptr) != MCNLA_B200_OK) return 2;
  double *a, *omega, *q[2], *qbar[2];
  if (cudaMalloc(&a, m * n * 8) != cudaSuccess || cudaMalloc(&omega, n * L * 8) != cudaSuccess) return 2;
  for (int i = 0; i < 2; ++i)
    if (cudaMalloc(&q[i], m * L * 8) != cudaSuccess || cudaMalloc(&qbar[i], m * l * 8) != cudaSuccess) return 2;
  ok(mcnla_b200_gaussian(ctx, 1, m * n, a), "gaussian");
  ok(mcnla_b200_gaussian(ctx, 2, n * L, omega), "gaussian");
  int64_t launches[2];
  for (int i = 0; i < 2; ++i) {
    ctx->int8 = i == 0;
    const int64_t before = mcnla_b200_kernels_launched(ctx);
    ok(mcnla_b200_sketch(ctx, &p, a, MCNLA_B200_ROW_MAJOR, n, omega, 0, q[i]), "sketch");
    launches[i] = mcnla_b200_kernels_launched(ctx) - before;
  }
  const double sketch = difference(q[0], q[1], size_t(m) * L);
  std::printf("sketch: %lld and %lld launches, difference %.1e\n", (long long)launches[0], (long long)launches[1], sketch);
  if (!(launches[0] > launches[1]) || !(sketch < 1e-14)) ++fails;
  ok(mcnla_b200_orthogonalize(ctx, &p, q[0]), "orthogonalize");
  for (int kind : {MCNLA_B200_KOLMOGOROV_NAGUMO, MCNLA_B200_ROW_BLOCK_KOLMOGOROV_NAGUMO,
                   MCNLA_B200_ROW_BLOCK_GRAMIAN_KOLMOGOROV_NAGUMO}) {
    int it[2] = {0, 0};
    for (int i = 0; i < 2; ++i) {
      ctx->int8 = i == 0;
      ok(mcnla_b200_integrate(ctx, &p, kind, q[0], 12, 1e-9, qbar[i], &it[i]), "integrate");
    }
    const double d = difference(qbar[0], qbar[1], size_t(m) * l);
    std::printf("integrator %d: %d and %d iterations, difference %.1e\n", kind, it[0], it[1], d);
    if (it[0] != it[1] || !(d < 1e-13)) ++fails;
  }
  mcnla_b200_destroy(ctx);
  std::printf("%s\n", fails ? "FAILED" : "OK");
  return fails != 0;
}
