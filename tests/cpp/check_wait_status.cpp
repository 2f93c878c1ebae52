// A bounded wait of an int8 product that ran out is reported by the call it ran out in: the sketch and the integrator are
// given a device status as such a wait leaves it (written here, nothing is made to wait), and have to return it, once.
#include <cstddef>
#include <cstdio>

#include "../../mcnla_b200/csrc/common.cuh"

static int fails = 0;
static void expect(int got, int want, const char* what) {
  std::printf("%s: %d (expected %d)\n", what, got, want);
  if (got != want) ++fails;
}

int main() {
  const int64_t m = 2048, n = 4096;
  mcnla_b200_params p{m, n, 64, 32, 8};
  const int64_t l = 96, L = l * 8;
  const mcnla_b200_params pi{16384, 64, 64, 32, 16};     // its Gramian is an int8 product
  mcnla_b200_ctx* ctx = nullptr;
  if (mcnla_b200_create(&ctx, 0, nullptr) != MCNLA_B200_OK) return 2;
  double *a, *omega, *q, *qs, *qbar;
  if (cudaMalloc(&a, m * n * 8) != cudaSuccess || cudaMalloc(&omega, n * L * 8) != cudaSuccess ||
      cudaMalloc(&q, m * L * 8) != cudaSuccess || cudaMalloc(&qs, pi.nrow * l * 16 * 8) != cudaSuccess ||
      cudaMalloc(&qbar, pi.nrow * l * 8) != cudaSuccess)
    return 2;
  if (mcnla_b200_gaussian(ctx, 1, m * n, a) != MCNLA_B200_OK ||
      mcnla_b200_gaussian(ctx, 2, n * L, omega) != MCNLA_B200_OK ||
      mcnla_b200_gaussian(ctx, 3, pi.nrow * l * 16, qs) != MCNLA_B200_OK)
    return 2;
  auto sketch = [&] { return mcnla_b200_sketch(ctx, &p, a, MCNLA_B200_ROW_MAJOR, n, omega, 0, q); };
  int it = 0;
  auto integrate = [&] {
    return mcnla_b200_integrate(ctx, &pi, MCNLA_B200_ROW_BLOCK_GRAMIAN_KOLMOGOROV_NAGUMO, qs, 0, 1e-4, qbar, &it);
  };
  auto plant = [&] {
    const int status = MCNLA_B200_ERR_DEVICE_TIMEOUT;
    if (cudaMemcpy(&ctx->scal->wait_status, &status, sizeof(int), cudaMemcpyHostToDevice) != cudaSuccess) ++fails;
  };
  expect(sketch(), MCNLA_B200_OK, "sketch");
  plant();
  expect(sketch(), MCNLA_B200_ERR_DEVICE_TIMEOUT, "sketch in which a wait ran out");
  expect(sketch(), MCNLA_B200_OK, "sketch after it");
  expect(integrate(), MCNLA_B200_OK, "integrate, no iterations");
  plant();
  expect(integrate(), MCNLA_B200_ERR_DEVICE_TIMEOUT, "integrate in which a wait ran out");
  expect(integrate(), MCNLA_B200_OK, "integrate after it");
  cudaFree(a);
  cudaFree(omega);
  cudaFree(q);
  cudaFree(qs);
  cudaFree(qbar);
  mcnla_b200_destroy(ctx);
  std::printf("%s\n", fails ? "FAILED" : "OK");
  return fails != 0;
}
