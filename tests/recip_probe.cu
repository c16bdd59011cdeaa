// The functions of csrc/recip.cuh, the approximations under them and CUDA's own, entry by entry.
#include <cuda_runtime.h>

#include "recip.cuh"

namespace {

__global__ void fp64_kernel(int n, const double* x, const double* v, double* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double a, b;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(a) : "d"(x[i]));
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(b) : "d"(x[i]));
  const double r = bem::reciprocal(x[i]);
  const double o[7] = {a, bem::rsqrt_h3(x[i]), rsqrt(x[i]), b, r, bem::corrected_quotient(v[i], x[i], r), v[i] / x[i]};
  for (int k = 0; k < 7; ++k) out[(size_t)k * n + i] = o[k];
}

__global__ void fp32_kernel(int n, const float* x, const float* v, float* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float r = bem::reciprocal_newton(x[i]), c = bem::reciprocal(x[i]);
  const float o[5] = {r, bem::corrected_quotient(v[i], x[i], r), v[i] / x[i], c, bem::corrected_quotient(v[i], x[i], c)};
  for (int k = 0; k < 5; ++k) out[(size_t)k * n + i] = o[k];
}

}  // namespace

// x, v, out: device addresses, n entries each (out: 7 or 5 times n)
extern "C" int probe_fp64(int n, const double* x, const double* v, double* out) {
  fp64_kernel<<<(n + 255) / 256, 256>>>(n, x, v, out);
  return (int)cudaDeviceSynchronize();
}
extern "C" int probe_fp32(int n, const float* x, const float* v, float* out) {
  fp32_kernel<<<(n + 255) / 256, 256>>>(n, x, v, out);
  return (int)cudaDeviceSynchronize();
}
