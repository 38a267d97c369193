// The FP64 reciprocal square root and exponential of csrc/fastmath.cuh beside CUDA's, over an array (test only).
#include "fastmath.cuh"

namespace fb {
void set_error(const char *, ...) {}

__global__ void probe_kernel(int n, const double *x, const double *s, double *out) {
  __shared__ double tab[kExpTab];
  load_exp_tab(tab);
  __syncthreads();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  out[i] = rsqrt_pos(x[i]);
  out[n + i] = rsqrt(x[i]);
  out[2 * n + i] = exp_tab(s[i], tab);
  out[3 * n + i] = exp2(s[i] * (1.0 / 64.0));
}
}  // namespace fb

// out: rsqrt_pos(x), rsqrt(x), exp_tab(s), exp2(s / 64), n values each
extern "C" int fastmath_probe(int n, const double *x, const double *s, double *out) {
  double *d = nullptr;
  const size_t b = n * sizeof(double);
  if (!fb::init_exp_tab() || cudaMalloc(&d, 6 * b) != cudaSuccess) return 0;
  bool ok = cudaMemcpy(d, x, b, cudaMemcpyHostToDevice) == cudaSuccess &&
            cudaMemcpy(d + n, s, b, cudaMemcpyHostToDevice) == cudaSuccess;
  if (ok) fb::probe_kernel<<<(n + 255) / 256, 256>>>(n, d, d + n, d + 2 * (size_t)n);
  ok = ok && cudaGetLastError() == cudaSuccess &&
       cudaMemcpy(out, d + 2 * (size_t)n, 4 * b, cudaMemcpyDeviceToHost) == cudaSuccess;
  cudaFree(d);
  return ok;
}
