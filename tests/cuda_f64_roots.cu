// The FP64 reciprocals and roots of fj_physics.cuh at n given arguments, for
// test_gpu_f64_roots.py: out = rcp_normal | rsqrt_normal | sqrt_normal | rcp_any.
#include "fj_physics.cuh"

__global__ void k_roots(const double* x, double* out, int n) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const double r = fj::rsqrt_normal(x[t]);
  out[t] = fj::rcp_normal(x[t]);
  out[n + t] = r;
  out[2 * n + t] = fj::sqrt_normal(x[t], r);
  out[3 * n + t] = fj::rcp_any(x[t]);
}

extern "C" int f64_roots(const double* x, double* out, int n, void* stream) {
  if (n <= 0) return 1;
  k_roots<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(x, out, n);
  return (int)cudaGetLastError();
}
