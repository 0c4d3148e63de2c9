// The engine's own arithmetic in place of library functions (csrc/sph_device.cuh), over arrays:
// built by test_gpu_device_math.py.
#include "sph_device.cuh"

namespace {

// op 0: inv_sqrt(a), 1: its seed, 2: quotient(a, b), 3: the seed of 1 / b,
// 4: length_of(a, inv_sqrt(a))
__global__ void k_eval(int op, const double* a, const double* b, double* out, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double y = 0.0;
  if (op == 0) y = sph::inv_sqrt(a[i]);
  if (op == 1) asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a[i]));
  if (op == 2) y = sph::quotient(a[i], b[i]);
  if (op == 3) asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b[i]));
  if (op == 4) y = sph::length_of(a[i], sph::inv_sqrt(a[i]));
  out[i] = y;
}

}  // namespace

// Host arrays of n; returns a CUDA error code.
extern "C" int eval_host(int op, const double* a, const double* b, double* out, int n) {
  double* d = nullptr;
  const size_t bytes = (size_t)n * sizeof(double);
  cudaError_t e = cudaMalloc(&d, 3 * bytes);
  if (e != cudaSuccess) return (int)e;
  e = cudaMemcpy(d, a, bytes, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d + n, b, bytes, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    k_eval<<<(n + 255) / 256, 256>>>(op, d, d + n, d + 2 * (size_t)n, n);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(out, d + 2 * (size_t)n, bytes, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return (int)e;
}
