// Device results of csrc/fp64_steps.cuh and of CUDA's operators (built and called by test_gpu_fp64_steps.py).
#include <cuda_runtime.h>

#include "fp64_steps.cuh"

using namespace nnpp;

__global__ void k_eval(int op, int n, const double* a, const double* b, double* out, double* cuda) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (op == 0) {
    out[i] = div_newton(a[i], b[i]);
    cuda[i] = a[i] / b[i];
  } else if (op == 1) {
    out[i] = div_corrected(a[i], b[i], 1.0 / b[i]);
    cuda[i] = a[i] / b[i];
  } else {
    out[i] = op == 2 ? rsqrt_newton(a[i]) : rsqrt_step(a[i]);
    cuda[i] = 1.0 / sqrt(a[i]);
  }
}

extern "C" int fp64_steps(int op, int n, const double* a, const double* b, double* out, double* cuda) {
  double* d[4] = {};
  const size_t bytes = sizeof(double) * (size_t)n;
  bool ok = n > 0;
  for (double*& p : d) ok = ok && cudaMalloc(&p, bytes) == cudaSuccess;
  ok = ok && cudaMemcpy(d[0], a, bytes, cudaMemcpyHostToDevice) == cudaSuccess &&
       cudaMemcpy(d[1], b, bytes, cudaMemcpyHostToDevice) == cudaSuccess;
  if (ok) {
    k_eval<<<(n + 255) / 256, 256>>>(op, n, d[0], d[1], d[2], d[3]);
    ok = cudaGetLastError() == cudaSuccess && cudaMemcpy(out, d[2], bytes, cudaMemcpyDeviceToHost) == cudaSuccess &&
         cudaMemcpy(cuda, d[3], bytes, cudaMemcpyDeviceToHost) == cudaSuccess;
  }
  for (double* p : d)
    if (p) cudaFree(p);
  return ok ? 0 : 1;
}
