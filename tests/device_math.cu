// rcp3 and exp2_tab on arrays, for test_gpu_device_math.py (compiled by it)
#define OCFD_DEFINE_CONST
#include "ocfd_device.cuh"
#include "ocfd_exp2.cuh"

__global__ void k_eval(int n, const double* x, double* rcp, double* ex) {
  __shared__ double tab[ocfd::E2_N];
  ocfd::exp2_tab_load(tab);
  __syncthreads();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  rcp[i] = ocfd::rcp3(x[i]);
  ex[i] = ocfd::exp2_tab(x[i], tab);
}

extern "C" int device_math(int n, const double* x, double* rcp, double* ex) {
  double* d = nullptr;
  const size_t b = sizeof(double) * (size_t)n;
  cudaError_t e = ocfd::exp2_tab_setup();
  if (e == cudaSuccess) e = cudaMalloc(&d, 3 * b);
  if (e == cudaSuccess) e = cudaMemcpy(d, x, b, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    k_eval<<<(n + 255) / 256, 256>>>(n, d, d + n, d + 2 * (size_t)n);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(rcp, d + n, b, cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) e = cudaMemcpy(ex, d + 2 * (size_t)n, b, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return (int)e;
}
