// The fast reciprocals of the explicit path on n values: out [3][n] = 1/x, 1/sqrt(x), sqrt(x).
#include "../../bes_gb300/csrc/side_kernels.cuh"

__global__ void reciprocals_kernel(const double* x, int64_t n, double* out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  out[i] = bes::fast_rcp(x[i]);
  out[n + i] = bes::fast_rsqrt(x[i]);
  const bes::RootFactors r = bes::fast_sqrt(x[i]);
  out[2 * n + i] = r.s * r.y;
}

extern "C" int reciprocals(const double* x, int64_t n, double* out) {
  double *dx = nullptr, *dout = nullptr;
  cudaError_t e = cudaMalloc(&dx, n * sizeof(double));
  if (e == cudaSuccess) e = cudaMalloc(&dout, 3 * n * sizeof(double));
  if (e == cudaSuccess) e = cudaMemcpy(dx, x, n * sizeof(double), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    reciprocals_kernel<<<(unsigned)((n + 255) / 256), 256>>>(dx, n, dout);
    e = cudaMemcpy(out, dout, 3 * n * sizeof(double), cudaMemcpyDeviceToHost);
  }
  cudaFree(dx);
  cudaFree(dout);
  return (int)e;
}
