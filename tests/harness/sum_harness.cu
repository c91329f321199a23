// The mixed form's adjoint channel sums (channel_sum_fixed_kernel) on host rows.
#include "odps_kernels.cuh"

extern "C" int run_channel_sum(const float* rows, long long n, int L, double* out) {
  float* d = nullptr;
  double* o = nullptr;
  int rc = cudaMalloc(&d, sizeof(float) * n * L) != cudaSuccess || cudaMalloc(&o, sizeof(double) * n) != cudaSuccess ||
           cudaMemcpy(d, rows, sizeof(float) * n * L, cudaMemcpyHostToDevice) != cudaSuccess;
  if (!rc) {
    crtm::channel_sum_fixed_kernel<<<(unsigned)((n * 32 + 255) / 256), 256>>>(d, n, L, o);
    rc = cudaGetLastError() != cudaSuccess ||
         cudaMemcpy(out, o, sizeof(double) * n, cudaMemcpyDeviceToHost) != cudaSuccess;
  }
  cudaFree(d);
  cudaFree(o);
  return rc;
}
