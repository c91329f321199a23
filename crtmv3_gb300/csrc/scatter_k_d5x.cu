// The mixed form's scattering layers of constant angle counts (up to 5 angles):
// the layer records and the reverse sweep through the layers' optics.
#include "scatter_kernels.cuh"
#include "scatter_launch.h"

namespace crtm {

int scatter_k_d5x_set_gauss(const GaussTable& g) {
  return cudaMemcpyToSymbol(c_gauss, &g, sizeof g) == cudaSuccess ? 0 : 1;
}

int launch_layers_fixed(const ScatterArgs<float>& a, float* rec, const ItemLists& ls, cudaStream_t st) {
  layers_fixed_kernel<5, 4><<<list_ctas(ls, 6), SCATTER_THREADS, 0, st>>>(a, rec, ls);
  layers_fixed_kernel<5, 3><<<list_ctas(ls, 5), SCATTER_THREADS, 0, st>>>(a, rec, ls);
  layers_fixed_kernel<5, 2><<<list_ctas(ls, 4), SCATTER_THREADS, 0, st>>>(a, rec, ls);
  return 3;
}
int launch_reverse_fixed(const ScatterArgs<float>& a, const ItemLists& ls, cudaStream_t st) {
  reverse_fixed_kernel<5, 4><<<list_ctas(ls, 6), SCATTER_THREADS, 0, st>>>(a, ls);
  reverse_fixed_kernel<5, 3><<<list_ctas(ls, 5), SCATTER_THREADS, 0, st>>>(a, ls);
  reverse_fixed_kernel<5, 2><<<list_ctas(ls, 4), SCATTER_THREADS, 0, st>>>(a, ls);
  return 3;
}

}  // namespace crtm
