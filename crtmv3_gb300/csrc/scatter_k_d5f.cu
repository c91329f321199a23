// The mixed form's per-thread scattering kernels for NZ = 5 angles (the stream rule's 2-6 streams):
// the layer records, what precedes the adding, and the reverse sweep through
// the layers' optics.
#include "scatter_kernels.cuh"
#include "scatter_launch.h"

namespace crtm {

int scatter_k_d5f_set_gauss(const GaussTable& g) {
  return cudaMemcpyToSymbol(c_gauss, &g, sizeof g) == cudaSuccess ? 0 : 1;
}

template <int NZ>
void launch_layers_listed(const ScatterArgs<float>& a, float* rec, const ItemLists& ls, int pass, cudaStream_t st) {
  layers_listed_kernel<NZ><<<list_ctas(ls, pass), list_threads(pass), 0, st>>>(a, rec, ls, pass);
}

template <int NZ>
void launch_adding_front(const ScatterArgs<float>& a, dim3 grid, cudaStream_t st) {
  adding_front_kernel<NZ><<<grid, SCATTER_THREADS, 0, st>>>(a);
}

template <int NZ>
void launch_reverse_listed(const ScatterArgs<float>& a, const ItemLists& ls, int pass, cudaStream_t st) {
  reverse_listed_kernel<NZ><<<list_ctas(ls, pass), list_threads(pass), 0, st>>>(a, ls, pass);
}

template void launch_layers_listed<5>(const ScatterArgs<float>&, float*, const ItemLists&, int, cudaStream_t);
template void launch_adding_front<5>(const ScatterArgs<float>&, dim3, cudaStream_t);
template void launch_reverse_listed<5>(const ScatterArgs<float>&, const ItemLists&, int, cudaStream_t);

}  // namespace crtm
