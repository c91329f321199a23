// Host launchers of the scattering K-matrix/adjoint kernels.  R is the gas
// optics' arithmetic (double in the FP64 form, float in the mixed form), C
// the layer solver's (the same); the adding and its adjoint are in R too.
// A batch with SOI profiles runs in the FP64 form.  Translation units per
// angle capacity (d5: the stream rule's 2-6 streams, d10: Options%n_Streams
// up to 16): scatter_k_*.cu (FP64 form: records, adding adjoint, reverse sweep of
// the ADA layers; the f units the mixed form's layers by lists, the x unit those
// of known angle counts), scatter_team.cu (the mixed form's adding) and
// scatter_soi_*.cu (the SOI layers' derivative-number contraction); they compile
// in parallel.
#pragma once

#include <cuda_runtime.h>

namespace crtm {

struct GaussTable;
template <class R> struct ScatterArgs;
struct ItemLists;

// Upload the Gauss table into each unit's constant memory; 0 on success.
int scatter_k_d5_set_gauss(const GaussTable& g);
int scatter_k_d10_set_gauss(const GaussTable& g);
int scatter_k_d5f_set_gauss(const GaussTable& g);
int scatter_k_d10f_set_gauss(const GaussTable& g);
int scatter_soi_d5_set_gauss(const GaussTable& g);
int scatter_soi_d10_set_gauss(const GaussTable& g);
int scatter_team_set_gauss(const GaussTable& g);
int scatter_k_d5x_set_gauss(const GaussTable& g);
inline int scatter_k_set_gauss(const GaussTable& g) {
  return scatter_k_d5_set_gauss(g) | scatter_k_d10_set_gauss(g) | scatter_k_d5f_set_gauss(g) |
         scatter_k_d10f_set_gauss(g) | scatter_soi_d5_set_gauss(g) | scatter_soi_d10_set_gauss(g) |
         scatter_team_set_gauss(g) | scatter_k_d5x_set_gauss(g);
}

// FP64 form: layer records (in R) with the layer solver in C
template <int NZ, class R, class C>
void launch_scatter_layers_k(const ScatterArgs<R>& a, unsigned grid, cudaStream_t st);
// FP64 form: the ADA adding adjoint, then (soi) the SOI orders' adjoint of the SOI profiles
template <int NZ, class R>
void launch_scatter_kmatrix(const ScatterArgs<R>& a, dim3 grid, cudaStream_t st, bool soi);
// mixed form: the clear columns and refused stream sets, then the ADA adding
// and its adjoint by teams of lanes (NC: angle capacity of the records; returns
// the number of kernels launched)
template <int NZ>
void launch_adding_front(const ScatterArgs<float>& a, dim3 grid, cudaStream_t st);
int launch_adding_team(const ScatterArgs<float>& a, int NC, cudaStream_t st);
// mixed form: the listed layers' records and their reverse sweep; pass 0 the
// classes' lists, then 1 (layers) or 2 (reverse) what it deferred
template <int NZ>
void launch_layers_listed(const ScatterArgs<float>& a, float* rec, const ItemLists& ls, int pass, cudaStream_t st);
template <int NZ>
void launch_reverse_listed(const ScatterArgs<float>& a, const ItemLists& ls, int pass, cudaStream_t st);
// 5 angles: the classes of constant angle counts (number of kernels launched)
int launch_layers_fixed(const ScatterArgs<float>& a, float* rec, const ItemLists& ls, cudaStream_t st);
int launch_reverse_fixed(const ScatterArgs<float>& a, const ItemLists& ls, cudaStream_t st);
// FP64 form: the ADA profiles' layer contraction (reverse sweep in C)
template <int NZ, class R, class C>
void launch_scatter_reverse(const ScatterArgs<R>& a, unsigned grid, cudaStream_t st);
// the SOI profiles' layer contraction (derivative numbers, FP64 form)
template <int NZ, class C>
void launch_scatter_contract(const ScatterArgs<double>& a, unsigned grid, cudaStream_t st);

}  // namespace crtm
