// The mixed form's adding by teams of lanes, per angle class NZ and angle
// capacity NC of the records.
#include "scatter_launch.h"
#include "scatter_team.cuh"

namespace crtm {

int scatter_team_set_gauss(const GaussTable& g) {
  return cudaMemcpyToSymbol(c_gauss, &g, sizeof g) == cudaSuccess ? 0 : 1;
}

namespace {
template <int NZ>
int adding(const ScatterArgs<float>& a, int NC, cudaStream_t st) {
  constexpr int per = TEAM_WARPS * (32 / team_size<NZ>());   // channels per CTA
  constexpr size_t smem = adding_team_smem<NZ>();
  static_assert(smem <= 48 * 1024, "the default shared-memory limit");
  adding_team_kernel<NZ><<<dim3((a.L + per - 1) / per, a.n_chunk), 32 * TEAM_WARPS, smem, st>>>(a, NC);
  return 1;
}
}  // namespace

// Angle classes of a capacity: up to 6 streams make 2-5 angles, 8 and 16
// streams 5, 6, 9 or 10.
int launch_adding_team(const ScatterArgs<float>& a, int NC, cudaStream_t st) {
  if (NC == 5) return adding<4>(a, NC, st) + adding<5>(a, NC, st);
  return adding<5>(a, NC, st) + adding<6>(a, NC, st) + adding<10>(a, NC, st);
}

}  // namespace crtm
