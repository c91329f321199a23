// The mixed form's adding and its adjoint on host records: the per-thread kernel
// (scatter_kmatrix_kernel in FP32), or what the library runs in its place
// (adding_front_kernel, then the teams of lanes).
#include <vector>

#include "scatter_kernels.cuh"
#include "scatter_launch.h"
#include "scatter_team.cuh"

using namespace crtm;

namespace {
struct Pool {
  std::vector<void*> p;
  bool ok = true;
  template <class T>
  T* up(const T* h, size_t n) {
    void* d = nullptr;
    ok = ok && cudaMalloc(&d, n * sizeof(T)) == cudaSuccess &&
         (!h || cudaMemcpy(d, h, n * sizeof(T), cudaMemcpyHostToDevice) == cudaSuccess);
    p.push_back(d);
    return (T*)d;
  }
  template <class T>
  void down(T* h, const T* d, size_t n) {
    ok = ok && cudaMemcpy(h, d, n * sizeof(T), cudaMemcpyDeviceToHost) == cudaSuccess;
  }
  ~Pool() {
    for (void* d : p) cudaFree(d);
  }
};

template <int NZ>
void team(const ScatterArgs<float>& a, int NC) {
  constexpr int per = TEAM_WARPS * (32 / team_size<NZ>());
  adding_team_kernel<NZ><<<dim3((a.L + per - 1) / per, a.n_chunk), 32 * TEAM_WARPS, adding_team_smem<NZ>()>>>(a, NC);
}

template <int NC>
void run(const ScatterArgs<float>& a, bool teams) {
  const dim3 grid((a.L + SCATTER_THREADS - 1) / SCATTER_THREADS, a.n_chunk);
  if (!teams) {
    scatter_kmatrix_kernel<NC, float><<<grid, SCATTER_THREADS>>>(a);
    return;
  }
  adding_front_kernel<NC><<<grid, SCATTER_THREADS>>>(a);
  if (NC == 5) {
    team<4>(a, NC);
    team<5>(a, NC);
  } else {
    team<5>(a, NC);
    team<6>(a, NC);
    team<10>(a, NC);
  }
}
}  // namespace

extern "C" double gauss_angle(int n, int i) {
  GaussTable g;
  gauss_table_host(g);
  return g.mu[n][i];
}

// ints: n_layers, n_clouds, n_streams [P]; prof: mu_sensor, surface temperature,
// cover [P]; spec: c1, c2, b1, b2, cosmic background, wavenumber [L]; rec: [P][Kmax][NE][L]
extern "C" int run_adding(int teams, int NC, int P, int L, int Kmax, const int* ints, const double* prof,
                          const double* spec, const double* temperature, const double* emissivity, const float* rec,
                          const float* tau, float* lba, double* cb, int* status, int* nfs, int* error) {
  GaussTable g;
  gauss_table_host(g);
  if (cudaMemcpyToSymbol(c_gauss, &g, sizeof g) != cudaSuccess) return 1;
  Pool d;
  const size_t NE = 2 + 2 * NC * NC + NC, pairs = (size_t)P * L, nrec = pairs * Kmax * NE;
  std::vector<double> scal((size_t)P * PREP_SCAL, 0.0), one(P, 1.0), zero(P, 0.0);
  std::vector<int> out(L), zi(P, 0);
  for (int p = 0; p < P; p++) scal[(size_t)p * PREP_SCAL + 1] = prof[p];
  for (int l = 0; l < L; l++) out[l] = L - 1 - l;   // the caller's columns in another order
  ScatterArgs<float> a{};
  a.L = L; a.Kmax = Kmax; a.n_chunk = P;
  const int* di = d.up(ints, 3 * (size_t)P);
  const double* ds = d.up(spec, 6 * (size_t)L);
  const double* w = d.up(one.data(), P), *z = d.up(zero.data(), P);
  a.b.n_profiles = P; a.b.max_layers = Kmax; a.b.n_layers = di; a.n_clouds = di + P; a.n_streams = di + 2 * P;
  a.b.temperature = d.up(temperature, (size_t)P * Kmax);
  a.b.emissivity = d.up(emissivity, pairs);
  a.b.water_cov = w; a.b.land_cov = a.b.snow_cov = a.b.ice_cov = z;
  a.b.water_t = d.up(prof + P, P); a.b.land_t = a.b.snow_t = a.b.ice_t = z;
  a.sp.c1 = ds; a.sp.c2 = ds + L; a.sp.b1 = ds + 2 * L; a.sp.b2 = ds + 3 * L; a.sp.cbr = ds + 4 * L;
  a.sp.wn = a.sp.freq = ds + 5 * L;
  a.sp.out = d.up(out.data(), L);
  a.pv.scal = d.up(scal.data(), scal.size());
  a.pv.status = d.up(zi.data(), P);
  a.lut.nleg = 40;
  a.max_clouds = 1;
  a.cover = d.up(prof + 2 * P, P);
  a.maxreff = d.up(zero.data(), P);
  a.TAU = d.up(tau, pairs * Kmax);
  a.LBK = d.up(rec, nrec);
  a.AS = d.up((const float*)nullptr, pairs * (Kmax + 1) * (NC * NC + NC));
  a.LBA = d.up((const float*)lba, nrec);
  a.CB = d.up((const double*)cb, 4 * pairs);
  a.status = d.up((const int*)status, P);
  a.x.nfs = d.up((const int*)nfs, pairs);
  a.error = d.up(zi.data(), 1);
  if (!d.ok) return 2;
  if (NC == 5) run<5>(a, teams); else run<10>(a, teams);
  if (cudaGetLastError() != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess) return 3;
  d.down(lba, a.LBA, nrec);
  d.down(cb, a.CB, 4 * pairs);
  d.down(status, a.status, P);
  d.down(nfs, a.x.nfs, pairs);
  d.down(error, a.error, 1);
  return d.ok ? 0 : 4;
}
