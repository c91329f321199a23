// scatter_fixed.cuh (known angle counts) against the run-time forms it stands
// for: values that differ, bit for bit, over random layers.
#include <cmath>
#include <cstdlib>
#include <cstring>

#include "scatter_adjoint.cuh"

using namespace crtm;

namespace {
constexpr int NZ = 5;
double rnd() { return std::rand() / (double)RAND_MAX; }
bool differ(float a, float b) { return std::memcmp(&a, &b, 4) != 0 && !(a == 0.f && b == 0.f); }

template <int NS>
long layers(int n, double tau_lo, double tau_hi, double w_hi) {
  constexpr int nZ = NS + 1, nleg = 2 * NS - 2;
  double x[16], w[16];
  double_gauss_host(NS, x, w);
  long bad = 0;
  for (int it = 0; it < n; it++) {
    float mu[NZ], wt[NZ], P[NZ][SC_NLEG_MAX + 1], pc[SC_NLEG_MAX + 1], sb[NZ];
    Mat<NZ, float> Tb, Rb;
    for (int i = 0; i < NS; i++) { mu[i] = x[i]; wt[i] = w[i]; }
    mu[NS] = 0.3 + 0.7 * rnd();
    wt[NS] = 0.f;
    const float ssa = w_hi * rnd(), tau = tau_lo * std::pow(tau_hi / tau_lo, rnd()), B = 50 * rnd();
    const double g = rnd() < 0.3 ? -0.3 : 0.9 * rnd();
    for (int l = 0; l <= nleg; l++) pc[l] = 0.5 * (2 * l + 1) * std::pow(g, l);
    for (int i = 0; i < nZ; i++) {
      P[i][0] = 1.f;
      P[i][1] = mu[i];
      for (int j = 1; j < nleg; j++) P[i][j + 1] = ((2 * j + 1) * mu[i] * P[i][j] - j * P[i][j - 1]) / (j + 1);
      sb[i] = rnd() - 0.5;
      for (int j = 0; j < nZ; j++) { Tb.a[i][j] = rnd() - 0.5; Rb.a[i][j] = rnd() - 0.5; }
    }
    Mat<NZ, float> ff[2], bb[2], U[2], R[2], fb[2], bq[2];
    float src[2][NZ], wb[2], tb[2], Bb[2], pb[2][SC_NLEG_MAX + 1];
    double gap[2] = {1.0, 1.0};
    bool ok[2];
    phase_blocks<NZ, float>(NS, nZ, nleg, pc, P, wt, ff[0], bb[0]);
    fixed::phase_blocks<NZ, NS>(pc, P, wt, ff[1], bb[1]);
    ok[0] = ada_layer_loss<NZ, float>(NS, nZ, ssa, tau, mu, wt, ff[0], bb[0], B, U[0], R[0], src[0], &gap[0]);
    ok[1] = fixed::ada_layer_loss<NZ, NS>(ssa, tau, mu, wt, ff[1], bb[1], B, U[1], R[1], src[1], &gap[1]);
    bad += ok[0] != ok[1] || gap[0] != gap[1];
    if (!ok[0] || !ok[1]) continue;
    ok[0] = ada_layer_adjoint<NZ, float>(NS, nZ, ssa, tau, mu, wt, ff[0], bb[0], B, Tb, Rb, sb, &wb[0], &tb[0], fb[0],
                                         bq[0], &Bb[0], &gap[0]);
    ok[1] = fixed::ada_layer_adjoint<NZ, NS>(ssa, tau, mu, wt, ff[1], bb[1], B, Tb, Rb, sb, &wb[1], &tb[1], fb[1],
                                             bq[1], &Bb[1], &gap[1]);
    bad += ok[0] != ok[1] || gap[0] != gap[1];
    if (!ok[0] || !ok[1]) continue;
    phase_blocks_adjoint<NZ, float>(NS, nZ, nleg, pc, P, wt, fb[0], bq[0], pb[0]);
    fixed::phase_blocks_adjoint<NZ, NS>(pc, P, wt, fb[1], bq[1], pb[1]);
    for (int i = 0; i < nZ; i++) {
      bad += differ(src[0][i], src[1][i]);
      for (int j = 0; j < nZ; j++)
        bad += differ(ff[0].a[i][j], ff[1].a[i][j]) + differ(bb[0].a[i][j], bb[1].a[i][j]) +
               differ(U[0].a[i][j], U[1].a[i][j]) + differ(R[0].a[i][j], R[1].a[i][j]) +
               differ(fb[0].a[i][j], fb[1].a[i][j]) + differ(bq[0].a[i][j], bq[1].a[i][j]);
    }
    bad += differ(wb[0], wb[1]) + differ(tb[0], tb[1]) + differ(Bb[0], Bb[1]);
    for (int l = 0; l < nleg; l++) bad += differ(pb[0][l], pb[1][l]);
  }
  return bad;
}
}  // namespace

extern "C" long run_layers(int NS, int n, double tau_lo, double tau_hi, double w_hi) {
  std::srand(NS);
  switch (NS) {
    case 2: return layers<2>(n, tau_lo, tau_hi, w_hi);
    case 3: return layers<3>(n, tau_lo, tau_hi, w_hi);
    case 4: return layers<4>(n, tau_lo, tau_hi, w_hi);
  }
  return -1;
}
