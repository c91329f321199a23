// The adding and its adjoint in the mixed form (cloudy_adjoint in FP32), a team
// of lanes per (profile, channel): one lane per angle, which holds its row of
// every NZ x NZ matrix in registers, the other operand's rows broadcast from
// shared memory, the elimination's pivot row by shuffles.
//
// Bound and layout.  The recursion over the layers is serial, and one thread per
// pair kept its ten matrices in local memory: a microwave sounder's pairs made 7
// warps per SM, waiting on local memory (53.8 ms for 2000 profiles x 16
// channels of 2 ... 5 angles; 6.6 ms now).  With teams of 4, 8 or 16 lanes a layer's matrices
// stay on the SM, the next layer's record and state load while this one is
// worked on, and there are 4 to 16 times the warps.
//
// Every matrix element sees the per-thread functions' operations in their
// order, and a product that they store before it meets a sum is rounded here
// too, so the results are the same bits.
#pragma once

#include "scatter_kernels.cuh"
#include "scatter_team_math.cuh"

namespace crtm {

constexpr int TEAM_WARPS = 4;

// Angle class of a team kernel.
template <int NZ>
__device__ __forceinline__ bool in_class(int nZ) {
  return NZ == 4 ? nZ <= 4 : (NZ == 10 ? nZ > 6 : nZ == NZ);
}

constexpr int ADD_MATS = 10, ADD_VECS = 4;
template <int NZ>
constexpr size_t adding_team_smem() {
  return sizeof(float) * TEAM_WARPS * (32 / team_size<NZ>()) * (size_t)team_floats<NZ, ADD_MATS, ADD_VECS>();
}

template <int NZ>
__global__ void __launch_bounds__(32 * TEAM_WARPS) adding_team_kernel(ScatterArgs<float> a, int NC) {
  extern __shared__ __align__(16) float tsm[];
  constexpr int TPW = 32 / team_size<NZ>(), MS = team_mat<NZ>(), LD = team_ld<NZ>();
  Team<NZ> t;
  t.lane = threadIdx.x & 31;
  t.r = t.lane & (team_size<NZ>() - 1);
  t.base = t.lane - t.r;
  const int wib = threadIdx.x >> 5, team = t.base / team_size<NZ>();
  const int L = a.L, Kmax = a.Kmax, NE = 2 + 2 * NC * NC + NC, S0 = 2 + 2 * NC * NC, R0 = 2 + NC * NC,
            NS = NC * NC + NC;
  const int p = blockIdx.y, gp = batch_profile(a.b, a.p_begin + p);
  const int l0 = (blockIdx.x * TEAM_WARPS + wib) * TPW, l = l0 + team, lc = l < L ? l : L - 1;
  if (l0 >= L || a.pv.status[p] != 0) return;
  const CloudyColumn c = column_inputs(a, p, gp, lc);
  if (c.n_clouds == 0 && c.n_aerosols == 0) return;
  StreamShape sh{NZ - 1, NZ, 0};
  const int bad = stream_shape(c.nleg, c.mu_sensor, c.n_clouds > 0 ? a.lut.nleg : -1, NC, sh);
  t.live = l < L && !bad && in_class<NZ>(sh.nZ);
  if (!__any_sync(FULL, t.live)) return;
  if (!t.live) sh = StreamShape{NZ == 10 ? 9 : NZ - 1, NZ, 0};
  t.n = sh.nZ;
  t.nS = sh.nS;
  const int nz = t.nz(), r = t.row() ? t.r : 0, Ku = c.Ku;
  float* M = tsm + (size_t)(wib * TPW + team) * team_floats<NZ, ADD_MATS, ADD_VECS>();
  double* MD = reinterpret_cast<double*>(M);
  float* MT = M + 2 * MS, *MR = M + 3 * MS, *MU = M + 4 * MS, *MUb = M + 5 * MS, *MG = M + 6 * MS, *MA = M + 7 * MS,
       *MB = M + 8 * MS, *MC = M + 9 * MS;
  float* V0 = M + 10 * MS, *V1 = V0 + LD, *V2 = V1 + LD, *V3 = V2 + LD;
  if (t.live && t.r == 0 && a.x.nfs) a.x.nfs[(size_t)gp * L + a.sp.out[l]] = c.nleg + 2;
  const double mu = r < sh.nS ? c_gauss.mu[sh.nS][r] : c.mu_sensor;
  const float muf = float(mu);
  const float b1 = float(c.b1), b2 = float(c.b2), c1 = float(c.c1), c2 = float(c.c2);
  auto planck = [&](int k) {
    const float te = b1 + b2 * float(c.temperature[k]);
    return c1 / (exp(c2 / te) - 1.0f);
  };
  const float* rec0 = a.LBK + (size_t)p * Kmax * NE * L + lc;
  float* adj0 = a.LBA + (size_t)p * Kmax * NE * L + lc;
  float* as0 = a.AS + (size_t)p * (Kmax + 1) * NS * L + lc;
  float Tm[NZ], Rm[NZ], src = 0.f, kindf = 0.f, odf = 0.f;
  auto fetch = [&](int k) {   // layer k's record, the own rows
    const float* rec = rec0 + (size_t)k * NE * L;
    kindf = rec[0];
    odf = rec[(size_t)L];
#pragma unroll
    for (int j = 0; j < NZ; j++) {
      Tm[j] = j < nz ? rec[(size_t)(2 + r * NC + j) * L] : 0.f;
      Rm[j] = j < nz ? rec[(size_t)(R0 + r * NC + j) * L] : 0.f;
    }
    src = rec[(size_t)(S0 + r) * L];
  };
  float rup[NZ], rad = float(c.emissivity * c.planck_surface);
#pragma unroll
  for (int j = 0; j < NZ; j++) rup[j] = t.r == j ? float(1.0 - c.emissivity) : 0.f;
  int code = 0;
  auto save = [&](int lev) {
    if (!t.live || !t.row() || code) return;
    float* as = as0 + (size_t)lev * NS * L;
#pragma unroll
    for (int j = 0; j < NZ; j++)
      if (j < nz) as[(size_t)(r * NC + j) * L] = rup[j];
    as[(size_t)(NC * NC + r) * L] = rad;
  };
  save(Ku);
  fetch(Ku - 1);
  for (int k = Ku - 1; k >= 0; k--) {
    float T[NZ], R[NZ];
#pragma unroll
    for (int j = 0; j < NZ; j++) { T[j] = Tm[j]; R[j] = Rm[j]; }
    const float s = src, odk = odf;
    const int kind = (int)kindf;
    if (k > 0) fetch(k - 1);
    if (kind < 0 && !code) code = -kind;
    const bool scat = t.live && !code && kind == 1;
    if (__any_sync(FULL, scat)) {
      __syncwarp();
      st_row(t, MT, T);
      st_row(t, MR, R);
      st_vec(t, V0, s);
      __syncwarp();
      float g[NZ];
      row_mul(t, rup, MR, g);
#pragma unroll
      for (int j = 0; j < NZ; j++) g[j] = (t.r == j ? 1.0f : 0.0f) - g[j];
      const bool ok = team_invert_adding(t, g, MG, MD);
      if (scat && !ok) code = 6;
      float tmp = rad;
#pragma unroll
      for (int j = 0; j < NZ; j++)
        if (j < nz) tmp += rup[j] * V0[j];
      float rt[NZ], igt[NZ];
      row_mul(t, rup, MT, rt);
      st_vec(t, V1, tmp);
      st_row(t, MB, rt);
      __syncwarp();
      row_mul(t, T, MG, igt);
      float rn = s;
#pragma unroll
      for (int j = 0; j < NZ; j++)
        if (j < nz) rn += igt[j] * V1[j];
      float un[NZ];
      row_mul(t, igt, MB, un);
      if (scat) {
        rad = rn;
#pragma unroll
        for (int j = 0; j < NZ; j++) {
          rup[j] = un[j];
          rup[j] += R[j];
        }
      }
    }
    if (__any_sync(FULL, t.live && !code && kind != 1)) {
      const float x = float(-double(odk) / mu);
      const float tr = exp(x), sc = mul_rn(-planck(k), expm1(x));
      float v = rad, ru[NZ];
#pragma unroll
      for (int j = 0; j < NZ; j++) {
        const float sj = t.bc(sc, j), tj = t.bc(tr, j);
        if (j < nz) v += rup[j] * sj;
        ru[j] = rup[j] * (tr * tj);
      }
      if (kind != 1) {
        rad = sc + tr * v;
#pragma unroll
        for (int j = 0; j < NZ; j++) rup[j] = ru[j];
      }
    }
    save(k);
  }
  // TOA radiance (adding_toa)
  double radiance = 0.0;
  {
    double sum = 0.0;
#pragma unroll
    for (int j = 0; j < NZ; j++)
      if (j < nz) sum += double(rup[j]);
    radiance = double(rad) + sum * c.cosmic;   // on the lane of the sensor angle
  }
  // ---- adjoint of the TOA radiance, top down
  float rupb[NZ], radb = t.r == sh.isat ? 1.0f : 0.0f;
#pragma unroll
  for (int j = 0; j < NZ; j++) rupb[j] = t.r == sh.isat ? float(c.cosmic) : 0.0f;
  fetch(0);
  float rupn[NZ], radn = 0.f;
  auto load = [&](int lev) {
    const float* as = as0 + (size_t)lev * NS * L;
#pragma unroll
    for (int j = 0; j < NZ; j++) rupn[j] = j < nz ? as[(size_t)(r * NC + j) * L] : 0.f;
    radn = as[(size_t)(NC * NC + r) * L];
  };
  load(1);
  for (int k = 0; k < Ku; k++) {
    float T[NZ], R[NZ], ru[NZ];
#pragma unroll
    for (int j = 0; j < NZ; j++) { T[j] = Tm[j]; R[j] = Rm[j]; ru[j] = rupn[j]; }
    const float s = src, odk = odf, ra = radn;
    const int kind = (int)kindf;
    if (k + 1 < Ku) {
      fetch(k + 1);
      load(k + 2);
    }
    float* adj = adj0 + (size_t)k * NE * L;
    const bool on = t.live && !code;
    const bool scat = on && kind == 1;
    __syncwarp();
    st_row(t, MU, ru);
    st_row(t, MUb, rupb);
    if (__any_sync(FULL, scat)) {
      st_row(t, MT, T);
      st_row(t, MR, R);
      st_vec(t, V0, s);
      st_vec(t, V1, radb);
      __syncwarp();
      float g[NZ], igt[NZ], rt[NZ];
      row_mul(t, ru, MR, g);
#pragma unroll
      for (int j = 0; j < NZ; j++) g[j] = (t.r == j ? 1.0f : 0.0f) - g[j];
      const bool ok = team_invert_adding(t, g, MG, MD);
      row_mul(t, ru, MT, rt);
      float tv = ra;
#pragma unroll
      for (int j = 0; j < NZ; j++)
        if (j < nz) tv += ru[j] * V0[j];
      st_row(t, MB, rt);
      st_vec(t, V2, tv);
      __syncwarp();
      row_mul(t, T, MG, igt);
      st_row(t, MA, igt);
      // IGT_b = rad'_b t^T + Rup'_b RT^T
      float m1[NZ];
#pragma unroll
      for (int j = 0; j < NZ; j++) {
        m1[j] = 0.f;
        if (j >= nz) continue;
        float b[NZ];
        ld_row<NZ>(MB + j * LD, b);
        float v = mul_rn(radb, V2[j]);
#pragma unroll
        for (int m = 0; m < NZ; m++)
          if (m < nz) v += rupb[m] * b[m];
        m1[j] = v;
      }
      st_row(t, MC, m1);
      __syncwarp();
      // t_b = IGT^T rad'_b;  RT_b = IGT^T Rup'_b
      float tbv = 0.f;
#pragma unroll
      for (int i = 0; i < NZ; i++)
        if (i < nz) tbv += MA[i * LD + r] * V1[i];
      float m2[NZ], Rb[NZ], Tb[NZ], Un[NZ];
      row_mul_tn(t, MA, MUb, m2);
#pragma unroll
      for (int j = 0; j < NZ; j++) Rb[j] = rupb[j];
      st_vec(t, V3, tbv);
      st_row(t, MB, m2);
      __syncwarp();
      row_mul_nt(t, m2, MT, Un);    // Rup_b = RT_b T^T
      row_mul_tn(t, MU, MB, Tb);    // T_b = Rup^T RT_b
      float sb = radb;
#pragma unroll
      for (int i = 0; i < NZ; i++)
        if (i < nz) sb += V3[i] * MU[i * LD + r];
#pragma unroll
      for (int j = 0; j < NZ; j++)
        if (j < nz) Un[j] += tbv * V0[j];
      // IGT = T Gamma
      float w1[NZ], w2[NZ];
      row_mul_nt(t, m1, MG, w1);
#pragma unroll
      for (int j = 0; j < NZ; j++) Tb[j] += w1[j];
      row_mul_tn(t, MT, MC, w2);
      // Gamma = G^-1:  G_b = -Gamma^T (Gamma_b Gamma^T)
      row_mul_nt(t, w2, MG, w1);
      __syncwarp();
      st_row(t, MA, w1);
      __syncwarp();
      row_mul_tn(t, MG, MA, m1);
#pragma unroll
      for (int j = 0; j < NZ; j++) m1[j] = -m1[j];
      st_row(t, MC, m1);
      __syncwarp();
      // G = I - Rup R
      row_mul_nt(t, m1, MR, w1);
      row_mul_tn(t, MU, MC, w2);
#pragma unroll
      for (int j = 0; j < NZ; j++) {
        Un[j] -= w1[j];
        Rb[j] -= w2[j];
      }
      if (scat && !ok) code = 6;
      if (scat && ok) {
        radb = tbv;
        if (t.row()) {
#pragma unroll
          for (int j = 0; j < NZ; j++)
            if (j < nz) {
              adj[(size_t)(2 + r * NC + j) * L] = Tb[j];
              adj[(size_t)(R0 + r * NC + j) * L] = Rb[j];
            }
          adj[(size_t)(S0 + r) * L] = sb;
        }
        if (t.r == 0) {
          adj[0] = 1.0f;
          adj[(size_t)L] = 0.0f;
        }
#pragma unroll
        for (int j = 0; j < NZ; j++) rupb[j] = Un[j];
      }
    }
    if (__any_sync(FULL, on && kind != 1)) {
      __syncwarp();
      const float B = planck(k);
      const float x = float(-double(odk) / mu);
      const float tr = exp(x), om = -expm1(x), sc = mul_rn(B, om);
      float trv[NZ], scv[NZ];
#pragma unroll
      for (int j = 0; j < NZ; j++) { trv[j] = t.bc(tr, j); scv[j] = t.bc(sc, j); }
      float tv = ra;
#pragma unroll
      for (int j = 0; j < NZ; j++)
        if (j < nz) tv += ru[j] * scv[j];
      float sb = radb, trb = mul_rn(radb, tv);
      const float tbv = radb * tr;
      // trb takes the terms of a loop over i, then j, in that order
      float ub[NZ];
#pragma unroll
      for (int i = 0; i < NZ; i++)
        if (i < nz) {
          if (i == t.r) {
#pragma unroll
            for (int j = 0; j < NZ; j++)
              if (j < nz) {
                trb += rupb[j] * ru[j] * trv[j];
                if (j == t.r) trb += rupb[j] * tr * ru[j];
              }
          } else {
            trb += MUb[i * LD + r] * trv[i] * MU[i * LD + r];
          }
        }
#pragma unroll
      for (int j = 0; j < NZ; j++) {
        ub[j] = mul_rn(rupb[j] * tr, trv[j]);
        ub[j] += tbv * scv[j];
      }
#pragma unroll
      for (int i = 0; i < NZ; i++) {
        const float ti = t.bc(tbv, i);
        if (i < nz) sb += ti * MU[i * LD + r];
      }
      trb -= sb * B;
      const float q = trb * tr / muf;
      float ob = 0.f, bbs = 0.f;
#pragma unroll
      for (int i = 0; i < NZ; i++) {
        const float si = t.bc(sb, i), oi = t.bc(om, i), qi = t.bc(q, i);
        if (i < nz) { bbs += si * oi; ob -= qi; }
      }
      if (on && kind != 1) {
        radb = tbv;
#pragma unroll
        for (int j = 0; j < NZ; j++) rupb[j] = ub[j];
        if (t.r == 0) {
          adj[0] = float(kind);
          adj[(size_t)L] = ob;
          adj[2 * (size_t)L] = bbs;
        }
      }
    }
  }
  double tr = 0.0, sr = 0.0;
#pragma unroll
  for (int i = 0; i < NZ; i++) {
    float d = 0.f;
#pragma unroll
    for (int j = 0; j < NZ; j++)
      if (j == t.r) d = rupb[j];
    const float di = t.bc(d, i), ri = t.bc(radb, i);
    if (i < nz) { tr += double(di); sr += double(ri); }
  }
  if (!t.live) return;
  double* cb = a.CB + (size_t)p * 4 * L + l;
  if (t.r == sh.isat) {
    cb[0] = code ? 0.0 : radiance;
    cb[(size_t)L] = code ? 0.0 : -tr + c.planck_surface * sr;
    cb[2 * (size_t)L] = code ? 0.0 : c.emissivity * sr;
  }
  if (code && t.r == 0) {
    atomicCAS(a.error, 0, code);
    if (a.status) atomicOr(a.status + gp, 1 << 4);
    for (int k = 0; k < Ku; k++) adj0[(size_t)k * NE * L] = -1.0f;
  }
}

}  // namespace crtm
