// Small matrices by a team of lanes, one lane per angle (a matrix row):
// products and the adding's inverse, every element with the operations of the
// per-thread functions in their order.  See scatter_team.cuh for the kernel and
// the reasons; the tests run this header on an emulated warp.
#pragma once

#include "scatter_physics.cuh"

namespace crtm {

// lanes of a team, floats per matrix row (16-byte rows) and per matrix
template <int NZ> constexpr int team_size() { return NZ <= 4 ? 4 : (NZ <= 8 ? 8 : 16); }
template <int NZ> constexpr int team_ld() { return (NZ + 3) / 4 * 4; }
template <int NZ> constexpr int team_mat() { return NZ * team_ld<NZ>(); }
// Shared floats of a team of NM matrices and NV vectors, padded so that the
// teams of a warp start 8 banks (16 lanes: 16 banks) apart.
template <int NZ, int NM, int NV>
constexpr int team_floats() {
  const int want = team_size<NZ>() == 16 ? 16 : (team_size<NZ>() == 8 ? 8 : 4);
  int n = NM * team_mat<NZ>() + NV * team_ld<NZ>();
  while (n % 32 != want) n += 4;
  return n;
}

// A product that the per-thread functions keep in a matrix: rounded there, so
// rounded here before it meets a sum.
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }

template <int NZ>
struct Team {
  static constexpr int TS = team_size<NZ>(), LD = team_ld<NZ>(), MS = team_mat<NZ>();
  // fixed angle count: the classes of 5 and 6 angles
  static constexpr bool EXACT = NZ == 5 || NZ == 6;
  int lane, r, base, n, nS;   // warp lane, row, first lane of the team, angles, quadrature angles
  bool live;                  // the team has a layer
  __device__ bool row() const { return r < (EXACT ? NZ : n); }
  __device__ int nz() const { return EXACT ? NZ : n; }
  template <class T>
  __device__ T bc(T v, int row) const { return __shfl_sync(FULL, v, base + row); }
};

template <int NZ>
__device__ __forceinline__ void ld_row(const float* p, float* v) {
#pragma unroll
  for (int j = 0; j < team_ld<NZ>(); j += 4) {
    const float4 q = *reinterpret_cast<const float4*>(p + j);
    v[j] = q.x;
    if (j + 1 < NZ) v[j + 1] = q.y;
    if (j + 2 < NZ) v[j + 2] = q.z;
    if (j + 3 < NZ) v[j + 3] = q.w;
  }
}
template <int NZ>
__device__ __forceinline__ void st_row(const Team<NZ>& t, float* M, const float* v) {
  if (!t.row()) return;
  float* p = M + t.r * team_ld<NZ>();
#pragma unroll
  for (int j = 0; j < team_ld<NZ>(); j += 4)
    *reinterpret_cast<float4*>(p + j) = make_float4(v[j], j + 1 < NZ ? v[j + 1] : 0.f, j + 2 < NZ ? v[j + 2] : 0.f,
                                                    j + 3 < NZ ? v[j + 3] : 0.f);
}
// the team's vector of one value per lane
template <int NZ>
__device__ __forceinline__ void st_vec(const Team<NZ>& t, float* V, float v) {
  if (t.row()) V[t.r] = v;
}

// Row r of A B: a the own row of A, B in shared memory.
template <int NZ>
__device__ __forceinline__ void row_mul(const Team<NZ>& t, const float* a, const float* B, float* c) {
#pragma unroll
  for (int j = 0; j < NZ; j++) c[j] = 0.f;
#pragma unroll
  for (int k = 0; k < NZ; k++) {
    if (k >= t.nz()) break;
    float b[NZ];
    ld_row<NZ>(B + k * team_ld<NZ>(), b);
#pragma unroll
    for (int j = 0; j < NZ; j++) c[j] += a[k] * b[j];
  }
}
// Row r of A^T B, both in shared memory.
template <int NZ>
__device__ __forceinline__ void row_mul_tn(const Team<NZ>& t, const float* A, const float* B, float* c) {
  const int r = t.row() ? t.r : 0;
#pragma unroll
  for (int j = 0; j < NZ; j++) c[j] = 0.f;
#pragma unroll
  for (int k = 0; k < NZ; k++) {
    if (k >= t.nz()) break;
    const float a = A[k * team_ld<NZ>() + r];
    float b[NZ];
    ld_row<NZ>(B + k * team_ld<NZ>(), b);
#pragma unroll
    for (int j = 0; j < NZ; j++) c[j] += a * b[j];
  }
}
// Row r of A B^T: a the own row of A, B in shared memory.
template <int NZ>
__device__ __forceinline__ void row_mul_nt(const Team<NZ>& t, const float* a, const float* B, float* c) {
#pragma unroll
  for (int j = 0; j < NZ; j++) {
    c[j] = 0.f;
    if (j >= t.nz()) continue;
    float b[NZ];
    ld_row<NZ>(B + j * team_ld<NZ>(), b);
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < NZ; k++)
      if (k < t.nz()) s += a[k] * b[k];
    c[j] = s;
  }
}

// Inverse by Gauss-Jordan elimination with partial pivoting (mat_invert): own
// row in a (destroyed), the inverse to M.  Rows stay in their lanes; pos is
// the row's place after the interchanges, so the lane at place j is the
// original row perm[j].
template <int NZ, class T>
__device__ __forceinline__ bool team_invert(const Team<NZ>& t, T* a, T* M, int ldm) {
  int pos = t.r;
  bool ok = true;
#pragma unroll
  for (int k = 0; k < NZ; k++) {
    // (no early exit: the warp's teams may have different angle counts)
    const bool act = k < t.nz();
    T bv = T(-1);
    if (t.row() && pos >= k) {
      const T m = fabs(a[k]);
      bv = m == m ? m : T(0);
    }
    int bi = (pos << 5) | t.lane;
#pragma unroll
    for (int o = Team<NZ>::TS / 2; o > 0; o >>= 1) {
      const T ov = __shfl_xor_sync(FULL, bv, o);
      const int oi = __shfl_xor_sync(FULL, bi, o);
      if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
    }
    ok = ok && (!act || bv > T(1.0e-40));
    const int pl = bi & 31, pp = bi >> 5;
    if (act && t.lane == pl) pos = k;
    else if (act && pos == k) pos = pp;
    const T d = T(1.0) / __shfl_sync(FULL, a[k], pl);
    if (act && t.lane == pl) {
#pragma unroll
      for (int j = 0; j < NZ; j++) a[j] = mul_rn(a[j], d);
      a[k] = d;
    }
    const T f = a[k];
    const bool upd = act && t.lane != pl && !is_zero(f);
#pragma unroll
    for (int j = 0; j < NZ; j++) {
      const T b = __shfl_sync(FULL, a[j], pl);
      if (upd) a[j] -= f * b;
    }
    if (upd) a[k] = mul_rn(-f, d);
  }
  // undo the row interchanges as column interchanges of the inverse
  unsigned long long w = t.row() ? (unsigned long long)t.r << (4 * pos) : 0ull;
#pragma unroll
  for (int o = Team<NZ>::TS / 2; o > 0; o >>= 1) w |= __shfl_xor_sync(FULL, w, o);
  if (t.row()) {
    T* p = M + pos * ldm;
#pragma unroll
    for (int j = 0; j < NZ; j++)
      if (j < t.nz()) p[(int)(w >> (4 * j)) & 15] = a[j];
  }
  return ok;
}

// Gamma = G^-1 (invert_fp64): own row g of G (destroyed), the inverse to M.
// FP32 where the coupling is weak, else FP64 (MD: a matrix of doubles).
template <int NZ>
__device__ __forceinline__ bool team_invert_adding(const Team<NZ>& t, float* g, float* M, double* MD) {
  constexpr int LD = team_ld<NZ>();
  float c = 0.f;
#pragma unroll
  for (int j = 0; j < NZ; j++)
    if (j < t.nz()) c += fabs((t.r == j ? 1.0f : 0.0f) - g[j]);
  if (!t.row() || !(c > 0.f)) c = 0.f;
#pragma unroll
  for (int o = Team<NZ>::TS / 2; o > 0; o >>= 1) {
    const float v = __shfl_xor_sync(FULL, c, o);
    c = v > c ? v : c;
  }
  const bool wide = t.live && !(c < float(ADDING_FP32_COUPLING));
  bool ok64 = true;
  const bool any = __any_sync(FULL, wide);
  if (any) {
    double d[NZ];
#pragma unroll
    for (int j = 0; j < NZ; j++) d[j] = double(g[j]);
    ok64 = team_invert<NZ>(t, d, MD, LD);
    __syncwarp();
  }
  const bool ok32 = team_invert<NZ>(t, g, M, LD);
  if (any) {
    __syncwarp();
    if (wide && t.row()) {
#pragma unroll
      for (int j = 0; j < NZ; j++)
        if (j < t.nz()) M[t.r * LD + j] = float(MD[t.r * LD + j]);
    }
  }
  return wide ? ok64 : ok32;
}

}  // namespace crtm
