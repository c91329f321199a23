// The layer solver, its adjoint and the phase blocks of scatter_physics.cuh and
// scatter_adjoint.cuh for NS quadrature angles and the sensor's apart, in FP32:
// the same operations in the same order with loops of known bounds, for the
// kernels of a known angle count.
//
// With run-time bounds a multiply-add costs five to ten instructions (index
// arithmetic, loads and stores of matrices in local memory); here the matrices
// are in registers: 1503 -> 472 million instructions and 8.3 -> 4.3 ms for the
// reverse sweep of 16 x 616 channels of 100 layers (layers: 569 -> 226 million,
// 2.2 -> 1.5 ms).  In registers the compiler would also fuse a
// product with a later sum that the run-time form reads back from memory, so
// every product whose rounding matters is explicit: prod is rounded before it
// is added to anything, add_prod and sub_prod round once (c + a b, c - a b),
// two_prods rounds c d and then a b + c d.  These are the roundings of the
// run-time form's kernels with 5 angles, and results are the same bits.
#pragma once

#include "scatter_physics.cuh"

namespace crtm {

// C = A^T B, C = A B^T, adjoint of an inverse: scatter_adjoint.cuh
template <int NZ, class T> CRTM_HD void mat_mul_tn(int n, const Mat<NZ, T>& A, const Mat<NZ, T>& B, Mat<NZ, T>& C);
template <int NZ, class T> CRTM_HD void mat_mul_nt(int n, const Mat<NZ, T>& A, const Mat<NZ, T>& B, Mat<NZ, T>& C);
template <int NZ, class T>
CRTM_HD void inverse_adjoint(int n, const Mat<NZ, T>& Y, const Mat<NZ, T>& Yb, Mat<NZ, T>& Xb, Mat<NZ, T>& tmp);

namespace fixed {

CRTM_HD float prod(float a, float b) {
#ifdef __CUDA_ARCH__
  return __fmul_rn(a, b);
#else
  return a * b;
#endif
}
CRTM_HD float add_prod(float c, float a, float b) {
#ifdef __CUDA_ARCH__
  return __fmaf_rn(a, b, c);
#else
  return c + a * b;
#endif
}
CRTM_HD float sub_prod(float c, float a, float b) { return add_prod(c, -a, b); }
CRTM_HD float two_prods(float a, float b, float c, float d) { return add_prod(prod(c, d), a, b); }

// mat_invert: in place, partial pivoting.
template <int NZ, int NS>
CRTM_HD bool mat_invert(Mat<NZ, float>& A) {
  constexpr int n = NS + 1;
  int perm[NZ];
  for (int i = 0; i < n; i++) perm[i] = i;
  for (int k = 0; k < n; k++) {
    int p = k;
    float best = fabs(A.a[k][k]);
    for (int i = k + 1; i < n; i++)
      if (fabs(A.a[i][k]) > best) { best = fabs(A.a[i][k]); p = i; }
    if (!(best > 1.0e-40f)) return false;
    if (p != k) {
      for (int j = 0; j < n; j++) { const float t = A.a[p][j]; A.a[p][j] = A.a[k][j]; A.a[k][j] = t; }
      const int t = perm[p]; perm[p] = perm[k]; perm[k] = t;
    }
    const float d = 1.0f / A.a[k][k];
    for (int j = 0; j < n; j++) A.a[k][j] = prod(A.a[k][j], d);
    A.a[k][k] = d;
    for (int i = 0; i < n; i++) {
      if (i == k) continue;
      const float f = A.a[i][k];
      if (is_zero(f)) continue;
      for (int j = 0; j < n; j++) A.a[i][j] -= f * A.a[k][j];
      A.a[i][k] = prod(-f, d);
    }
  }
  // undo the row interchanges as column interchanges of the inverse
  float tmp[NZ];
  for (int i = 0; i < n; i++) {
    for (int j = 0; j < n; j++) tmp[perm[j]] = A.a[i][j];
    for (int j = 0; j < n; j++) A.a[i][j] = tmp[j];
  }
  return true;
}

// mom_eigen: the eigenpairs of MOM's (PP - PM)(PP + PM), the sensor angle's from the
// block-triangular structure.
template <int NZ, int NS>
CRTM_HD bool mom_eigen(float s, const float* mu, const float* wt, const Mat<NZ, float>& ff, const Mat<NZ, float>& bb,
                       Mat<NZ, float>& E, float* lam, Mat<NZ, float>& X, Mat<NZ, float>& Y, Mat<NZ, float>& V,
                       Mat<NZ, float>& W, double* gap) {
  constexpr int nS = NS, nZ = NS + 1;
  // symmetric form of the quadrature block
  float sq[NZ];
  for (int i = 0; i < nS; i++) sq[i] = sqrt(wt[i]);
  for (int i = 0; i < nS; i++)
    for (int j = 0; j < nS; j++) {
      const float sw = s * sq[i] * sq[j], dd = 1.0f / sqrt(mu[i] * mu[j]);
      const float id = (i == j) ? 1.0f : 0.0f;
      X.a[i][j] = prod(id - sw * (ff.a[i][j] - bb.a[i][j]), dd);
      Y.a[i][j] = prod(id - sw * (ff.a[i][j] + bb.a[i][j]), dd);
    }
  // Cholesky Y = L L^T (lower triangle of Y overwritten by L)
  for (int j = 0; j < nS; j++) {
    float d = Y.a[j][j];
    for (int k = 0; k < j; k++) d = sub_prod(d, Y.a[j][k], Y.a[j][k]);
    if (!(d > 0.0f)) return false;
    d = sqrt(d);
    Y.a[j][j] = d;
    for (int i = j + 1; i < nS; i++) {
      float v = Y.a[i][j];
      for (int k = 0; k < j; k++) v -= Y.a[i][k] * Y.a[j][k];
      Y.a[i][j] = v / d;
    }
  }
  // S = L^T X L in V (temporary X L in W)
  for (int i = 0; i < nS; i++)
    for (int j = 0; j < nS; j++) {
      float v = 0.0f;
      for (int k = j; k < nS; k++) v += X.a[i][k] * Y.a[k][j];
      W.a[i][j] = v;
    }
  for (int i = 0; i < nS; i++)
    for (int j = i; j < nS; j++) {
      float v = 0.0f;
      for (int k = i; k < nS; k++) v += Y.a[k][i] * W.a[k][j];
      V.a[i][j] = v;
    }
  for (int i = 0; i < nS; i++)
    for (int j = 0; j < i; j++) V.a[i][j] = V.a[j][i];
  jacobi(nS, V, lam, X);   // eigenvectors u in the columns of X
  // E = W^-1/2 D^-1/2 L^-T u: eigenvectors of HH, in E
  for (int c = 0; c < nS; c++) {
    for (int i = nS - 1; i >= 0; i--) {
      float v = X.a[i][c];
      for (int k = i + 1; k < nS; k++) v -= Y.a[k][i] * E.a[k][c];
      E.a[i][c] = v / Y.a[i][i];
    }
    for (int i = 0; i < nS; i++) E.a[i][c] /= sqrt(wt[i] * mu[i]);
  }
  // PP, PM for the full set of angles: PPM = PP - PM kept in X, PPP in Y
  for (int i = 0; i < nZ; i++) {
    const float c = s / mu[i];
    for (int j = 0; j < nZ; j++) {
      const float f = add_prod(i == j ? -(1.0f / mu[i]) : 0.0f, c * ff.a[i][j], wt[j]), b = c * bb.a[i][j];
      X.a[i][j] = sub_prod(f, b, wt[j]);
      Y.a[i][j] = add_prod(f, b, wt[j]);
    }
  }
  if (nZ > nS) {   // sensor angle (weight 0): HH is block lower triangular
    const int z = nZ - 1;
    float hz[NZ];
    for (int k = 0; k < nZ; k++) {
      float v = 0.0f;
      for (int m = 0; m < nZ; m++) v += X.a[z][m] * Y.a[m][k];
      hz[k] = v;   // row z of HH
    }
    for (int c = 0; c < nS; c++) {
      float v = 0.0f;
      for (int k = 0; k < nS; k++) v += hz[k] * E.a[k][c];
      E.a[z][c] = v / (lam[c] - hz[z]);
      if (gap) {
        const double g = fabs(value_of(lam[c]) - value_of(hz[z])) / fabs(value_of(lam[c]));
        if (g < *gap) *gap = g;
      }
    }
    for (int i = 0; i < nS; i++) E.a[i][z] = 0.0f;
    E.a[z][z] = 1.0f;
    lam[z] = hz[z];
  }
  return true;
}

// ada_layer_loss: U = I - T, R and the source.
template <int NZ, int NS>
CRTM_HD bool ada_layer_loss(float w, float tau, const float* mu, const float* wt, const Mat<NZ, float>& ff,
                            const Mat<NZ, float>& bb, float B, Mat<NZ, float>& Um, Mat<NZ, float>& Rm, float* src,
                            double* gap) {
  constexpr int nS = NS, nZ = NS + 1;
  if (gap) *gap = 1.0;
  if (tau < float(DELTA_OPTICAL_DEPTH)) {   // thin layer: first-order scattering
    const float s = tau * w;
    for (int i = 0; i < nZ; i++) {
      const float c = s / mu[i];
      float a = 0.0f;
      for (int j = 0; j < nZ; j++) {
        Rm.a[i][j] = c * bb.a[i][j] * wt[j];
        Um.a[i][j] = (i == j ? tau / mu[i] : 0.0f) - c * ff.a[i][j] * wt[j];
        a += Um.a[i][j] - Rm.a[i][j];
      }
      src[i] = a * B;
    }
    return true;
  }
  const float s = w < float(MAX_ALBEDO) ? w : float(MAX_ALBEDO);
  Mat<NZ, float> X, Y, V;
  float lam[NZ];
  if (!mom_eigen<NZ, NS>(s, mu, wt, ff, bb, Rm, lam, X, Y, V, Um, gap)) return false;
  // MOM with the eigenpairs (E in R, eigenvalues lam)
  if (!mat_invert<NZ, NS>(X)) return false;   // inverse of PP - PM
  float ex[NZ], dx[NZ];
  for (int i = 0; i < nZ; i++) {
    lam[i] = lam[i] > 0.0f ? sqrt(lam[i]) : 0.0f;
    ex[i] = exp(-lam[i] * tau);
    dx[i] = -expm1(-lam[i] * tau);
  }
  // EF = (PP-PM)^-1 E diag(lam);  Gp = (E + EF)/2 in Y, Gm = (E - EF)/2 in V
  for (int i = 0; i < nZ; i++)
    for (int j = 0; j < nZ; j++) {
      float v = 0.0f;
      for (int k = 0; k < nZ; k++) v += X.a[i][k] * Rm.a[k][j];
      Y.a[i][j] = prod(0.5f, add_prod(Rm.a[i][j], v, lam[j]));
      V.a[i][j] = prod(0.5f, sub_prod(Rm.a[i][j], v, lam[j]));
    }
  // P = Gm^-1 Gp (in Rm)
  for (int i = 0; i < nZ; i++)
    for (int j = 0; j < nZ; j++) X.a[i][j] = V.a[i][j];
  if (!mat_invert<NZ, NS>(X)) return false;    // Gm^-1
  mat_mul(nZ, X, Y, Rm);
  // W = D P e + P D (in X);  Q = Gm - Gp P (in Um)
  for (int i = 0; i < nZ; i++)
    for (int j = 0; j < nZ; j++) {
      X.a[i][j] = two_prods(dx[i] * Rm.a[i][j], ex[j], Rm.a[i][j], dx[j]);
      float v = 0.0f;
      for (int k = 0; k < nZ; k++) v += Y.a[i][k] * Rm.a[k][j];
      Um.a[i][j] = V.a[i][j] - v;
    }
  // GA = Q + Gp W (in A);  U numerator Q D + Gp W (in Um);  R numerator Gp D + Gm D P e (in Rn)
  Mat<NZ, float> A, Rn;
  for (int i = 0; i < nZ; i++)
    for (int j = 0; j < nZ; j++) {
      float gw = 0.0f, gd = 0.0f;
      for (int k = 0; k < nZ; k++) {
        gw += Y.a[i][k] * X.a[k][j];
        gd += V.a[i][k] * dx[k] * Rm.a[k][j];
      }
      A.a[i][j] = Um.a[i][j] + gw;
      Um.a[i][j] = Um.a[i][j] * dx[j] + gw;
      Rn.a[i][j] = two_prods(Y.a[i][j], dx[j], gd, ex[j]);
    }
  if (!mat_invert<NZ, NS>(A)) return false;    // GA^-1
  mat_mul(nZ, Um, A, X);
  mat_mul(nZ, Rn, A, V);
  for (int i = 0; i < nZ; i++)
    for (int j = 0; j < nZ; j++) { Um.a[i][j] = X.a[i][j]; Rm.a[i][j] = V.a[i][j]; }
  // source (1 - row sum of T + R) B over the quadrature columns (and T's
  // diagonal on the sensor row) = (row sum of U - row sum of R) B
  for (int i = 0; i < nZ; i++) {
    float a = 0.0f;
    for (int j = 0; j < nS; j++) a += Um.a[i][j] - Rm.a[i][j];
    if (i == nZ - 1) a += Um.a[i][i];
    src[i] = a * B;
  }
  return true;
}

// ada_layer_adjoint.
template <int NZ, int NS>
CRTM_HD bool ada_layer_adjoint(float w, float tau, const float* mu, const float* wt, const Mat<NZ, float>& ff,
                               const Mat<NZ, float>& bb, float B, const Mat<NZ, float>& T_b, const Mat<NZ, float>& R_b,
                               const float* src_b, float* w_b, float* tau_b, Mat<NZ, float>& ff_b,
                               Mat<NZ, float>& bb_b, float* B_b, double* gap) {
  constexpr int nS = NS, n = NS + 1;
  if (gap) *gap = 1.0;
  if (tau < float(DELTA_OPTICAL_DEPTH)) {   // thin layer (first-order scattering)
    const float s = tau * w;
    float s_b = 0.0f, tb = 0.0f, bsum = 0.0f;
    for (int i = 0; i < n; i++) {
      const float c = s / mu[i];
      float th = 0.0f;
      for (int j = 0; j < n; j++)
        th += c * (bb.a[i][j] + ff.a[i][j]) * wt[j] + (i == j ? 1.0f - tau / mu[i] : 0.0f);
      bsum += src_b[i] * (1.0f - th);
      const float th_b = prod(-src_b[i], B);
      float c_b = 0.0f;
      for (int j = 0; j < n; j++) {
        const float rb = R_b.a[i][j] + th_b, tbij = T_b.a[i][j] + th_b;
        c_b = add_prod(c_b, two_prods(rb, bb.a[i][j], tbij, ff.a[i][j]), wt[j]);
        bb_b.a[i][j] = prod(rb * c, wt[j]);
        ff_b.a[i][j] = prod(tbij * c, wt[j]);
        if (i == j) tb -= tbij / mu[i];
      }
      s_b += c_b / mu[i];
    }
    *tau_b = tb + s_b * w;
    *w_b = s_b * tau;
    *B_b = bsum;
    return true;
  }
  // ---- forward in the loss form of ada_layer_loss, keeping what the
  // reverse sweep reads.  With P = Gm^-1 Gp, D = diag(1 - exp(-ev tau)) and
  // e = diag(exp(-ev tau)):  W = D P e + P D,  Q = Gm - Gp P,  GA = Q + Gp W,
  // U = (Q D + Gp W) GA^-1 = I - T,  R = (Gp D + Gm D P e) GA^-1.  Every
  // term of U and R is O(tau) for a thin layer, and so is every adjoint that
  // reaches the eigen-decomposition below: the FP32 form keeps its relative
  // accuracy where the plain form T = Tt GA^-1 loses it to cancellation.
  const float s = w < float(MAX_ALBEDO) ? w : float(MAX_ALBEDO);
  Mat<NZ, float> E, iX, Gp, Gm, iGm, P, W, iGA, Um, Rm, T1, T2;
  float lam[NZ], ev[NZ], ex[NZ], dx[NZ], buf[NZ];
  if (!mom_eigen<NZ, NS>(s, mu, wt, ff, bb, E, lam, iX, T1, T2, Um, gap)) return false;
  if (!mat_invert<NZ, NS>(iX)) return false;   // (PP - PM)^-1
  for (int i = 0; i < n; i++) {
    ev[i] = lam[i] > 0.0f ? sqrt(lam[i]) : 0.0f;
    ex[i] = exp(-ev[i] * tau);
    dx[i] = -expm1(-ev[i] * tau);
  }
  // EF = (PP-PM)^-1 E diag(ev);  Gp = (E + EF)/2, Gm = (E - EF)/2
  for (int i = 0; i < n; i++)
    for (int j = 0; j < n; j++) {
      float v = 0.0f;
      for (int k = 0; k < n; k++) v += iX.a[i][k] * E.a[k][j];
      Gp.a[i][j] = prod(0.5f, add_prod(E.a[i][j], v, ev[j]));
      Gm.a[i][j] = prod(0.5f, sub_prod(E.a[i][j], v, ev[j]));
    }
  iGm = Gm;
  if (!mat_invert<NZ, NS>(iGm)) return false;
  mat_mul(n, iGm, Gp, P);
  for (int i = 0; i < n; i++)
    for (int j = 0; j < n; j++) W.a[i][j] = two_prods(dx[i] * P.a[i][j], ex[j], P.a[i][j], dx[j]);
  for (int i = 0; i < n; i++)   // Q (T1)
    for (int j = 0; j < n; j++) {
      float v = 0.0f;
      for (int k = 0; k < n; k++) v += Gp.a[i][k] * P.a[k][j];
      T1.a[i][j] = Gm.a[i][j] - v;
    }
  // GA (iGA), U numerator (T1, in place over Q), R numerator (T2)
  for (int i = 0; i < n; i++)
    for (int j = 0; j < n; j++) {
      float gw = 0.0f, gd = 0.0f;
      for (int k = 0; k < n; k++) {
        gw += Gp.a[i][k] * W.a[k][j];
        gd += Gm.a[i][k] * dx[k] * P.a[k][j];
      }
      iGA.a[i][j] = T1.a[i][j] + gw;
      T1.a[i][j] = T1.a[i][j] * dx[j] + gw;
      T2.a[i][j] = two_prods(Gp.a[i][j], dx[j], gd, ex[j]);
    }
  if (!mat_invert<NZ, NS>(iGA)) return false;
  mat_mul(n, T1, iGA, Um);
  mat_mul(n, T2, iGA, Rm);
  // ---- reverse ----
  // src_i = a_i B with a_i the row sum of U - R over the quadrature columns
  // (and U's diagonal on the sensor row); U_b = -T_b.  U_b in T1, R_b in T2.
  float bsum = 0.0f;
  for (int i = 0; i < n; i++) {
    float a = 0.0f;
    for (int j = 0; j < nS; j++) a += Um.a[i][j] - Rm.a[i][j];
    if (i == n - 1) a += Um.a[i][i];
    bsum += src_b[i] * a;
    const float sb = prod(src_b[i], B);
    for (int j = 0; j < n; j++) {
      const bool in_a = j < nS || (i == n - 1 && j == i);
      T1.a[i][j] = (in_a ? sb : 0.0f) - T_b.a[i][j];
      T2.a[i][j] = R_b.a[i][j] - (j < nS ? sb : 0.0f);
    }
  }
  *B_b = bsum;
  // U = Un GA^-1, R = Rn GA^-1:  Un_b = U_b GA^-T, Rn_b = R_b GA^-T (row by
  // row in place), then GA_b = -(U^T Un_b + R^T Rn_b) into iGA
  for (int i = 0; i < n; i++) {
    for (int j = 0; j < n; j++) {
      float v = 0.0f;
      for (int k = 0; k < n; k++) v += T1.a[i][k] * iGA.a[j][k];
      buf[j] = v;
    }
    for (int j = 0; j < n; j++) T1.a[i][j] = buf[j];
    for (int j = 0; j < n; j++) {
      float v = 0.0f;
      for (int k = 0; k < n; k++) v += T2.a[i][k] * iGA.a[j][k];
      buf[j] = v;
    }
    for (int j = 0; j < n; j++) T2.a[i][j] = buf[j];
  }
  for (int i = 0; i < n; i++)
    for (int j = 0; j < n; j++) {
      float v = 0.0f;
      for (int k = 0; k < n; k++) v += two_prods(Um.a[k][i], T1.a[k][j], Rm.a[k][i], T2.a[k][j]);
      iGA.a[i][j] = -v;
    }
  Mat<NZ, float>& GAb = iGA;
  Mat<NZ, float>& Qb = Um;   // U, R are dead
  Mat<NZ, float>& Wb = Rm;
  float dx_b[NZ], ex_b[NZ];
  for (int j = 0; j < n; j++) { dx_b[j] = 0.0f; ex_b[j] = 0.0f; }
  // Un = Q D + Gp W, GA = Q + Gp W:  Q_b = Un_b D + GA_b;  dx_b_j += sum_i Un_b_ij Q_ij;
  //   with S = Un_b + GA_b (T1):  W_b = Gp^T S;  Gp_b = S W^T
  for (int i = 0; i < n; i++)
    for (int j = 0; j < n; j++) {
      float v = 0.0f;
      for (int k = 0; k < n; k++) v += Gp.a[i][k] * P.a[k][j];
      dx_b[j] += T1.a[i][j] * (Gm.a[i][j] - v);
      Qb.a[i][j] = T1.a[i][j] * dx[j] + GAb.a[i][j];
      T1.a[i][j] += GAb.a[i][j];
    }
  mat_mul_tn(n, Gp, T1, Wb);
  Mat<NZ, float>& Gpb = iGA;   // GA_b is dead
  mat_mul_nt(n, T1, W, Gpb);
  Mat<NZ, float>& Gmb = T1;    // S is dead
  // Rn = Gp D + Gm D P e:  Gp_b += Rn_b D;  dx_b_j += sum_i Rn_b_ij Gp_ij;
  //   ex_b_j += sum_i Rn_b_ij (Gm D P)_ij;  with Z = Rn_b e:  Gm_b = Z P^T D,
  //   dx_b_k += sum_i Gm_ik (Z P^T)_ik;  P_b = D Gm^T Z (column by column into T2)
  for (int i = 0; i < n; i++)
    for (int j = 0; j < n; j++) {
      const float rb = T2.a[i][j];
      Gpb.a[i][j] += rb * dx[j];
      float g = 0.0f;
      for (int k = 0; k < n; k++) g += Gm.a[i][k] * dx[k] * P.a[k][j];
      dx_b[j] += rb * Gp.a[i][j];
      ex_b[j] += rb * g;
    }
  for (int i = 0; i < n; i++)
    for (int k = 0; k < n; k++) {
      float zp = 0.0f;
      for (int j = 0; j < n; j++) zp += T2.a[i][j] * ex[j] * P.a[k][j];
      Gmb.a[i][k] = prod(zp, dx[k]);
      dx_b[k] += Gm.a[i][k] * zp;
    }
  for (int j = 0; j < n; j++) {
    for (int k = 0; k < n; k++) {
      float v = 0.0f;
      for (int i = 0; i < n; i++) v += Gm.a[i][k] * T2.a[i][j];
      buf[k] = prod(dx[k] * v, ex[j]);
    }
    for (int k = 0; k < n; k++) T2.a[k][j] = buf[k];
  }
  Mat<NZ, float>& Pb = T2;
  // Q = Gm - Gp P:  Gm_b += Q_b;  Gp_b -= Q_b P^T;  P_b -= Gp^T Q_b
  for (int i = 0; i < n; i++)
    for (int j = 0; j < n; j++) {
      float a = 0.0f, b = 0.0f;
      for (int k = 0; k < n; k++) {
        a += Qb.a[i][k] * P.a[j][k];
        b += Gp.a[k][i] * Qb.a[k][j];
      }
      Gmb.a[i][j] += Qb.a[i][j];
      Gpb.a[i][j] -= a;
      Pb.a[i][j] -= b;
    }
  // W_ij = dx_i P_ij ex_j + P_ij dx_j
  for (int i = 0; i < n; i++)
    for (int j = 0; j < n; j++) {
      const float wb = Wb.a[i][j], pij = P.a[i][j];
      Pb.a[i][j] += wb * (dx[i] * ex[j] + dx[j]);
      dx_b[i] = add_prod(dx_b[i], prod(wb, pij), ex[j]);
      ex_b[j] = add_prod(ex_b[j], wb * dx[i], pij);
      dx_b[j] += prod(wb, pij);
    }
  // P = Gm^-1 Gp:  K = Gm^-T P_b;  Gp_b += K;  Gm_b -= K P^T
  Mat<NZ, float>& Kt = Um;   // Q_b is dead
  mat_mul_tn(n, iGm, Pb, Kt);
  for (int i = 0; i < n; i++)
    for (int j = 0; j < n; j++) {
      float v = 0.0f;
      for (int k = 0; k < n; k++) v += Kt.a[i][k] * P.a[j][k];
      Gpb.a[i][j] += Kt.a[i][j];
      Gmb.a[i][j] -= v;
    }
  // Gp = (E + EF)/2, Gm = (E - EF)/2
  Mat<NZ, float>& Eb = Gpb;
  Mat<NZ, float>& EFb = Gmb;
  for (int i = 0; i < n; i++)
    for (int j = 0; j < n; j++) {
      const float p = Gpb.a[i][j], q = Gmb.a[i][j];
      Eb.a[i][j] = prod(0.5f, p + q);
      EFb.a[i][j] = prod(0.5f, p - q);
    }
  // EF = iX E diag(ev):  iX_b = EF_b (E diag(ev))^T;  EV_b = iX^T EF_b;
  //   E_b += EV_b diag(ev);  ev_b_j = sum_i EV_b_ij E_ij
  Mat<NZ, float>& iXb = Um;   // K is dead
  Mat<NZ, float>& EVb = Rm;   // W_b is dead
  for (int i = 0; i < n; i++)
    for (int j = 0; j < n; j++) {
      float v = 0.0f;
      for (int k = 0; k < n; k++) v += EFb.a[i][k] * E.a[j][k] * ev[k];
      iXb.a[i][j] = v;
    }
  mat_mul_tn(n, iX, EFb, EVb);
  float lam_b[NZ];
  float tb = 0.0f;
  for (int j = 0; j < n; j++) {
    float v = 0.0f;
    for (int i = 0; i < n; i++) {
      v += EVb.a[i][j] * E.a[i][j];
      Eb.a[i][j] += EVb.a[i][j] * ev[j];
    }
    // ex_j = exp(-ev_j tau), dx_j = 1 - ex_j, ev_j = sqrt(lam_j)
    const float d = dx_b[j] - ex_b[j];
    const float ev_b = v + tau * ex[j] * d;
    tb += ev[j] * ex[j] * d;
    lam_b[j] = lam[j] > 0.0f ? 0.5f * ev_b / ev[j] : 0.0f;
  }
  *tau_b = tb;
  // X = PP - PM inverted:  X_b = -iX^T iX_b iX^T  (in P; W is scratch)
  Mat<NZ, float>& Xb = P;
  inverse_adjoint(n, iX, iXb, Xb, W);
  // HH = E diag(lam) E^-1:  HH_b = E^-T (diag(lam_b) + F o (E^T E_b)) E^T,
  // F_ij = 1 / (lam_j - lam_i) off the diagonal
  Mat<NZ, float>& Ei = Gp;    // Gp, Gm, iGm are dead
  Mat<NZ, float>& Mx = Gm;
  Ei = E;
  if (!mat_invert<NZ, NS>(Ei)) return false;
  mat_mul_tn(n, E, Eb, Mx);
  for (int i = 0; i < n; i++)
    for (int j = 0; j < n; j++)
      Mx.a[i][j] = (i == j) ? lam_b[i] : Mx.a[i][j] / (lam[j] - lam[i]);
  Mat<NZ, float>& HHb = Rm;   // EV_b is dead
  mat_mul_tn(n, Ei, Mx, T2);   // E^-T M  (P_b is dead)
  mat_mul_nt(n, T2, E, HHb);   // (E^-T M) E^T
  // HH = X Y with X = PP - PM, Y = PP + PM (rebuilt from the phase blocks):
  //   X_b += HH_b Y^T;  Y_b = X^T HH_b
  Mat<NZ, float>& X = iGm;
  Mat<NZ, float>& Y = W;
  for (int i = 0; i < n; i++) {
    const float c = s / mu[i];
    for (int j = 0; j < n; j++) {
      const float f = add_prod(i == j ? -(1.0f / mu[i]) : 0.0f, c * ff.a[i][j], wt[j]), b = c * bb.a[i][j];
      X.a[i][j] = sub_prod(f, b, wt[j]);
      Y.a[i][j] = add_prod(f, b, wt[j]);
    }
  }
  Mat<NZ, float>& Yb = T2;
  mat_mul_tn(n, X, HHb, Yb);
  mat_mul_nt(n, HHb, Y, Um);   // iX_b is dead
  // f = c_i ff_ij wt_j - delta_ij / mu_i, b = c_i bb_ij wt_j, c_i = s / mu_i;
  // X = f - b, Y = f + b
  float s_b = 0.0f;
  for (int i = 0; i < n; i++) {
    const float c = s / mu[i];
    float c_b = 0.0f;
    for (int j = 0; j < n; j++) {
      const float xb = Xb.a[i][j] + Um.a[i][j];
      const float fb = xb + Yb.a[i][j], bbv = Yb.a[i][j] - xb;
      ff_b.a[i][j] = prod(fb * c, wt[j]);
      bb_b.a[i][j] = prod(bbv * c, wt[j]);
      c_b = add_prod(c_b, two_prods(fb, ff.a[i][j], bbv, bb.a[i][j]), wt[j]);
    }
    s_b += c_b / mu[i];
  }
  *w_b = w < float(MAX_ALBEDO) ? s_b : 0.0f;
  return true;
}

// phase_blocks: the phase blocks from the Legendre terms, normalised.
template <int NZ, int NS>
CRTM_HD void phase_blocks(const float* pc, const float (*P)[SC_NLEG_MAX + 1],
                                 const float* wt, Mat<NZ, float>& ff, Mat<NZ, float>& bb) {
  constexpr int nS = NS, nZ = NS + 1, nleg = 2 * NS - 2;
  for (int i = 0; i < nZ; i++)
    for (int j = i; j < nZ; j++) {
      float f = 0.0f, b = 0.0f;
      for (int l = 0; l < nleg; l++) {
        const float u = pc[l] * P[i][l];
        f = add_prod(f, u, P[j][l]);
        b = (l & 1) ? sub_prod(b, u, P[j][l]) : add_prod(b, u, P[j][l]);
      }
      ff.a[i][j] = ff.a[j][i] = f < 0.0f ? float(PHASE_THRESHOLD) : f;
      bb.a[i][j] = bb.a[j][i] = b < 0.0f ? float(PHASE_THRESHOLD) : b;
    }
  float carried = 0.0f;
  for (int i = 0; i < nS; i++) {
    float nf = 0.0f;
    for (int j = i; j < nZ; j++) nf += (ff.a[i][j] + bb.a[i][j]) * wt[j];
    const float sc = (1.0f - carried) / nf;
    for (int j = i; j < nZ; j++) {
      ff.a[i][j] = prod(ff.a[i][j], sc); bb.a[i][j] = prod(bb.a[i][j], sc);
      ff.a[j][i] = ff.a[i][j]; bb.a[j][i] = bb.a[i][j];
    }
    carried = 0.0f;
    if (i + 1 < nZ)
      for (int j = 0; j <= i; j++) carried += (ff.a[i + 1][j] + bb.a[i + 1][j]) * wt[j];
  }
  if (nS < nZ) {
    const int z = nZ - 1;
    for (int j = 0; j < nZ; j++) {
      ff.a[j][z] /= carried; bb.a[j][z] /= carried;
      if (j < z) { ff.a[z][j] = ff.a[j][z]; bb.a[z][j] = bb.a[j][z]; }
    }
  }
}

// phase_blocks_adjoint.
template <int NZ, int NS>
CRTM_HD void phase_blocks_adjoint(const float* pc, const float (*P)[SC_NLEG_MAX + 1], const float* wt,
                                  const Mat<NZ, float>& ff_b, const Mat<NZ, float>& bb_b, float* pc_b) {
  constexpr int nS = NS, nZ = NS + 1, nleg = 2 * NS - 2;
  Mat<NZ, float> f0, b0, fb, bq;   // clamped unscaled blocks (upper triangle) and their adjoints
  unsigned clampf[NZ] = {0}, clampb[NZ] = {0};
  for (int i = 0; i < nZ; i++)
    for (int j = i; j < nZ; j++) {
      float f = 0.0f, b = 0.0f;
      for (int l = 0; l < nleg; l++) {
        const float u = pc[l] * P[i][l];
        f = add_prod(f, u, P[j][l]);
        b = (l & 1) ? sub_prod(b, u, P[j][l]) : add_prod(b, u, P[j][l]);
      }
      if (f < 0.0f) { f = float(PHASE_THRESHOLD); clampf[i] |= 1u << j; }
      if (b < 0.0f) { b = float(PHASE_THRESHOLD); clampb[i] |= 1u << j; }
      f0.a[i][j] = f;
      b0.a[i][j] = b;
      fb.a[i][j] = 0.0f;
      bq.a[i][j] = 0.0f;
    }
  // forward scales
  float sc[NZ], nf[NZ];
  float carried = 0.0f;
  for (int i = 0; i < nS; i++) {
    float v = 0.0f;
    for (int j = i; j < nZ; j++) v += (f0.a[i][j] + b0.a[i][j]) * wt[j];
    nf[i] = v;
    sc[i] = (1.0f - carried) / v;
    carried = 0.0f;
    if (i + 1 < nZ)
      for (int j = 0; j <= i; j++) carried += (f0.a[j][i + 1] + b0.a[j][i + 1]) * sc[j] * wt[j];
  }
  const bool sensor = nS < nZ;
  const int z = nZ - 1;
  const float cz = carried;   // the sensor column's divisor (when sensor)
  float sc_b[NZ];
  for (int i = 0; i < nZ; i++) sc_b[i] = 0.0f;
  float cz_b = 0.0f;
  // final entries: (i <= j) f0_ij sc_i, the sensor column further / cz
  for (int i = 0; i < nZ; i++)
    for (int j = i; j < nZ; j++) {
      const float hf = (i == j) ? ff_b.a[i][i] : ff_b.a[i][j] + ff_b.a[j][i];
      const float hb = (i == j) ? bb_b.a[i][i] : bb_b.a[i][j] + bb_b.a[j][i];
      const float si = i < nS ? sc[i] : 1.0f;
      if (sensor && j == z) {
        fb.a[i][j] += hf * si / cz;
        bq.a[i][j] += hb * si / cz;
        const float hs = two_prods(hf, f0.a[i][j], hb, b0.a[i][j]);
        if (i < nS) sc_b[i] += hs / cz;
        cz_b -= hs * si / (cz * cz);
      } else {
        fb.a[i][j] += prod(hf, si);
        bq.a[i][j] += prod(hb, si);
        sc_b[i] += two_prods(hf, f0.a[i][j], hb, b0.a[i][j]);
      }
    }
  if (sensor)   // cz = sum_{j < z} (f0_jz + b0_jz) sc_j wt_j
    for (int j = 0; j < z; j++) {
      fb.a[j][z] = add_prod(fb.a[j][z], cz_b * sc[j], wt[j]);
      bq.a[j][z] = add_prod(bq.a[j][z], cz_b * sc[j], wt[j]);
      sc_b[j] += cz_b * (f0.a[j][z] + b0.a[j][z]) * wt[j];
    }
  for (int i = nS - 1; i >= 0; i--) {   // sc_i = (1 - carried_i) / nf_i
    const float car_b = -sc_b[i] / nf[i], nf_b = -sc_b[i] * sc[i] / nf[i];
    for (int j = i; j < nZ; j++) {
      fb.a[i][j] = add_prod(fb.a[i][j], nf_b, wt[j]);
      bq.a[i][j] = add_prod(bq.a[i][j], nf_b, wt[j]);
    }
    for (int j = 0; j < i; j++) {   // carried_i = sum_{j < i} (f0_ji + b0_ji) sc_j wt_j
      fb.a[j][i] = add_prod(fb.a[j][i], car_b * sc[j], wt[j]);
      bq.a[j][i] = add_prod(bq.a[j][i], car_b * sc[j], wt[j]);
      sc_b[j] += car_b * (f0.a[j][i] + b0.a[j][i]) * wt[j];
    }
  }
  for (int l = 0; l < nleg; l++) pc_b[l] = 0.0f;
  for (int i = 0; i < nZ; i++)
    for (int j = i; j < nZ; j++) {
      const float gf = (clampf[i] >> j) & 1u ? 0.0f : fb.a[i][j];
      const float gb = (clampb[i] >> j) & 1u ? 0.0f : bq.a[i][j];
      for (int l = 0; l < nleg; l++) pc_b[l] += ((l & 1) ? gf - gb : gf + gb) * P[i][l] * P[j][l];
    }
}

}  // namespace fixed
}  // namespace crtm
