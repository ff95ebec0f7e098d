// g3_fatbra.cuh -- the composite-bra / pair-ket form of the four-particle
// geminal Coulomb integrals G4_MD_xgVepg and G4_MD_xgVeeg (XC1_G4_MD.f:
// 796-1125, 1559-1978) used by the gam_3 builder (k_gam3.cu, whose header
// comment gives the derivation).  Every function is __host__ __device__ so
// the tests can compare it, compiled as plain C++, with the element-wise
// md_math.cuh integrals.  R = double (FP64 path) or float (mixed path); the
// Boys function, the seeds (-alpha)^m F_m(T) and their sum are FP64 in both.
#pragma once
#include <math.h>
#include <string.h>

#include "md_math.cuh"

#if defined(__CUDACC__)
#define G3_HD __host__ __device__ __forceinline__
#else
#define G3_HD inline
#endif

namespace neoxc {
namespace g3 {

// C(t,i) 2^(2i-t) in the precision of the contraction
template <class R>
G3_HD R hermc_r(int t, int i) {
  if constexpr (sizeof(R) == sizeof(float)) return hermc32(t, i);
  else return (R)hermc(t, i);
}

// ---- pair records (FP64, 32 doubles each) ----------------------------------
// [0] p  [1..3] P  [4] c_a c_b  [5..19] E[d][t] (t <= 4)  [20..22] t_max[d]
// [23] S  [24] Q (screening magnitudes, see k_gam3.cu)
enum { kRP = 0, kRX = 1, kRC = 4, kRE = 5, kRT = 20, kRS = 23, kRQ = 24, kRLen = 32 };

G3_HD int pair_index(int i, int j) {
  return i >= j ? i * (i + 1) / 2 + j : j * (j + 1) / 2 + i;
}

// Record of one primitive pair (A, B) with contraction coefficients ca, cb
// (without Q, which comes from the record itself: g2::schwarz_factor).
G3_HD void fill_pair_record(const md::Prim& A, const md::Prim& B, double ca, double cb,
                            double* out) {
  md::Pair pr;
  md::gauss_pair(A, B, pr);
  out[kRP] = pr.p;
  for (int d = 0; d < 3; d++) out[kRX + d] = pr.P[d];
  out[kRC] = ca * cb;
  double ang = 1.0;
  const double sig = 1.0 / sqrt(pr.p);
  for (int d = 0; d < 3; d++) {
    double tmp[2 * md::TMX + 1];
    const int tl = A.l[d] + B.l[d];
    md::hermite_e(A.l[d], B.l[d], pr.K[d], A.a, B.a, pr.p, pr.q, pr.Q[d], tmp);
    for (int k = 0; k < 5; k++) out[kRE + 5 * d + k] = k <= tl ? tmp[k] : 0.0;
    out[kRT + d] = (double)tl;
    for (int k = 0; k < A.l[d]; k++) ang *= fabs(pr.P[d] - A.c[d]) + sig;
    for (int k = 0; k < B.l[d]; k++) ang *= fabs(pr.P[d] - B.c[d]) + sig;
  }
  const double cab = fabs(ca * cb);
  const double pi = 3.14159265358979323846;
  out[kRS] = cab * pow(pi / pr.p, 1.5) * pr.K[0] * pr.K[1] * pr.K[2] * ang;
  for (int k = kRQ; k < kRLen; k++) out[k] = 0.0;
}

// ---- composite bra -----------------------------------------------------------
template <class R, int NW>
struct Bra {
  R W[3][NW + 1];   // W'_d
  R Z;              // composite exponent (Tx4 for Vep, W1 for Vee)
  R C[3];           // composite centre
  R pref;           // C0 * CB0
  double wgt;       // sign x b_k b_l x contraction coefficients of the bra's pairs
  double est;       // screening estimate of the bra's factors
  int N[3];
};

// derivatives of prod_k exp(-xi_k (c_k . x)^2), x = (x0, x1, x2), at X;
// extents X0, X1, X2 (D[(n0*X1 + n1)*X2 + n2]); the recurrence of dgauss3.
template <class R, int X0, int X1, int X2>
G3_HD void dgauss3t(int nk, const R* xi, const R (*c)[3], const R* X,
                    const int* N, R* D) {
  R grad[3] = {0, 0, 0}, H[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
  R expo = R(0);
  for (int k = 0; k < nk; k++) {
    const R u = c[k][0] * X[0] + c[k][1] * X[1] + c[k][2] * X[2];
    expo -= xi[k] * u * u;
    for (int i = 0; i < 3; i++) {
      grad[i] += R(2) * xi[k] * u * c[k][i];
      for (int j = 0; j < 3; j++) H[i][j] += R(2) * xi[k] * c[k][i] * c[k][j];
    }
  }
  const R base = exp(expo);
#define DD(a, b, e) D[((a) * X1 + (b)) * X2 + (e)]
  for (int n0 = 0; n0 <= N[0]; n0++)
    for (int n1 = 0; n1 <= N[1]; n1++)
      for (int n2 = 0; n2 <= N[2]; n2++) {
        if (n0 + n1 + n2 == 0) { DD(0, 0, 0) = base; continue; }
        int m[3] = {n0, n1, n2};
        const int i = n0 > 0 ? 0 : (n1 > 0 ? 1 : 2);
        m[i] -= 1;
        R v = -grad[i] * DD(m[0], m[1], m[2]);
        for (int j = 0; j < 3; j++)
          if (m[j] > 0) {
            int r[3] = {m[0], m[1], m[2]};
            r[j] -= 1;
            v -= H[i][j] * (R)m[j] * DD(r[0], r[1], r[2]);
          }
        DD(n0, n1, n2) = v;
      }
#undef DD
}

// C(n, k), k <= n <= 4
G3_HD int binom4(int n, int k) {
  return k == 0 || k == n ? 1 : (n == 4 && k == 2 ? 6 : n);
}

// In place along one axis: v[x] <- sum_s v[s] E[s + x] C(s + x, x), s + x <= t.
G3_HD void fold_line(double* v, int stride, int t, const double* E) {
  const double v0 = v[0];
  if (t == 0) {
    v[0] = v0 * E[0];
    return;
  }
  const double v1 = v[stride];
  if (t == 1) {
    v[0] = fma(v1, E[1], v0 * E[0]);
    v[stride] = v0 * E[1];
    return;
  }
  const double v2 = v[2 * stride];
  if (t == 2) {
    v[0] = fma(v2, E[2], fma(v1, E[1], v0 * E[0]));
    v[stride] = fma(v1 + v1, E[2], v0 * E[1]);
    v[2 * stride] = v0 * E[2];
    return;
  }
  const double v3 = v[3 * stride];
  if (t == 3) {
    v[0] = fma(v3, E[3], fma(v2, E[2], fma(v1, E[1], v0 * E[0])));
    v[stride] = fma(3.0 * v2, E[3], fma(v1 + v1, E[2], v0 * E[1]));
    v[2 * stride] = fma(3.0 * v1, E[3], v0 * E[2]);
    v[3 * stride] = v0 * E[3];
    return;
  }
  const double v4 = v[4 * stride];
  v[0] = fma(v4, E[4], fma(v3, E[3], fma(v2, E[2], fma(v1, E[1], v0 * E[0]))));
  v[stride] = fma(4.0 * v3, E[4], fma(3.0 * v2, E[3], fma(v1 + v1, E[2], v0 * E[1])));
  v[2 * stride] = fma(6.0 * v2, E[4], fma(3.0 * v1, E[3], v0 * E[2]));
  v[3 * stride] = fma(4.0 * v1, E[4], v0 * E[3]);
  v[4 * stride] = v0 * E[4];
}

// W'_d[x0+x1+x2] = sum E0[t0] E1[t1] E2[t2] sum_x C(t,x) cof^x D(t - x):
// slots 0, 1 electrons (extent 2LE+1), slot 2 the proton (2LN+1).
template <class R, int LE, int LN, int NW>
G3_HD void fold_bra(const double* r0, const double* r1, const double* r2, int nk,
                    const R* xi, const R (*c)[3], const R* cof, Bra<R, NW>& b) {
  constexpr int X0 = 2 * LE + 1, X2 = 2 * LN + 1;
  R D[X0 * X0 * X2];
  R pw[3][5];
  for (int i = 0; i < 3; i++) {
    pw[i][0] = R(1);
    for (int k = 1; k < 5; k++) pw[i][k] = pw[i][k - 1] * cof[i];
  }
  const double* rr[3] = {r0, r1, r2};
  for (int d = 0; d < 3; d++) {
    int tl[3];
    R X[3];
    for (int i = 0; i < 3; i++) {
      tl[i] = (int)rr[i][kRT + d];
      X[i] = (R)rr[i][kRX + d];
    }
    dgauss3t<R, X0, X0, X2>(nk, xi, c, X, tl, D);
    for (int n = 0; n <= NW; n++) b.W[d][n] = R(0);
    for (int t0 = 0; t0 <= tl[0]; t0++)
      for (int t1 = 0; t1 <= tl[1]; t1++)
        for (int t2 = 0; t2 <= tl[2]; t2++) {
          const R e = (R)r0[kRE + 5 * d + t0] * (R)r1[kRE + 5 * d + t1] *
                      (R)r2[kRE + 5 * d + t2];
          for (int x0 = 0; x0 <= t0; x0++)
            for (int x1 = 0; x1 <= t1; x1++)
              for (int x2 = 0; x2 <= t2; x2++) {
                const R cc = (R)(binom4(t0, x0) * binom4(t1, x1) * binom4(t2, x2)) *
                             pw[0][x0] * pw[1][x1] * pw[2][x2] *
                             D[((t0 - x0) * X0 + (t1 - x1)) * X2 + (t2 - x2)];
                b.W[d][x0 + x1 + x2] += e * cc;
              }
        }
    b.N[d] = tl[0] + tl[1] + tl[2];
  }
}

// The same in FP64 with far fewer operations: one exponential for the three
// directions (into *scale), and the sums over t one particle at a time.
template <int LE, int LN, int NW>
G3_HD void fold_bra(const double* r0, const double* r1, const double* r2, int nk,
                    const double* xi, const double (*c)[3], const double* cof,
                    Bra<double, NW>& b, double* scale) {
  constexpr int X0 = 2 * LE + 1, X2 = 2 * LN + 1;
  double H[6] = {0, 0, 0, 0, 0, 0};   // 2 sum_k xi_k c_k c_k^T: 00 01 02 11 12 22
  for (int k = 0; k < nk; k++) {
    const double x0 = 2.0 * xi[k] * c[k][0], x1 = 2.0 * xi[k] * c[k][1];
    H[0] = fma(x0, c[k][0], H[0]);
    H[1] = fma(x0, c[k][1], H[1]);
    H[2] = fma(x0, c[k][2], H[2]);
    H[3] = fma(x1, c[k][1], H[3]);
    H[4] = fma(x1, c[k][2], H[4]);
    H[5] = fma(2.0 * xi[k] * c[k][2], c[k][2], H[5]);
  }
  double ex = 0.0;
  for (int d = 0; d < 3; d++) {
    const double X[3] = {r0[kRX + d], r1[kRX + d], r2[kRX + d]};
    const int t0 = (int)r0[kRT + d], t1 = (int)r1[kRT + d], t2 = (int)r2[kRT + d];
    double g0 = 0.0, g1 = 0.0, g2 = 0.0;   // -gradient
    for (int k = 0; k < nk; k++) {
      const double u = c[k][0] * X[0] + c[k][1] * X[1] + c[k][2] * X[2], xu = xi[k] * u;
      ex = fma(xu, u, ex);
      g0 = fma(-2.0 * xu, c[k][0], g0);
      g1 = fma(-2.0 * xu, c[k][1], g1);
      g2 = fma(-2.0 * xu, c[k][2], g2);
    }
    const int w2 = t2 + 1, w1 = (t1 + 1) * w2;
    double V[X0 * X0 * X2];
    for (int n0 = 0; n0 <= t0; n0++)
      for (int n1 = 0; n1 <= t1; n1++)
        for (int n2 = 0; n2 <= t2; n2++) {
          const int o = n0 * w1 + n1 * w2 + n2;
          double v = 1.0;
          if (n0 > 0) {
            v = g0 * V[o - w1];
            if (n0 > 1) v = fma(-H[0] * (double)(n0 - 1), V[o - 2 * w1], v);
            if (n1 > 0) v = fma(-H[1] * (double)n1, V[o - w1 - w2], v);
            if (n2 > 0) v = fma(-H[2] * (double)n2, V[o - w1 - 1], v);
          } else if (n1 > 0) {
            v = g1 * V[o - w2];
            if (n1 > 1) v = fma(-H[3] * (double)(n1 - 1), V[o - 2 * w2], v);
            if (n2 > 0) v = fma(-H[4] * (double)n2, V[o - w2 - 1], v);
          } else if (n2 > 0) {
            v = g2 * V[o - 1];
            if (n2 > 1) v = fma(-H[5] * (double)(n2 - 1), V[o - 2], v);
          }
          V[o] = v;
        }
    for (int n0 = 0; n0 <= t0; n0++)
      for (int n1 = 0; n1 <= t1; n1++) fold_line(V + n0 * w1 + n1 * w2, 1, t2, r2 + kRE + 5 * d);
    for (int n0 = 0; n0 <= t0; n0++)
      for (int n2 = 0; n2 <= t2; n2++) fold_line(V + n0 * w1 + n2, w2, t1, r1 + kRE + 5 * d);
    for (int n1 = 0; n1 < w1; n1++) fold_line(V + n1, w1, t0, r0 + kRE + 5 * d);
    const int n = t0 + t1 + t2;
    for (int k = 0; k <= n; k++) b.W[d][k] = 0.0;
    const double* v = V;
    double p0 = 1.0;
    for (int x0 = 0; x0 <= t0; x0++) {
      double p01 = p0;
      for (int x1 = 0; x1 <= t1; x1++) {
        double p = p01;
        for (int x2 = 0; x2 <= t2; x2++) {
          b.W[d][x0 + x1 + x2] = fma(p, *v++, b.W[d][x0 + x1 + x2]);
          if (x2 < t2) p *= cof[2];
        }
        if (x1 < t1) p01 *= cof[1];
      }
      if (x0 < t0) p0 *= cof[0];
    }
    b.N[d] = n;
  }
  *scale = exp(-ex);
}

// G4_MD_xgVepg's composite (XC1_G4_MD.f:1559-1978): e1 (r1), e2 (r2), proton
// (rp); geminals gam14 = gk (e1-p), gam24 = gl (e2-p); Coulomb partner e3.
template <class R, int LE, int LN, int NW>
G3_HD void build_bra_vep(const double* r1, const double* r2, const double* rp,
                         R gk, R gl, Bra<R, NW>& b) {
  const R kPiT = R(3.14159265358979e+00);
  const R P1 = (R)r1[kRP], P2 = (R)r2[kRP], P4 = (R)rp[kRP];
  const R C0 = (kPiT / (P1 + gk)) * sqrt(kPiT / (P1 + gk));
  const R C1 = (P1 * gk) / (P1 + gk);
  const R S4 = C1 + P4;
  const R CB0 = (kPiT / (P2 + gl)) * sqrt(kPiT / (P2 + gl));
  const R CB1 = (P2 * gl) / (P2 + gl);
  const R Tx4 = S4 + CB1;
  const R xcof = (S4 + CB1) * (C1 + P4);
  const R cof[3] = {S4 * C1 / xcof, CB1 / (S4 + CB1), S4 * P4 / xcof};
  for (int d = 0; d < 3; d++) {
    const R sm4 = (C1 * (R)r1[kRX + d] + P4 * (R)rp[kRX + d]) / (C1 + P4);
    b.C[d] = (S4 * sm4 + CB1 * (R)r2[kRX + d]) / (S4 + CB1);
  }
  const R xi[3] = {(P4 * C1) / (P4 + C1), (S4 * CB1) / (S4 + CB1), R(0)};
  const R c[3][3] = {{R(1), R(0), R(-1)},
                     {C1 / (C1 + P4), R(-1), P4 / (C1 + P4)},
                     {R(0), R(0), R(0)}};
  R scale = R(1);
  if constexpr (sizeof(R) == sizeof(float)) fold_bra<R, LE, LN, NW>(r1, r2, rp, 2, xi, c, cof, b);
  else fold_bra<LE, LN, NW>(r1, r2, rp, 2, xi, c, cof, b, &scale);
  b.Z = Tx4;
  b.pref = C0 * CB0;
  if constexpr (sizeof(R) != sizeof(float)) b.pref *= scale;
}

// G4_MD_xgVeeg's composite (XC1_G4_MD.f:796-1125): e1 (r1), e3 (r3), proton
// (rp); geminals gam14 = gk (e1-p), gam34 = gl (e3-p); Coulomb partner e2.
template <class R, int LE, int LN, int NW>
G3_HD void build_bra_vee(const double* r1, const double* r3, const double* rp,
                         R gk, R gl, Bra<R, NW>& b) {
  const R kPiT = R(3.14159265358979e+00);
  const R P1 = (R)r1[kRP], P3 = (R)r3[kRP], P4 = (R)rp[kRP];
  const R xsum = P4 + gk + gl;
  const R C0 = (kPiT / xsum) * sqrt(kPiT / xsum);
  const R C1 = (P4 * gk) / xsum, C3 = (P4 * gl) / xsum;
  const R C13 = (gk * gl) / xsum;
  const R S1 = P1 + C1, S3 = P3 + C3;
  const R CB0 = (kPiT / (S3 + C13)) * sqrt(kPiT / (S3 + C13));
  const R CB1 = (S3 * C13) / (S3 + C13);
  const R W1 = S1 + CB1;
  const R cof[3] = {P1 / (S1 + CB1), (CB1 / (S1 + CB1)) * (P3 / (P3 + C3)),
                    (C1 / (S1 + CB1)) + (CB1 / (S1 + CB1)) * (C3 / (P3 + C3))};
  for (int d = 0; d < 3; d++)
    b.C[d] = cof[0] * (R)r1[kRX + d] + cof[1] * (R)r3[kRX + d] + cof[2] * (R)rp[kRX + d];
  const R xi[3] = {P1 * C1 / (P1 + C1), P3 * C3 / (P3 + C3), S1 * CB1 / (S1 + CB1)};
  const R c[3][3] = {{R(1), R(0), R(-1)},
                     {R(0), R(1), R(-1)},
                     {P1 / (P1 + C1), -P3 / (P3 + C3), C1 / (P1 + C1) - C3 / (P3 + C3)}};
  R scale = R(1);
  if constexpr (sizeof(R) == sizeof(float)) fold_bra<R, LE, LN, NW>(r1, r3, rp, 3, xi, c, cof, b);
  else fold_bra<LE, LN, NW>(r1, r3, rp, 3, xi, c, cof, b, &scale);
  b.Z = W1;
  b.pref = C0 * CB0;
  if constexpr (sizeof(R) != sizeof(float)) b.pref *= scale;
}

// One (bra, ket) Coulomb integral, pref C4 sum_tuv W_x W_y W_z R_tuv, with
// W_d = W'_d (*) Ek_d (Ek: the ket's Hermite coefficients times (-1)^t) and
// the Hermite-Coulomb sum in factorised form:
//   sum_m (-alpha)^m F_m(T) sum_{i+j+k=m} A_x[i] A_y[j] A_z[k],
//   A_d[i] = sum_t W_d[t] C(t,i) 2^(2i-t) R_d^(2i-t).
// With s functions only (NW = NK = 0) the orders are known here: read at run
// time they cost 1100 instructions an evaluation, mostly loops of one turn
// (examples/xchf, FP32, a Vee pass: 559 us, 430 so).
template <class R, int NW, int NK>
G3_HD double fb_eval(const Bra<R, NW>& b, R pk, const R* Xk, const R (*Ek)[NK + 1],
                     const int* tk) {
  constexpr int NT = NW + NK;
  const R zk = b.Z + pk;
  const R alpha = (b.Z * pk) / zk;
  R Rv[3], R2 = R(0);
  for (int d = 0; d < 3; d++) {
    Rv[d] = b.C[d] - Xk[d];
    R2 += Rv[d] * Rv[d];
  }
  const R T = alpha * R2;
  const R kPiT = R(3.14159265358979e+00);
  const R C4 = (R(2) * kPiT * kPiT * sqrt(kPiT)) / (b.Z * pk * sqrt(zk));
  R A[3][NT + 1];
  int L = 0;
  for (int d = 0; d < 3; d++) {
    const int nb = NW > 0 ? b.N[d] : 0, nkd = NK > 0 ? tk[d] : 0, n = nb + nkd;
    R W[NT + 1];
    for (int m = 0; m <= n; m++) {
      R acc = R(0);
      const int lo = m - nb > 0 ? m - nb : 0, hi = m < nkd ? m : nkd;
      for (int t = lo; t <= hi; t++) acc += b.W[d][m - t] * Ek[d][t];
      W[m] = acc;
    }
    R xp[NT + 1];
    xp[0] = R(1);
    for (int k = 1; k <= n; k++) xp[k] = xp[k - 1] * Rv[d];
    for (int i = 0; i <= n; i++) A[d][i] = R(0);
    for (int t = 0; t <= n; t++)
      for (int i = (t + 1) / 2; i <= t; i++) A[d][i] += W[t] * hermc_r<R>(t, i) * xp[2 * i - t];
    L += n;
  }
  const int nx = (NW > 0 ? b.N[0] : 0) + (NK > 0 ? tk[0] : 0),
            ny = (NW > 0 ? b.N[1] : 0) + (NK > 0 ? tk[1] : 0),
            nz = (NW > 0 ? b.N[2] : 0) + (NK > 0 ? tk[2] : 0);
  R Bxy[2 * NT + 1];
  for (int m = 0; m <= nx + ny; m++) Bxy[m] = R(0);
  for (int i = 0; i <= nx; i++)
    for (int j = 0; j <= ny; j++) Bxy[i + j] += A[0][i] * A[1][j];
  // seeds (-alpha)^m F_m(T) and the final sum in FP64
  const double s = boys_sum(L, T, (double)alpha, [&](int m) {
    R bm = R(0);
    const int lo = m - nz > 0 ? m - nz : 0, hi = m < nx + ny ? m : nx + ny;
    for (int i = lo; i <= hi; i++) bm += Bxy[i] * A[2][m - i];
    return bm;
  });
  return (double)(b.pref * C4) * s;
}

// ---- FP64 evaluation -----------------------------------------------------------
// The same integral with the fewest FP64 instructions (2 per SM and clock on
// this GPU; integer and memory instructions beside them are free): one rsqrt
// serves alpha and the prefactor, bra and ket are normalised so that the
// common low orders multiply by nothing, (-alpha)^m is part of the Hermite
// powers, and the Boys recursion has one loop for both ranges of T.  About
// 120 instructions an evaluation where fb_eval<double> takes 230.

#if defined(__CUDACC__)
#define NX_LOOP _Pragma("unroll 1")
#else
#define NX_LOOP
#endif

G3_HD double rsqrt64(double x) {
#if defined(__CUDA_ARCH__)
  return rsqrt(x);
#else
  return 1.0 / sqrt(x);
#endif
}

G3_HD long long bits64(double x) {
#if defined(__CUDA_ARCH__)
  return __double_as_longlong(x);
#else
  long long b;
  memcpy(&b, &x, sizeof(b));
  return b;
#endif
}

// |x| < 1e-100 -> 0 (underflow.f:2-11), compared as integers (the bits of 1e-100)
G3_HD double underflow_bits(double x) {
  return (bits64(x) & 0x7fffffffffffffffLL) < 0x2b2bff2ee48e0530LL ? 0.0 : x;
}

// Gamma(L + 1/2) / 2, L = 0..16: F_L(T) ~ Gamma(L + 1/2) / (2 T^(L + 1/2))
#define NX_ASYM_VALUES \
    0.886226925452758, 0.443113462726379, 0.6646701940895685, 1.6616754852239213, \
    5.815864198283724, 26.17138889227676, 143.94263890752217, 935.6271528988942, \
    7017.2036467417065, 59646.230997304505, 566639.1944743928, 5949711.541981124, \
    68421682.73278293, 855271034.1597866, 11546158961.15712, 167419304936.77823, \
    2594999226520.0625
#if defined(__CUDACC__)
static __device__ const double kAsymDev[17] = {NX_ASYM_VALUES};
#endif
static const double kAsymHost[17] = {NX_ASYM_VALUES};
#undef NX_ASYM_VALUES
G3_HD double asym(int L) {
#if defined(__CUDA_ARCH__)
  return __ldg(&kAsymDev[L]);
#else
  return kAsymHost[L];
#endif
}

// Largest Hermite order of one direction: d electrons in the bra's two pairs
// and the ket (4 each) and a d proton pair (4).
constexpr int kHermMax = 16;

// t! / ((2i-t)! (t-i)! 2^(t-i)), t, i <= kHermMax (zero unless i <= t <= 2i)
#define NX_HERMX_VALUES \
    1.0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, \
    0, 1.0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, \
    0, 1.0, 1.0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, \
    0, 0, 3.0, 1.0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, \
    0, 0, 3.0, 6.0, 1.0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, \
    0, 0, 0, 15.0, 10.0, 1.0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, \
    0, 0, 0, 15.0, 45.0, 15.0, 1.0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, \
    0, 0, 0, 0, 105.0, 105.0, 21.0, 1.0, 0, 0, 0, 0, 0, 0, 0, 0, 0, \
    0, 0, 0, 0, 105.0, 420.0, 210.0, 28.0, 1.0, 0, 0, 0, 0, 0, 0, 0, 0, \
    0, 0, 0, 0, 0, 945.0, 1260.0, 378.0, 36.0, 1.0, 0, 0, 0, 0, 0, 0, 0, \
    0, 0, 0, 0, 0, 945.0, 4725.0, 3150.0, 630.0, 45.0, 1.0, 0, 0, 0, 0, 0, 0, \
    0, 0, 0, 0, 0, 0, 10395.0, 17325.0, 6930.0, 990.0, 55.0, 1.0, 0, 0, 0, 0, 0, \
    0, 0, 0, 0, 0, 0, 10395.0, 62370.0, 51975.0, 13860.0, 1485.0, 66.0, 1.0, 0, 0, 0, 0, \
    0, 0, 0, 0, 0, 0, 0, 135135.0, 270270.0, 135135.0, 25740.0, 2145.0, 78.0, 1.0, 0, 0, 0, \
    0, 0, 0, 0, 0, 0, 0, 135135.0, 945945.0, 945945.0, 315315.0, 45045.0, 3003.0, 91.0, 1.0, 0, 0, \
    0, 0, 0, 0, 0, 0, 0, 0, 2027025.0, 4729725.0, 2837835.0, 675675.0, 75075.0, 4095.0, 105.0, 1.0, 0, \
    0, 0, 0, 0, 0, 0, 0, 0, 2027025.0, 16216200.0, 18918900.0, 7567560.0, 1351350.0, 120120.0, 5460.0, 120.0, 1.0
#if defined(__CUDACC__)
static __device__ const double kHermXDev[(kHermMax + 1) * (kHermMax + 1)] = {NX_HERMX_VALUES};
#endif
static const double kHermXHost[(kHermMax + 1) * (kHermMax + 1)] = {NX_HERMX_VALUES};
#undef NX_HERMX_VALUES
G3_HD double hermx(int t, int i) {
#if defined(__CUDA_ARCH__)
  return __ldg(&kHermXDev[t * (kHermMax + 1) + i]);
#else
  return kHermXHost[t * (kHermMax + 1) + i];
#endif
}

// The factors of F_i(alpha R^2) in sum_t W[t] d^t/dR^t F_0(alpha R^2), i <= n:
//   A[i] = sum_t W[t] t! / ((2i-t)! (t-i)!) (-2 alpha R)^(2i-t) (-alpha)^(t-i)
// with y = -2 alpha R and z = -2 alpha, n <= kHermMax.  Orders up to 4 straight
// (s, p and most d pairs), beyond by Horner in y.
G3_HD void hermite_scaled(int n, const double* W, double y, double z, double* A) {
  A[0] = W[0];
  if (n == 0) return;
  if (n == 1) {
    A[1] = W[1] * y;
    return;
  }
  const double a1 = fma(W[1], y, W[2] * z);
  if (n == 2) {
    A[1] = a1;
    A[2] = W[2] * y * y;
    return;
  }
  if (n == 3) {
    const double w3 = W[3], y2 = y * y;
    A[2] = fma(W[2], y, 3.0 * (w3 * z)) * y;
    A[1] = a1;
    A[3] = w3 * y2 * y;
    return;
  }
  if (n == 4) {
    const double w3 = W[3], w4 = W[4], y2 = y * y, w4z = w4 * z;
    A[2] = fma(W[2], y2, 3.0 * (z * fma(w3, y, w4z)));
    A[1] = a1;
    A[3] = y2 * fma(w3, y, 6.0 * w4z);
    A[4] = w4 * y2 * y2;
    return;
  }
  double zp[kHermMax / 2 + 1];
  zp[0] = 1.0;
  for (int k = 1; k <= n / 2; k++) zp[k] = zp[k - 1] * z;
  double yp = 1.0;   // y^(2i - min(2i, n))
  for (int i = 1; i <= n; i++) {
    const int hi = 2 * i < n ? 2 * i : n;
    double a = W[i];
    for (int t = i + 1; t <= hi; t++) a = fma(a, y, W[t] * (hermx(t, i) * zp[t - i]));
    if (2 * i > n) {
      yp *= (2 * i == n + 1) ? y : y * y;
      a *= yp;
    }
    A[i] = a;
  }
}

// sum_m F_m(T) B[m], m <= L <= 16, with boys()'s Boys function: F_L from the
// Taylor expansion (T <= 20) or the asymptotic form, and one downward
// recursion F_m = (2T F_(m+1) + e) / (2m + 1) for both, e = exp(-T) or 0 (with
// e = 0 it is the asymptotic form's F_(m+1) = F_m (m + 1/2) / T).
G3_HD double boys_dot(int L, double T, const double* B) {
  double f, e = 0.0;
  if (bits64(T) <= 0x4034000000000000LL) {   // T <= 20 (T >= 0; NaN goes below)
    const double kMagic = 6755399441055744.0;   // 1.5 * 2^52: its sum rounds 16 T to an integer
    const double t = fma(T, 16.0, kMagic);
    int g = (int)bits64(t);
    g = g < 0 ? 0 : (g > kBoysRows - 1 ? kBoysRows - 1 : g);
    const double d = fma(t - kMagic, 0.0625, -T);
    const int row = g * kBoysCols;
    const double d2 = d * 0.5, d3 = d * (1.0 / 3.0), d4 = d * 0.25, d5 = d * 0.2,
                 d6 = d * (1.0 / 6.0);
    f = boys_tab(row + L + 6);
    f = fma(f, d6, boys_tab(row + L + 5));
    f = fma(f, d5, boys_tab(row + L + 4));
    f = fma(f, d4, boys_tab(row + L + 3));
    f = fma(f, d3, boys_tab(row + L + 2));
    f = fma(f, d2, boys_tab(row + L + 1));
    f = fma(f, d, boys_tab(row + L));
    if (L == 0) return f * B[0];
    e = 1.0 + d6;   // exp(d), the same seven terms
    e = fma(e, d5, 1.0);
    e = fma(e, d4, 1.0);
    e = fma(e, d3, 1.0);
    e = fma(e, d2, 1.0);
    e = fma(e, d, 1.0);
    e *= boys_tab(row + kBoysCols - 1);
  } else {
    const double rs = rsqrt64(T), rT = rs * rs;
    if (!(T < 1.0e15)) {   // T^-L would leave the range: upwards (and NaN)
      double s = B[L];
      for (int m = L; m >= 1; m--) s = fma(s, rT * ((double)m - 0.5), B[m - 1]);
      return (0.886226925452758 * rs) * s;
    }
    f = asym(L) * rs;
    double p = rT;
    for (int k = L; k > 0; k >>= 1) {
      if (k & 1) f *= p;
      if (k > 1) p *= p;
    }
  }
  double s = f * B[L];
  const double t2 = T + T;
  NX_LOOP
  for (int m = L - 1; m >= 0; m--) {
    f = fma(f, t2, e) * boys_rinv(m);
    s = fma(f, B[m], s);
  }
  return s;
}

// B <- B (*) A, orders L and n (B has room for L + n + 1)
G3_HD void convolve(double* B, int L, const double* A, int n) {
  NX_LOOP
  for (int m = L + n; m >= 0; m--) {
    const int lo = m > L ? m - L : 0, hi = m < n ? m : n;
    double b = A[lo] * B[m - lo];
    for (int i = lo + 1; i <= hi; i++) b = fma(A[i], B[m - i], b);
    B[m] = b;
  }
}

// A bra of build_bra_* made ready: the ket-independent part of the Coulomb
// prefactor into pref, and orderless directions' W into it as well.
template <int NW>
G3_HD void finish_bra(Bra<double, NW>& b) {
  b.pref *= 34.98683665524963 / b.Z;   // 2 pi^(5/2) of the truncated pi
  for (int d = 0; d < 3; d++)
    if (b.N[d] == 0) {
      b.pref *= b.W[d][0];
      b.W[d][0] = 1.0;
    }
}

// The free electron's pair density, from its record: Hermite coefficients
// with (-1)^t over the top one, whose product is in f (with 1/p).
template <int NK>
struct Ket {
  double p, f, X[3], e[3][NK > 0 ? NK : 1];
  int t[3];
};
template <int NK>
G3_HD void load_ket(const double* rk, Ket<NK>& k) {
  k.p = rk[kRP];
  double f = 1.0 / k.p;
  for (int d = 0; d < 3; d++) {
    const int n = (int)rk[kRT + d];
    const double* E = rk + kRE + 5 * d;
    k.X[d] = rk[kRX + d];
    k.t[d] = n;
    // E[n] = K / (2p)^n.  With K underflowing its reciprocal would overflow and
    // the coefficients lose their digits: the whole density, K times a few
    // powers of its widths, is then far below 1e-250 and is left out.
    const bool on = n == 0 || !(fabs(E[n]) < 1e-280);   // (NaN goes on)
    const double top = on ? E[n] : 0.0, r = on ? 1.0 / top : 0.0;
    f *= (n & 1) ? -top : top;
    if (NK > 0)
      for (int q = 0; q < n; q++) k.e[d][q] = ((n - q) & 1) ? -(E[q] * r) : E[q] * r;
  }
  k.f = f;
}

// One (finished bra, ket) integral.
template <int NW, int NK>
G3_HD double fb_value(const Bra<double, NW>& b, const Ket<NK>& k) {
  constexpr int NT = NW + NK;
  static_assert(NT <= kHermMax, "hermite_scaled's tables");
  const double rs = rsqrt64(b.Z + k.p), z = b.Z * k.p * (rs * rs);   // z: alpha
  double R[3], R2 = 0.0;
  for (int d = 0; d < 3; d++) {
    R[d] = b.C[d] - k.X[d];
    R2 = fma(R[d], R[d], R2);
  }
  const double T = z * R2, m2 = -(z + z);
  double B[3 * NT + 1];
  B[0] = 1.0;
  int L = 0;
  NX_LOOP
  for (int d = 0; d < 3; d++) {
    const int nb = NW > 0 ? b.N[d] : 0, tk = NK > 0 ? k.t[d] : 0, n = nb + tk;
    if (n == 0) continue;   // W = 1 after the normalisations
    double Wc[NT + 1];
    const double* W = b.W[d];
    if (tk > 0) {   // Wc[m] = W[m - tk] + sum_q e[q] W[m - q]
      for (int m = 0; m <= n; m++) {
        double w = m >= tk ? b.W[d][m - tk] : 0.0;
        for (int q = 0; q < tk; q++)
          if (m >= q && m - q <= nb) w = fma(k.e[d][q], b.W[d][m - q], w);
        Wc[m] = w;
      }
      W = Wc;
    }
    const double y = m2 * R[d];
    if (L == 0) {
      hermite_scaled(n, W, y, m2, B);
    } else {
      double A[NT + 1];
      hermite_scaled(n, W, y, m2, A);
      convolve(B, L, A, n);
    }
    L += n;
  }
  return (b.pref * k.f) * rs * boys_dot(L, T, B);
}

}  // namespace g3
}  // namespace neoxc
