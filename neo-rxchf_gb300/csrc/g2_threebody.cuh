// g2_threebody.cuh -- the gam_2 primitive integrals over pair densities
// (gam_2_OMP.f:546-1077 xcalc_GAM2_MD, rxchfne_gam_2_OMP.f:2-530), used by the
// gam_2 builder (k_gam2.cu, whose header comment gives the decomposition).
// Every function is __host__ __device__ so that it can be compiled as plain
// C++ and compared with the element-wise md_math.cuh integrals.  All FP64.
//
// Three pair densities rho_1, rho_2 (electrons) and rho_p (proton), each a
// sum of Hermite Gaussians of exponent P_i at centre c_i, coupled by
// exp(-gk r_1p^2 - gl r_2p^2).  With M the 3x3 matrix of the total quadratic
// form, N = diag(P) and G = M^-1:
//   * the s-type overlap is (pi^3/det M)^(3/2) exp(-sum_{i<j} k_ij (c_i-c_j)^2),
//     k_ij = P_i G_ij P_j; Hermite functions differentiate it by the centres;
//   * along a unit combination q.r (q = e1-e2, e1-p, e2-p, e1, e2, p) the
//     Gaussian has the mean q.GN c and the exponent alpha = 1/(q.G q), so
//     1/|q.r - C| integrates to 2 sqrt(alpha/pi) F_0(alpha |q.GN c - C|^2)
//     times the overlap, differentiated by the centres as well.
// Every entry of adj(M), the determinant and the q.adj(M) q below are sums of
// positive terms, so no digits cancel.
//   Per Cartesian direction, with D(s) the derivatives of the Gaussian:
//   V(x) = sum_s D(s) prod_i E_i[s_i + x_i] C(s_i + x_i, x_i) does not depend
//   on the operator; the operator's Hermite vector is
//   W[n] = sum_{|x| = n} prod_i b_i^x_i V(x), b = q.GN.
//   Kinetic energy, by partial integration over a particle's own density:
//   <f w|T|f'> + <T f|w|f'> = sum_d int w (f_d f'_d - rho_dd / 2) for a
//   multiplicative w (electrons), and the proton's <f gk|T|f' gl> averaged
//   over the exchange of the two electrons (which the gam_2 symmetrisation
//   does) is sum_d int [f_d f'_d / 2 - (d_c1^2 + d_c2^2) / 4] -- so all of
//   them are sums over the same D with one density's Hermite vector replaced.
#pragma once
#include "g3_fatbra.cuh"

namespace neoxc {
namespace g2 {

using g3::fold_line;
using g3::kRC;
using g3::kRE;
using g3::kRLen;
using g3::kRP;
using g3::kRT;
using g3::kRX;
using g3::rsqrt64;

// gradient record of a pair: EG[d][t], t <= 6, the Hermite coefficients of
// (d phi_a / dx_d)(d phi_b / dx_d) in direction d
constexpr int kGLen = 24, kGRow = 7;

G3_HD void fill_gradient_record(const md::Prim& A, const md::Prim& B, double* out) {
  md::Pair pr;
  md::gauss_pair(A, B, pr);
  for (int d = 0; d < 3; d++) {
    double e[kGRow];
    for (int t = 0; t < kGRow; t++) e[t] = 0.0;
    const int la = A.l[d], lb = B.l[d];
    for (int u = 0; u < 2; u++)
      for (int v = 0; v < 2; v++) {
        const int i = u ? la + 1 : la - 1, j = v ? lb + 1 : lb - 1;
        if (i < 0 || j < 0) continue;
        const double f = (u ? -2.0 * A.a : (double)la) * (v ? -2.0 * B.a : (double)lb);
        double tmp[2 * md::TMX + 1];
        md::hermite_e(i, j, pr.K[d], A.a, B.a, pr.p, pr.q, pr.Q[d], tmp);
        for (int t = 0; t <= i + j; t++) e[t] += f * tmp[t];
      }
    for (int t = 0; t < kGRow; t++) out[kGRow * d + t] = e[t];
  }
  for (int t = 3 * kGRow; t < kGLen; t++) out[t] = 0.0;
}

// sum_m F_m(T) sum_{i+j+k=m} A_x[i] A_y[j] A_z[k], T = alpha |R|^2
template <int NT>
G3_HD double coulomb_sum(const int* n, const double (*W)[NT + 1], const double* R, double T,
                         double alpha) {
  static_assert(NT <= g3::kHermMax, "hermite_scaled's tables");
  const double z = -(alpha + alpha);
  double B[3 * NT + 1], A[NT + 1];
  g3::hermite_scaled(n[0], W[0], z * R[0], z, B);
  NX_LOOP
  for (int d = 1; d < 3; d++) {
    g3::hermite_scaled(n[d], W[d], z * R[d], z, A);
    g3::convolve(B, d == 1 ? n[0] : n[0] + n[1], A, n[d]);
  }
  return g3::boys_dot(n[0] + n[1] + n[2], T, B);
}

// What three_body evaluates: everything of the symmetrised gam_2 integrand
// that couples all three particles, 1/r_12 alone, or the overlap alone.
enum TripleMode { kAll = 0, kCoulomb12 = 1, kOverlap = 2 };

// One primitive triple and geminal pair.  kAll: *x1 = the Coulomb, nuclear
// and kinetic terms of the symmetrised gam_2 integrand that couple all three
// particles, <gk(1p) gl(2p)| 1/r_12 - 1/r_1p - 1/r_2p + sum_C Z (1/r_pC -
// 1/r_1C - 1/r_2C) + T_p + (T_1 + T_2)/2 as above |>, *x2 = the overlap;
// kCoulomb12: *x2 = the 1/r_12 term (the RXCHF-ne exchange tensor);
// kOverlap: *x2 = the overlap.
template <int LE, int LN, int MODE>
G3_HD void three_body(const double* r1, const double* r2, const double* rp, const double* e1,
                      const double* e2, const double* ep, double gk, double gl, int nat,
                      const double* cat, const double* zan, double rpmass, double* x1,
                      double* x2) {
  constexpr bool FULL = MODE == kAll;
  constexpr int M1 = 2 * LE, M3 = 2 * LN;         // largest Hermite orders of a pair
  constexpr int K = FULL ? 2 : 0;                 // kinetic extension of D
  constexpr int S2 = M3 + K + 1, S1 = (M1 + K + 1) * S2;   // strides of D
  constexpr int NT = 2 * M1 + M3;                 // Coulomb order per direction
  constexpr int NV = (M1 + 1) * (M1 + 1) * (M3 + 1);
  const double P1 = r1[kRP], P2 = r2[kRP], P3 = rp[kRP];
  const double s3 = P3 + gk + gl, A1 = P1 + gk, A2 = P2 + gl;
  const double u1 = fma(P2, s3, gl * P3), u2 = fma(P1, s3, gk * P3);   // adj11 - adj12, adj22 - adj12
  const double g12 = gk * gl;
  const double a11 = u1 + g12, a22 = u2 + g12, a33 = A1 * A2, a13 = gk * A2, a23 = gl * A1;
  const double det = fma(P1, a11, gk * fma(P2, P3 + gl, gl * P3));
  const double rsd = rsqrt64(det), rdet = rsd * rsd;
  const double k12 = P1 * P2 * g12 * rdet, k13 = P1 * P3 * a13 * rdet, k23 = P2 * P3 * a23 * rdet;
  double c13[3], c23[3], c3[3], ex = 0.0;
  for (int d = 0; d < 3; d++) {
    c3[d] = rp[kRX + d];
    c13[d] = r1[kRX + d] - c3[d];
    c23[d] = r2[kRX + d] - c3[d];
    const double c12 = c13[d] - c23[d];
    ex = fma(k12 * c12, c12, fma(k13 * c13[d], c13[d], fma(k23 * c23[d], c23[d], ex)));
  }
  const double base = exp(-ex);
  int T1[3], T2[3], T3[3], n[3];
  double V[3][NV];
  double kin1[3], kin2[3], kin3[3];
  {
    const double h12 = -2.0 * k12, h13 = -2.0 * k13, h23 = -2.0 * k23;
    const double h11 = -(h12 + h13), h22 = -(h12 + h23), h33 = -(h13 + h23);
    double D[(M1 + K + 1) * S1];
    NX_LOOP
    for (int d = 0; d < 3; d++) {
      const int t1 = (int)r1[kRT + d], t2 = (int)r2[kRT + d], t3 = (int)rp[kRT + d];
      T1[d] = t1;
      T2[d] = t2;
      T3[d] = t3;
      n[d] = t1 + t2 + t3;
      const double c12 = c13[d] - c23[d];
      const double g1 = fma(h12, c12, h13 * c13[d]), g2 = fma(h23, c23[d], -h12 * c12);
      const double g3 = -(g1 + g2);   // = -dQ/dc_i: the gradients enter with this sign
      // D[s1][s2][s3]: the box (t1,t2,t3) and, for the kinetic terms, two
      // more orders along each axis (not along two at once)
      NX_LOOP
      for (int a = 0; a <= t1 + K; a++) {
        const int bm = a <= t1 ? t2 + K : t2;
        NX_LOOP
        for (int b = 0; b <= bm; b++) {
          const int cm = (a <= t1 && b <= t2) ? t3 + K : t3;
          NX_LOOP
          for (int c = 0; c <= cm; c++) {
            const int o = a * S1 + b * S2 + c;
            double v;
            if (a > 0) {
              v = g1 * D[o - S1];
              if (a > 1) v = fma(-h11 * (double)(a - 1), D[o - 2 * S1], v);
              if (b > 0) v = fma(-h12 * (double)b, D[o - S1 - S2], v);
              if (c > 0) v = fma(-h13 * (double)c, D[o - S1 - 1], v);
            } else if (b > 0) {
              v = g2 * D[o - S2];
              if (b > 1) v = fma(-h22 * (double)(b - 1), D[o - 2 * S2], v);
              if (c > 0) v = fma(-h23 * (double)c, D[o - S2 - 1], v);
            } else if (c > 0) {
              v = g3 * D[o - 1];
              if (c > 1) v = fma(-h33 * (double)(c - 1), D[o - 2], v);
            } else {
              v = d == 0 ? base : 1.0;
            }
            D[o] = v;
          }
        }
      }
      const double* E1 = r1 + kRE + 5 * d;
      const double* E2 = r2 + kRE + 5 * d;
      const double* E3 = rp + kRE + 5 * d;
      if constexpr (FULL) {
        const double* G1 = e1 + kGRow * d;
        const double* G2 = e2 + kGRow * d;
        const double* G3 = ep + kGRow * d;
        // Y(s): two densities contracted, the third's order left open
        double q1 = 0.0, q2 = 0.0, q3 = 0.0, d1 = 0.0, d2 = 0.0;
        NX_LOOP
        for (int a = 0; a <= t1 + 2; a++) {
          double y = 0.0;
          for (int b = 0; b <= t2; b++) {
            double z = D[a * S1 + b * S2] * E3[0];
            for (int c = 1; c <= t3; c++) z = fma(D[a * S1 + b * S2 + c], E3[c], z);
            y = fma(z, E2[b], y);
          }
          q1 = fma(y, G1[a], q1);
          if (a >= 2) d1 = fma(y, E1[a - 2], d1);
        }
        NX_LOOP
        for (int b = 0; b <= t2 + 2; b++) {
          double y = 0.0;
          for (int a = 0; a <= t1; a++) {
            double z = D[a * S1 + b * S2] * E3[0];
            for (int c = 1; c <= t3; c++) z = fma(D[a * S1 + b * S2 + c], E3[c], z);
            y = fma(z, E1[a], y);
          }
          q2 = fma(y, G2[b], q2);
          if (b >= 2) d2 = fma(y, E2[b - 2], d2);
        }
        NX_LOOP
        for (int c = 0; c <= t3 + 2; c++) {
          double y = 0.0;
          for (int a = 0; a <= t1; a++) {
            double z = D[a * S1 + c] * E2[0];
            for (int b = 1; b <= t2; b++) z = fma(D[a * S1 + b * S2 + c], E2[b], z);
            y = fma(z, E1[a], y);
          }
          q3 = fma(y, G3[c], q3);
        }
        kin1[d] = fma(-0.5, d1, q1);
        kin2[d] = fma(-0.5, d2, q2);
        kin3[d] = fma(0.5, q3, -0.25 * (d1 + d2));
      }
      if constexpr (MODE == kOverlap) {
        double x = 0.0;
        for (int a = 0; a <= t1; a++) {
          double y = 0.0;
          for (int b = 0; b <= t2; b++) {
            double z = D[a * S1 + b * S2] * E3[0];
            for (int c = 1; c <= t3; c++) z = fma(D[a * S1 + b * S2 + c], E3[c], z);
            y = fma(z, E2[b], y);
          }
          x = fma(y, E1[a], x);
        }
        V[d][0] = x;
        continue;
      }
      // V(x1,x2,x3), compact strides, one axis at a time in place
      double* v = V[d];
      const int w2 = t3 + 1, w1 = (t2 + 1) * w2;
      for (int a = 0; a <= t1; a++)
        for (int b = 0; b <= t2; b++) {
          for (int c = 0; c <= t3; c++) v[a * w1 + b * w2 + c] = D[a * S1 + b * S2 + c];
          fold_line(v + a * w1 + b * w2, 1, t3, E3);
        }
      for (int a = 0; a <= t1; a++)
        for (int c = 0; c <= t3; c++) fold_line(v + a * w1 + c, w2, t2, E2);
      for (int b = 0; b < w1; b++) fold_line(v + b, w1, t1, E1);
    }
  }
  const double kPi = 3.14159265358979e+00;   // the MD kernels' truncated pi
  if constexpr (MODE == kOverlap) {
    *x1 = 0.0;
    *x2 = (kPi * kPi * kPi * kPi) * sqrt(kPi) * (rdet * rsd) * (V[0][0] * V[1][0] * V[2][0]);
    return;
  }
  double acc = 0.0;
  // the operators: 1/r_12, then (FULL) 1/r_1p, 1/r_2p and the nuclear
  // attraction of 1, 2 and p
  NX_LOOP
  for (int op = 0; op < (FULL ? 6 : 1); op++) {
    double v, b1, b2, b3;   // q.adj(M) q and q.adj(M) N (times rdet below)
    switch (op) {
      case 0:
        v = fma(P1 + P2, s3, P3 * (gk + gl));
        b1 = u1 * P1; b2 = -u2 * P2; b3 = (gk * P2 - gl * P1) * P3;
        break;
      case 1:
        v = fma(P2, P3 + gl, fma(gl, P3, P1 * A2));
        b1 = fma(P2, P3 + gl, gl * P3) * P1; b2 = -gl * P1 * P2; b3 = -P1 * A2 * P3;
        break;
      case 2:
        v = fma(P1, P3 + gk, fma(gk, P3, P2 * A1));
        b1 = -gk * P1 * P2; b2 = fma(P1, P3 + gk, gk * P3) * P2; b3 = -P2 * A1 * P3;
        break;
      case 3: v = a11; b1 = a11 * P1; b2 = g12 * P2; b3 = a13 * P3; break;
      case 4: v = a22; b1 = g12 * P1; b2 = a22 * P2; b3 = a23 * P3; break;
      default: v = a33; b1 = a13 * P1; b2 = a23 * P2; b3 = a33 * P3; break;
    }
    b1 *= rdet;
    b2 *= rdet;
    b3 *= rdet;
    const double rv = rsqrt64(v), alpha = det * rv * rv;
    // W per direction
    double W[3][NT + 1], R0[3];
    NX_LOOP
    for (int d = 0; d < 3; d++) {
      const int t1 = T1[d], t2 = T2[d], t3 = T3[d];
      R0[d] = fma(b1, c13[d], b2 * c23[d]);
      const double* vv = V[d];
      if (n[d] == 0) {
        W[d][0] = vv[0];
        continue;
      }
      for (int k = 0; k <= n[d]; k++) W[d][k] = 0.0;
      double p1 = 1.0;
      for (int x1i = 0; x1i <= t1; x1i++) {
        double p12 = p1;
        for (int x2i = 0; x2i <= t2; x2i++) {
          double p = p12;
          for (int x3i = 0; x3i <= t3; x3i++) {
            W[d][x1i + x2i + x3i] = fma(p, *vv++, W[d][x1i + x2i + x3i]);
            if (x3i < t3) p *= b3;
          }
          if (x2i < t2) p12 *= b2;
        }
        if (x1i < t1) p1 *= b1;
      }
    }
    const int nc = op < 3 ? 1 : nat;
    double sum = 0.0;
    NX_LOOP
    for (int c = 0; c < nc; c++) {
      double R[3], R2 = 0.0;
      for (int d = 0; d < 3; d++) {
        R[d] = op < 3 ? R0[d] : (R0[d] + c3[d]) - cat[3 * c + d];
        R2 = fma(R[d], R[d], R2);
      }
      const double x = coulomb_sum<NT>(n, W, R, alpha * R2, alpha);
      sum = op < 3 ? x : fma(zan[c], x, sum);
    }
    acc = (op == 0 || op == 5) ? fma(sum, rv, acc) : fma(-sum, rv, acc);
  }
  const double f = (2.0 * kPi * kPi * kPi * kPi) * rdet;   // 2 pi^4 / det (x rv)
  if constexpr (FULL) {
    const double so = (kPi * kPi * kPi * kPi) * sqrt(kPi) * (rdet * rsd);   // pi^(9/2) / det^(3/2)
    const double sxy = V[0][0] * V[1][0], syz = V[1][0] * V[2][0], sxz = V[0][0] * V[2][0];
    double kin = 0.0;
    for (int d = 0; d < 3; d++) {
      const double k = fma(0.5, kin1[d] + kin2[d], kin3[d] * rpmass);
      kin = fma(k, d == 0 ? syz : (d == 1 ? sxz : sxy), kin);
    }
    *x1 = fma(f, acc, so * kin);
    *x2 = so * (sxy * V[2][0]);
  } else {
    *x1 = 0.0;
    *x2 = f * acc;
  }
}

// S-type overlap factor and Hermite overlap of two pair densities coupled by
// exp(-g r^2) (G2_MD_xggs, XC1_G2_MD.f:3-187), without contraction coefficients.
G3_HD double two_body_overlap(const double* r1, const double* rp, double g) {
  const double kPi = 3.14159265358979e+00;
  const double P1 = r1[kRP], P3 = rp[kRP];
  const double rs = rsqrt64(fma(P1, P3, g * (P1 + P3))), rd = rs * rs;
  const double q = P1 * P3 * g * rd;
  double res = 1.0, ex = 0.0;
  NX_LOOP
  for (int d = 0; d < 3; d++) {
    const int t1 = (int)r1[kRT + d], t3 = (int)rp[kRT + d];
    const double u = r1[kRX + d] - rp[kRX + d];
    ex = fma(q * u, u, ex);
    double gd[9];   // derivatives of exp(-q u^2) over exp(-q u^2)
    gd[0] = 1.0;
    for (int k = 1; k <= t1 + t3; k++)
      gd[k] = -2.0 * q * (k > 1 ? fma(u, gd[k - 1], (double)(k - 1) * gd[k - 2]) : u * gd[0]);
    double acc = 0.0;
    for (int a = 0; a <= t1; a++) {
      double y = 0.0;
      for (int c = 0; c <= t3; c++) y = fma((c & 1) ? -gd[a + c] : gd[a + c], rp[kRE + 5 * d + c], y);
      acc = fma(y, r1[kRE + 5 * d + a], acc);
    }
    res *= acc;
  }
  return (kPi * kPi * kPi) * (rd * rs) * exp(-ex) * res;
}

// (r | s): Coulomb integral of two pair densities (gfvee, vee.f:3-78; gam_ep).
template <int NT>
G3_HD double pair_coulomb(const double* r, const double* s) {
  const double kPi = 3.14159265358979323846;
  const double p = r[kRP], q = s[kRP], rs = rsqrt64(p + q), pq = p * q, alpha = pq * (rs * rs);
  double W[3][NT + 1], R[3], R2 = 0.0;
  int n[3];
  for (int d = 0; d < 3; d++) {
    const int t = (int)r[kRT + d], u = (int)s[kRT + d];
    const double* E = r + kRE + 5 * d;
    const double* F = s + kRE + 5 * d;
    n[d] = t + u;
    for (int k = 0; k <= n[d]; k++) W[d][k] = 0.0;
    for (int b = 0; b <= u; b++) {
      const double f = (b & 1) ? -F[b] : F[b];
      for (int a = 0; a <= t; a++) W[d][a + b] = fma(E[a], f, W[d][a + b]);
    }
    R[d] = r[kRX + d] - s[kRX + d];
    R2 = fma(R[d], R[d], R2);
  }
  return (2.0 * kPi * kPi * sqrt(kPi)) * rs / pq * coulomb_sum<NT>(n, W, R, alpha * R2, alpha);
}

// |c_a c_b| sqrt((ab|ab)) of a pair record.  (As an integral over four
// primitives this was the longest chain of g3_records_kernel: examples/xchf,
// 86 us, and nebf = 4 s/p, 128 us; 63 on average from the record.)
G3_HD double schwarz_factor(const double* r) {
  return fabs(r[kRC]) * sqrt(fabs(pair_coulomb<8>(r, r)));
}

// The multiplicative terms of xcalc_GAM1_MD's integrand (gam_1_OMP.f:398-836)
// for an electron and a proton pair density coupled by exp(-g r^2):
// *e = -Z/r_eC + Z/r_pC - 1/r_ep, *ov = the overlap.
template <int LE, int LN>
G3_HD void two_body(const double* r1, const double* rp, double g, int nat, const double* cat,
                    const double* zan, double* e, double* ov) {
  constexpr int M1 = 2 * LE, M3 = 2 * LN, NT = M1 + M3;
  const double kPi = 3.14159265358979e+00;
  const double P1 = r1[kRP], P3 = rp[kRP], a11 = P3 + g, a33 = P1 + g;
  const double det = fma(P1, P3, g * (P1 + P3));
  const double rs = rsqrt64(det), rd = rs * rs, K = P1 * P3 * g * rd;
  double V[3][(M1 + 1) * (M3 + 1)], u[3], ex = 0.0;
  int T1[3], T3[3], n[3];
  NX_LOOP
  for (int d = 0; d < 3; d++) {
    const int t1 = (int)r1[kRT + d], t3 = (int)rp[kRT + d];
    T1[d] = t1;
    T3[d] = t3;
    n[d] = t1 + t3;
    u[d] = r1[kRX + d] - rp[kRX + d];
    ex = fma(K * u[d], u[d], ex);
    double gd[NT + 1];
    gd[0] = 1.0;
    const double h = -2.0 * K;
    for (int k = 1; k <= n[d]; k++)
      gd[k] = h * (k > 1 ? fma(u[d], gd[k - 1], (double)(k - 1) * gd[k - 2]) : u[d] * gd[0]);
    const int w = t3 + 1;
    for (int i = 0; i <= t1; i++) {
      for (int c = 0; c <= t3; c++) V[d][i * w + c] = (c & 1) ? -gd[i + c] : gd[i + c];
      fold_line(V[d] + i * w, 1, t3, rp + kRE + 5 * d);
    }
    for (int c = 0; c <= t3; c++) fold_line(V[d] + c, w, t1, r1 + kRE + 5 * d);
  }
  const double base = exp(-ex);
  double acc = 0.0;
  NX_LOOP
  for (int op = 0; op < 3; op++) {   // 1/r_ep, 1/r_eC, 1/r_pC
    const double v = op == 0 ? P1 + P3 : (op == 1 ? a11 : a33);
    const double b1 = (op == 0 ? P3 * P1 : (op == 1 ? a11 * P1 : g * P1)) * rd;
    const double b3 = op == 0 ? -b1 : (op == 1 ? g * P3 : a33 * P3) * rd;
    const double rv = rsqrt64(v), alpha = det * rv * rv;
    double W[3][NT + 1];
    NX_LOOP
    for (int d = 0; d < 3; d++) {
      for (int k = 0; k <= n[d]; k++) W[d][k] = 0.0;
      const double* vv = V[d];
      double p1 = 1.0;
      for (int i = 0; i <= T1[d]; i++) {
        double p = p1;
        for (int c = 0; c <= T3[d]; c++) {
          W[d][i + c] = fma(p, *vv++, W[d][i + c]);
          p *= b3;
        }
        p1 *= b1;
      }
    }
    const int nc = op == 0 ? 1 : nat;
    double sum = 0.0;
    NX_LOOP
    for (int c = 0; c < nc; c++) {
      double R[3], R2 = 0.0;
      for (int d = 0; d < 3; d++) {
        R[d] = b1 * u[d];   // the mean of e or p lies at c_p + b1 u
        if (op > 0) R[d] = (R[d] + rp[kRX + d]) - cat[3 * c + d];
        R2 = fma(R[d], R[d], R2);
      }
      const double x = coulomb_sum<NT>(n, W, R, alpha * R2, alpha);
      sum = op == 0 ? x : fma(zan[c], x, sum);
    }
    acc = op == 2 ? fma(sum, rv, acc) : fma(-sum, rv, acc);
  }
  *e = 2.0 * kPi * kPi * sqrt(kPi) * rd * base * acc;
  *ov = (kPi * kPi * kPi) * (rd * rs) * base * (V[0][0] * V[1][0] * V[2][0]);
}

// pgike1 (g2.f:545-651): kinetic energy of particle 1 with geminal exponents
// gA (bra) and gB (ket), by the formulas of md::pgike1 operation by operation
// (the kinetic terms of a nearly dependent basis cancel to the last digits of
// the reference's logged energies, so its rounding is kept), with the Hermite
// vectors, the Gaussian derivatives and the exponentials shared by the ten
// 1-D overlaps of a direction instead of rebuilt for each.
G3_HD double pair_kinetic(const md::Prim& A1, const md::Prim& A2, const md::Prim& B1,
                          const md::Prim& B2, double gA, double gB, double xmass) {
  constexpr int N = 2 * md::LP + 3;   // Hermite entries with the ket raised by two
  const double g = gA + gB, PI = 3.141592650;   // pgi_hint0_1D's pi (g2.f:200-234)
  double S[3], T[3];
  NX_LOOP
  for (int d = 0; d < 3; d++) {
    const double a1 = A1.a, a2 = A2.a, b1 = B1.a, b2 = B2.a;
    const double X1 = A1.c[d], X2 = A2.c[d], Y1 = B1.c[d], Y2 = B2.c[d];
    const int I1 = A1.l[d], I2 = A2.l[d], L1 = B1.l[d], L2 = B2.l[d];
    const double p1 = a1 + b1, q1 = (a1 * b1) / (a1 + b1), Q1 = X1 - Y1;
    const double p2 = a2 + b2, q2 = (a2 * b2) / (a2 + b2), Q2 = X2 - Y2;
    const double Pm1 = (a1 * X1 + b1 * Y1) / (a1 + b1);
    const double Pm2 = (a2 * X2 + b2 * Y2) / (a2 + b2);
    const double K1 = exp(-q1 * Q1 * Q1), K2 = exp(-q2 * Q2 * Q2);
    const double s = (p1 * p2) + (p1 * g) + (p2 * g);
    const double q = (p1 * p2 * g) / s, pre = sqrt(PI * PI / s);
    double E1[5][2 * md::TMX + 1], E2[3][2 * md::TMX + 1], gd[2 * N + 1];
    md::gauss_derivs(I1 + L1 + I2 + L2 + 4, q, Pm1 - Pm2, gd);
    NX_LOOP
    for (int k = 0; k < 5; k++)   // ket L1 - 2 .. L1 + 2
      if (L1 + k - 2 >= 0) md::hermite_e(I1, L1 + k - 2, K1, a1, b1, p1, q1, Q1, E1[k]);
    NX_LOOP
    for (int k = 0; k < 3; k++) md::hermite_e(I2, L2 + k, K2, a2, b2, p2, q2, Q2, E2[k]);
    auto ov = [&](int k, int m) {
      double acc = 0.0;
      for (int t1 = 0; t1 <= I1 + L1 + k - 2; t1++)
        for (int t2 = 0; t2 <= I2 + L2 + m; t2++)
          acc += E1[k][t1] * E2[m][t2] * (((t2 & 1) ? -1.0 : 1.0) * pre * gd[t1 + t2]);
      return acc;
    };
    const double X12 = Y1 - Y2;
    const double o00 = ov(2, 0), o01 = ov(2, 1), o02 = ov(2, 2), o10 = ov(3, 0), o11 = ov(3, 1),
                 o20 = ov(4, 0);
    const double om0 = L1 >= 1 ? ov(1, 0) : 0.0, om1 = L1 >= 1 ? ov(1, 1) : 0.0;
    const double omm = L1 >= 2 ? ov(0, 0) : 0.0;
    const double d1 = (double)(L1 * (L1 - 1)), d2 = -2.0 * b1 * (double)((2 * L1) + 1);
    const double d3 = 4.0 * b1 * b1, c1 = (double)L1, c2 = -2.0 * b1;
    const double W1 = (d1 * omm) + (d2 * o00) + (d3 * o20);
    const double z1 = L1 >= 1 ? o00 - om1 + (X12 * om0) : 0.0;
    const double z2 = o20 - o11 + (X12 * o10);
    const double W2 = -2.0 * gB * ((c1 * z1) + (c2 * z2));
    const double t2 = o20 + o02 + (X12 * X12 * o00) - (2.0 * o11) - (2.0 * X12 * o01) + (2.0 * X12 * o10);
    const double W3 = (-2.0 * gB * o00) + (4.0 * gB * gB * t2);
    S[d] = o00;
    T[d] = -(W1 + (2.0 * W2) + W3) * 0.50 / xmass;
  }
  return (T[0] * S[1] * S[2]) + (S[0] * T[1] * S[2]) + (S[0] * S[1] * T[2]);
}

// Composite bra of pair densities A (kept) and B (integrated out with the
// geminal exp(-g r_AB^2)): the charge density of A's particle dressed by B.
template <int MA, int MB, int NW>
G3_HD void build_bra_pair(const double* ra, const double* rb, double g, g3::Bra<double, NW>& b) {
  const double kPi = 3.14159265358979e+00;
  const double PA = ra[kRP], PB = rb[kRP];
  const double x = PB + g, rx = 1.0 / x;
  const double C2 = PB * g * rx, Z = PA + C2, rZ = 1.0 / Z;
  const double bA = PA * rZ, bB = C2 * rZ, xi = PA * C2 * rZ;
  double ex = 0.0;
  NX_LOOP
  for (int d = 0; d < 3; d++) {
    const int ta = (int)ra[kRT + d], tb = (int)rb[kRT + d], n = ta + tb;
    const double u = ra[kRX + d] - rb[kRX + d];
    ex = fma(xi * u, u, ex);
    double gd[MA + MB + 1];
    gd[0] = 1.0;
    for (int k = 1; k <= n; k++)
      gd[k] = -2.0 * xi * (k > 1 ? fma(u, gd[k - 1], (double)(k - 1) * gd[k - 2]) : u * gd[0]);
    double V[(MA + 1) * (MB + 1)];
    for (int s = 0; s <= ta; s++) {
      for (int t = 0; t <= tb; t++) V[s * (tb + 1) + t] = (t & 1) ? -gd[s + t] : gd[s + t];
      fold_line(V + s * (tb + 1), 1, tb, rb + kRE + 5 * d);
    }
    for (int t = 0; t <= tb; t++) fold_line(V + t, tb + 1, ta, ra + kRE + 5 * d);
    for (int k = 0; k <= n; k++) b.W[d][k] = 0.0;
    double pa = 1.0;
    for (int s = 0; s <= ta; s++) {
      double p = pa;
      for (int t = 0; t <= tb; t++) {
        b.W[d][s + t] = fma(p, V[s * (tb + 1) + t], b.W[d][s + t]);
        p *= bB;
      }
      pa *= bA;
    }
    b.N[d] = n;
    b.C[d] = fma(bA, ra[kRX + d], bB * rb[kRX + d]);
  }
  b.Z = Z;
  const double px = kPi * rx;
  b.pref = px * sqrt(px) * exp(-ex);
}

}  // namespace g2
}  // namespace neoxc
