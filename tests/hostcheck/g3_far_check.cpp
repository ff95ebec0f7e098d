// g3_far_check.cpp -- test helper: the integrals of the gam_2 and gam_3 builders
// with one pair density whose two primitives lie so far apart that its Gaussian
// product factor exp(-q Q^2) passes through the subnormal numbers to zero.
// A row a case: q Q^2, the two powers along the axis, then fb_value and fb_eval
// of that pair as the ket.  Exits with 1 if anything else is not finite.
#include <cstdio>

#include "../../neo-rxchf_gb300/csrc/g2_threebody.cuh"

using namespace neoxc;
using namespace neoxc::g3;
using md::Prim;

static Prim prim(int axis, int l, double a, double x, double y, double z) {
  Prim p;
  p.a = a;
  for (int d = 0; d < 3; d++) p.l[d] = d == axis ? l : 0;
  p.c[0] = x;
  p.c[1] = y;
  p.c[2] = z;
  return p;
}

template <int NW>
static void row(double qq, int la, int lb, Bra<double, NW> b, const double* rk) {
  double Ek[3][5], X[3];
  int t[3];
  for (int d = 0; d < 3; d++) {
    X[d] = rk[kRX + d];
    t[d] = (int)rk[kRT + d];
    for (int k = 0; k < 5; k++) Ek[d][k] = (k & 1) ? -rk[kRE + 5 * d + k] : rk[kRE + 5 * d + k];
  }
  const double ref = fb_eval<double, NW, 4>(b, rk[kRP], X, Ek, t);
  finish_bra<NW>(b);
  Ket<4> k;
  load_ket<4>(rk, k);
  printf("%.6g %d %d %.17g %.17g\n", qq, la, lb, fb_value<NW, 4>(b, k), ref);
}

int main() {
  const double alphas[4][2] = {{20, 20}, {10, 3000}, {0.5, 40}, {1000, 1000}};
  const double cat[6] = {0.0, 0.0, 0.0, 4.0, 1.0, 0.0}, zan[2] = {1.0, 3.0};
  int bad = 0;
  for (const auto& al : alphas)
    for (int axis = 0; axis < 2; axis++)
      for (int la = 0; la <= 2; la++)
        for (int lb = 0; lb <= 2; lb++)
          for (double qq = 660.0; qq <= 770.0; qq += 0.5) {
            const double Q = sqrt(qq * (al[0] + al[1]) / (al[0] * al[1]));
            double far[kRLen], fg[g2::kGLen], r1[kRLen], e1[g2::kGLen], rp[kRLen], ep[g2::kGLen];
            const Prim A = prim(axis, la, al[0], 0.1, 0.2, 0.0), B = prim(axis, lb, al[1], 0.1 + Q, 0.2, 0.0);
            const Prim C = prim(0, 1, 0.8, 0.0, 0.3, 0.0), D = prim(1, 2, 1.7, 0.5, 0.0, 0.4);
            const Prim P = prim(0, 1, 12.0, 0.0, 0.0, 0.0), R = prim(2, 2, 7.0, 0.0, 0.0, 0.0);
            fill_pair_record(A, B, 1.3, 0.7, far);
            g2::fill_gradient_record(A, B, fg);
            fill_pair_record(C, D, 1.0, 1.0, r1);
            g2::fill_gradient_record(C, D, e1);
            fill_pair_record(P, R, 1.0, 1.0, rp);
            g2::fill_gradient_record(P, R, ep);
            Bra<double, 12> vep, vee;
            build_bra_vep<double, 2, 2, 12>(r1, r1, rp, 0.9, 2.0, vep);
            build_bra_vee<double, 2, 2, 12>(r1, r1, rp, 0.9, 2.0, vee);
            row<12>(qq, la, lb, vep, far);
            row<12>(qq, la, lb, vee, far);
            Bra<double, 8> b;
            g2::build_bra_pair<4, 4, 8>(r1, rp, 0.9, b);
            row<8>(qq, la, lb, b, far);
            g2::build_bra_pair<4, 4, 8>(rp, r1, 0.9, b);
            row<8>(qq, la, lb, b, far);
            // the same pair in every other place
            double v[12] = {0};
            g2::three_body<2, 2, g2::kAll>(far, r1, rp, fg, e1, ep, 0.9, 2.0, 2, cat, zan, 1.0 / 1836, v, v + 1);
            g2::three_body<2, 2, g2::kCoulomb12>(r1, far, rp, e1, fg, ep, 0.9, 2.0, 2, cat, zan, 1.0 / 1836, v + 2, v + 3);
            v[4] = g2::two_body_overlap(far, rp, 0.9);
            v[5] = g2::pair_coulomb<8>(far, r1);
            v[6] = g2::schwarz_factor(far);
            g2::two_body<2, 2>(far, rp, 0.9, 2, cat, zan, v + 7, v + 8);
            Ket<4> k;
            load_ket<4>(r1, k);
            build_bra_vep<double, 2, 2, 12>(far, r1, rp, 0.9, 2.0, vep);
            build_bra_vee<double, 2, 2, 12>(r1, far, rp, 0.9, 2.0, vee);
            g2::build_bra_pair<4, 4, 8>(far, rp, 0.9, b);
            finish_bra<12>(vep);
            finish_bra<12>(vee);
            finish_bra<8>(b);
            v[9] = fb_value<12, 4>(vep, k);
            v[10] = fb_value<12, 4>(vee, k);
            v[11] = fb_value<8, 4>(b, k);
            for (double x : v) bad |= !(fabs(x) < 1e-200);
          }
  return bad;
}
