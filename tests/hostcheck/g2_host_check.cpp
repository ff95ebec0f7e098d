// g2_host_check.cpp -- test helper: the gam_2 pair-density integrals
// (csrc/g2_threebody.cuh) and the element-wise MD integrals (csrc/md_math.cuh)
// of the same primitives, both compiled as plain C++.
#include "../../neo-rxchf_gb300/csrc/md_math.cuh"
#include "../../neo-rxchf_gb300/csrc/g2_threebody.cuh"

using namespace neoxc;
using md::G3;
using md::Prim;

struct HP { int l[3]; double a; double c[3]; };

static Prim cv(const HP& h) {
  Prim p;
  p.a = h.a;
  for (int d = 0; d < 3; d++) { p.l[d] = h.l[d]; p.c[d] = h.c[d]; }
  return p;
}

static void order(const Prim* X, int a, int b, int c, Prim* Y) { Y[0] = X[a]; Y[1] = X[b]; Y[2] = X[c]; }

enum { A12 = 0, A13, A23, B12, B13, B23 };

// xcalc_GAM2_MD's terms that couple all three particles, of one (k, l)
static void item(const Prim* A, const Prim* B, double gk, double gl, int nat, const double* cat,
                 const double* zan, double pmass, double* out) {
  static thread_local G3 st;
  double g[6];
  auto gem = [&](int sa, int sb) { for (double& x : g) x = 0.0; g[sa] = gk; g[sb] = gl; };
  auto vxc = [&]() { double a = 0.0; for (int i = 0; i < nat; i++) a += zan[i] * md::g3_vxc(st, cat + 3 * i); return a; };
  Prim a[3], b[3];
  order(A, 2, 0, 1, a); order(B, 2, 0, 1, b);
  gem(A12, B13); md::g3_setup(st, a, b, g, 2);
  const double tp = md::g3_ke(st, gl, pmass), vpc = vxc();
  gem(A13, B23); md::g3_setup(st, A, B, g, 2);
  const double te1 = md::g3_ke(st, 0.0, 1.0), vec = vxc(), vee = md::g3_vee(st), s = md::g3_overlap(st);
  gem(A23, B13); md::g3_setup(st, A, B, g, 2);
  const double te2 = md::g3_ke(st, gl, 1.0);
  order(A, 0, 2, 1, a); order(B, 0, 2, 1, b);
  gem(A12, B23); md::g3_setup(st, a, b, g, 0);
  const double vep = md::g3_vee(st);
  out[0] += 0.5 * (tp + vpc + te1 + te2 - 2.0 * (vep + vec) + vee);
  out[1] += 0.5 * s;
  out[2] += 0.5 * vee;
  out[3] += fabs(tp) + fabs(vpc) + fabs(te1) + fabs(te2) + fabs(vep) + fabs(vec) + fabs(vee);
}

extern "C" {
// ref[4]: the symmetrised sums over (k, l) by the element-wise integrals
// (energy terms, overlap, 1/r12 alone) and the sum of magnitudes; got[3] the
// same by three_body.  pair[4]: composite-bra values (VEE, VEP) and theirs
// from g3_vee; ov[2]: two_body_overlap and g2_xggs.
void hc_gam2(const HP* hA, const HP* hB, int ng, const double* gm, int nat, const double* cat,
             const double* zan, double pmass, double* ref, double* got, double* pair, double* ov) {
  Prim A[3], B[3], A2[3], B2[3];
  for (int i = 0; i < 3; i++) { A[i] = cv(hA[i]); B[i] = cv(hB[i]); }
  order(A, 1, 0, 2, A2);
  order(B, 1, 0, 2, B2);
  double r[3][g3::kRLen], e[3][g2::kGLen];
  for (int i = 0; i < 3; i++) {
    g3::fill_pair_record(A[i], B[i], 1.0, 1.0, r[i]);
    g2::fill_gradient_record(A[i], B[i], e[i]);
  }
  for (int i = 0; i < 4; i++) ref[i] = 0.0;
  for (int i = 0; i < 3; i++) got[i] = 0.0;
  for (int k = 0; k < ng; k++)
    for (int l = 0; l < ng; l++) {
      item(A, B, gm[k], gm[l], nat, cat, zan, pmass, ref);
      item(A2, B2, gm[k], gm[l], nat, cat, zan, pmass, ref);
      double x, y;
      g2::three_body<2, 2, g2::kAll>(r[0], r[1], r[2], e[0], e[1], e[2], gm[k], gm[l], nat, cat, zan,
                                 1.0 / pmass, &x, &y);
      got[0] += x;
      got[1] += y;
      double z;
      g2::three_body<2, 2, g2::kOverlap>(r[0], r[1], r[2], e[0], e[1], e[2], gm[k], gm[l], nat, cat,
                                         zan, 1.0 / pmass, &x, &z);
      if (!(fabs(z - y) <= 1e-12 * fabs(y))) got[1] = NAN;   // one overlap, two ways
      g2::three_body<2, 2, g2::kCoulomb12>(r[0], r[1], r[2], e[0], e[1], e[2], gm[k], gm[l], nat, cat, zan,
                                  1.0 / pmass, &x, &y);
      got[2] += y;
    }
  static thread_local G3 st;
  const double gm6[6] = {0.0, 0.0, gm[0], 0.0, 0.0, 0.0};
  g3::Bra<double, 8> b;
  g3::Ket<4> ket;
  g3::load_ket<4>(r[0], ket);
  g2::build_bra_pair<4, 4, 8>(r[1], r[2], gm[0], b);
  g3::finish_bra<8>(b);
  pair[0] = g3::fb_value<8, 4>(b, ket);
  g2::build_bra_pair<4, 4, 8>(r[2], r[1], gm[0], b);
  g3::finish_bra<8>(b);
  pair[1] = g3::fb_value<8, 4>(b, ket);
  md::g3_setup(st, A, B, gm6, 0);
  pair[2] = md::g3_vee(st);
  Prim A3[3], B3[3];
  order(A, 0, 2, 1, A3);
  order(B, 0, 2, 1, B3);
  md::g3_setup(st, A3, B3, gm6, 0);
  pair[3] = md::g3_vee(st);
  ov[0] = g2::two_body_overlap(r[0], r[2], gm[0]);
  ov[1] = md::g2_xggs(A[0], A[2], B[0], B[2], gm[0], 0.0);
}

double hc_boys_dot(int L, double T, const double* B) { return g3::boys_dot(L, T, B); }
double hc_boys_ref(int L, double T, const double* B) {
  double F[32], s = 0.0;
  boys(L, T, F);
  for (int m = 0; m <= L; m++) s += F[m] * B[m];
  return s;
}

// got/ref pairs of one (electron, proton) pair: pair_kinetic, the
// multiplicative terms and the overlap of two_body, pair_coulomb; mag: the
// size of the multiplicative terms.
void hc_gam1(const HP* hA, const HP* hB, double gk, double gl, int nat, const double* cat,
             const double* zan, double m, double* got, double* ref, double* mag) {
  Prim A[2], B[2];
  for (int i = 0; i < 2; i++) { A[i] = cv(hA[i]); B[i] = cv(hB[i]); }
  double r[2][g3::kRLen];
  for (int i = 0; i < 2; i++) g3::fill_pair_record(A[i], B[i], 1.0, 1.0, r[i]);
  got[0] = g2::pair_kinetic(A[0], A[1], B[0], B[1], gk, gl, m);
  ref[0] = md::pgike1(A[0], A[1], B[0], B[1], gk, gl, m);
  g2::two_body<2, 2>(r[0], r[1], gk + gl, nat, cat, zan, &got[1], &got[2]);
  double ve = 0.0, vp = 0.0, me = 0.0;
  for (int c = 0; c < nat; c++) {
    const double x = zan[c] * md::g2_xggvec(A[0], A[1], B[0], B[1], gk, gl, cat + 3 * c);
    const double y = zan[c] * md::g2_xggvec(A[1], A[0], B[1], B[0], gk, gl, cat + 3 * c);
    ve += x; vp += y; me += fabs(x) + fabs(y);
  }
  const double vm = md::g2_xggvee(A[0], A[1], B[0], B[1], gk, gl);
  ref[1] = vp - ve - vm;
  *mag = me + fabs(vm);
  ref[2] = md::g2_xggs(A[0], A[1], B[0], B[1], gk, gl);
  got[3] = g2::pair_coulomb<8>(r[0], r[1]);
  ref[3] = md::gfvee(A[0], A[1], B[0], B[1]);
}
}
