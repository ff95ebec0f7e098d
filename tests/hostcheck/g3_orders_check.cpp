// g3_orders_check.cpp -- test helper: the FP64 (bra, ket) integral of the gam_3
// and gam_2 builders (csrc/g3_fatbra.cuh, fb_value) compiled as plain C++ with
// the address and bounds checkers, at every Hermite order a direction can have.
// A row a case: order, fb_value, the same sum in long double, and the sum of
// its terms' magnitudes.
#include <cstdio>
#include <random>

#include "../../neo-rxchf_gb300/csrc/g3_fatbra.cuh"

using namespace neoxc;
using namespace neoxc::g3;
using md::Prim;
typedef long double ld;

static std::mt19937_64 rng(5);
static double uni(double a, double b) { return std::uniform_real_distribution<double>(a, b)(rng); }

static Prim prim(int axis, int l, double lo, double hi, const double* c) {
  Prim p;
  p.a = exp(uni(log(lo), log(hi)));
  for (int d = 0; d < 3; d++) {
    p.l[d] = d == axis ? l : 0;
    p.c[d] = c ? c[d] : uni(-1.0, 1.0);
  }
  return p;
}

static ld fact(int n) { return n < 2 ? 1.0L : n * fact(n - 1); }

// sum_m F_m(T) sum_{i+j+k=m} A_x[i] A_y[j] A_z[k] with the factors of F_i in
// sum_t W[t] d^t/dR^t F_0(alpha R^2) written out
static void reference(const Bra<double, 12>& b, const double* rk, ld* val, ld* mag) {
  const ld pi = 3.14159265358979L, p = rk[kRP], Z = b.Z, alpha = Z * p / (Z + p);
  ld A[2][3][17], R2 = 0.0L;
  int n[3];
  for (int d = 0; d < 3; d++) {
    const ld R = b.C[d] - rk[kRX + d];
    R2 += R * R;
    const int t = (int)rk[kRT + d];
    n[d] = b.N[d] + t;
    ld W[2][17] = {};
    for (int i = 0; i <= b.N[d]; i++)
      for (int q = 0; q <= t; q++) {
        const ld x = (ld)b.W[d][i] * rk[kRE + 5 * d + q];
        W[0][i + q] += (q & 1) ? -x : x;
        W[1][i + q] += fabsl(x);
      }
    for (int i = 0; i <= n[d]; i++) {
      A[0][d][i] = A[1][d][i] = 0.0L;
      for (int k = i; k <= n[d] && k <= 2 * i; k++) {
        const ld h = fact(k) / (fact(2 * i - k) * fact(k - i) * powl(2.0L, k - i)) *
                     powl(-2.0L * alpha * R, 2 * i - k) * powl(-2.0L * alpha, k - i);
        A[0][d][i] += W[0][k] * h;
        A[1][d][i] += W[1][k] * fabsl(h);
      }
    }
  }
  double F[40];
  boys(n[0] + n[1] + n[2], (double)(alpha * R2), F);
  ld s[2] = {0.0L, 0.0L};
  for (int w = 0; w < 2; w++)
    for (int i = 0; i <= n[0]; i++)
      for (int j = 0; j <= n[1]; j++)
        for (int k = 0; k <= n[2]; k++) s[w] += F[i + j + k] * A[w][0][i] * A[w][1][j] * A[w][2][k];
  const ld pre = b.pref * 2.0L * pi * pi * sqrtl(pi) / (Z * p * sqrtl(Z + p));
  *val = pre * s[0];
  *mag = fabsl(pre) * s[1];
}

int main() {
  // electron pairs of l = 2 + 2 along one axis, ket and proton pair from 0 to 4
  for (int axis = 0; axis < 3; axis++)
    for (int vee = 0; vee < 2; vee++)
      for (int tk = 0; tk <= 4; tk++)
        for (int tp = 0; tp <= 4; tp++)
          for (int rep = 0; rep < 6; rep++) {
            double r[4][kRLen], cp[3] = {uni(-1, 1), uni(-1, 1), uni(-1, 1)};
            for (int i = 0; i < 4; i++) {
              const int l = i < 2 ? 4 : (i == 2 ? tk : tp), la = (l + 1) / 2;
              const double* c = i == 3 ? cp : nullptr;
              const double lo = i == 3 ? 4.0 : 0.1, hi = i == 3 ? 32.0 : 20.0;
              fill_pair_record(prim(axis, la, lo, hi, c), prim(axis, l - la, lo, hi, c), 1.0, 1.0, r[i]);
            }
            Bra<double, 12> b;
            if (vee) build_bra_vee<double, 2, 2, 12>(r[0], r[1], r[3], uni(0.5, 20.0), uni(0.5, 20.0), b);
            else build_bra_vep<double, 2, 2, 12>(r[0], r[1], r[3], uni(0.5, 20.0), uni(0.5, 20.0), b);
            ld ref, mag;
            reference(b, r[2], &ref, &mag);
            finish_bra<12>(b);
            Ket<4> k;
            load_ket<4>(r[2], k);
            printf("%d %.17g %.20Lg %.6Lg\n", 8 + tk + tp, fb_value<12, 4>(b, k), ref, mag);
          }
  return 0;
}
