// k_md.cu -- contracted geminal-integral builders on sm_103a (FP64).
//
// Reference:
//   gam_ee.f:2-169 (calc_GAM_ee)                 -> gam_ee_kernel
//   gam_3_OMP.f:617-984 (xcalc_GAM3_MD) separable terms
//                                                -> gam3_w1/w3/hcore_kernel
//     (the four-particle terms: k_gam3.cu; gam_2: k_gam2.cu)
//   gam3_IC1_OMP.f:143-262                       -> gam3_sym_kernel
//
// Work decomposition: one warp per contracted tuple (its packed index is
// the warp id, since the reference's loop order equals the packing order);
// the lanes split the tuple's primitive combinations and the contraction
// is a warp-shuffle reduction.  Each lane evaluates the reference's
// per-primitive integrand with the factorised MD kernels of md_math.cuh,
// re-using one Boys'-lemma/derivative setup for every integral that shares
// a particle order and geminal assignment.
#include "md_math.cuh"
#include "neoxc_internal.h"

namespace neoxc {
namespace {

using md::G3;
using md::Prim;

__device__ __forceinline__ Prim to_prim(const DevPrim& d) {
  Prim p;
  p.a = d.a;
  for (int k = 0; k < 3; k++) {
    p.c[k] = d.c[k];
    p.l[k] = d.l[k];
  }
  return p;
}

__device__ __forceinline__ double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

template <class R>
__device__ __forceinline__ void gam6(R* g, int slot_a, R va, int slot_b, R vb) {
  for (int k = 0; k < 6; k++) g[k] = R(0.0);
  if (slot_a >= 0) g[slot_a] = va;
  if (slot_b >= 0) g[slot_b] = vb;
}
enum { A12 = 0, A13, A23, B12, B13, B23 };

template <class P>
__device__ __forceinline__ void perm3(const P* X, int a, int b, int c, P* Y) {
  Y[0] = X[a];
  Y[1] = X[b];
  Y[2] = X[c];
}

// ---- GAM_ee: warp per contracted (iec1,jec1,iec2,jec2) ----------------------
// lanes share the primitive quartets; warp-shuffle contraction.
__global__ void __launch_bounds__(128)
gam_ee_kernel(DevSystem S, double* __restrict__ gee) {
  const int ne = S.nebf;
  const long long n4 = (long long)ne * ne * ne * ne;
  const int lane = threadIdx.x & 31;
  const long long nw = (long long)gridDim.x * blockDim.x / 32;
  for (long long t = (blockIdx.x * (long long)blockDim.x + threadIdx.x) / 32; t < n4;
       t += nw) {
    // pack_4D(jec2, iec2, jec1, iec1) - 1 == t
    long long r = t;
    const int jc2 = (int)(r % ne); r /= ne;
    const int ic2 = (int)(r % ne); r /= ne;
    const int jc1 = (int)(r % ne); r /= ne;
    const int ic1 = (int)r;
    const int s1 = S.kpestr[ic1], n1 = S.kpeend[ic1] - s1 + 1;
    const int t1 = S.kpestr[jc1], m1 = S.kpeend[jc1] - t1 + 1;
    const int s2 = S.kpestr[ic2], n2 = S.kpeend[ic2] - s2 + 1;
    const int t2 = S.kpestr[jc2], m2 = S.kpeend[jc2] - t2 + 1;
    const int nq = n1 * m1 * n2 * m2;
    double acc = 0.0;
    for (int q = lane; q < nq; q += 32) {
      int qq = q;
      const int j2 = t2 + qq % m2; qq /= m2;
      const int i2 = s2 + qq % n2; qq /= n2;
      const int j1 = t1 + qq % m1; qq /= m1;
      const int i1 = s1 + qq;
      const DevPrim &a1 = S.eprim[i1], &a2 = S.eprim[i2];
      const DevPrim &b1 = S.eprim[j1], &b2 = S.eprim[j2];
      double v = md::gfvee(to_prim(a1), to_prim(a2), to_prim(b1), to_prim(b2));
      acc = acc + v * a1.coef * b1.coef * a2.coef * b2.coef;
    }
    acc = warp_sum(acc);
    if (lane == 0) gee[t] = acc;
  }
}

// ---- separable gam_3 factors (contracted, FP64) ---------------------------
// W1[ip][jp][i1][j1] = sum_prims c c c_p c_p' [sum_k b_k G2xggs(g_k,0)
//                       + 1/2 sum_kl b_k b_l G2xggs(g_k,g_l)]       (e1, p)
__global__ void gam3_w1_kernel(DevSystem S, double* __restrict__ W1) {
  const int ne = S.nebf, np = S.npbf;
  const int lane = threadIdx.x & 31;
  const long long w = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
  if (w >= (long long)np * np * ne * ne) return;
  long long r = w;
  const int j1 = (int)(r % ne); r /= ne;
  const int i1 = (int)(r % ne); r /= ne;
  const int jp = (int)(r % np);
  const int ip = (int)(r / np);
  const int s1 = S.kpestr[i1], n1 = S.kpeend[i1] - s1 + 1;
  const int s2 = S.kpestr[j1], n2 = S.kpeend[j1] - s2 + 1;
  const Prim P1 = to_prim(S.pprim[ip]), P2 = to_prim(S.pprim[jp]);
  double o = 0.0;
  for (int q = lane; q < n1 * n2; q += 32) {
    const int a = s1 + q / n2, bq = s2 + q % n2;
    const Prim A = to_prim(S.eprim[a]), B = to_prim(S.eprim[bq]);
    double v = 0.0;
    for (int k = 0; k < S.ngtg; k++)
      v = v + S.bgem[k] * md::underflow(md::g2_xggs(A, P1, B, P2, S.ggem[k], 0.0));
    double v2 = 0.0;
    for (int k = 0; k < S.ngtg; k++)
      for (int l = 0; l < S.ngtg; l++)
        v2 = v2 + S.bgem[k] * S.bgem[l] *
                      md::underflow(md::g2_xggs(A, P1, B, P2, S.ggem[k], S.ggem[l]));
    o = o + (v + 0.5 * v2) * (S.eprim[a].coef * S.eprim[bq].coef *
                              S.pprim[ip].coef * S.pprim[jp].coef);
  }
  o = warp_sum(o);
  if (lane == 0) W1[w] = o;
}

// W3[ip][jp][i1][j1][i2][j2] = sum_prims c^6 sum_kl b_k b_l
//                              G3xggs(e1,e2,p; A13 = g_k, B23 = g_l)
__global__ void __launch_bounds__(64)
gam3_w3_kernel(DevSystem S, double* __restrict__ W3) {
  const int ne = S.nebf, np = S.npbf;
  const int lane = threadIdx.x & 31;
  const long long w = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
  if (w >= (long long)np * np * ne * ne * ne * ne) return;
  long long r = w;
  int c[4];
  for (int k = 3; k >= 0; k--) {
    c[k] = (int)(r % ne);
    r /= ne;
  }
  const int jp = (int)(r % np);
  const int ip = (int)(r / np);
  int st0[4], cnt[4], nq = 1;
  for (int k = 0; k < 4; k++) {
    st0[k] = S.kpestr[c[k]];
    cnt[k] = S.kpeend[c[k]] - st0[k] + 1;
    nq *= cnt[k];
  }
  G3 st;
  double o = 0.0, g[6];
  for (int q = lane; q < nq; q += 32) {
    int qq = q, idx[4];
    for (int k = 3; k >= 0; k--) {
      idx[k] = st0[k] + qq % cnt[k];
      qq /= cnt[k];
    }
    const Prim A[3] = {to_prim(S.eprim[idx[0]]), to_prim(S.eprim[idx[2]]),
                       to_prim(S.pprim[ip])};
    const Prim B[3] = {to_prim(S.eprim[idx[1]]), to_prim(S.eprim[idx[3]]),
                       to_prim(S.pprim[jp])};
    md::Pair pr[3];
    for (int i = 0; i < 3; i++) md::gauss_pair(A[i], B[i], pr[i]);
    double v = 0.0;
    for (int k = 0; k < S.ngtg; k++)
      for (int l = 0; l < S.ngtg; l++) {
        gam6(g, A13, S.ggem[k], B23, S.ggem[l]);
        md::g3_setup_pairs(st, A, B, pr, g, 0);
        v = v + S.bgem[k] * S.bgem[l] * md::underflow(md::g3_overlap(st));
      }
    double cc = S.pprim[ip].coef * S.pprim[jp].coef;
    for (int k = 0; k < 4; k++) cc = cc * S.eprim[idx[k]].coef;
    o = o + v * cc;
  }
  o = warp_sum(o);
  if (lane == 0) W3[w] = o;
}

// Hcore[i][j] = sum_prims c c [T - sum_C Z V_C]  (xcalc_GAM3_MD's h(e3))
__global__ void gam3_hcore_kernel(DevSystem S, double* __restrict__ Hc) {
  const int ne = S.nebf;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= ne * ne) return;
  const int i = t / ne, j = t - i * ne;
  double h = 0.0;
  for (int a = S.kpestr[i]; a <= S.kpeend[i]; a++)
    for (int bq = S.kpestr[j]; bq <= S.kpeend[j]; bq++) {
      const Prim A = to_prim(S.eprim[a]), B = to_prim(S.eprim[bq]);
      const double xke = md::gfke(A, B, 1.0);
      double Vc = 0.0;
      for (int ia = 0; ia < S.nat; ia++)
        Vc = Vc + (S.zan[ia] * md::gfvec(A, B, S.cat + 3 * ia));
      h = h + (xke + (Vc * -1.0)) * (S.eprim[a].coef * S.eprim[bq].coef);
    }
  Hc[t] = h;
}

// Six-permutation symmetrisation in place: each orbit is handled by the
// tuple with the largest packed index (the reference's last writer), which
// averages in its own permutation order and writes the whole orbit.
__global__ void gam3_sym_kernel(int ne, int np, double* __restrict__ g,
                                long long n) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x) {
    long long r = t;
    const int j3 = (int)(r % ne); r /= ne;
    const int i3 = (int)(r % ne); r /= ne;
    const int j2 = (int)(r % ne); r /= ne;
    const int i2 = (int)(r % ne); r /= ne;
    const int j1 = (int)(r % ne); r /= ne;
    const int i1 = (int)(r % ne); r /= ne;
    const long long pp = r;
    auto idx = [&](int a, int b, int c, int d, int e, int f) -> long long {
      return f + (long long)ne * (e + (long long)ne * (d + (long long)ne * (c +
             (long long)ne * (b + (long long)ne * (a + (long long)ne * pp)))));
    };
    const long long a132 = idx(i1, j1, i3, j3, i2, j2);
    const long long a213 = idx(i2, j2, i1, j1, i3, j3);
    const long long a231 = idx(i2, j2, i3, j3, i1, j1);
    const long long a312 = idx(i3, j3, i1, j1, i2, j2);
    const long long a321 = idx(i3, j3, i2, j2, i1, j1);
    if (a132 > t || a213 > t || a231 > t || a312 > t || a321 > t) continue;
    const double xx = (g[t] + g[a132] + g[a213] + g[a231] + g[a312] + g[a321]) / 6.0;
    g[t] = xx;
    g[a132] = xx;
    g[a213] = xx;
    g[a231] = xx;
    g[a312] = xx;
    g[a321] = xx;
  }
}

}  // namespace

cudaError_t launch_gam_ee(const DevSystem& sys, double* gee, cudaStream_t s) {
  const long long n4 = (long long)sys.nebf * sys.nebf * sys.nebf * sys.nebf;
  long long blocks = (n4 * 32 + 127) / 128;   // a warp per contracted quartet
  if (blocks > 152 * 64) blocks = 152 * 64;
  gam_ee_kernel<<<(unsigned)blocks, 128, 0, s>>>(sys, gee);
  return cudaGetLastError();
}

cudaError_t launch_gam3_aux(const DevSystem& sys, double* aux, cudaStream_t s,
                            const double* gee_in, const double* hc_in) {
  const int ne = sys.nebf, np = sys.npbf;
  const long long n2 = (long long)ne * ne, n4 = n2 * n2;
  double* gee = aux;
  double* hc = gee + n4;
  double* W1 = hc + n2;
  double* W3 = W1 + (long long)np * np * n2;
  cudaError_t e = gee_in ? cudaMemcpyAsync(gee, gee_in, sizeof(double) * n4,
                                           cudaMemcpyDeviceToDevice, s)
                         : launch_gam_ee(sys, gee, s);
  if (e != cudaSuccess) return e;
  if (hc_in)
    e = cudaMemcpyAsync(hc, hc_in, sizeof(double) * n2, cudaMemcpyDeviceToDevice, s);
  else
    gam3_hcore_kernel<<<(unsigned)((n2 + 127) / 128), 128, 0, s>>>(sys, hc);
  if (e != cudaSuccess) return e;
  const long long w1 = (long long)np * np * n2, w3 = w1 * n2;
  gam3_w1_kernel<<<(unsigned)((w1 * 32 + 127) / 128), 128, 0, s>>>(sys, W1);
  gam3_w3_kernel<<<(unsigned)((w3 * 32 + 63) / 64), 64, 0, s>>>(sys, W3);
  return cudaGetLastError();
}

cudaError_t launch_gam3_symmetrize(int ne, int np, double* g3,
                                   cudaStream_t s) {
  const long long n = (long long)ne * ne * ne * ne * ne * ne * np * np;
  long long blocks = (n + 255) / 256;
  if (blocks > 152 * 32) blocks = 152 * 32;
  gam3_sym_kernel<<<(unsigned)blocks, 256, 0, s>>>(ne, np, g3, n);
  return cudaGetLastError();
}

}  // namespace neoxc
