// k_md.cu -- the gam_3 tensor around its four-particle terms (k_gam3.cu) for
// sm_103a: the separable factors GAM_ee, Hcore, W1 and W3 of gam_3_OMP.f:617-984
// (xcalc_GAM3_MD), built by k_pair.cu and k_gam2.cu, and the six-permutation
// symmetrisation of gam3_IC1_OMP.f:143-262.
#include "neoxc_internal.h"

namespace neoxc {
namespace {

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

cudaError_t launch_gam3_aux(const DevSystem& sys, double* aux, double* scratch, cudaStream_t s,
                            const double* gee_in, const double* hc_in, const double* w3_in) {
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
  if (hc_in) {
    e = cudaMemcpyAsync(hc, hc_in, sizeof(double) * n2, cudaMemcpyDeviceToDevice, s);
    if (e != cudaSuccess) return e;
  }
  return launch_gam3_factors(sys, scratch, w3_in, W1, W3, hc_in ? nullptr : hc, s);
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
