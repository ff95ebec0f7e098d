// k_pair.cu -- the one- and two-particle integral tables on sm_103a (FP64).
//
// Reference: pure_ovlap.f:2-202 (elec_ovlap, nuc_ovlap), gam_epcore.f:2-270,
// gam_ee.f:2-169 (calc_GAM_ee), gam_ep.f:2-219, gam_1_OMP.f:2-836 and
// rxchf/rxchf_gam_1_OMP.f (GAM1_OMP_MD, RXCHF_GAM1_OMP_MD).
//
// Every table depends on its particles' pair densities alone (the kinetic
// terms after the sum over geminals), so each is computed once per
// canonical pair (i >= j) from the pair records of stage_system, and written
// to all the places of that pair.  A warp (GAM_1: a CTA) owns an output and
// its lanes take primitive pairs x nuclei or geminal terms: the tables are
// small, so what bounds them is the longest chain of FP64 instructions of a
// thread, not their number.  One thread per output, walking its primitives
// with the general MD routines, took 5.6 ms for GAM_1 of examples/xchf (36
// outputs), 0.64 ms for the one-body matrices and 0.25 ms for GAM_ep; with
// them, and with the separable gam_3 factors taken from the gam_2 build, a
// whole examples/xchf solve took 17.3 ms and now takes 9.3 ms.
#include "g2_threebody.cuh"
#include "neoxc_internal.h"

namespace neoxc {
namespace {

using namespace g2;

__device__ __forceinline__ void unpair(int P, int& i, int& j) {
  int a = (int)((sqrtf(8.0f * (float)P + 1.0f) - 1.0f) * 0.5f);
  while (a * (a + 1) / 2 > P) a--;
  while ((a + 1) * (a + 2) / 2 <= P) a++;
  i = a;
  j = P - a * (a + 1) / 2;
}

__device__ __forceinline__ double warp_all(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ md::Prim to_md(const DevPrim& d) {
  md::Prim p;
  p.a = d.a;
  for (int k = 0; k < 3; k++) {
    p.c[k] = d.c[k];
    p.l[k] = d.l[k];
  }
  return p;
}

// Overlap and core Hamiltonian (xcalc_GAM_epcore) of a contracted pair: lanes
// take (primitive pair, overlap and kinetic energy or one nucleus).  The
// reference's two-centre formulas are kept operation by operation: the basis
// sets of its regression decks are nearly linearly dependent, so the guess
// orbitals, and with them the logged energies' last digits, carry the
// rounding of exactly these two matrices.
__device__ __forceinline__ void onebody_terms(const DevSystem& S, const DevPrim* bra, int na,
                                              const DevPrim* ket, int nb, double mass,
                                              double sign, int lane, double& ov, double& h) {
  ov = h = 0.0;
  const int nk = na * nb;
  for (int q = lane; q < nk * (S.nat + 1); q += 32) {
    const int k = q % nk, c = q / nk;
    const DevPrim &pa = bra[k / nb], &pb = ket[k % nb];
    const md::Prim A = to_md(pa), B = to_md(pb);
    if (c == 0) {
      double o = 1.0;
      for (int d = 0; d < 3; d++) o *= md::ovl1d(A.l[d], A.a, A.c[d], B.l[d], B.a, B.c[d]);
      ov = ov + o * pa.coef * pb.coef;
      h = h + md::gfke(A, B, mass) * pa.coef * pb.coef;
    } else {
      const double C[3] = {S.cat[3 * c - 3], S.cat[3 * c - 2], S.cat[3 * c - 1]};
      h = h + sign * S.zan[c - 1] * md::gfvec(A, B, C) * pa.coef * pb.coef;
    }
  }
  ov = warp_all(ov);
  h = warp_all(h);
}

// warps: electronic pairs, then proton pairs
__global__ void __launch_bounds__(64)
onebody_kernel(DevSystem S, double* __restrict__ Se, double* __restrict__ Sp,
               double* __restrict__ Hce, double* __restrict__ Hcp) {
  const int nPe = S.nebf * (S.nebf + 1) / 2, nPp = S.npbf * (S.npbf + 1) / 2;
  const int lane = threadIdx.x & 31, w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (w >= nPe + nPp) return;
  const bool el = w < nPe;
  const int n = el ? S.nebf : S.npbf;
  int i, j;
  unpair(el ? w : w - nPe, i, j);
  double ov, h;
  if (el)
    onebody_terms(S, S.eprim + S.kpestr[i], S.kpeend[i] - S.kpestr[i] + 1, S.eprim + S.kpestr[j],
                  S.kpeend[j] - S.kpestr[j] + 1, 1.0, -1.0, lane, ov, h);
  else
    onebody_terms(S, S.pprim + i, 1, S.pprim + j, 1, S.pmass, 1.0, lane, ov, h);
  if (lane == 0) {
    double* So = el ? Se : Sp;
    double* Ho = el ? Hce : Hcp;
    So[i * n + j] = So[j * n + i] = ov;
    Ho[i * n + j] = Ho[j * n + i] = h;
  }
}

// GAM_ep[ip][jp][ie][je] = -(e | p); a warp per (Pp, Pe)
template <int LE, int LN>
__global__ void __launch_bounds__(64) gam_ep_kernel(DevSystem S, double* __restrict__ Gep) {
  const int ne = S.nebf, np = S.npbf, nPe = ne * (ne + 1) / 2, nPp = np * (np + 1) / 2;
  const int lane = threadIdx.x & 31;
  const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (w >= (long long)nPp * nPe) return;
  const int P = (int)(w % nPe), Pp = (int)(w / nPe);
  const int* kofs = S.g3i + 2 * S.g3_nket;
  const double* rp = S.g3rec + (size_t)kRLen * (S.g3_nket + Pp);
  double acc = 0.0;
  for (int k = kofs[P] + lane; k < kofs[P + 1]; k += 32) {
    const double* r = S.g3rec + (size_t)kRLen * k;
    acc = fma(-pair_coulomb<2 * LE + 2 * LN>(r, rp), r[kRC], acc);
  }
  acc = warp_all(acc) * rp[kRC];
  if (lane < 4) {   // (ip,jp), (jp,ip) x (ie,je), (je,ie)
    int i, j, a, b;
    unpair(P, i, j);
    unpair(Pp, a, b);
    const long long pp = (lane & 1) ? (long long)b * np + a : (long long)a * np + b;
    const int ee = (lane & 2) ? j * ne + i : i * ne + j;
    Gep[pp * ne * ne + ee] = acc;
  }
}

// GAM_ee, pack_4D order; a warp per unordered (P1 >= P2)
template <int LE>
__global__ void __launch_bounds__(64) gam_ee_kernel(DevSystem S, double* __restrict__ gee) {
  const int ne = S.nebf, nPe = ne * (ne + 1) / 2, lane = threadIdx.x & 31;
  const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (w >= (long long)nPe * (nPe + 1) / 2) return;
  long long a = (long long)((sqrt(8.0 * (double)w + 1.0) - 1.0) * 0.5);
  while (a * (a + 1) / 2 > w) a--;
  while ((a + 1) * (a + 2) / 2 <= w) a++;
  const int P1 = (int)a, P2 = (int)(w - a * (a + 1) / 2);
  const int* kofs = S.g3i + 2 * S.g3_nket;
  const int k1 = kofs[P1], n1 = kofs[P1 + 1] - k1, k2 = kofs[P2], n2 = kofs[P2 + 1] - k2;
  double acc = 0.0;
  for (int q = lane; q < n1 * n2; q += 32) {
    const double* r = S.g3rec + (size_t)kRLen * (k1 + q / n2);
    const double* s = S.g3rec + (size_t)kRLen * (k2 + q % n2);
    acc = fma(pair_coulomb<4 * LE>(r, s), r[kRC] * s[kRC], acc);
  }
  acc = warp_all(acc);
  if (lane < 8) {   // (12) or (21), and the two orders within each pair
    int i, j, k, l;
    unpair(P1, i, j);
    unpair(P2, k, l);
    const int e1 = (lane & 1) ? j * ne + i : i * ne + j, e2 = (lane & 2) ? l * ne + k : k * ne + l;
    const long long m = (long long)ne * ne;
    gee[(lane & 4) ? e2 * m + e1 : e1 * m + e2] = acc;
  }
}

// GAM_1 / GAM_1s[ip][jp][ie][je]; a CTA per (Pp, Pe).  Its threads take first
// the multiplicative terms of (primitive pair, geminal exponent), then the
// kinetic ones of (primitive pair, geminals on bra and ket, particle): both
// depend on the pair only after the sum over geminals, so (ie,je), (je,ie) and
// the proton's two orders share the result.  pairs_only: RXCHF_GAM1_OMP_MD.
constexpr int kGam1Threads = 256;
template <int LE, int LN>
__global__ void __launch_bounds__(kGam1Threads)
gam1_kernel(DevSystem S, int pairs_only, double* __restrict__ G1, double* __restrict__ G1s) {
  __shared__ double se[kGam1Threads / 32], ss[kGam1Threads / 32];
  const int ne = S.nebf, np = S.npbf, nPe = ne * (ne + 1) / 2;
  const long long u = blockIdx.x;
  const int P = (int)(u % nPe), Pp = (int)(u / nPe);
  const int* kofs = S.g3i + 2 * S.g3_nket;
  const int k0 = kofs[P], nk = kofs[P + 1] - k0, ng = S.ngtg;
  const int npr = ng * (ng + 1) / 2, nt = npr + (pairs_only ? 0 : ng);
  const int nkin = ng * ng + (pairs_only ? 0 : 2 * ng);
  const double* rp = S.g3rec + (size_t)kRLen * (S.g3_nket + Pp);
  int ip, jp;
  unpair(Pp, ip, jp);
  double e = 0.0, o = 0.0;
  for (int q = threadIdx.x; q < nk * (nt + 2 * nkin); q += kGam1Threads) {
    const int k = k0 + q % nk;
    int t = q / nk;
    const double* r = S.g3rec + (size_t)kRLen * k;
    if (t < nt) {
      // pairs k <= l first (b_k b_l, twice off the diagonal), then singles (2 b_k)
      double g, w;
      if (t < npr) {
        int b, a;
        unpair(t, b, a);
        g = S.ggem[a] + S.ggem[b];
        w = S.bgem[a] * S.bgem[b] * (a == b ? 1.0 : 2.0);
      } else {
        g = S.ggem[t - npr];
        w = 2.0 * S.bgem[t - npr];
      }
      double x, y;
      two_body<LE, LN>(r, rp, g, S.nat, S.cat, S.zan, &x, &y);
      w *= r[kRC];
      e = fma(w, x, e);
      o = fma(w, y, o);
    } else {
      t -= nt;
      const bool proton = t >= nkin;
      if (proton) t -= nkin;
      double gA = 0.0, gB = 0.0, w = r[kRC];
      if (t < ng * ng) {
        gA = S.ggem[t / ng];
        gB = S.ggem[t % ng];
        w *= S.bgem[t / ng] * S.bgem[t % ng];
      } else {
        t -= ng * ng;
        (t < ng ? gA : gB) = S.ggem[t % ng];
        w *= S.bgem[t % ng];
      }
      const md::Prim E1 = to_md(S.eprim[S.g3i[2 * k]]), E2 = to_md(S.eprim[S.g3i[2 * k + 1]]);
      const md::Prim Q1 = to_md(S.pprim[ip]), Q2 = to_md(S.pprim[jp]);
      const double x = proton ? pair_kinetic(Q1, E1, Q2, E2, gA, gB, S.pmass)
                              : pair_kinetic(E1, Q1, E2, Q2, gA, gB, 1.0);
      e = fma(w, x, e);
    }
  }
  e = warp_all(e);
  o = warp_all(o);
  if ((threadIdx.x & 31) == 0) {
    se[threadIdx.x >> 5] = e;
    ss[threadIdx.x >> 5] = o;
  }
  __syncthreads();
  if (threadIdx.x < 4) {
    double x = 0.0, y = 0.0;
    for (int k = 0; k < kGam1Threads / 32; k++) {
      x += se[k];
      y += ss[k];
    }
    int i, j;
    unpair(P, i, j);
    const long long pp = (threadIdx.x & 1) ? (long long)jp * np + ip : (long long)ip * np + jp;
    const int ee = (threadIdx.x & 2) ? j * ne + i : i * ne + j;
    G1[pp * ne * ne + ee] = x * rp[kRC];
    G1s[pp * ne * ne + ee] = y * rp[kRC];
  }
}

unsigned warps2(long long w) { return (unsigned)((w + 1) / 2); }   // CTAs of two warps

}  // namespace

cudaError_t launch_scf_onebody(const DevSystem& S, double* Se, double* Sp, double* Hce,
                               double* Hcp, cudaStream_t s) {
  const long long n = (long long)S.nebf * (S.nebf + 1) / 2 + (long long)S.npbf * (S.npbf + 1) / 2;
  onebody_kernel<<<warps2(n), 64, 0, s>>>(S, Se, Sp, Hce, Hcp);
  return cudaGetLastError();
}

cudaError_t launch_gam_ep(const DevSystem& S, double* Gep, cudaStream_t s) {
  const long long n = (long long)S.nebf * (S.nebf + 1) / 2 * S.npbf * (S.npbf + 1) / 2;
  switch (S.lmax_e * 3 + (S.lmax_p == 0 ? 0 : 2)) {
    case 0: gam_ep_kernel<0, 0><<<warps2(n), 64, 0, s>>>(S, Gep); break;
    case 2: gam_ep_kernel<0, 2><<<warps2(n), 64, 0, s>>>(S, Gep); break;
    case 3: gam_ep_kernel<1, 0><<<warps2(n), 64, 0, s>>>(S, Gep); break;
    case 5: gam_ep_kernel<1, 2><<<warps2(n), 64, 0, s>>>(S, Gep); break;
    case 6: gam_ep_kernel<2, 0><<<warps2(n), 64, 0, s>>>(S, Gep); break;
    default: gam_ep_kernel<2, 2><<<warps2(n), 64, 0, s>>>(S, Gep); break;
  }
  return cudaGetLastError();
}

cudaError_t launch_gam_ee(const DevSystem& S, double* gee, cudaStream_t s) {
  const long long nPe = (long long)S.nebf * (S.nebf + 1) / 2, n = nPe * (nPe + 1) / 2;
  switch (S.lmax_e) {
    case 0: gam_ee_kernel<0><<<warps2(n), 64, 0, s>>>(S, gee); break;
    case 1: gam_ee_kernel<1><<<warps2(n), 64, 0, s>>>(S, gee); break;
    default: gam_ee_kernel<2><<<warps2(n), 64, 0, s>>>(S, gee); break;
  }
  return cudaGetLastError();
}

cudaError_t launch_gam1(const DevSystem& S, double* G1, double* G1s, cudaStream_t s,
                        int pairs_only) {
  const unsigned n = (unsigned)((long long)S.nebf * (S.nebf + 1) / 2 * (S.npbf * (S.npbf + 1LL) / 2));
  switch (S.lmax_e * 3 + (S.lmax_p == 0 ? 0 : 2)) {
    case 0: gam1_kernel<0, 0><<<n, kGam1Threads, 0, s>>>(S, pairs_only, G1, G1s); break;
    case 2: gam1_kernel<0, 2><<<n, kGam1Threads, 0, s>>>(S, pairs_only, G1, G1s); break;
    case 3: gam1_kernel<1, 0><<<n, kGam1Threads, 0, s>>>(S, pairs_only, G1, G1s); break;
    case 5: gam1_kernel<1, 2><<<n, kGam1Threads, 0, s>>>(S, pairs_only, G1, G1s); break;
    case 6: gam1_kernel<2, 0><<<n, kGam1Threads, 0, s>>>(S, pairs_only, G1, G1s); break;
    default: gam1_kernel<2, 2><<<n, kGam1Threads, 0, s>>>(S, pairs_only, G1, G1s); break;
  }
  return cudaGetLastError();
}

}  // namespace neoxc
