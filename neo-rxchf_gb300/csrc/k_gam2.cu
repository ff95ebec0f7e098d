// k_gam2.cu -- the contracted gam_2 tensors on sm_103a (FP64).
//
// Reference: gam_2_OMP.f:546-1077 (xcalc_GAM2_MD), gam2_CONV_OMP.f:388-579
// (contract_omega2_conv), gam2_IC1_OMP.f:136-337 (GAM2_IC1 with its pair
// symmetrisation), rxchfne/rxchfne_gam_2_OMP.f:2-530 and
// rxchfne_gam2_IC1_OMP.f:184-340 (RXCHFne_GAM2_IC1).
//
// What bounds it: FP64 instructions (2 per SM and clock on this GPU).  The
// element-by-element form evaluated all of xcalc_GAM2_MD for every ordered
// primitive quartet; this one evaluates each distinct quantity once:
//
//  1. The symmetrised tensors depend on each particle only through its pair
//     density, also in the kinetic terms (g2_threebody.cuh), so they are
//     computed for canonical pairs (i >= j) of every particle and gathered
//     onto index_GAM_2PK: 8x fewer tuples, and the terms that couple all
//     three particles once per unordered electron pair: 2x again.
//  2. Terms in which one electron meets no geminal -- xgVEE, xgVEP, xgVEEg1,
//     xgVEPg2 -- are two-centre Coulomb integrals between that electron's
//     pair density and a composite density of the other two particles (the
//     bra / ket form of k_gam3.cu).  They see only the sum of the geminal
//     exponents, so the ng single and ng^2 pair terms are ng + ng(ng+1)/2
//     exponents (gam2_pair_kernel, array Y[bra pair][ket]).
//  3. xgTPg, xgTEg1/2, xgVPCg, xgVECg1, xgVEEg2, xgVEPg1 and the overlap of
//     one (k, l) all integrate the same three-particle Gaussian: one
//     derivative table and one set of Hermite folds serves the six Coulomb
//     operators, the kinetic terms and the overlap (gam2_triple_kernel,
//     arrays R1, R2).
//  4. xgTE, xgVEC, xgTEg3 and xgVECg2 factor into the core Hamiltonian of
//     electron 1 and a two-particle overlap of (e2, p) (gam2_factor_kernel).
//
// Measured (one GB300, neoxc_gam2_ic1 / _rxchfne_gam2_ic1 from host arrays):
// nebf = 8 s/p of 2 primitives, npbf = 3 s/p/d, NG = 3: 494 ms element by
// element, 5.6 ms so; RXCHF-ne, nebf = 9 s/p/d, npbf = 4, NG = 4: 815 ms and
// 11.7 ms.  The former FP32-first form (dynamic precision) was 1.8x faster
// than the first of each pair, so it is gone.
//
// A warp owns one canonical (proton pair, electron pair) and a share of its
// primitive pairs x geminal terms; its lanes take 32 primitive pairs of the
// other electron, so bra data are uniform and nothing is summed across
// lanes.  Lane sums go to a per-primitive-pair scratch array (one slot per
// share), which gam2_contract_kernel adds up in a fixed order: results are
// deterministic.  The tensor is built in chunks of proton pairs so that the
// scratch stays bounded.
#include <algorithm>

#include "g2_threebody.cuh"
#include "neoxc_internal.h"

namespace neoxc {
namespace {

using namespace g2;
using g3::Bra;

constexpr int kWarps = 2;   // independent warps of a CTA

__host__ __device__ __forceinline__ void unpair(int P, int& i, int& j) {
  int a = (int)((sqrtf(8.0f * (float)P + 1.0f) - 1.0f) * 0.5f);
  while (a * (a + 1) / 2 > P) a--;
  while ((a + 1) * (a + 2) / 2 <= P) a++;
  i = a;
  j = P - a * (a + 1) / 2;
}

struct Gam2View {   // the pair tables of DevSystem (stage_system)
  const double *erec, *prec;      // pair records
  const double *egrad, *pgrad;    // gradient records
  const int *kofs, *kperm;        // primitive pairs of a contracted pair; class order
  int nket, nPe;
};

__host__ __device__ __forceinline__ Gam2View view(const DevSystem& S) {
  Gam2View v;
  v.nPe = S.nebf * (S.nebf + 1) / 2;
  v.nket = S.g3_nket;
  v.erec = S.g3rec;
  v.prec = S.g3rec + (size_t)kRLen * v.nket;
  v.egrad = S.g3grad;
  v.pgrad = S.g3grad + (size_t)kGLen * v.nket;
  v.kofs = S.g3i + 2 * v.nket;
  // after kofs[nPe + 1]: tile_k and tile_P [ntile + 1 each], then the permutation
  v.kperm = v.kofs + v.nPe + 1 + 2 * (S.g3_ntile_all + 1);
  return v;
}

__device__ __forceinline__ double warp_add(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// exponent and weight of the q-th two-particle geminal term: g_k with 2 b_k,
// then g_k + g_l, k <= l, with b_k b_l (twice off the diagonal)
__device__ __forceinline__ void pair_term(const DevSystem& S, int q, double& g, double& w) {
  const int ng = S.ngtg;
  if (q < ng) {
    g = S.ggem[q];
    w = 2.0 * S.bgem[q];
    return;
  }
  int l, k;
  unpair(q - ng, l, k);
  g = S.ggem[k] + S.ggem[l];
  w = S.bgem[k] * S.bgem[l] * (k == l ? 1.0 : 2.0);
}

// One warp per output: W[Pp][Pe] = sum over primitives and the terms above of
// the two-particle overlap; then H[Pe], the contracted core Hamiltonian.
template <int LE>
__global__ void __launch_bounds__(32 * kWarps)
gam2_factor_kernel(DevSystem S, int nPp,
                   double* __restrict__ W, double* __restrict__ H) {
  const Gam2View v = view(S);
  const int lane = threadIdx.x & 31;
  const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nw = (long long)nPp * v.nPe;
  if (w >= nw + v.nPe) return;
  const int P = (int)(w % v.nPe);
  const int k0 = v.kofs[P], nk = v.kofs[P + 1] - k0;
  double acc = 0.0;
  if (w < nw) {
    const double* rp = v.prec + (size_t)kRLen * (w / v.nPe);
    const int nt = S.ngtg + S.ngtg * (S.ngtg + 1) / 2;
    for (int q = lane; q < nk * nt; q += 32) {
      const double* r = v.erec + (size_t)kRLen * (k0 + q % nk);
      double g, wt;
      pair_term(S, q / nk, g, wt);
      acc = fma(wt * r[kRC], two_body_overlap(r, rp, g), acc);
    }
    acc = warp_add(acc);
    if (lane == 0) W[w] = acc * rp[kRC];
  } else {
    const int nat = S.nat;
    const double kPi = 3.14159265358979323846;
    for (int q = lane; q < nk * (nat + 1); q += 32) {
      const int k = k0 + q % nk, c = q / nk;
      const double* r = v.erec + (size_t)kRLen * k;
      const double p = r[kRP], ip = kPi / p;
      double x;
      if (c == nat) {   // <T>: half the gradient product
        const double* e = v.egrad + (size_t)kGLen * k;
        const double ex = r[kRE], ey = r[kRE + 5], ez = r[kRE + 10];
        x = 0.5 * (e[0] * ey * ez + ex * e[kGRow] * ez + ex * ey * e[2 * kGRow]) * ip * sqrt(ip);
      } else {
        int n[3];
        double E[3][2 * LE + 1], R[3], R2 = 0.0;
        for (int d = 0; d < 3; d++) {
          n[d] = (int)r[kRT + d];
          for (int t = 0; t <= n[d]; t++) E[d][t] = r[kRE + 5 * d + t];
          R[d] = r[kRX + d] - S.cat[3 * c + d];
          R2 = fma(R[d], R[d], R2);
        }
        x = -S.zan[c] * 2.0 * ip * coulomb_sum<2 * LE>(n, E, R, p * R2, p);
      }
      acc = fma(x, r[kRC], acc);
    }
    acc = warp_add(acc);
    if (lane == 0) H[P] = acc;
  }
}

// Y[split][Pp - Pp0][Pb][ket]: bras (two per geminal exponent: electron b
// dressed by the proton, positive, and the proton dressed by electron b,
// negative) of (Pp, Pb) against the ket's electron.  PAIRS: the pair
// exponents only (RXCHF-ne).  grid (nPp * nPe, ket groups, splits) of warps.
template <int LE, int LN, bool PAIRS>
__global__ void __launch_bounds__(32 * kWarps)
gam2_pair_kernel(DevSystem S, int Pp0, long long nunit,
                 double* __restrict__ Y) {
  constexpr int NW = 2 * LE + 2 * LN, NK = 2 * LE;
  __shared__ Bra<double, NW> s_bra[kWarps][32];
  const Gam2View v = view(S);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const long long u = (long long)blockIdx.x * kWarps + wid;
  if (u >= nunit) return;
  const int grp = blockIdx.y, split = blockIdx.z, nsplit = gridDim.z;
  const int Pb = (int)(u % v.nPe), Pp = Pp0 + (int)(u / v.nPe);
  const int kb = v.kofs[Pb], nb = v.kofs[Pb + 1] - kb;
  const int q0 = PAIRS ? S.ngtg : 0;
  const int nt = S.ngtg + S.ngtg * (S.ngtg + 1) / 2 - q0;
  const int nbra = 2 * nb * nt;
  const int b0 = (int)((long long)nbra * split / nsplit), b1 = (int)((long long)nbra * (split + 1) / nsplit);
  const double* rp = v.prec + (size_t)kRLen * Pp;
  const int pos = grp * 32 + lane;
  const bool on = pos < v.nket;
  const int kid = on ? v.kperm[pos] : 0;
  const double* rk = v.erec + (size_t)kRLen * kid;
  g3::Ket<NK> ket;
  g3::load_ket<NK>(rk, ket);
  Bra<double, NW>* bras = s_bra[wid];
  double acc = 0.0;
  for (int c0 = b0; c0 < b1; c0 += 32) {
    __syncwarp();
    const int nv = b1 - c0 < 32 ? b1 - c0 : 32;
    if (lane < nv) {
      int q = c0 + lane;
      const int kind = q & 1;
      q >>= 1;
      const double* rb = v.erec + (size_t)kRLen * (kb + q % nb);
      double g, w;
      pair_term(S, q0 + q / nb, g, w);
      Bra<double, NW>& b = bras[lane];
      if (kind == 0) build_bra_pair<2 * LE, 2 * LN, NW>(rb, rp, g, b);
      else build_bra_pair<2 * LN, 2 * LE, NW>(rp, rb, g, b);
      g3::finish_bra<NW>(b);
      b.wgt = (kind == 0 ? w : -w) * rb[kRC] * rp[kRC];
    }
    __syncwarp();
    if (on)
      for (int i = 0; i < nv; i++)
        acc = fma(bras[i].wgt, g3::fb_value<NW, NK>(bras[i], ket), acc);
  }
  if (on) Y[((long long)split * nunit + u) * v.nket + kid] = acc * rk[kRC];
}

// R1 / R2[split][Pp - Pp0][Pa][ket] for the kets of pairs P <= Pa.  Lanes take
// those kets in class order (a queue filled by ballots over the permutation).
template <int LE, int LN, int MODE>
__global__ void __launch_bounds__(32 * kWarps)
gam2_triple_kernel(DevSystem S, int Pp0, long long nunit,
                   double* __restrict__ R1, double* __restrict__ R2) {
  constexpr bool FULL = MODE == kAll;
  __shared__ int s_q[kWarps][64];
  const Gam2View v = view(S);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  // the last pairs have the most kets: take them first
  const long long u = nunit - 1 - ((long long)blockIdx.x * kWarps + wid);
  if (u < 0) return;
  const int split = blockIdx.y, nsplit = gridDim.y;
  const int Pp = Pp0 + (int)(u % (nunit / v.nPe)), Pa = (int)(u / (nunit / v.nPe));
  const long long row = (long long)(Pp - Pp0) * v.nPe + Pa;
  const int ka = v.kofs[Pa], na = v.kofs[Pa + 1] - ka, kmax = v.kofs[Pa + 1];
  const int ng = S.ngtg, nbra = na * ng * ng;
  const int b0 = (int)((long long)nbra * split / nsplit), b1 = (int)((long long)nbra * (split + 1) / nsplit);
  const double* rp = v.prec + (size_t)kRLen * Pp;
  const double* ep = v.pgrad + (size_t)kGLen * Pp;
  const double rpm = 1.0 / S.pmass;
  int* que = s_q[wid];
  int nq = 0;
  const long long o = ((long long)split * nunit + row) * v.nket;
  int turn = 0;   // the warps of grid z take every gridDim.z-th 32 kets
  for (int p0 = 0; p0 < v.nket || nq > 0;) {
    while (nq < 32 && p0 < v.nket) {
      const int pos = p0 + lane;
      const int kid = pos < v.nket ? v.kperm[pos] : kmax;
      const bool in = kid < kmax;
      const unsigned m = __ballot_sync(0xffffffffu, in);
      if (in) que[nq + __popc(m & ((1u << lane) - 1u))] = kid;
      nq += __popc(m);
      p0 += 32;
      __syncwarp();
    }
    const int nv = nq < 32 ? nq : 32;
    const bool mine = turn++ % gridDim.z == blockIdx.z;
    if (lane < nv && mine) {
      const int kid = que[lane];
      const double* r2 = v.erec + (size_t)kRLen * kid;
      const double* e2 = v.egrad + (size_t)kGLen * kid;
      double s1 = 0.0, s2 = 0.0;
      for (int b = b0; b < b1; b++) {
        const int kl = b % (ng * ng), k = kl / ng, l = kl - k * ng, ua = b / (ng * ng);
        const double* r1 = v.erec + (size_t)kRLen * (ka + ua);
        const double* e1 = v.egrad + (size_t)kGLen * (ka + ua);
        double x1, x2;
        three_body<LE, LN, MODE>(r1, r2, rp, e1, e2, ep, S.ggem[k], S.ggem[l], S.nat, S.cat,
                                 S.zan, rpm, &x1, &x2);
        const double w = S.bgem[k] * S.bgem[l] * r1[kRC];
        if (FULL) s1 = fma(w, x1, s1);
        s2 = fma(w, x2, s2);
      }
      const double c = r2[kRC] * rp[kRC];
      if (FULL) R1[o + kid] = s1 * c;
      R2[o + kid] = s2 * c;
    }
    __syncwarp();
    const int rest = nq - nv;   // < 32
    const int mv = lane < rest ? que[nv + lane] : 0;
    __syncwarp();
    if (lane < rest) que[lane] = mv;
    __syncwarp();
    nq = rest;
  }
}

// out[row][P] = sum_split sum_{ket of P} in[split][row][ket]; lower = only P <= row % nPe.
// lanes (a power of two) threads share a sum over the splits: with one, a small
// system's 64 splits were 57 us of dependent adds (examples/xchf; 6 so).
__global__ void gam2_contract_kernel(DevSystem S, long long nrow, int nsplit, int lower, int lanes,
                                     const double* __restrict__ in, double* __restrict__ out) {
  const int nPe = S.nebf * (S.nebf + 1) / 2, nket = S.g3_nket;
  const int* kofs = S.g3i + 2 * nket;
  const long long n = nrow * nPe * lanes;
  const int sub = threadIdx.x & (lanes - 1);
  // (a warp's threads stay in the loop together)
  for (long long u0 = blockIdx.x * (long long)blockDim.x; u0 < n; u0 += (long long)gridDim.x * blockDim.x) {
    const long long t = (u0 + threadIdx.x) / lanes;
    const long long row = t / nPe;
    const int P = (int)(t - row * nPe);
    const bool on = row < nrow && !(lower && P > (int)(row % nPe));
    double s = 0.0;
    if (on)
      for (int q = sub; q < nsplit; q += lanes) {
        const double* x = in + ((long long)q * nrow + row) * nket;
        for (int k = kofs[P]; k < kofs[P + 1]; k++) s += x[k];
      }
    for (int o = lanes >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (on && sub == 0) out[t] = s;
  }
}

void contract(const DevSystem& S, long long nrow, int nsplit, int lower, const double* in,
              double* out, cudaStream_t s) {
  const int nPe = S.nebf * (S.nebf + 1) / 2;
  int lanes = 1;
  while (lanes < 32 && 2 * lanes < nsplit) lanes *= 2;
  const unsigned nb = (unsigned)std::min<long long>((nrow * nPe * lanes + 127) / 128, 152 * 16);
  gam2_contract_kernel<<<nb, 128, 0, s>>>(S, nrow, nsplit, lower, lanes, in, out);
}

// The contracted canonical arrays onto the packed order: block y is the
// (Pp - Pp0)-th proton pair, written at (ip,jp) and (jp,ip) (ONE: at the
// single slice x1 / x2 point at).
template <bool RX, bool ONE>
__global__ void gam2_expand_kernel(int ne, int np, int Pp0, const double* __restrict__ Yc,
                                   const double* __restrict__ R1, const double* __restrict__ R2,
                                   const double* __restrict__ W, const double* __restrict__ H,
                                   double* __restrict__ x1, double* __restrict__ x2) {
  const int n2 = ne * ne, nPe = ne * (ne + 1) / 2;
  const long long n4 = (long long)n2 * n2;
  const int Pl = blockIdx.y;
  int ip, jp;
  unpair(Pp0 + Pl, ip, jp);
  const long long oa = ONE ? 0 : ((long long)ip * np + jp) * n4;
  const long long ob = ONE ? 0 : ((long long)jp * np + ip) * n4;
  const long long base = (long long)Pl * nPe * nPe;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n4;
       t += (long long)gridDim.x * blockDim.x) {
    const int e1 = (int)(t / n2), e2 = (int)(t - (long long)e1 * n2);
    const int P1 = g3::pair_index(e1 / ne, e1 % ne), P2 = g3::pair_index(e2 / ne, e2 % ne);
    const int a = P1 > P2 ? P1 : P2, b = P1 > P2 ? P2 : P1;
    const long long ab = base + (long long)a * nPe + b, ba = base + (long long)b * nPe + a;
    double v1;
    if (RX) {
      v1 = Yc[base + (long long)P1 * nPe + P2];
    } else {
      const double* w = W + (long long)(Pp0 + Pl) * nPe;
      v1 = R1[ab] + 0.5 * ((Yc[ab] + Yc[ba]) + (H[a] * w[b] + H[b] * w[a]));
    }
    const double v2 = R2[ab];
    x1[oa + t] = v1;
    x2[oa + t] = v2;
    if (!ONE && oa != ob) {
      x1[ob + t] = v1;
      x2[ob + t] = v2;
    }
  }
}

// ---- sizes --------------------------------------------------------------------
// Warps wanted on the GPU: 16 for each of the 152 SMs keep the FP64 pipes
// busy; fewer (Pp, P) pairs than that are split over their primitives.
constexpr long long kWantWarps = 152 * 16;
constexpr size_t kChunkDoubles = (size_t)1 << 25;   // scratch aim of a chunk: 256 MiB

struct Plan {
  int nPe, nPp, nket, chunk, spY, spR;
  size_t fac, per;   // W and H; doubles per proton pair of a chunk
};

// max_prim: primitive pairs of the largest contracted pair (bounds the splits)
Plan make_plan(int ne, int np, int nket, int max_prim, int ng, bool rx, int nPp_want) {
  Plan p;
  p.nPe = ne * (ne + 1) / 2;
  p.nPp = np * (np + 1) / 2;
  p.nket = nket;
  const long long units = (long long)nPp_want * p.nPe;
  const long long groups = (nket + 31) / 32;
  auto split = [](long long want, long long most) {
    return (int)std::max(1LL, std::min(std::min(want, most), 64LL));
  };
  const long long nt = ng + ng * (ng + 1) / 2;
  p.spY = split((kWantWarps + units * groups - 1) / (units * groups), (2 * max_prim * nt + 31) / 32);
  p.spR = split((kWantWarps + units - 1) / units, (long long)max_prim * ng * ng);
  p.fac = (size_t)p.nPp * p.nPe + p.nPe;
  const size_t row = (size_t)p.nPe * nket;
  p.per = row * ((size_t)p.spY + (rx ? 1 : 2) * (size_t)p.spR) + 3 * (size_t)p.nPe * p.nPe;
  size_t c = kChunkDoubles / p.per;
  p.chunk = (int)std::max<size_t>(1, std::min<size_t>(std::min<size_t>(c, (size_t)nPp_want), 32768));
  return p;
}

template <int LE, int LN, bool RX>
cudaError_t build_t(const DevSystem& S, const Plan& p, double* scratch, int Pp0, int nPp, bool one,
                    double* x1, double* x2, cudaStream_t s) {
  double* W = scratch;
  double* H = W + (size_t)p.nPp * p.nPe;
  double* buf = W + p.fac;
  const size_t row = (size_t)p.nPe * p.nket;
  const int ne = S.nebf, np = S.npbf;
  for (int c0 = Pp0; c0 < Pp0 + nPp; c0 += p.chunk) {
    const int nc = std::min(p.chunk, Pp0 + nPp - c0);
    const long long units = (long long)nc * p.nPe;
    double* Y = buf;
    double* R1 = Y + row * p.spY * nc;
    double* R2 = RX ? R1 : R1 + row * p.spR * nc;
    double* Yc = R2 + row * p.spR * nc;
    double* R1c = Yc + (size_t)units * p.nPe;
    double* R2c = R1c + (size_t)units * p.nPe;
    const unsigned nb = (unsigned)((units + kWarps - 1) / kWarps);
    // too few warps even with a bra each: the 32-ket turns of one over several
    // (examples/xchf, 1344 warps of three turns: 283 us, 150 so)
    const unsigned nz = units * p.spR < kWantWarps ? std::min((p.nket + 31) / 32, 4) : 1;
    gam2_triple_kernel<LE, LN, RX ? kCoulomb12 : kAll><<<dim3(nb, p.spR, nz), 32 * kWarps, 0, s>>>(
        S, c0, units, R1, R2);
    gam2_pair_kernel<LE, LN, RX><<<dim3(nb, (p.nket + 31) / 32, p.spY), 32 * kWarps, 0, s>>>(
        S, c0, units, Y);
    contract(S, units, p.spY, 0, Y, Yc, s);
    if (!RX) contract(S, units, p.spR, 1, R1, R1c, s);
    contract(S, units, p.spR, 1, R2, R2c, s);
    const long long n4 = (long long)ne * ne * ne * ne;
    const dim3 eg((unsigned)std::min<long long>((n4 + 255) / 256, 1024), (unsigned)nc);
    if (one)
      gam2_expand_kernel<RX, true><<<eg, 256, 0, s>>>(ne, np, c0, Yc, R1c, R2c, W, H, x1, x2);
    else
      gam2_expand_kernel<RX, false><<<eg, 256, 0, s>>>(ne, np, c0, Yc, R1c, R2c, W, H, x1, x2);
  }
  return cudaGetLastError();
}

template <bool RX>
cudaError_t build(const DevSystem& S, const Plan& p, double* scratch, int Pp0, int nPp, bool one,
                  double* x1, double* x2, cudaStream_t s) {
  const int LN = S.lmax_p == 0 ? 0 : 2;
  switch (S.lmax_e * 3 + LN) {
    case 0: return build_t<0, 0, RX>(S, p, scratch, Pp0, nPp, one, x1, x2, s);
    case 2: return build_t<0, 2, RX>(S, p, scratch, Pp0, nPp, one, x1, x2, s);
    case 3: return build_t<1, 0, RX>(S, p, scratch, Pp0, nPp, one, x1, x2, s);
    case 5: return build_t<1, 2, RX>(S, p, scratch, Pp0, nPp, one, x1, x2, s);
    case 6: return build_t<2, 0, RX>(S, p, scratch, Pp0, nPp, one, x1, x2, s);
    case 8: return build_t<2, 2, RX>(S, p, scratch, Pp0, nPp, one, x1, x2, s);
    default: return cudaErrorInvalidValue;
  }
}

Plan plan_of(const DevSystem& S, int rx, int nPp_want) {
  return make_plan(S.nebf, S.npbf, S.g3_nket, S.g3_max_prim, S.ngtg, rx != 0, nPp_want);
}

// W3 on the packed order from the canonical overlaps (grid y: proton pairs of a chunk)
__global__ void overlap_expand_kernel(int ne, int np, int Pp0, const double* __restrict__ R2,
                                      double* __restrict__ W3) {
  const int n2 = ne * ne, nPe = ne * (ne + 1) / 2;
  const long long n4 = (long long)n2 * n2;
  int ip, jp;
  unpair(Pp0 + blockIdx.y, ip, jp);
  const double* r = R2 + (long long)blockIdx.y * nPe * nPe;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n4;
       t += (long long)gridDim.x * blockDim.x) {
    const int e1 = (int)(t / n2), e2 = (int)(t - (long long)e1 * n2);
    const int P1 = g3::pair_index(e1 / ne, e1 % ne), P2 = g3::pair_index(e2 / ne, e2 % ne);
    const double v = P1 > P2 ? r[(long long)P1 * nPe + P2] : r[(long long)P2 * nPe + P1];
    W3[((long long)ip * np + jp) * n4 + t] = v;
    W3[((long long)jp * np + ip) * n4 + t] = v;
  }
}

// W1 = W / 2 on [ip][jp][i][j] and the core Hamiltonian on [i][j]
__global__ void factor_expand_kernel(int ne, int np, const double* __restrict__ W,
                                     const double* __restrict__ H, double* __restrict__ W1,
                                     double* __restrict__ hc) {
  const int n2 = ne * ne, nPe = ne * (ne + 1) / 2;
  const long long total = (long long)np * np * n2;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    const int e = (int)(t % n2), pp = (int)(t / n2);
    const int P = g3::pair_index(e / ne, e % ne);
    W1[t] = 0.5 * W[(long long)g3::pair_index(pp / np, pp % np) * nPe + P];
    if (hc && pp == 0) hc[e] = H[P];
  }
}

template <int LE, int LN>
void overlap_t(const DevSystem& S, const Plan& p, int c0, long long units, double* R2, cudaStream_t s) {
  gam2_triple_kernel<LE, LN, kOverlap><<<dim3((unsigned)((units + kWarps - 1) / kWarps), p.spR),
                                         32 * kWarps, 0, s>>>(S, c0, units, R2, R2);
}

}  // namespace

cudaError_t launch_gam3_factors(const DevSystem& S, double* scratch, const double* w3_in,
                                double* W1, double* W3, double* hc, cudaStream_t s) {
  const int ne = S.nebf, np = S.npbf;
  const long long n4 = (long long)ne * ne * ne * ne;
  cudaError_t e = launch_gam2_prepare(S, scratch, s);
  if (e != cudaSuccess) return e;
  const Plan p = plan_of(S, 1, np * (np + 1) / 2);
  double* W = scratch;
  const long long n1 = (long long)np * np * ne * ne;
  factor_expand_kernel<<<(unsigned)std::min<long long>((n1 + 255) / 256, 152 * 16), 256, 0, s>>>(
      ne, np, W, W + (size_t)p.nPp * p.nPe, W1, hc);
  if (w3_in)
    return cudaMemcpyAsync(W3, w3_in, sizeof(double) * n4 * np * np, cudaMemcpyDeviceToDevice, s);
  double* buf = W + p.fac;
  for (int c0 = 0; c0 < p.nPp; c0 += p.chunk) {
    const int nc = std::min(p.chunk, p.nPp - c0);
    const long long units = (long long)nc * p.nPe;
    double* R2 = buf;
    double* R2c = R2 + (size_t)p.nPe * p.nket * p.spR * nc;
    switch (S.lmax_e * 3 + (S.lmax_p == 0 ? 0 : 2)) {
      case 0: overlap_t<0, 0>(S, p, c0, units, R2, s); break;
      case 2: overlap_t<0, 2>(S, p, c0, units, R2, s); break;
      case 3: overlap_t<1, 0>(S, p, c0, units, R2, s); break;
      case 5: overlap_t<1, 2>(S, p, c0, units, R2, s); break;
      case 6: overlap_t<2, 0>(S, p, c0, units, R2, s); break;
      case 8: overlap_t<2, 2>(S, p, c0, units, R2, s); break;
      default: return cudaErrorInvalidValue;
    }
    contract(S, units, p.spR, 1, R2, R2c, s);
    overlap_expand_kernel<<<dim3((unsigned)std::min<long long>((n4 + 255) / 256, 1024), nc), 256, 0, s>>>(
        ne, np, c0, R2c, W3);
  }
  return cudaGetLastError();
}

size_t gam2_scratch_doubles(const DevSystem& S, int rx, int nPp_want) {
  const Plan p = plan_of(S, rx, nPp_want);
  return p.fac + p.per * (size_t)p.chunk;
}

size_t gam2_scratch_bound(int ne, int np, int nket, int max_prim, int ng) {
  const Plan p = make_plan(ne, np, nket, max_prim, ng, false, np * (np + 1) / 2);
  return p.fac + p.per * (size_t)p.chunk;
}

size_t gam3_factors_scratch(int ne, int np, int nket, int max_prim, int ng, bool w3_given) {
  const Plan p = make_plan(ne, np, nket, max_prim, ng, true, np * (np + 1) / 2);
  return w3_given ? p.fac : p.fac + p.per * (size_t)p.chunk;
}

cudaError_t launch_gam2_prepare(const DevSystem& S, double* scratch, cudaStream_t s) {
  if (S.nebf < 1 || S.npbf < 1 || !S.g3i || !S.g3rec || !S.g3grad) return cudaErrorInvalidValue;
  const int nPe = S.nebf * (S.nebf + 1) / 2, nPp = S.npbf * (S.npbf + 1) / 2;
  double* W = scratch;
  double* H = W + (size_t)nPp * nPe;
  const long long warps = (long long)nPp * nPe + nPe;
  const unsigned nb = (unsigned)((warps + kWarps - 1) / kWarps);
  switch (S.lmax_e) {
    case 0: gam2_factor_kernel<0><<<nb, 32 * kWarps, 0, s>>>(S, nPp, W, H); break;
    case 1: gam2_factor_kernel<1><<<nb, 32 * kWarps, 0, s>>>(S, nPp, W, H); break;
    default: gam2_factor_kernel<2><<<nb, 32 * kWarps, 0, s>>>(S, nPp, W, H); break;
  }
  return cudaGetLastError();
}

cudaError_t launch_gam2_build(const DevSystem& S, int rx, double* scratch, double* x1, double* x2,
                              cudaStream_t s) {
  const int nPp = S.npbf * (S.npbf + 1) / 2;
  const Plan p = plan_of(S, rx, nPp);
  cudaError_t e = launch_gam2_prepare(S, scratch, s);
  if (e != cudaSuccess) return e;
  return rx ? build<true>(S, p, scratch, 0, nPp, false, x1, x2, s)
            : build<false>(S, p, scratch, 0, nPp, false, x1, x2, s);
}

cudaError_t launch_gam2_slice(const DevSystem& S, int Pp, double* scratch, double* x1, double* x2,
                              cudaStream_t s) {
  return build<false>(S, plan_of(S, 0, 1), scratch, Pp, 1, true, x1, x2, s);
}

}  // namespace neoxc
