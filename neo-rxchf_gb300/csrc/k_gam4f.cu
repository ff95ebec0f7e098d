// k_gam4f.cu -- factorised gam_4 Fock build for sm_103a.
//
// Same results as the fused element-wise GAM4_DSCF (gam4_DSCF_OMP.f:2-320,
// element from gam_4_OMP.f:712-1192) at O(nebf^4 npbf^2 + nebf^5) work
// instead of O(nebf^8 npbf^2), for the reference's actual inputs: GAM_2s
// pair-symmetric, gs(p; ab; cd) = gs(p; cd; ab) (GAM2_IC1 stores
// (x12+x21)/2, gam2_IC1_OMP.f:141-176), and GAM_ee symmetric under pair
// exchange, (ab|cd) = (cd|ab) (an ERI tensor).
//
// Derivation.  With k_m = je_sigma(m) the element is
//   gam4 = 1/16 sum_sigma c_sigma 1/6 sum_{splits (ab|cd)} 1/2
//          ee(ie_c k_c | ie_d k_d) gs(p; ie_a k_a; ie_b k_b),
// c_sigma = 16 (-1/2)^(4 - cycles(sigma)).  Summed against
// DP(p) DE(ie1,je1)..DE(ie4,je4), relabelling the four electrons maps every
// split onto (12|34) without changing c_sigma (a class function), so
//   E = 1/32 sum_sigma c_sigma sum_{i1..i4} G'(i1,i_s1,i2,i_s2) E'(i3,i_s3,i4,i_s4)
// with G = sum_p DP(p) gs(p) and the ket legs carried to bra labels by DE:
//   T'(a,x,c,y) = sum_{b,d} T(a,b,c,d) DE(x,b) DE(y,d).
// E is linear in DP and quartic in DE, and the same relabelling symmetry
// makes the reference's Fock contractions (4 DP DE^3 gam4 into focke(ie1,je1),
// DE^4 gam4 into fockp) exactly its gradients:
//   fockp(p)  = <gs(p), W>,   W = back-transform of W' = dE/dG',
//   focke(x,b)= sum_{a,c,y} [W'+W'^swap](a,x,c,y) H_G(a,b,c,y)
//             + [V'+V'^swap](a,x,c,y) H_E(a,b,c,y),   V' = dE/dE',
// H_T(a,b,c,y) = sum_d T(a,b,c,d) DE(y,d) the half-transformed tensor and
// ^swap the pair exchange (a,x,c,y) -> (c,y,a,x).  E = sum_p DP(p) fockp(p).
//
// dE/dG' at (a,x,c,y) is, per sigma, either a gather of E' with permuted
// legs, a Kronecker delta times a partial trace (one index pair of E'
// contracted), or two deltas times a full double trace; the 24 cases are the
// switch table sig_code below (the same table serves dE/dE' with G').
//
// Every 4-index tensor is stored C-order [l0][l1][l2][l3] (the layout of
// GAM_ee = pack_4D(je2,ie2,je1,ie1) and of one proton pair of GAM_2s =
// index_GAM_2PK), so a table read is a linear offset.  All arithmetic is
// FP64; table reads pass through the reference's underflow (|x|<1e-100 -> 0).
#include <utility>

#include "neoxc_internal.h"
#include "tc_gemm.cuh"

namespace neoxc {
namespace {

// |x| < 1e-100 -> 0 (underflow.f:2-11), compared as integers: an FP64 compare
// would cost as much as the FMA that uses the element
__device__ __forceinline__ double flush(double x) {
  return (__double_as_longlong(x) & 0x7fffffffffffffffLL) < 0x2b2bff2ee48e0530LL ? 0.0 : x;
}

// ---- 3. partial and double traces ------------------------------------------
// leg pairs (0,1) (0,2) (0,3) (1,2) (1,3) (2,3) -> 0..5
__host__ __device__ constexpr int pair_leg(int p, int which) {
  return which == 0 ? (p < 3 ? 0 : (p < 5 ? 1 : 2))
                    : (p < 3 ? p + 1 : (p < 5 ? p - 1 : 3));
}

__device__ __forceinline__ long long idx4(int n, int l0, int l1, int l2, int l3) {
  return ((long long)((long long)l0 * n + l1) * n + l2) * n + l3;
}

// PT[t][p][u][v] = sum_z T_t with the legs of pair p at z and the other two
// legs (in leg order) at u, v.  blockIdx.y picks the tensor.
__global__ void traces_kernel(int n, const double* __restrict__ T0,
                              const double* __restrict__ T1,
                              double* __restrict__ PT) {
  const double* T = blockIdx.y ? T1 : T0;
  double* out = PT + (size_t)blockIdx.y * 6 * n * n;
  const int total = 6 * n * n;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += gridDim.x * blockDim.x) {
    const int p = e / (n * n), r = e - p * n * n, u = r / n, v = r - u * n;
    const int k = pair_leg(p, 0), m = pair_leg(p, 1);
    int l[4];
    int q = 0;
    double acc = 0.0;
    for (int z = 0; z < n; z++) {
      q = 0;
      for (int g = 0; g < 4; g++) {
        if (g == k || g == m) l[g] = z;
        else l[g] = (q++ == 0) ? u : v;
      }
      acc += T[idx4(n, l[0], l[1], l[2], l[3])];
    }
    out[e] = acc;
  }
}

// ST[t][0..2] = double traces (01)(23), (02)(13), (03)(12) = traces of
// PT[t][0], PT[t][1], PT[t][2].  One warp per tensor.
__global__ void dtraces_kernel(int n, const double* __restrict__ PT,
                               double* __restrict__ ST) {
  const int t = threadIdx.x / 32, lane = threadIdx.x & 31;
  if (t >= 2) return;
  for (int s = 0; s < 3; s++) {
    const double* P = PT + ((size_t)t * 6 + s) * n * n;
    double acc = 0.0;
    for (int u = lane; u < n; u += 32) acc += P[u * n + u];
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if (lane == 0) ST[t * 4 + s] = acc;
  }
}

// ---- 4. dE/dG' and dE/dE' --------------------------------------------------
// Term t of the 24 permutations, for the gradient with respect to the tensor
// on slots (0,1) at output legs o = (a,x,c,y).  Bits: [0:2) k with
// coefficient 1/2 (-1/2)^k (= c_sigma/32); [2:6) Kronecker deltas between
// output legs (0,1), (2,3), (0,3), (1,2); [6:8) kind (0 gather, 1 partial
// trace, 2 double trace); [8:11) trace id (leg pair, or pairing for kind
// 2); then for legs 0..3 of the other tensor, 3 bits each: the output leg
// that supplies its value, 7 = traced.  Derived by following each label of
// the permutation through the two tensors' legs; by the exchange symmetry of
// slots (0,1) <-> (2,3) the same table gives the gradient with respect to
// the tensor on slots (2,3).
__device__ __forceinline__ int sig_code(int t) {
  switch (t) {
    case 0: return 8386700;   // sigma = id:          +1/2,  d01 d23, (01)(23)
    case 1: return 8387213;   // -1/4, d01 d23, (03)(12)
    case 2: return 8297797;   // -1/4, d01, PT(23) of legs (y,c)
    case 3: return 3136326;   // +1/8, d01, PT(12) of legs (y,c)
    case 4: return 7780934;   // +1/8, d01, PT(03) of legs (c,y)
    case 5: return 2619461;   // -1/4, d01, PT(01) of legs (y,c)
    case 6: return 8386737;   // -1/4, d03 d12, (01)(23)
    case 7: return 8387250;   // +1/8, d03 d12, (03)(12)
    case 8: return 8265058;   // +1/8, d12, PT(23) of legs (y,a)
    case 9: return 1039203;   // -1/16, d12, PT(12) of legs (y,a)
    case 10: return 7748195;  // -1/16, d12, PT(03) of legs (a,y)
    case 11: return 522338;   // +1/8, d12, PT(01) of legs (y,a)
    case 12: return 8293714;  // +1/8, d03, PT(23) of legs (x,c)
    case 13: return 3132243;  // -1/16, d03, PT(12) of legs (x,c)
    case 14: return 8260937;  // -1/4, d23, PT(23) of legs (x,a)
    case 15: return 1035082;  // +1/8, d23, PT(12) of legs (x,a)
    case 16: return 2492418;  // +1/8, gather (x,a,y,c)
    case 17: return 428035;   // -1/16, gather (x,c,y,a)
    case 18: return 7518803;  // -1/16, d03, PT(03) of legs (c,x)
    case 19: return 2357330;  // +1/8, d03, PT(01) of legs (x,c)
    case 20: return 7486026;  // +1/8, d23, PT(03) of legs (a,x)
    case 21: return 260169;   // -1/4, d23, PT(01) of legs (x,a)
    case 22: return 2234371;  // -1/16, gather (y,a,x,c)
    case 23: return 169986;   // +1/8, gather (y,c,x,a)
    default: return 0;
  }
}

__device__ __forceinline__ double sig_coef(int k) {
  return k == 0 ? 0.5 : (k == 1 ? -0.25 : (k == 2 ? 0.125 : -0.0625));
}

// dE/d(the tensor on slots 0, 1) at legs l, from the other tensor T, its leg-pair
// traces P and its double traces S (sig_code's table)
__device__ __forceinline__ double grad_term(int n, const int* l, const double* __restrict__ T,
                                            const double* __restrict__ P, const double* S) {
  double acc = 0.0;
#pragma unroll
  for (int t = 0; t < 24; t++) {
    const int code = sig_code(t);
    const int dm = (code >> 2) & 15;
    if ((dm & 1) && l[0] != l[1]) continue;
    if ((dm & 2) && l[2] != l[3]) continue;
    if ((dm & 4) && l[0] != l[3]) continue;
    if ((dm & 8) && l[1] != l[2]) continue;
    const int kind = (code >> 6) & 3, tid = (code >> 8) & 7;
    const int s0 = (code >> 11) & 7, s1 = (code >> 14) & 7,
              s2 = (code >> 17) & 7, s3 = (code >> 20) & 7;
    double v;
    if (kind == 0) {
      v = __ldg(T + idx4(n, l[s0], l[s1], l[s2], l[s3]));
    } else if (kind == 1) {
      int uv[2], q = 0;
      if (s0 != 7) uv[q++] = l[s0];
      if (s1 != 7) uv[q++] = l[s1];
      if (s2 != 7) uv[q++] = l[s2];
      if (s3 != 7) uv[q++] = l[s3];
      v = __ldg(P + ((size_t)tid * n + uv[0]) * n + uv[1]);
    } else {
      v = S[tid];
    }
    acc = fma(sig_coef(code & 3), v, acc);
  }
  return acc;
}

// Tensor-core build, Wp = dE/dG' from (E', PT_E, ST_E) and Vp = dE/dE' from (G',
// PT_G, ST_G), in two kernels: off every delta an element is four gathers and
// four FMAs; the 4 n^3 elements on a delta are done over by gam4f_delta_kernel.
// (In one kernel the rare delta terms, up to twenty of them one lane at a time,
// filled the FP64 pipe of whole warps: n = 48, 472 us; 146 us so.)
// grid (n, ceil(n/4), 2 * kGradSplit): a CTA owns (x, four consecutive a, a
// share of c), a thread (a, y): two of the gathers read the four a of one
// 32-byte sector in one request, the other two the four c of one.
constexpr int kGradSplit = 4;
__global__ void __launch_bounds__(256)
gam4f_gather_kernel(int n, const double* __restrict__ Ep, const double* __restrict__ Gp,
                    double* __restrict__ Wp, double* __restrict__ Vp) {
  const int which = blockIdx.z / kGradSplit, part = blockIdx.z % kGradSplit;
  const double* T = which ? Gp : Ep;   // the other tensor
  double* out = which ? Vp : Wp;
  const int x = blockIdx.x, a = blockIdx.y * 4 + (threadIdx.x & 3), y = threadIdx.x >> 2;
  if (a >= n || y >= n) return;
  const int nb = (n + 3) / 4, c1 = min(n, nb * (part + 1) / kGradSplit * 4);
#pragma unroll 4
  for (int c = nb * part / kGradSplit * 4; c < c1; c++) {
    double acc = 0.125 * __ldg(T + idx4(n, x, a, y, c));   // grad_term's order
    acc = fma(-0.0625, __ldg(T + idx4(n, x, c, y, a)), acc);
    acc = fma(-0.0625, __ldg(T + idx4(n, y, a, x, c)), acc);
    out[idx4(n, a, x, c, y)] = fma(0.125, __ldg(T + idx4(n, y, c, x, a)), acc);
  }
}

// grid (x, 4 deltas, 2 tensors); an element on several deltas is written
// with the same value by each
__global__ void gam4f_delta_kernel(int n, const double* __restrict__ Ep,
                                   const double* __restrict__ Gp, const double* __restrict__ PT,
                                   const double* __restrict__ ST, double* __restrict__ Wp,
                                   double* __restrict__ Vp) {
  const int which = blockIdx.z, d = blockIdx.y;
  const double* T = which ? Gp : Ep;
  const double* P = PT + (size_t)(which ? 0 : 1) * 6 * n * n;
  const double* S = ST + (which ? 0 : 4);
  double* out = which ? Vp : Wp;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n * n * n; t += gridDim.x * blockDim.x) {
    const int u = t / (n * n), v = t / n % n, w = t % n;
    // legs (0,1), (2,3), (0,3), (1,2) equal
    const int l[4] = {u, d == 0 ? u : v, d == 1 ? w : (d == 3 ? v : (d == 0 ? v : w)),
                      d == 2 ? u : w};
    out[idx4(n, l[0], l[1], l[2], l[3])] = grad_term(n, l, T, P, S);
  }
}

// ---- 5. fockp(p) = <GAM_2s(p), W>;  E = sum_p DP(p) fockp(p) ----------------
constexpr int kDotTB = 256;
constexpr int kDotChunk = 16384;   // elements per CTA

__device__ __forceinline__ double block_sum(double v, double* sw) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int w = threadIdx.x / 32, lane = threadIdx.x & 31;
  __syncthreads();
  if (lane == 0) sw[w] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x < 32) {
    t = threadIdx.x < (blockDim.x + 31) / 32 ? sw[threadIdx.x] : 0.0;
    for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
  }
  return t;   // valid in thread 0
}

// One CTA, a warp per p: fockp(ip,jp) (+)= sum_chunk part; E = sum_p DP(p) *
// (new part).
__global__ void __launch_bounds__(1024)
fockp_reduce_kernel(int np, int nchunk, const double* __restrict__ part,
                    const double* __restrict__ DP, int accumulate,
                    double* __restrict__ fockp, double* __restrict__ E) {
  __shared__ double sw[32];
  const int lane = threadIdx.x & 31;
  double e = 0.0;
  for (int p = threadIdx.x >> 5; p < np * np; p += 32) {
    double s = 0.0;
    for (int c = lane; c < nchunk; c += 32) s += part[(long long)p * nchunk + c];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (lane == 0) {
      const int ip = p / np, jp = p - ip * np;
      const int f = ip + np * jp;                  // column-major fockp(ip,jp)
      fockp[f] = accumulate ? fockp[f] + s : s;
      e = fma(DP[f], s, e);
    }
  }
  const double t = block_sum(e, sw);
  if (threadIdx.x == 0) *E = t;
}

// ---- mixed-precision forms of the two GAM_2s passes (tensor-core build) ----
// The FP64 forms above issue one FP64 FMA per GAM_2s element, which on this
// GPU (FP64 at 1/64 of the FP32 rate) costs more than reading the element
// from HBM.  These narrow each element to FP32 on the integer pipes
// (tc::narrow_f64) and multiply in FP32; partial sums are FP32 over at most
// kMixChunk terms and FP64 beyond, so the result carries ~1e-7 relative
// rounding (the GAM_2s values themselves are FP64 in memory).  GAM_2s is
// read once per pass with evict-first loads (__ldcs), which leaves L2 to
// the re-read operands (DP, the narrowed W).
constexpr int kMixChunk = 64;
constexpr int kDpShared = 12288;   // np^2 up to this: DP staged in shared memory

// G[r] = sum_p DP(p) GAM_2s[p][r]  (DP column-major, p = ip*np + jp as above);
// vec: two consecutive elements per thread (16-byte loads), for a 16-byte
// aligned table whose rows p * n4 stay so, i.e. n4 even.
__global__ void dp_contract_mixed_kernel(long long n4, int np, bool vec, const double* __restrict__ g2s,
                         const double* __restrict__ DP, double* __restrict__ G) {
  extern __shared__ float sdp[];   // [np*np] in the loop order of g2s, if staged
  const int np2 = np * np;
  const bool staged = np2 <= kDpShared;
  if (staged)
    for (int p = threadIdx.x; p < np2; p += blockDim.x) {
      const int ip = p / np, jp = p - ip * np;
      sdp[p] = tc::narrow_f64(DP[ip + np * jp]);
    }
  __syncthreads();
  const long long nv = vec ? n4 / 2 : n4;
  // one item a thread: a grid-strided loop of four and a quarter rounds left
  // the last one three quarters empty
  const long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (v < nv) {
    double acc0 = 0.0, acc1 = 0.0;
    for (int p0 = 0; p0 < np2; p0 += kMixChunk) {
      const int p1 = p0 + kMixChunk < np2 ? p0 + kMixChunk : np2;
      float a0 = 0.0f, a1 = 0.0f;
      if (!vec) {
#pragma unroll 8
        for (int p = p0; p < p1; p++) {
          const float d = staged ? sdp[p] : tc::narrow_f64(DP[(p / np) + np * (p % np)]);
          a0 = fmaf(d, tc::narrow_f64(__ldcs(g2s + (long long)p * n4 + v)), a0);
        }
      } else {
#pragma unroll 16
        for (int p = p0; p < p1; p++) {
          const float d = staged ? sdp[p] : tc::narrow_f64(DP[(p / np) + np * (p % np)]);
          const double2 g = __ldcs(reinterpret_cast<const double2*>(g2s + (long long)p * n4) + v);
          a0 = fmaf(d, tc::narrow_f64(g.x), a0);
          a1 = fmaf(d, tc::narrow_f64(g.y), a1);
        }
      }
      acc0 += (double)a0;
      acc1 += (double)a1;
    }
    if (!vec) {
      G[v] = acc0;
    } else {
      G[2 * v] = acc0;
      G[2 * v + 1] = acc1;
    }
  }
}

// Wf[r] = narrow_f64(W[r])
__global__ void narrow_kernel(long long n, const double* __restrict__ in,
                              float* __restrict__ out) {
  for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r < n;
       r += (long long)gridDim.x * blockDim.x)
    out[r] = tc::narrow_f64(in[r]);
}

// part[p*nchunk + chunk] = sum_{r in chunk} GAM_2s[p][r] Wf[r], FP32
// products; each thread sums its kDotChunk / kDotTB (= kMixChunk) terms in
// FP32, the block in FP64.  Wf: W narrowed once (narrow_kernel), so the
// np^2 re-reads of it come from L2 at half the bytes.
// A CTA takes kDotP consecutive p (grid (nchunk, ceil(np^2 / kDotP))) so
// that each Wf element it loads serves kDotP products.
static_assert(kDotChunk / kDotTB == kMixChunk, "one FP32 partial sum per thread");
constexpr int kDotP = 2, kDotBatch = 8;
__global__ void __launch_bounds__(kDotTB)
fockp_dot_mixed_kernel(long long n4, int nchunk, int np2,
                       const double* __restrict__ g2s,
                       const float* __restrict__ Wf,
                       double* __restrict__ part) {
  __shared__ double sw[kDotP][kDotTB / 32];
  const int p0 = blockIdx.y * kDotP;
  const int pn = np2 - p0 < kDotP ? np2 - p0 : kDotP;
  const long long base = (long long)blockIdx.x * kDotChunk;
  const long long end = base + kDotChunk < n4 ? base + kDotChunk : n4;
  float a[kDotP];
#pragma unroll
  for (int j = 0; j < kDotP; j++) a[j] = 0.0f;
  if (pn == kDotP && end - base == kDotChunk) {
    // whole chunks: kDotBatch steps' loads in flight before the first product
    const double* g = g2s + (long long)p0 * n4 + base + threadIdx.x;
    const float* w = Wf + base + threadIdx.x;
#pragma unroll 1
    for (int k = 0; k < kMixChunk; k += kDotBatch) {
      double x[kDotP][kDotBatch];
      float v[kDotBatch];
#pragma unroll
      for (int q = 0; q < kDotBatch; q++) {
#pragma unroll
        for (int j = 0; j < kDotP; j++) x[j][q] = __ldcs(g + j * n4 + (k + q) * kDotTB);
        v[q] = __ldg(w + (k + q) * kDotTB);
      }
#pragma unroll
      for (int q = 0; q < kDotBatch; q++)
#pragma unroll
        for (int j = 0; j < kDotP; j++) a[j] = fmaf(tc::narrow_f64(x[j][q]), v[q], a[j]);
    }
  } else {
    for (long long r = base + threadIdx.x; r < end; r += kDotTB) {
      const float w = __ldg(Wf + r);
#pragma unroll
      for (int j = 0; j < kDotP; j++)
        if (j < pn) a[j] = fmaf(tc::narrow_f64(__ldcs(g2s + (long long)(p0 + j) * n4 + r)), w, a[j]);
    }
  }
  // kDotP block sums in FP64: warp shuffles, then one warp over the warps
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int j = 0; j < kDotP; j++) {
    double v = (double)a[j];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) sw[j][warp] = v;
  }
  __syncthreads();
  if (warp < kDotP && warp < pn) {
    double v = lane < kDotTB / 32 ? sw[warp][lane] : 0.0;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) part[(long long)(p0 + warp) * nchunk + blockIdx.x] = v;
  }
}

// ---- FP64 build: four launches, a CTA per leg pair (a, c) --------------------
// Fixing the bra legs a and c of both electron pairs leaves an n x n tile in
// (b, d) or (x, y), on which every step but the traces is local: the sum over
// proton pairs, both one-index transforms, the gradient, the back transforms,
// the dot with GAM_2s and the focke products.  So one kernel goes from GAM_2s
// and GAM_ee to H and T', one forms the traces, one goes from T' to partial
// fockp and focke, and one adds the partials up; a tile stays in shared
// memory in between.  (As fourteen kernels over whole tensors the build at
// n = 12, np = 8 spent its time on launches and on threads that walked 64
// proton pairs or 144 partials one load at a time: 109 us; see
// launch_gam4_factored for the time now.)  At large n the n^5 products and
// the two FMAs per GAM_2s element are FP64-bound.

// out[i][j] = sum_k A(i, k) B(k, j), the products of n x n tiles below.
// AT / BT: that factor stored transposed.  Rows are ld = n | 1 doubles apart:
// with an odd pitch neither rows nor columns of a tile fall on one bank.
template <bool AT, bool BT>
__device__ __forceinline__ void tile_mul(int n, int ld, const double* A, const double* B, double* out) {
  for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
    const int i = e / n, j = e - i * n;
    double s = 0.0;
#pragma unroll 4
    for (int k = 0; k < n; k++)
      s = fma(AT ? A[k * ld + i] : A[i * ld + k], BT ? B[j * ld + k] : B[k * ld + j], s);
    out[i * ld + j] = s;
  }
}

// grid (n^2, 2): y = 0: G = sum_p DP(p) GAM_2s(p) -> HG, Gp; y = 1: GAM_ee -> HE, Ep.
// H(a,b,c,y) = sum_d T(a,b,c,d) DE(y,d), T'(a,x,c,y) = sum_b DE(x,b) H(a,b,c,y).
constexpr int kForwardThreads = 1024;
__global__ void __launch_bounds__(kForwardThreads)
gam4f_forward_kernel(int n, int np, const double* __restrict__ gee,
                     const double* __restrict__ g2s, const double* __restrict__ DE,
                     const double* __restrict__ DP, double* __restrict__ HG,
                     double* __restrict__ Gp, double* __restrict__ HE, double* __restrict__ Ep,
                     unsigned* __restrict__ counter) {
  extern __shared__ double sm[];
  const int n2 = n * n, np2 = np * np, ld = n | 1;
  const long long n4 = (long long)n2 * n2;
  double* sDE = sm;            // DE(i,j) at [j][i] (column-major)
  double* sT = sDE + n * ld;
  double* sH = sT + n * ld;
  double* sred = sH + n * ld;  // [blockDim]
  const int a = blockIdx.x / n, c = blockIdx.x - a * n;
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *counter = 0u;
  for (int e = threadIdx.x; e < n2; e += blockDim.x) sDE[(e / n) * ld + e % n] = DE[e];
  const long long base = (long long)a * n * n2 + (long long)c * n;   // + b n^2 + d
  if (blockIdx.y) {
    for (int e = threadIdx.x; e < n2; e += blockDim.x) {
      const int b = e / n, d = e - b * n;
      sT[b * ld + d] = flush(__ldg(gee + base + (long long)b * n2 + d));
    }
  } else if (n2 >= (int)blockDim.x) {
    for (int e = threadIdx.x; e < n2; e += blockDim.x) {
      const int b = e / n, d = e - b * n;
      const double* g = g2s + base + (long long)b * n2 + d;
      double acc = 0.0;
      int ip = 0, jp = 0;
#pragma unroll 8
      for (int p = 0; p < np2; p++) {
        acc = fma(__ldg(DP + ip + np * jp), flush(__ldg(g + p * n4)), acc);
        if (++jp == np) { jp = 0; ip++; }
      }
      sT[b * ld + d] = acc;
    }
  } else {
    // fewer elements than threads: groups of n^2 threads share the proton pairs
    const int ng = blockDim.x / n2, grp = threadIdx.x / n2, e = threadIdx.x - grp * n2;
    double acc = 0.0;
    if (grp < ng) {
      const int b = e / n, d = e - b * n;
      const double* g = g2s + base + (long long)b * n2 + d;
#pragma unroll 8
      for (int p = grp; p < np2; p += ng)
        acc = fma(__ldg(DP + p / np + np * (p % np)), flush(__ldg(g + p * n4)), acc);
    }
    sred[threadIdx.x] = acc;
    __syncthreads();
    if ((int)threadIdx.x < n2) {
      double s = 0.0;
      for (int k = 0; k < ng; k++) s += sred[k * n2 + threadIdx.x];
      sT[(threadIdx.x / n) * ld + threadIdx.x % n] = s;
    }
  }
  __syncthreads();
  double* H = blockIdx.y ? HE : HG;
  double* T = blockIdx.y ? Ep : Gp;
  // H[b][y] = sum_d T[b][d] DE(y,d), DE(y,d) at [d][y]
  tile_mul<false, false>(n, ld, sT, sDE, sH);
  __syncthreads();
  // T'[x][y] = sum_b DE(x,b) H[b][y], DE(x,b) at [b][x]
  tile_mul<true, false>(n, ld, sDE, sH, sT);
  __syncthreads();
  for (int e = threadIdx.x; e < n2; e += blockDim.x) {
    const int b = e / n, d = e - b * n;
    H[base + (long long)b * n2 + d] = sH[b * ld + d];
    T[base + (long long)b * n2 + d] = sT[b * ld + d];
  }
}

// Off every delta only its four gathers are left (terms 16, 17, 22, 23).
__device__ __forceinline__ double grad_gather(int n, const int* l, const double* __restrict__ T) {
  double acc = 0.125 * __ldg(T + idx4(n, l[1], l[0], l[3], l[2]));
  acc = fma(-0.0625, __ldg(T + idx4(n, l[1], l[2], l[3], l[0])), acc);
  acc = fma(-0.0625, __ldg(T + idx4(n, l[3], l[0], l[1], l[2])), acc);
  return fma(0.125, __ldg(T + idx4(n, l[3], l[2], l[1], l[0])), acc);
}

// Sums of v[0..3] over the warp: lane's result is that of v[(lane >> 3) & 3]
// (six additions instead of twenty).
__device__ __forceinline__ double warp_sum4(double v0, double v1, double v2, double v3, int lane) {
  const bool hi = lane & 16, h2 = lane & 8;
  double a = hi ? v2 : v0, b = hi ? v3 : v1;
  a += __shfl_xor_sync(0xffffffffu, hi ? v0 : v2, 16);
  b += __shfl_xor_sync(0xffffffffu, hi ? v1 : v3, 16);
  double r = h2 ? b : a;
  r += __shfl_xor_sync(0xffffffffu, h2 ? a : b, 8);
  r += __shfl_xor_sync(0xffffffffu, r, 4);
  r += __shfl_xor_sync(0xffffffffu, r, 2);
  r += __shfl_xor_sync(0xffffffffu, r, 1);
  return r;
}

// grid n^2: tile (a, c) of dE/dG', dE/dE' -> epart[(a,c)][x*n + b] and
// fpart[p][(a,c)] = sum_bd GAM_2s(p; ab; cd) W(ab; cd).  LEAN: three tiles of
// shared memory for six; DE, H_G and H_E are read from memory, an element at a
// time for all lanes of a warp, and epart is [(a,c)][b*n + x].
constexpr int kBackwardThreads = 512;
template <bool LEAN>
__global__ void __launch_bounds__(kBackwardThreads)
gam4f_backward_kernel(int n, int np, const double* __restrict__ g2s,
                      const double* __restrict__ DE, const double* __restrict__ HG,
                      const double* __restrict__ Gp, const double* __restrict__ HE,
                      const double* __restrict__ Ep, const double* __restrict__ PT,
                      double* __restrict__ epart, double* __restrict__ fpart) {
  extern __shared__ double sm[];
  const int n2 = n * n, np2 = np * np, ld = n | 1, tl = n * ld;
  const long long n4 = (long long)n2 * n2;
  double* sDE = sm;
  double* sW = LEAN ? sm : sDE + tl;   // Wp(a,x,c,y)
  double* sX = sW + tl;        // Wp(a,x,c,y) + Wp(c,y,a,x)
  double* sY = sX + tl;        // the same of Vp
  double* sHG = sY + tl;       // [b][y]
  double* sHE = sHG + tl;
  __shared__ double sST[8];
  const int a = blockIdx.x / n, c = blockIdx.x - a * n;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long base = (long long)a * n * n2 + (long long)c * n;
  const double* PG = PT;
  const double* PE = PT + 6 * n2;
  // double traces (01)(23), (02)(13), (03)(12): traces of the first three tables
  if (warp < 6) {
    const double* P = (warp < 3 ? PG : PE) + (size_t)(warp % 3) * n2;
    double s = 0.0;
    for (int u = lane; u < n; u += 32) s += P[u * n + u];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (lane == 0) sST[(warp / 3) * 4 + warp % 3] = s;
  }
  if (!LEAN)
    for (int e = threadIdx.x; e < n2; e += blockDim.x) {
      const int b = e / n, d = e - b * n;
      sDE[b * ld + d] = DE[e];
      sHG[b * ld + d] = HG[base + (long long)b * n2 + d];
      sHE[b * ld + d] = HE[base + (long long)b * n2 + d];
    }
  __syncthreads();
  for (int e = threadIdx.x; e < n2; e += blockDim.x) {
    const int x = e / n, y = e - x * n;
    const int l[4] = {a, x, c, y}, m[4] = {c, y, a, x};
    const double w = grad_gather(n, l, Ep);
    sW[x * ld + y] = w;
    sX[x * ld + y] = w + grad_gather(n, m, Ep);
    sY[x * ld + y] = grad_gather(n, l, Gp) + grad_gather(n, m, Gp);
  }
  __syncthreads();
  // the rows x = a, x = c and columns y = a, y = c lie on deltas (a lane with
  // delta terms in the loop above would hold up its whole warp)
  for (int e = threadIdx.x; e < 4 * n; e += blockDim.x) {
    const int k = e / n, u = e - k * n, q = (k & 1) ? c : a;
    const int x = k < 2 ? q : u, y = k < 2 ? u : q;
    const int l[4] = {a, x, c, y}, m[4] = {c, y, a, x};
    const double w = grad_term(n, l, Ep, PE, sST + 4);
    sW[x * ld + y] = w;
    sX[x * ld + y] = w + grad_term(n, m, Ep, PE, sST + 4);
    sY[x * ld + y] = grad_term(n, l, Gp, PG, sST) + grad_term(n, m, Gp, PG, sST);
  }
  __syncthreads();
  // focke(x,b) of this tile: sum_y X[x][y] HG[b][y] + Y[x][y] HE[b][y]
  for (int e = threadIdx.x; e < n2; e += blockDim.x) {
    const int q = e / n, r = e - q * n, x = LEAN ? r : q, b = LEAN ? q : r;
    const double* hg = LEAN ? HG + base + (long long)b * n2 : sHG + b * ld;
    const double* he = LEAN ? HE + base + (long long)b * n2 : sHE + b * ld;
    double s = 0.0, t = 0.0;
#pragma unroll 4
    for (int y = 0; y < n; y++) {
      s = fma(sX[x * ld + y], LEAN ? __ldg(hg + y) : hg[y], s);
      t = fma(sY[x * ld + y], LEAN ? __ldg(he + y) : he[y], t);
    }
    epart[(long long)blockIdx.x * n2 + e] = s + t;
  }
  __syncthreads();
  // W[b][d] = sum_xy Wp[x][y] DE(x,b) DE(y,d), through Ht[x][d] (in sX) into sY;
  // DE(y,d) at [d][y], DE(x,b) at [b][x]
  if (LEAN) {
    for (int e = threadIdx.x; e < n2; e += blockDim.x) {
      const int d = e / n, x = e - d * n;
      double s = 0.0;
#pragma unroll 4
      for (int y = 0; y < n; y++) s = fma(sW[x * ld + y], __ldg(DE + d * n + y), s);
      sX[x * ld + d] = s;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < n2; e += blockDim.x) {
      const int b = e / n, d = e - b * n;
      double s = 0.0;
#pragma unroll 4
      for (int x = 0; x < n; x++) s = fma(__ldg(DE + b * n + x), sX[x * ld + d], s);
      sY[b * ld + d] = s;
    }
  } else {
    tile_mul<false, true>(n, ld, sW, sDE, sX);
    __syncthreads();
    tile_mul<false, false>(n, ld, sDE, sX, sY);
  }
  __syncthreads();
  // four proton pairs of a warp at a time
  const int nw = blockDim.x >> 5;
  for (int p0 = warp * 4; p0 < np2; p0 += nw * 4) {
    double v[4] = {0.0, 0.0, 0.0, 0.0};
    for (int e = lane; e < n2; e += 32) {
      const int b = e / n, d = e - b * n;
      const double* g = g2s + base + (long long)b * n2 + d;
      const double w = sY[b * ld + d];
#pragma unroll
      for (int k = 0; k < 4; k++)
        if (p0 + k < np2) v[k] = fma(flush(__ldg(g + (p0 + k) * n4)), w, v[k]);
    }
    const double r = warp_sum4(v[0], v[1], v[2], v[3], lane);
    if ((lane & 7) == 0 && p0 + (lane >> 3) < np2)
      fpart[(long long)(p0 + (lane >> 3)) * n2 + blockIdx.x] = r;
  }
}

// lean: the layout of epart.  CTAs [0, ne_ctas): 32 focke elements each, 32 warps sharing the n^2 tiles; the
// others: 32 proton pairs each.  The last of those to finish adds E up.
__global__ void __launch_bounds__(1024)
gam4f_reduce_kernel(int n, int np, int ne_ctas, bool lean, const double* __restrict__ epart,
                    const double* __restrict__ fpart, const double* __restrict__ DP,
                    int accumulate, double* __restrict__ focke, double* __restrict__ fockp,
                    double* __restrict__ evals, unsigned* __restrict__ counter,
                    double* __restrict__ E) {
  __shared__ double sr[32][33];
  __shared__ bool last;
  const int n2 = n * n, np2 = np * np, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if ((int)blockIdx.x < ne_ctas) {
    const int e = blockIdx.x * 32 + lane;
    double s = 0.0;
    if (e < n2) {
#pragma unroll 8
      for (int t = warp; t < n2; t += 32) s += epart[(long long)t * n2 + e];
    }
    sr[warp][lane] = s;
    __syncthreads();
    double v = sr[lane][warp];   // warp = element now, lane = share
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int q = blockIdx.x * 32 + warp;
    if (lane == 0 && q < n2) {
      const int f = lean ? q : q / n + n * (q % n);   // focke(x,b), column-major
      focke[f] = accumulate ? focke[f] + v : v;
    }
    return;
  }
  const int p = (blockIdx.x - ne_ctas) * 32 + warp;
  double v = 0.0;
  if (p < np2) {
    for (int t = lane; t < n2; t += 32) v += fpart[(long long)p * n2 + t];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) {
      const int f = p / np + np * (p % np);
      fockp[f] = accumulate ? fockp[f] + v : v;
      evals[p] = DP[f] * v;
      __threadfence();
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(counter, 1u) == gridDim.x - ne_ctas - 1;
  __syncthreads();
  if (last && warp == 0) {
    __threadfence();
    double s = 0.0;
    for (int k = lane; k < np2; k += 32) s += __ldcg(evals + k);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (lane == 0) *E = s;
  }
}

// Per-CTA maxima of |T(l0,l1,l2,l3) - T(l2,l3,l0,l1)| and |T| for GAM_ee
// (n^4) and GAM_2s (np^2 blocks of n^4): out[4*blockIdx.x + {0,1,2,3}].
__global__ void pair_symmetry_kernel(int n, int np, const double* __restrict__ gee,
                                     const double* __restrict__ g2s,
                                     double* __restrict__ out) {
  __shared__ double sw[4][32];
  const long long n4 = (long long)n * n * n * n;
  const long long total = n4 * (1 + (long long)np * np);
  double m[4] = {0.0, 0.0, 0.0, 0.0};
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < total;
       g += stride) {
    const long long blk = g / n4, r = g - blk * n4;
    const double* T = blk == 0 ? gee : g2s + (blk - 1) * n4;
    long long q = r;
    const int l3 = (int)(q % n); q /= n;
    const int l2 = (int)(q % n); q /= n;
    const int l1 = (int)(q % n); q /= n;
    const int l0 = (int)q;
    const double v = T[r];
    const double d = fabs(v - T[idx4(n, l2, l3, l0, l1)]);
    const int t = blk == 0 ? 0 : 2;
    m[t] = fmax(m[t], d);
    m[t + 1] = fmax(m[t + 1], fabs(v));
  }
  const int w = threadIdx.x / 32, lane = threadIdx.x & 31;
  for (int k = 0; k < 4; k++) {
    double v = m[k];
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, o));
    if (lane == 0) sw[k][w] = v;
  }
  __syncthreads();
  if (threadIdx.x < 4) {
    double v = 0.0;
    for (int i = 0; i < (int)(blockDim.x + 31) / 32; i++) v = fmax(v, sw[threadIdx.x][i]);
    out[4 * blockIdx.x + threadIdx.x] = v;
  }
}

int grid_for(long long work, int tb) {
  long long g = (work + tb - 1) / tb;
  const long long cap = 152LL * 16;
  return (int)(g < 1 ? 1 : (g > cap ? cap : g));
}

// out = underflow(in), element by element
__global__ void flush_copy_kernel(long long n, const double* __restrict__ in,
                                  double* __restrict__ out) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    out[i] = flush(in[i]);
}

// ---- mixed-precision variant: the transforms and focke on tensor cores -----
// Rows [0, rows) x K [kt, kt + 64) of an operand into its two TF32 halves in
// the canonical layout, by warps [w0, nw) of the CTA: a warp takes 8 rows x 8
// k, a lane two neighbouring k, so that its two 8-byte stores per half fill
// whole 128-byte core matrices (a lane per k hit four banks eight times over)
// and eight such loads are in flight before the first is converted.  VEC: the
// pairs are 16-byte aligned.
template <bool VEC>
__device__ __forceinline__ void tc_load(const double* __restrict__ X, long long ld, long long x0,
                                        int rows, long long kt, int kv, unsigned char* hi,
                                        unsigned char* lo) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int nw = tc::kThreads / 32, kBatch = 8;
  const int kh = (kv + 7) / 8, nt = ((rows + 7) / 8) * kh;
  const int r = (lane >> 1) & 7, k = ((lane >> 4) << 2) + ((lane & 1) << 1);
  for (int t0 = warp; t0 < nt; t0 += nw * kBatch) {
    double2 v[kBatch];
#pragma unroll
    for (int q = 0; q < kBatch; q++) {
      const int t = t0 + q * nw;
      v[q] = make_double2(0.0, 0.0);
      if (t < nt) {
        const int rr = (t / kh) * 8 + r, kk = (t % kh) * 8 + k;
        const double* p = X + (x0 + rr) * ld + kt + kk;
        if (rr < rows) {
          if (VEC && kk + 1 < kv) {
            v[q] = __ldg(reinterpret_cast<const double2*>(p));
          } else {
            if (kk < kv) v[q].x = __ldg(p);
            if (kk + 1 < kv) v[q].y = __ldg(p + 1);
          }
        }
      }
    }
#pragma unroll
    for (int q = 0; q < kBatch; q++) {
      const int t = t0 + q * nw;
      if (t < nt) {
        uint2 h, l;
        tc::split_tf32(v[q].x, h.x, l.x);
        tc::split_tf32(v[q].y, h.y, l.y);
        const int off = tc::canon_off((t / kh) * 8 + r, (t % kh) * 8 + k);
        *reinterpret_cast<uint2*>(hi + off) = h;
        *reinterpret_cast<uint2*>(lo + off) = l;
      }
    }
  }
}

// 2^ea v in FP64 by integer operations, for normal numbers and zeros: their
// fields move over.  (A conversion, an addition and a multiplication per
// result, all on the FP64 pipe, were a transform's largest part.)
__device__ __forceinline__ double widen(float v, int ea) {
  const uint32_t u = __float_as_uint(v), e = (u >> 23) & 255u;
  const uint32_t hi = (u & 0x80000000u) | (e == 0u ? 0u : (((e + 896u + (uint32_t)ea) << 20) | ((u & 0x7fffffu) >> 3)));
  return __hiloint2double((int)hi, (int)(u << 29));
}
// subnormal, infinite or NaN: what widen does not carry over
__device__ __forceinline__ bool not_plain(float v) {
  const uint32_t u = __float_as_uint(v) & 0x7fffffffu;
  return u - 0x00800000u >= 0x7f000000u && u != 0u;
}

// C[m*ldc + n] = 2^ea sum_{k in split} A[m*lda + k] B[n*ldb + k]
// grid (ceil(M/128), ceil(N/64), nsplit); split z covers K range
// [z*kchunk, min(K, (z+1)*kchunk)) and writes C + z*split_stride.
// Rows past M or N are not loaded (their results are not stored), K steps past
// the end not multiplied; a K tail inside a step is zero.
// Measured at n = 48 (M = 110592, N = K = 48): 257 us a call with 128 threads
// loading one element at a time and converting on the FP64 pipe, 65 us so.
template <bool VEC>
__global__ void __launch_bounds__(tc::kThreads, 2)
tc_gemm_kernel(const double* __restrict__ A, long long lda, long long M,
               const double* __restrict__ B, long long ldb, long long N, long long K,
               long long kchunk, int ea, double* __restrict__ C, long long ldc,
               long long split_stride, int* __restrict__ err) {
  extern __shared__ __align__(1024) unsigned char tc_sm[];
  unsigned char* a_hi = tc_sm;
  unsigned char* a_lo = tc_sm + tc::kABytes;
  unsigned char* b_hi = tc_sm + 2 * tc::kABytes;
  unsigned char* b_lo = b_hi + tc::kBBytes;
  uint64_t* mbar = reinterpret_cast<uint64_t*>(b_lo + tc::kBBytes);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(b_lo + tc::kBBytes + 8);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const long long m0 = (long long)blockIdx.x * tc::kTileM;
  const long long n0 = (long long)blockIdx.y * tc::kTileN;
  const int mv = (int)(M - m0 < tc::kTileM ? M - m0 : tc::kTileM);
  const int nv = (int)(N - n0 < tc::kTileN ? N - n0 : tc::kTileN);
  const long long kbeg = (long long)blockIdx.z * kchunk;
  const long long kend = kbeg + kchunk < K ? kbeg + kchunk : K;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 64;"
                 :: "r"(tc::smem_u32(tmem_slot)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(tc::smem_u32(mbar))
                 : "memory");
  }
  // rows that are never loaded are multiplied all the same: give them a value
  if (mv < tc::kTileM || nv < tc::kTileN)
    for (int e = tid * 16; e < 2 * (tc::kABytes + tc::kBBytes); e += tc::kThreads * 16)
      *reinterpret_cast<uint4*>(tc_sm + e) = make_uint4(0u, 0u, 0u, 0u);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  const uint32_t mb = tc::smem_u32(mbar);
  uint32_t phase = 0;
  bool ok = true;
  const uint32_t idesc = tc::instr_desc();
  // kFoldTiles 64-wide K tiles are accumulated in TMEM (FP32) and then folded
  // into FP64: this thread's half row of the result (a warp reads the 32
  // tensor-memory lanes of its number modulo four)
  constexpr int kHalf = tc::kTileN / 2;
  const int half = warp >> 2, rloc = (warp & 3) * 32 + lane;
  const bool used = (warp & 3) * 32 < mv && half * kHalf < nv;   // any result of this warp stored
  const bool one = kend - kbeg <= tc::kTileK * tc::kFoldTiles;   // a single fold
  const double scale = ldexp(1.0, ea);
  double acc[kHalf];
#pragma unroll
  for (int i = 0; i < kHalf; i++) acc[i] = 0.0;
  const uint32_t trow = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(half * kHalf);
  int tile = 0;
  for (long long kt = kbeg; kt < kend && ok; kt += tc::kTileK, tile++) {
    const bool first = tile % tc::kFoldTiles == 0;
    const bool fold = (tile + 1) % tc::kFoldTiles == 0 || kt + tc::kTileK >= kend;
    const int kv = (int)(kend - kt < tc::kTileK ? kend - kt : tc::kTileK);
    tc_load<VEC>(A, lda, m0, mv, kt, kv, a_hi, a_lo);
    tc_load<VEC>(B, ldb, n0, nv, kt, kv, b_hi, b_lo);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (tid == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t ah = tc::smem_u32(a_hi), al = tc::smem_u32(a_lo);
      const uint32_t bh = tc::smem_u32(b_hi), bl = tc::smem_u32(b_lo);
      for (int st = 0; st < (kv + 7) / 8; st++) {
        const uint32_t o = st * 256;   // two 128-byte core matrices per K step
        tc::mma_tf32(tmem, tc::smem_desc(ah + o), tc::smem_desc(bh + o), idesc,
                     (st > 0 || !first) ? 1 : 0);
        tc::mma_tf32(tmem, tc::smem_desc(ah + o), tc::smem_desc(bl + o), idesc, 1);
        tc::mma_tf32(tmem, tc::smem_desc(al + o), tc::smem_desc(bh + o), idesc, 1);
      }
      tc::mma_commit(mb);
    }
    ok = __syncthreads_and(tc::mbar_wait(mb, phase) ? 1 : 0) != 0;
    phase ^= 1u;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (ok && fold && used) {
#pragma unroll
      for (int c = 0; c < kHalf / 16; c++) {
        float v[16];
        tc::tmem_ld16(trow + (uint32_t)(c * 16), v);
        bool odd = !one;
#pragma unroll
        for (int i = 0; i < 16; i++) odd = odd || not_plain(v[i]);
        if (__any_sync(0xffffffffu, odd)) {
          const double f = one ? scale : 1.0;
#pragma unroll
          for (int i = 0; i < 16; i++) acc[c * 16 + i] = fma((double)v[i], f, acc[c * 16 + i]);
        } else {
#pragma unroll
          for (int i = 0; i < 16; i++) acc[c * 16 + i] = widen(v[i], ea);
        }
      }
    }
    // every lane's reads are done before the next tile's MMA overwrites TMEM
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
  }
  if (!ok) {
    if (tid == 0) atomicExch(err, 1);
  } else {
    // every MMA has completed (last wait) and the operand tiles are dead:
    // stage the 128 x 64 FP64 tile in their shared memory (row stride 65)
    // and write it row-segment by row-segment, coalesced
    double* sc = reinterpret_cast<double*>(tc_sm);
#pragma unroll
    for (int i = 0; i < kHalf; i++)
      sc[rloc * (tc::kTileN + 1) + half * kHalf + i] = one ? acc[i] : scale * acc[i];
    __syncthreads();
    double* out = C + (long long)blockIdx.z * split_stride;
    for (int e = tid; e < mv * nv; e += tc::kThreads) {
      const int r = e / nv, c = e - r * nv;
      out[(m0 + r) * ldc + n0 + c] = sc[r * (tc::kTileN + 1) + c];
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 64;" :: "r"(tmem)
                 : "memory");
  }
}

// out(i,j,k,l) = in(k,l,i,j) + beta in(i,j,k,l): a transpose of the
// (n^2 x n^2) matrix view, through 32 x 32 shared-memory tiles.
__global__ void pair_swap_kernel(int n2, const double* __restrict__ in, double beta,
                                 double* __restrict__ out) {
  __shared__ double t[32][33];
  const int bx = blockIdx.x * 32, by = blockIdx.y * 32;
  for (int j = threadIdx.y; j < 32; j += blockDim.y) {
    const int r = by + j, c = bx + threadIdx.x;
    if (r < n2 && c < n2) t[j][threadIdx.x] = in[(long long)r * n2 + c];
  }
  __syncthreads();
  for (int j = threadIdx.y; j < 32; j += blockDim.y) {
    const int r = bx + j, c = by + threadIdx.x;   // out[r][c] = in[c][r]
    if (r < n2 && c < n2) {
      const long long o = (long long)r * n2 + c;
      out[o] = t[threadIdx.x][j] + (beta != 0.0 ? beta * in[o] : 0.0);
    }
  }
}

// out(x,a,c,y) = in(a,x,c,y)
__global__ void swap12_kernel(int n, const double* __restrict__ in, double* __restrict__ out) {
  const long long n2 = (long long)n * n, total = n2 * n2;
  for (long long o = blockIdx.x * (long long)blockDim.x + threadIdx.x; o < total;
       o += (long long)gridDim.x * blockDim.x) {
    const long long j = o % n2, xa = o / n2;
    const long long a = xa % n, x = xa / n;
    out[o] = in[(a * n + x) * n2 + j];
  }
}

// DEt[y*n + d] = DE(y,d) (column-major DE)
__global__ void transpose_n_kernel(int n, const double* __restrict__ DE, double* __restrict__ t) {
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n * n; e += gridDim.x * blockDim.x) {
    const int y = e / n, d = e - y * n;
    t[e] = DE[y + n * d];
  }
}

// focke(x,b) (+)= sum_split part[split][x*64 + b], a warp per output
__global__ void focke_tc_reduce_kernel(int n, int nsplit, const double* __restrict__ part,
                                       int accumulate, double* __restrict__ focke) {
  const int e = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (e >= n * n) return;
  const int x = e / n, b = e - x * n;
  double s = 0.0;
  for (int z = lane; z < nsplit; z += 32) s += part[(long long)z * 128 * 64 + x * 64 + b];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (lane == 0) {
    const int f = x + n * b;
    focke[f] = accumulate ? focke[f] + s : s;
  }
}

// Two 256-wide FP32 folds a CTA: enough of them for the SMs at n = 48 (216)
constexpr long long kFockeKChunk = 512;

cudaError_t tc_gemm(const double* A, long long lda, long long M, const double* B,
                    long long ldb, long long N, long long K, long long kchunk, int ea,
                    double* C, long long ldc, long long split_stride, int* err,
                    cudaStream_t s) {
  const bool vec = !(lda & 1) && !(ldb & 1) && !(kchunk & 1) &&
                   !((uintptr_t)A & 15) && !((uintptr_t)B & 15);
  const auto fn = vec ? tc_gemm_kernel<true> : tc_gemm_kernel<false>;
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       tc::kSmemBytes);
  if (e != cudaSuccess) return e;
  const long long nsplit = (K + kchunk - 1) / kchunk;
  const dim3 grid((unsigned)((M + tc::kTileM - 1) / tc::kTileM),
                  (unsigned)((N + tc::kTileN - 1) / tc::kTileN), (unsigned)(nsplit < 1 ? 1 : nsplit));
  fn<<<grid, tc::kThreads, tc::kSmemBytes, s>>>(A, lda, M, B, ldb, N, K, kchunk, ea, C, ldc,
                                               split_stride, err);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_pair_symmetry_check(int ne, int np, const double* gee,
                                       const double* g2s, double* out,
                                       int* grid, cudaStream_t s) {
  if (ne < 1 || np < 1) return cudaErrorInvalidValue;
  const long long n4 = (long long)ne * ne * ne * ne;
  const int g = grid_for(n4 * (1 + (long long)np * np), 256);
  *grid = g;
  pair_symmetry_kernel<<<g, 256, 0, s>>>(ne, np, gee, g2s, out);
  return cudaGetLastError();
}

size_t gam4f_scratch_doubles(int ne, int np) {
  const size_t n2 = (size_t)ne * ne, n4 = n2 * n2, p2 = (size_t)np * np;
  // H_G, G', H_E, E', focke partials; leg-pair traces; fockp partials,
  // energy terms; counter
  return 5 * n4 + 12 * n2 + p2 * n2 + p2 + 1;
}

// Measured (one GB300): n = 12, np = 8: 46 us a call, 71 us by itself (109 us and 301 us as fourteen launches).
cudaError_t launch_gam4_factored(int ne, int np, const double* gee,
                                 const double* g2s, const double* DE,
                                 const double* DP, double* scratch,
                                 double* focke, double* fockp, double* E,
                                 int accumulate, cudaStream_t s) {
  if (ne < 1 || ne > kGam4FactMaxNE || np < 1 || np > 255)
    return cudaErrorInvalidValue;
  const int n = ne, n2 = n * n;
  const size_t n4 = (size_t)n2 * n2, p2 = (size_t)np * np;
  double* HG = scratch;
  double* Gp = HG + n4;
  double* HE = Gp + n4;
  double* Ep = HE + n4;
  double* epart = Ep + n4;
  double* PT = epart + n4;
  double* fpart = PT + 12 * n2;
  double* evals = fpart + p2 * n2;
  unsigned* counter = reinterpret_cast<unsigned*>(evals + p2);
  // Threads beyond the n^2 elements of a tile share its proton pairs, so small
  // n takes wide CTAs too (n = 12: seven groups of 144; 256 threads, one group
  // walking all pairs, were 2.5x slower).  Beyond n = 22 there is one group, and
  // one wide CTA fills an SM, whose memory and FP64 phases then wait for each
  // other (and from n = 33 its loops over the n^2 elements take a second, nearly
  // empty turn): CTAs of which two share an SM are the better ones.  The forward
  // kernel has them with 640 threads; the backward one, by its 128 registers,
  // with 256, and with the three tiles of LEAN up to n = 64 (six: n = 48).  That
  // pays while its sums over proton pairs, which want all 16 warps, are short,
  // up to np = 5.  Whole calls, us, threads (1024, 512) with six tiles / (640, 256)
  // with six / (640, 512) LEAN / (640, 256) LEAN:
  //   n = 24, np = 1   244  192  235  194    n = 40, np = 1  2129 1886 2071 1880
  //   n = 24, np = 10  473  377  409  377    n = 40, np = 6  2546 2403 2385 2392
  //   n = 30, np = 4   677  567  646  561    n = 40, np = 10 3595 3327 3272 3302
  //   n = 30, np = 10  997 1010 1027 1000    n = 50, np = 2  5992 5901 5832 5374
  //   n = 33, np = 1   912  759  863  759    n = 60, np = 1 13573 13458 12933 12069
  //   n = 33, np = 10 1882 1471 1534 1461    n = 60, np = 10 20268 23020 18470 18396
  //   n = 36, np = 6  1670 1580 1511 1567    n = 64, np = 4 19749 19432 18067 17967
  // Six tiles stay below n = 23 (n = 12, np = 8: 45.6 us, LEAN 47.7).  The results
  // do not depend on the choice.
  const bool lean = n > 22, few = lean && np <= 5;
  const int tforward = few || n > 32 ? 640 : kForwardThreads;
  const int tbackward = few ? 256 : kBackwardThreads;
  const auto backward = lean ? gam4f_backward_kernel<true> : gam4f_backward_kernel<false>;
  const size_t tile = (size_t)n * (n | 1);
  const size_t smf = sizeof(double) * (3 * tile + kForwardThreads);
  const size_t smb = sizeof(double) * (lean ? 3 : 6) * tile;
  for (const auto& k : {std::make_pair((const void*)gam4f_forward_kernel, smf),
                        std::make_pair((const void*)backward, smb)})
    if (k.second > 48 * 1024) {
      cudaError_t e = cudaFuncSetAttribute(k.first, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)k.second);
      if (e != cudaSuccess) return e;
    }
  gam4f_forward_kernel<<<dim3(n2, 2), tforward, smf, s>>>(n, np, gee, g2s, DE, DP, HG, Gp, HE, Ep, counter);
  traces_kernel<<<dim3(grid_for(6LL * n2, 128), 2), 128, 0, s>>>(n, Gp, Ep, PT);
  backward<<<n2, tbackward, smb, s>>>(n, np, g2s, DE, HG, Gp, HE, Ep, PT, epart, fpart);
  const int ne_ctas = (n2 + 31) / 32;
  gam4f_reduce_kernel<<<ne_ctas + (int)((p2 + 31) / 32), 1024, 0, s>>>(
      n, np, ne_ctas, lean, epart, fpart, DP, accumulate, focke, fockp, evals, counter, E);
  return cudaGetLastError();
}

size_t gam4f_tc_scratch_doubles(int ne, int np) {
  const size_t n4 = (size_t)ne * ne * ne * ne;
  const size_t nchunk = (n4 + kDotChunk - 1) / kDotChunk;
  const size_t nsplit = (size_t)((n4 / ne + kFockeKChunk - 1) / kFockeKChunk);
  // 8 n^4 tensors, DE^T, PT(2x6 n^2), ST(8), fockp partials, focke partials,
  // error flag
  return 8 * n4 + (size_t)ne * ne + 12 * (size_t)ne * ne + 8 + (size_t)np * np * nchunk +
         2 * nsplit * 128 * 64 + 2;
}

// Same focke / fockp / E as launch_gam4_factored, with the one-index
// transforms and the focke contraction on the tensor cores (tc_gemm.cuh:
// 3xTF32 products, FP32 accumulation, FP64 results) and everything else
// (the two passes over GAM_2s, traces, gradients, reductions) FP64.  The
// second-index transforms use the pair-exchange symmetry of the tables:
// sum_b T(a,b,c,d) DE(x,b) = H(c,d,a,x) with H the last-index transform, so
// T' = last(swap(last(T))); likewise the back transform of the symmetrised
// gradient.  *err (device int, optional) is set when a tensor-core wait ran
// out; the call then returns cudaErrorLaunchTimeout after the stream drains.
cudaError_t launch_gam4_factored_tc(int ne, int np, const double* gee,
                                    const double* g2s, const double* DE,
                                    const double* DP, double* scratch,
                                    double* focke, double* fockp, double* E,
                                    int accumulate, cudaStream_t s) {
  if (ne < 1 || ne > 64 || np < 1 || np > 255) return cudaErrorInvalidValue;
  const int n = ne;
  const long long n2 = (long long)n * n, n3 = n2 * n, n4 = n2 * n2;
  const int nchunk = (int)((n4 + kDotChunk - 1) / kDotChunk);
  const long long nsplit = (n3 + kFockeKChunk - 1) / kFockeKChunk;
  double* buf[8];
  for (int i = 0; i < 8; i++) buf[i] = scratch + (size_t)i * n4;
  double* DEt = scratch + 8 * n4;
  double* PT = DEt + n2;
  double* ST = PT + 12 * n2;
  double* fpart = ST + 8;
  double* epart = fpart + (size_t)np * np * nchunk;   // [2][nsplit][128*64]
  int* err = reinterpret_cast<int*>(epart + 2 * nsplit * 128 * 64);
  const int TB = 256;
  const int g_n4 = grid_for(n4, TB);
  const dim3 tgrid((unsigned)((n2 + 31) / 32), (unsigned)((n2 + 31) / 32));
  const dim3 tblk(32, 8);
  cudaError_t e;
#define TRY(x) do { e = (x); if (e != cudaSuccess) return e; } while (0)
  TRY(cudaMemsetAsync(err, 0, sizeof(int), s));
  transpose_n_kernel<<<grid_for(n2, TB), TB, 0, s>>>(n, DE, DEt);
  // last-index transforms: T'(..,y) = sum_d T(..,d) DE(y,d)  [B = DE^T rows]
  auto last_f = [&](const double* in, double* out) {
    return tc_gemm(in, n, n3, DEt, n, n, n, n, 0, out, n, 0, err, s);
  };
  // back transforms: T'(..,d) = sum_y T(..,y) DE(y,d)  [B = DE rows]
  auto last_b = [&](const double* in, double* out, int ea) {
    return tc_gemm(in, n, n3, DE, n, n, n, n, ea, out, n, 0, err, s);
  };
  // 1. G = DP . GAM_2s (FP32 products, HBM)
  const bool vec = !(n4 & 1) && !((uintptr_t)g2s & 15);
  const long long nv = vec ? n4 / 2 : n4;
  dp_contract_mixed_kernel<<<(unsigned)((nv + 255) / 256), 256, np * np <= kDpShared ? sizeof(float) * np * np : 0, s>>>(
      n4, np, vec, g2s, DP, buf[0]);
  // 2. H_G, G' and H_E, E'
  TRY(last_f(buf[0], buf[1]));                                        // H_G
  pair_swap_kernel<<<tgrid, tblk, 0, s>>>((int)n2, buf[1], 0.0, buf[2]);
  TRY(last_f(buf[2], buf[3]));                                        // G'
  flush_copy_kernel<<<g_n4, TB, 0, s>>>(n4, gee, buf[0]);             // flushed GAM_ee
  TRY(last_f(buf[0], buf[4]));                                        // H_E
  pair_swap_kernel<<<tgrid, tblk, 0, s>>>((int)n2, buf[4], 0.0, buf[2]);
  TRY(last_f(buf[2], buf[5]));                                        // E'
  // 3-4. traces and gradients (FP64)
  traces_kernel<<<dim3(grid_for(6LL * n * n, TB), 2), TB, 0, s>>>(n, buf[3], buf[5], PT);
  dtraces_kernel<<<1, 64, 0, s>>>(n, PT, ST);
  gam4f_gather_kernel<<<dim3(n, (n + 3) / 4, 2 * kGradSplit), 4 * n, 0, s>>>(n, buf[5], buf[3], buf[6], buf[7]);
  gam4f_delta_kernel<<<dim3((unsigned)((n3 + 127) / 128), 4, 2), 128, 0, s>>>(n, buf[5], buf[3], PT, ST, buf[6], buf[7]);
  // Ws = Wp + Wp^swap, Vs = Vp + Vp^swap
  pair_swap_kernel<<<tgrid, tblk, 0, s>>>((int)n2, buf[6], 1.0, buf[0]);
  pair_swap_kernel<<<tgrid, tblk, 0, s>>>((int)n2, buf[7], 1.0, buf[2]);
  // 5. W = back(Ws / 2), fockp = <GAM_2s, W>, E
  TRY(last_b(buf[0], buf[3], -1));
  pair_swap_kernel<<<tgrid, tblk, 0, s>>>((int)n2, buf[3], 0.0, buf[5]);
  TRY(last_b(buf[5], buf[6], 0));                                   // W
  float* Wf = reinterpret_cast<float*>(buf[7]);   // free until swap12 below
  narrow_kernel<<<g_n4, TB, 0, s>>>(n4, buf[6], Wf);
  fockp_dot_mixed_kernel<<<dim3(nchunk, (np * np + kDotP - 1) / kDotP), kDotTB, 0, s>>>(
      n4, nchunk, np * np, g2s, Wf, fpart);
  fockp_reduce_kernel<<<1, 1024, 0, s>>>(np, nchunk, fpart, DP, accumulate, fockp, E);
  // 6. focke(x,b) = sum_{a,c,y} Ws(a,x,c,y) H_G(a,b,c,y) + Vs(a,x,c,y) H_E(a,b,c,y)
  swap12_kernel<<<g_n4, TB, 0, s>>>(n, buf[0], buf[3]);   // Ws  -> [x][a][c][y]
  swap12_kernel<<<g_n4, TB, 0, s>>>(n, buf[1], buf[5]);   // H_G -> [b][a][c][y]
  swap12_kernel<<<g_n4, TB, 0, s>>>(n, buf[2], buf[7]);   // Vs
  swap12_kernel<<<g_n4, TB, 0, s>>>(n, buf[4], buf[1]);   // H_E
  TRY(tc_gemm(buf[3], n3, n, buf[5], n3, n, n3, kFockeKChunk, 0, epart, 64, 128 * 64, err, s));
  TRY(tc_gemm(buf[7], n3, n, buf[1], n3, n, n3, kFockeKChunk, 0, epart + nsplit * 128 * 64,
              64, 128 * 64, err, s));
  focke_tc_reduce_kernel<<<(unsigned)((n2 * 32 + TB - 1) / TB), TB, 0, s>>>(n, (int)(2 * nsplit), epart,
                                                        accumulate, focke);
#undef TRY
  return cudaGetLastError();
}

}  // namespace neoxc
