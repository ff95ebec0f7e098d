// k_contract.cu -- in-core Fock/energy contractions for sm_103a and the
// deterministic partial-sum reducer shared by every contraction kernel.
//
// Reference: gam2_IC1_OMP.f:339-570 (EG2IC1 / thread_EG2ICR),
// gam3_IC1_OMP.f:433-725 (EG3IC1 / thread_EG3ICR; its kernel: k_rank3.cu),
// rxchfne/rxchfne_omg2.f (RXCHFne_FAE/FP/FBE_OMG2),
// xchf1_independent/xchf1_fock.f:728-783 (XCfock_correction),
// CS_Integrals/Spot_Check/pack_GAM.f (index maps).
//
// All kernels here stream over the stored integral tensor: every element is
// read from HBM once (FP64 instructions bound the wider ones, see each), and
// partial sums are written per CTA and reduced by a
// second, deterministic kernel (no floating-point atomics), so repeated
// calls give bit-identical results.
#include <algorithm>

#include "neoxc_internal.h"

namespace neoxc {

// part[((ipjp*ne + i1)*nsub + s)*ne + j1] -> Fock/energy.
//   fe(i1,j1) (+)= fe_scale * sum_{ipjp} DP(ipjp) * sum_s part
//   fp(ipjp)  (+)= sum_{i1,j1} DE(i1,j1) * sum_s part
//   E = sum_{ipjp} DP(ipjp) * [that fp contribution]
// Two kernels, both wide: the sub-block sums of every (ipjp, i1, j1) with
// their share of fp, then the sums over ipjp.  (One thread per output walked
// all of them in a row: 3.2 ms at ne = 12, np = 8, nsub = 144; now 10 us.)
// A CTA of the first takes 1024 outputs of one ipjp, so that up to ne = 32
// fp needs one partial per ipjp (the scratch size of the gam_4 calls).
constexpr int kRedThreads = 128, kRedOut = 1024;

__device__ __forceinline__ double block_add(double v, double* sw) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  if (lane == 0) sw[w] = v;
  __syncthreads();
  double t = 0.0;
  for (int k = 0; k < (int)(blockDim.x + 31) / 32; k++) t += sw[k];
  return t;   // every thread gets the same value
}

// grid (ceil(ne^2 / kRedOut), np^2); the sums replace sub-block 0
__global__ void __launch_bounds__(kRedThreads)
fock_reduce_sub_kernel(int ne, int np, int nsub, double* __restrict__ part,
                       const double* __restrict__ DE, double* __restrict__ fp_part) {
  __shared__ double sw[kRedThreads / 32];
  const int ipjp = blockIdx.y;
  const int t0 = blockIdx.x * kRedOut, t1 = min(ne * ne, t0 + kRedOut);
  double w = 0.0;
  for (int t = t0 + threadIdx.x; t < t1; t += kRedThreads) {
    const int i1 = t / ne, j1 = t - i1 * ne;
    double* p = part + ((size_t)ipjp * ne + i1) * nsub * ne + j1;
    double s = 0.0;
#pragma unroll 8
    for (int k = 0; k < nsub; k++) s += p[(size_t)k * ne];
    p[0] = s;
    w = fma(DE[i1 + ne * j1], s, w);
  }
  const double sum = block_add(w, sw);
  if (threadIdx.x == 0) fp_part[(size_t)ipjp * gridDim.x + blockIdx.x] = sum;
}

// CTAs 0..: a warp per (i1,j1), lanes over ipjp; the last CTA: fp and E
__global__ void __launch_bounds__(kRedThreads)
fock_reduce_out_kernel(int ne, int np, int nsub, int nfp, const double* __restrict__ part,
                       const double* __restrict__ fp_part, const double* __restrict__ DP,
                       double fe_scale, int accumulate, double* fe, double* fp, double* E) {
  __shared__ double sw[kRedThreads / 32];
  const int n2 = ne * ne, p2 = np * np;
  if (blockIdx.x == gridDim.x - 1) {
    double e = 0.0;
    for (int p = threadIdx.x; p < p2; p += kRedThreads) {
      double s = 0.0;
      for (int k = 0; k < nfp; k++) s += fp_part[(size_t)p * nfp + k];
      const int f = p / np + np * (p % np);
      if (fp) fp[f] = accumulate ? fp[f] + s : s;
      e = fma(DP[f], s, e);
    }
    e = block_add(e, sw);
    if (threadIdx.x == 0) *E = e;
    return;
  }
  const int t = (int)((blockIdx.x * kRedThreads + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (t >= n2 || !fe) return;
  const int i1 = t / ne, j1 = t - i1 * ne;
  double s = 0.0;
  for (int p = lane; p < p2; p += 32)
    s = fma(DP[p / np + np * (p % np)], part[((size_t)p * ne + i1) * nsub * ne + j1], s);
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (lane == 0) {
    const int f = i1 + ne * j1;
    fe[f] = accumulate ? fe[f] + fe_scale * s : fe_scale * s;
  }
}

__global__ void sum_vec_kernel(int n, const double* __restrict__ v,
                               double* out) {
  __shared__ double red[256];
  double s = 0.0;
  for (int k = threadIdx.x; k < n; k += blockDim.x) s += v[k];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = red[0];
}

size_t fock_reduce_doubles(int ne, int np) {
  return (size_t)np * np * (((size_t)ne * ne + kRedOut - 1) / kRedOut);
}

cudaError_t launch_fock_reduce(int ne, int np, int nsub, double* part,
                               const double* DE, const double* DP,
                               double fe_scale, int accumulate, double* fe,
                               double* fp, double* fp_part, double* E,
                               cudaStream_t s) {
  const int nfp = (ne * ne + kRedOut - 1) / kRedOut;
  for (int p0 = 0; p0 < np * np; p0 += 65535)   // grid.y limit
    fock_reduce_sub_kernel<<<dim3(nfp, std::min(np * np - p0, 65535)), kRedThreads, 0, s>>>(
        ne, np, nsub, part + (size_t)p0 * ne * nsub * ne, DE, fp_part + (size_t)p0 * nfp);
  fock_reduce_out_kernel<<<(ne * ne + 3) / 4 + 1, kRedThreads, 0, s>>>(
      ne, np, nsub, nfp, part, fp_part, DP, fe_scale, accumulate, fe, fp, E);
  return cudaGetLastError();
}

namespace {

// ---- EG2IC1 --------------------------------------------------------------
// CTA per (ip,jp,i1,i2); thread per j1 (strided), loop over j2.
__global__ void eg2_kernel(int ne, int np, const double* __restrict__ DE,
                           const double* __restrict__ g2,
                           const double* __restrict__ g2s,
                           double* __restrict__ pv, double* __restrict__ ps,
                           long long ipjp0) {
  int cta = blockIdx.x;
  const int i2 = cta % ne; cta /= ne;
  const int i1 = cta % ne; cta /= ne;
  const long long ipjp = cta;
  for (int j1 = threadIdx.x; j1 < ne; j1 += blockDim.x) {
    double av = 0.0, as = 0.0;
    for (int j2 = 0; j2 < ne; j2++) {
      // a12 = (i1,j1,i2,j2), a21 = (i1,j2,i2,j1)
      long long b1 = i1 + (long long)ne * ipjp;
      long long a12 = j2 + (long long)ne * (i2 + (long long)ne * (j1 + (long long)ne * b1));
      long long a21 = j1 + (long long)ne * (i2 + (long long)ne * (j2 + (long long)ne * b1));
      double v = g2[a12] - 0.5 * g2[a21];
      double vs = g2s[a12] - 0.5 * g2s[a21];
      double d = DE[i2 + ne * j2];
      av = fma(d, v, av);
      as = fma(d, vs, as);
    }
    const size_t c = (size_t)blockIdx.x + (size_t)ipjp0 * ne * ne;
    pv[c * ne + j1] = av;
    ps[c * ne + j1] = as;
  }
}

// ---- RXCHF-ne OMG2 (fused FAE / FP / FBE / energy) -----------------------
// GM2ICR viewed as M[r][c], r = (ip,jp,i1,j1), c = (i2,j2) (c fastest).
//   FAE[c]     += sum_r DP(ip,jp) DBE(i1,j1) M[r][c]
//   v[r]        = sum_c DAE[c] M[r][c]
//   FBE(i1,j1) += sum_{ip,jp} DP v[r];  FP(ip,jp) += sum_{i1,j1} DBE v[r]
// Two FP64 FMAs an element are what bounds it (2 per SM and clock: 3.9 ms of
// FMAs at ne = 40, np = 20 against 1.2 ms of HBM), so everything beside them
// is kept off the FP64 pipe and out of its way: a warp works alone (no barrier
// holds back the others' loads) on a panel of 32 * COLS columns, whose DAE and
// FAE stay in registers; it loads the next column's eight rows while it
// multiplies this one's, forms 32 row weights at a time, and sums eight rows'
// dots over its lanes by a transposing butterfly (one addition per row instead
// of five).  Measured there: 7.75 ms with a CTA of 256 threads per row and a
// tree per row, 6.5 ms with register columns but barriers every eight rows,
// 3.7 ms so (95 % of the FP64 pipe).
constexpr int kOmgRows = 8, kOmgCols = 10, kOmgWarps = 2;

// Columns a lane holds: as many as fit, in panels of even size.
__host__ __device__ inline int omg2_panels(int n2) {
  return (n2 + 32 * kOmgCols - 1) / (32 * kOmgCols);
}
inline int omg2_cols(int n2) {
  const int per = (n2 + omg2_panels(n2) - 1) / omg2_panels(n2);
  return (per + 31) / 32;
}

// warps: (row block, column panel), the panels of a row block side by side
template <int COLS>
__global__ void __launch_bounds__(32 * kOmgWarps, 16 / kOmgWarps)
omg2_kernel(int ne, int np, long long nrows, int rows_per_block, int nblocks, int npanels,
            const double* __restrict__ DAE, const double* __restrict__ DBE,
            const double* __restrict__ DP, const double* __restrict__ g2,
            double* __restrict__ fae_part, double* __restrict__ vrow) {
  const int n2 = ne * ne, lane = threadIdx.x & 31;
  const long long w = (long long)blockIdx.x * kOmgWarps + (threadIdx.x >> 5);
  if (w >= (long long)nblocks * npanels) return;
  const int panel = (int)(w % npanels), blk = (int)(w / npanels);
  const int c0 = panel * 32 * COLS + lane;
  const long long r0 = (long long)blk * rows_per_block;
  const long long r1 = min(nrows, r0 + rows_per_block);
  double dae[COLS], fae[COLS];
#pragma unroll
  for (int i = 0; i < COLS; i++) {
    const int c = c0 + i * 32;
    dae[i] = c < n2 ? DAE[c] : 0.0;
    fae[i] = 0.0;
  }
  double u = 0.0;   // weight of row (r - r0) % 32 == lane of the current 32 rows
  for (long long rb = r0; rb < r1; rb += kOmgRows) {
    if (((rb - r0) & 31) == 0) {
      u = 0.0;
      long long rr = rb + lane;
      if (rr < r1) {
        const int j1 = (int)(rr % ne); rr /= ne;
        const int i1 = (int)(rr % ne); rr /= ne;
        const int jp = (int)(rr % np), ip = (int)(rr / np);
        u = DP[ip + np * jp] * DBE[i1 + ne * j1];
      }
    }
    double su[kOmgRows], dot[kOmgRows];
    const int sh = (int)((rb - r0) & 31);
#pragma unroll
    for (int k = 0; k < kOmgRows; k++) {
      su[k] = __shfl_sync(0xffffffffu, u, sh + k);
      dot[k] = 0.0;
    }
    const double* g = g2 + rb * n2 + c0;
    if (rb + kOmgRows <= r1) {
      double m[2][kOmgRows];
#pragma unroll
      for (int k = 0; k < kOmgRows; k++) m[0][k] = c0 < n2 ? __ldcs(g + (long long)k * n2) : 0.0;
#pragma unroll
      for (int i = 0; i < COLS; i++) {
        if (i + 1 < COLS) {
#pragma unroll
          for (int k = 0; k < kOmgRows; k++)
            m[(i + 1) & 1][k] = c0 + (i + 1) * 32 < n2 ? __ldcs(g + (long long)k * n2 + (i + 1) * 32) : 0.0;
        }
#pragma unroll
        for (int k = 0; k < kOmgRows; k++) {
          fae[i] = fma(su[k], m[i & 1][k], fae[i]);
          dot[k] = fma(dae[i], m[i & 1][k], dot[k]);
        }
      }
    } else {
#pragma unroll
      for (int i = 0; i < COLS; i++)
        if (c0 + i * 32 < n2)
#pragma unroll
          for (int k = 0; k < kOmgRows; k++)
            if (rb + k < r1) {
              const double m = __ldcs(g + (long long)k * n2 + i * 32);
              fae[i] = fma(su[k], m, fae[i]);
              dot[k] = fma(dae[i], m, dot[k]);
            }
    }
    // eight rows over 32 lanes: halve the rows a lane holds, then the lanes
#pragma unroll
    for (int h = 4, o = 16; h >= 1; h >>= 1, o >>= 1) {
      const bool up = lane & o;
#pragma unroll
      for (int k = 0; k < h; k++) {
        const double keep = up ? dot[k + h] : dot[k], send = up ? dot[k] : dot[k + h];
        dot[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
      }
    }
    double v = dot[0];   // row 4*(lane bit 4) + 2*(bit 3) + (bit 2)
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    if ((lane & 3) == 0 && rb + (lane >> 2) < r1) vrow[panel * nrows + rb + (lane >> 2)] = v;
  }
#pragma unroll
  for (int i = 0; i < COLS; i++) {
    const int c = c0 + i * 32;
    if (c < n2) fae_part[(size_t)blk * n2 + c] = fae[i];
  }
}

// One warp per output over the row blocks (FAE) or the rows (FBE: over p, FP:
// over (i1,j1)); vrow's column panels are added as they are read.
__global__ void __launch_bounds__(128)
omg2_reduce(int ne, int np, int nparts, int npanels, const double* __restrict__ fae_part,
            const double* __restrict__ vrow, const double* __restrict__ DBE,
            const double* __restrict__ DP, double* FAE, double* FP, double* FBE,
            double* __restrict__ fp_tmp) {
  const int n2 = ne * ne, p2 = np * np, lane = threadIdx.x & 31;
  const long long nrows = (long long)p2 * n2;
  const int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  double s = 0.0;
  auto row = [&](long long r) {
    double v = vrow[r];
    for (int q = 1; q < npanels; q++) v += vrow[q * nrows + r];
    return v;
  };
  if (t < n2) {                       // FAE column c = i2*ne + j2
    for (int k = lane; k < nparts; k += 32) s += fae_part[(size_t)k * n2 + t];
  } else if (t < 2 * n2) {            // FBE(i1,j1)
    for (int p = lane; p < p2; p += 32)
      s = fma(DP[p / np + np * (p % np)], row((long long)p * n2 + t - n2), s);
  } else if (t < 2 * n2 + p2) {       // FP(ip,jp)
    const int p = t - 2 * n2;
    for (int k = lane; k < n2; k += 32)
      s = fma(DBE[k / ne + ne * (k % ne)], row((long long)p * n2 + k), s);
  } else {
    return;
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (lane) return;
  if (t < n2) {
    if (FAE) FAE[t / ne + ne * (t % ne)] += s;
  } else if (t < 2 * n2) {
    const int c = t - n2;
    if (FBE) FBE[c / ne + ne * (c % ne)] += s;
  } else {
    const int p = t - 2 * n2, f = p / np + np * (p % np);
    if (FP) FP[f] += s;
    fp_tmp[p] = DP[f] * s;
  }
}

// Row blocks: 16 warps a SM (the registers' limit), four rounds of them where
// the tensor is long.
int omg2_blocks(long long nrows, int panels) {
  long long want = 152LL * 16 / panels;
  if (want < 1) want = 1;
  if (nrows > want * kOmgRows * 64) want *= 4;
  long long per = (nrows + want - 1) / want;
  per = ((per + kOmgRows - 1) / kOmgRows) * kOmgRows;
  return (int)((nrows + per - 1) / per);
}

__global__ void xcfock_kernel(int ne, int np, double S_total, double H,
                              const double* se1, const double* sp1,
                              const double* se2, const double* sp2,
                              double* focke, double* fockp) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  const double one = 1.0, two = 2.0;
  if (t < ne * ne) {
    focke[t] = (one / S_total) * focke[t] - H * (se1[t] + two * se2[t]);
  } else if (t < ne * ne + np * np) {
    int k = t - ne * ne;
    fockp[k] = (one / S_total) * fockp[k] - H * (sp1[k] + sp2[k]);
  }
}

// ---- index maps (pack_GAM.f) on the device ------------------------------
// kind 0: pack_4D(ne,ne,ne) over (i4,i3,i2,i1) loop order  [GAM_ee]
// kind 2: index_GAM_2PK, 3: index_GAM_3PK, 4: index_GAM_4PK2, each over the
// reference's loop order (ip,jp,ie1,je1,... with the last ket fastest).
__global__ void index_fill_kernel(int kind, int ne, int np, long long count,
                                  long long* __restrict__ out) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
       t < count; t += (long long)gridDim.x * blockDim.x) {
    long long r = t;
    int nidx = kind == 0 ? 4 : 2 + 2 * kind;
    int idx[10];
    for (int k = nidx - 1; k >= 0; k--) {
      int dim = (kind != 0 && k < 2) ? np : ne;
      idx[k] = (int)(r % dim) + 1;
      r /= dim;
    }
    long long ia;
    if (kind == 0) {
      // loop (ie1, je1, ie2, je2) -> pack_4D(je2, ie2, je1, ie1)
      ia = 1 + (idx[3] - 1) + (long long)ne * ((idx[2] - 1) + (long long)ne *
           ((idx[1] - 1) + (long long)ne * (idx[0] - 1)));
    } else {
      // innermost ket first: je_k, ie_k, ..., je1, ie1, jp, ip
      long long acc = idx[0] - 1;                 // ip
      acc = (idx[1] - 1) + (long long)np * acc;   // jp
      for (int k = 2; k < nidx; k++) acc = (idx[k] - 1) + (long long)ne * acc;
      ia = 1 + acc;
    }
    out[t] = ia;
  }
}

}  // namespace

size_t eg3_partial_doubles(int ne, int np) {
  return rank3_weight_doubles(ne, 1) + (size_t)np * np * ne * ne * ne + fock_reduce_doubles(ne, np);
}

cudaError_t launch_eg3_weights(int ne, const double* DE, double* scratch, cudaStream_t s) {
  return launch_rank3_weights_closed(ne, DE, scratch, s);
}

cudaError_t launch_eg3_partials(int ne, int np, long long ipjp0, long long nipjp,
                                const double* g3_slice, double* scratch, cudaStream_t s) {
  if (ne < 1 || ne > 20 || np < 1) return cudaErrorInvalidValue;
  double* part = scratch + rank3_weight_doubles(ne, 1) + (size_t)ipjp0 * ne * ne * ne;
  return launch_rank3_closed(ne, nipjp, g3_slice, scratch, part, s);
}

cudaError_t launch_eg3_reduce(int ne, int np, double* scratch, const double* DE, const double* DP,
                              double* focke, double* fockp, double* E, cudaStream_t s) {
  double* part = scratch + rank3_weight_doubles(ne, 1);
  return launch_fock_reduce(ne, np, ne, part, DE, DP, 3.0, 1, focke, fockp,
                            part + (size_t)np * np * ne * ne * ne, E, s);
}

cudaError_t launch_eg3ic1(int ne, int np, const double* DE, const double* DP,
                          const double* g3, double* scratch, double* focke,
                          double* fockp, double* E, cudaStream_t s) {
  cudaError_t e = launch_eg3_weights(ne, DE, scratch, s);
  if (e != cudaSuccess) return e;
  e = launch_eg3_partials(ne, np, 0, (long long)np * np, g3, scratch, s);
  if (e != cudaSuccess) return e;
  return launch_eg3_reduce(ne, np, scratch, DE, DP, focke, fockp, E, s);
}

size_t eg2_partial_doubles(int ne, int np) {
  return 2 * (size_t)np * np * ne * ne * ne + 2 * fock_reduce_doubles(ne, np);
}

cudaError_t launch_eg2ic1(int ne, int np, const double* DE, const double* DP,
                          const double* g2, const double* g2s,
                          double* scratch, double* FE, double* SE, double* FP,
                          double* SP, double* E, double* S, cudaStream_t s) {
  if (ne < 1 || np < 1) return cudaErrorInvalidValue;
  const size_t npart = (size_t)np * np * ne * ne * ne;
  double* pv = scratch;
  double* ps = scratch + npart;
  double* ftmp = scratch + 2 * npart;
  eg2_kernel<<<(unsigned)(np * np * ne * ne), 32, 0, s>>>(ne, np, DE, g2, g2s,
                                                          pv, ps, 0);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  // FE, FP accumulate (add2fock); SE, SP are overwritten (:379-381)
  e = launch_fock_reduce(ne, np, ne, pv, DE, DP, 2.0, 1, FE, FP, ftmp, E, s);
  if (e != cudaSuccess) return e;
  return launch_fock_reduce(ne, np, ne, ps, DE, DP, 1.0, 0, SE, SP,
                            ftmp + fock_reduce_doubles(ne, np), S, s);
}

cudaError_t launch_eg2_partials(int ne, int np, long long ipjp0,
                                long long nipjp, const double* DE,
                                const double* g2_slice,
                                const double* g2s_slice, double* pv,
                                double* ps, cudaStream_t s) {
  if (ne < 1 || np < 1 || nipjp < 1) return cudaErrorInvalidValue;
  eg2_kernel<<<(unsigned)(nipjp * ne * ne), 32, 0, s>>>(
      ne, np, DE, g2_slice, g2s_slice, pv, ps, ipjp0);
  return cudaGetLastError();
}

size_t omg2_partial_doubles(int ne, int np) {
  const long long nrows = (long long)np * np * ne * ne;
  const int n2 = ne * ne, panels = omg2_panels(n2);
  return (size_t)omg2_blocks(nrows, panels) * ne * ne + (size_t)nrows * panels + np * np;
}

cudaError_t launch_rxchfne_omg2(int ne, int np, const double* DAE,
                                const double* DBE, const double* DP,
                                const double* g2, double* scratch, double* FAE,
                                double* FP, double* FBE, double* E,
                                cudaStream_t s) {
  if (ne < 1 || np < 1 || ne * ne > 16384) return cudaErrorInvalidValue;
  const int n2 = ne * ne, panels = omg2_panels(n2);
  const long long nrows = (long long)np * np * n2;
  const int want = omg2_blocks(nrows, panels);
  const long long per = (nrows + want - 1) / want;
  const int rows = (int)(((per + kOmgRows - 1) / kOmgRows) * kOmgRows);
  const int grid = (int)((nrows + rows - 1) / rows);
  double* fae_part = scratch;
  double* vrow = scratch + (size_t)want * n2;
  double* fp_tmp = vrow + nrows * panels;
  const unsigned ctas = (unsigned)(((long long)grid * panels + kOmgWarps - 1) / kOmgWarps);
#define OMG(C) omg2_kernel<C><<<ctas, 32 * kOmgWarps, 0, s>>>(ne, np, nrows, rows, grid, panels, DAE, DBE, DP, g2, fae_part, vrow)
  switch (omg2_cols(n2)) {   // no empty columns in the panels
    case 1: OMG(1); break;
    case 2: OMG(2); break;
    case 3: OMG(3); break;
    case 4: OMG(4); break;
    case 5: OMG(5); break;
    case 6: OMG(6); break;
    case 7: OMG(7); break;
    case 8: OMG(8); break;
    case 9: OMG(9); break;
    default: OMG(10); break;
  }
#undef OMG
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  const int nout = 2 * n2 + np * np;
  omg2_reduce<<<(nout + 3) / 4, 128, 0, s>>>(ne, np, grid, panels, fae_part, vrow, DBE, DP, FAE,
                                             FP, FBE, fp_tmp);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  sum_vec_kernel<<<1, 256, 0, s>>>(np * np, fp_tmp, E);
  return cudaGetLastError();
}

cudaError_t launch_xcfock_correction(int ne, int np, double S_total,
                                     double H_expect, const double* se1,
                                     const double* sp1, const double* se2,
                                     const double* sp2, double* focke,
                                     double* fockp, cudaStream_t s) {
  int n = ne * ne + np * np;
  xcfock_kernel<<<(n + 127) / 128, 128, 0, s>>>(ne, np, S_total, H_expect,
                                                se1, sp1, se2, sp2, focke,
                                                fockp);
  return cudaGetLastError();
}

cudaError_t launch_index_fill(int kind, int ne, int np, int64_t count,
                              int64_t* out, cudaStream_t s) {
  if (!(kind == 0 || (kind >= 2 && kind <= 4))) return cudaErrorInvalidValue;
  long long blocks = (count + 255) / 256;
  if (blocks > 152 * 32) blocks = 152 * 32;
  if (blocks < 1) blocks = 1;
  index_fill_kernel<<<(unsigned)blocks, 256, 0, s>>>(
      kind, ne, np, count, reinterpret_cast<long long*>(out));
  return cudaGetLastError();
}

}  // namespace neoxc
