// k_rank3.cu -- contractions of a stored rank-3 tensor G(p; i1 x, i2 y, i3 z)
// (GM3ICR) with two densities, for sm_103a: EG3IC1 (gam3_IC1_OMP.f:433-725)
// and the open-shell FAE_OMG3 / UFP_OMG3 (xcuhf/xcuhf_omg3.f:2-588).
//
// The reference forms, for every ket tuple (j1,j2,j3), a combination of the
// six ket permutations of G and weights it with densities of electrons 2 and
// 3.  Read from the stored element instead, G(x,y,z) enters the Fock row of
// x, of y and of z (the row's ket sits in slot 0, 1 or 2), each time with a
// weight of the other two kets that depends only on (i2,i3) and the
// densities:
//   row[j] += sum_uv G(j,u,v) W0(u,v) + G(u,j,v) W1(u,v) + G(u,v,j) W2(u,v).
// The weights are tabulated once per call (they serve every proton pair and
// i1; see kFormNE for the smallest calls), so an element costs 3 FP64 FMAs a class instead of the 9 to 14 FP64
// operations of forming the combinations.  FP64 issue (2 per SM and clock)
// is still what bounds it: 3 FMAs take 4.4x the time of the element's 8
// bytes from HBM.  A CTA owns (p, i1, i2) and walks i3 or a share of it, so one
// partial row is written per (p, i1, i2) and share.
// Measured (one GB300, whole call): EG3IC1 at ne = 12, np = 8 (1.5 GB) 6.69 ms
// with the combinations formed per ket tuple and a serial reduction, 1.12 ms
// so (3 FMAs an element at the measured FP64 rate: 1.08 ms); open shell at
// ne = 12, np = 4 (0.38 GB, two classes) 1.48 and 0.61 ms (0.54 ms).
#include "neoxc_internal.h"

namespace neoxc {
namespace {

constexpr int kThreads = 256;

// Open shell with few protons: a CTA per (p, i1, i2) that walks all of i3 leaves
// most of the chip idle (np = 1: 16 CTAs at ne = 4, 100 at ne = 10), so the walk
// is cut into shares until there are kFillCtas of them; up to kFormNE the CTAs
// then form the weights themselves, for the table is one launch more.  Whole
// calls (one GB300, us; the kernel without tables, one step per CTA / one share /
// shares / shares that form the weights): ne = 4, np = 1 40 / 45 / 39 / 33;
// ne = 6, np = 2 50 / 54 / 45 / 41; ne = 8, np = 1 46 / 60 / 43 / 39; ne = 10, np = 1
// 74 / 76 / 54 / 54; ne = 12, np = 1 131 / 105 / 76 / 82.  Cut for 152 x 8 CTAs instead,
// ne = 8, np = 2 takes 64 us for 56, ne = 12, np = 1 83 for 76.
constexpr long long kFillCtas = 152 * 4;
constexpr int kFormNE = 8;

// x / d for x < 65536, 2 <= d <= 256, by one multiply-high
struct DivN {
  unsigned d, m;
  __device__ explicit DivN(int n)
      : d((unsigned)n), m((unsigned)(((1ull << 32) + (unsigned)n - 1) / (unsigned)n)) {}
  __device__ unsigned operator()(unsigned x) const { return d == 1 ? x : __umulhi(x, m); }
};

__global__ void weights_closed_kernel(int ne, const double* __restrict__ DE,
                                      double* __restrict__ W) {
  const int n2 = ne * ne;
  const long long n4 = (long long)n2 * n2;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n4;
       t += (long long)gridDim.x * blockDim.x) {
    const int uv = (int)(t % n2), i = (int)(t / n2);
    const int u = uv / ne, v = uv - u * ne, i2 = i / ne, i3 = i - i2 * ne;
    const double uu = DE[i2 + ne * u] * DE[i3 + ne * v];   // electrons 2, 3 at (u, v)
    const double vv = DE[i2 + ne * v] * DE[i3 + ne * u];   // and exchanged
    // (8 o123 - 4 o213 + 2 o312 - 4 o132 + 2 o231 - 4 o321) / 8
    W[t] = uu - 0.5 * vv;
    W[n4 + t] = 0.25 * vv - 0.5 * uu;
    W[2 * n4 + t] = 0.25 * uu - 0.5 * vv;
  }
}

// Weights of the ket pair (u,v) of electrons (i2,i3) for one class with flags f
// (bit 0: the six-term set, bit 1: the two mixed pairs, bit 2: the 23 pair;
// FAE_OMG3's LAA, LAB, LBB); A, B: the class's densities of its own and of the
// other spin
__device__ __forceinline__ void open_weights(int ne, const double* __restrict__ A,
                                             const double* __restrict__ B, unsigned f, int i2,
                                             int i3, int u, int v, double* w) {
  const double a2u = A[i2 + ne * u], a2v = A[i2 + ne * v], a3u = A[i3 + ne * u], a3v = A[i3 + ne * v];
  const double b2u = B[i2 + ne * u], b2v = B[i2 + ne * v], b3u = B[i3 + ne * u], b3v = B[i3 + ne * v];
  double w0 = 0.0, w1 = 0.0, w2 = 0.0;
  if (f & 1u) {
    const double x = a2u * a3v - a2v * a3u;
    w0 += x;
    w1 -= x;
    w2 += x;
  }
  if (f & 2u) {
    w0 += a2u * b3v + b2u * a3v;
    w1 -= a2u * b3v;
    w2 -= b2v * a3u;
  }
  if (f & 4u) w0 += b2u * b3v - b2v * b3u;
  w[0] = w0;
  w[1] = w1;
  w[2] = w2;
}

// class B exchanges the spins
__global__ void weights_open_kernel(int ne, const double* __restrict__ DA,
                                    const double* __restrict__ DB, unsigned fa, unsigned fb,
                                    double* __restrict__ W) {
  const int n2 = ne * ne;
  const long long n4 = (long long)n2 * n2;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < 2 * n4;
       t += (long long)gridDim.x * blockDim.x) {
    const int c = t >= n4;
    const long long r = t - c * n4;
    const int uv = (int)(r % n2), i = (int)(r / n2);
    double w[3];
    open_weights(ne, c ? DB : DA, c ? DA : DB, c ? fb : fa, i / ne, i % ne, uv / ne, uv % ne, w);
    for (int s = 0; s < 3; s++) W[((size_t)c * 3 + s) * n4 + r] = w[s];
  }
}

// NC classes; USED: bit c = class c has weights.  Threads (j, q): ket j of the
// row, q strides the pairs (u,v).  CTA y of a (p, i1, i2) takes its share of i3
// and writes a partial row of its own.  FORM (NC = 2): the weights are formed
// here, of flags fa and fb, and W is not read.  Eight CTAs an SM, six with FORM:
// with 40 registers for 32, ne = 12, np = 4 took 611 us for 601; with all that
// FORM would take, ne = 7, np = 2 57 for 48.
template <int NC, unsigned USED, bool FORM>
__global__ void __launch_bounds__(kThreads, FORM ? 6 : 8)
rank3_kernel(int ne, const double* __restrict__ G, const double* __restrict__ W,
             const double* __restrict__ DA, const double* __restrict__ DB, unsigned fa,
             unsigned fb, double* __restrict__ part, double* __restrict__ ppart) {
  extern __shared__ double sm[];
  const int n2 = ne * ne, n3 = n2 * ne;
  const long long n4 = (long long)n2 * n2;
  // odd pitches: lanes that differ in one ket index hit different banks
  const int pt1 = ne | 1, pt0 = (pt1 * ne) | 1;
  double* sG = sm;                       // [x * pt0 + y * pt1 + z]
  double* sW = sG + pt0 * ne;            // [class][slot][u * ne + v]
  double* sred = sW + 3 * NC * n2;       // [blockDim]
  const DivN dv(ne);
  const long long cta = blockIdx.x;
  const int i2 = (int)(cta % ne);
  const long long pi1 = cta / ne;        // p * ne + i1
  const int lanes = blockDim.x / ne;
  const int q0 = (int)dv(threadIdx.x), j = threadIdx.x - q0 * ne;
  // element (x, y, z) of (p, i1, i2, i3): ((pi1 ne + x) ne + i2) ne^3 + y n2 + i3 ne + z
  const double* g0 = G + (pi1 * ne * ne + i2) * (long long)n3;
  double acc[NC];
#pragma unroll
  for (int c = 0; c < NC; c++) acc[c] = 0.0;
  const int i3end = ne * ((int)blockIdx.y + 1) / (int)gridDim.y;
  for (int i3 = ne * (int)blockIdx.y / (int)gridDim.y; i3 < i3end; i3++) {
    __syncthreads();
    for (int k = threadIdx.x; k < n3; k += blockDim.x) {
      const int xy = (int)dv((unsigned)k), z = k - xy * ne;
      const int x = (int)dv((unsigned)xy), y = xy - x * ne;
      sG[x * pt0 + y * pt1 + z] = __ldg(g0 + (long long)x * n4 + (long long)y * n2 + i3 * ne + z);
    }
    if constexpr (FORM) {
      for (int k = threadIdx.x; k < NC * n2; k += blockDim.x) {
        const int c = k >= n2, uv = k - c * n2, u = (int)dv((unsigned)uv);
        double w[3];
        open_weights(ne, c ? DB : DA, c ? DA : DB, c ? fb : fa, i2, i3, u, uv - u * ne, w);
        for (int s = 0; s < 3; s++) sW[(3 * c + s) * n2 + uv] = w[s];
      }
    } else {
      const double* w = W + (long long)(i2 * ne + i3) * n2;
#pragma unroll
      for (int s = 0; s < 3 * NC; s++)
        if (USED & (1u << (s / 3)))
          for (int k = threadIdx.x; k < n2; k += blockDim.x) sW[s * n2 + k] = __ldg(w + s * n4 + k);
    }
    __syncthreads();
    if (q0 < lanes) {
#pragma unroll 2
      for (int q = q0; q < n2; q += lanes) {
        const int u = (int)dv((unsigned)q), v = q - u * ne;
        const double a = sG[j * pt0 + u * pt1 + v];
        const double b = sG[u * pt0 + j * pt1 + v];
        const double d = sG[u * pt0 + v * pt1 + j];
#pragma unroll
        for (int c = 0; c < NC; c++)
          if (USED & (1u << c)) {
            acc[c] = fma(a, sW[(3 * c) * n2 + q], acc[c]);
            acc[c] = fma(b, sW[(3 * c + 1) * n2 + q], acc[c]);
            acc[c] = fma(d, sW[(3 * c + 2) * n2 + q], acc[c]);
          }
      }
    }
  }
  double row[NC];
  const long long out = cta * gridDim.y + blockIdx.y;
#pragma unroll
  for (int c = 0; c < NC; c++) {
    __syncthreads();
    sred[threadIdx.x] = acc[c];
    __syncthreads();
    row[c] = 0.0;
    if ((int)threadIdx.x < ne) {
      for (int t = threadIdx.x; t < lanes * ne; t += ne) row[c] += sred[t];
      part[(out * NC + c) * ne + threadIdx.x] = row[c];
    }
  }
  if constexpr (NC == 2) {
    // the proton terms of this CTA, in a fixed order
    const int i1 = (int)(pi1 % ne);
    __syncthreads();
    if ((int)threadIdx.x < ne)
      sred[threadIdx.x] = DA[i1 + ne * threadIdx.x] * row[0] + DB[i1 + ne * threadIdx.x] * row[1];
    __syncthreads();
    if (threadIdx.x == 0) {
      double s = 0.0;
      for (int k = 0; k < ne; k++) s += sred[k];
      ppart[out * 2] = s;
    }
  }
}

template <int NC, unsigned USED, bool FORM>
cudaError_t launch_t(int ne, long long nipjp, int split, const double* G, const double* W,
                     const double* DA, const double* DB, unsigned fa, unsigned fb, double* part,
                     double* ppart, cudaStream_t s) {
  // no more groups of ne threads than ket pairs: small ne takes small CTAs
  int lanes = kThreads / ne;
  if (lanes > ne * ne) lanes = ne * ne;
  const int bs = lanes * ne, pt1 = ne | 1, pt0 = (pt1 * ne) | 1;
  const size_t smem = sizeof(double) * ((size_t)pt0 * ne + 3 * NC * (size_t)ne * ne + bs);
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(rank3_kernel<NC, USED, FORM>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  rank3_kernel<NC, USED, FORM><<<dim3((unsigned)(nipjp * ne * ne), split), bs, smem, s>>>(
      ne, G, W, DA, DB, fa, fb, part, ppart);
  return cudaGetLastError();
}

int wgrid(long long n) { return (int)((n + 255) / 256 < 152 * 16 ? (n + 255) / 256 : 152 * 16); }

}  // namespace

size_t rank3_weight_doubles(int ne, int ncls) {
  return 3 * (size_t)ncls * ne * ne * ne * ne;
}

cudaError_t launch_rank3_weights_closed(int ne, const double* DE, double* W, cudaStream_t s) {
  weights_closed_kernel<<<wgrid((long long)ne * ne * ne * ne), 256, 0, s>>>(ne, DE, W);
  return cudaGetLastError();
}

int rank3_split(int ne, long long nipjp) {
  const long long fill = kFillCtas / (nipjp * ne * ne);
  return (int)(fill < 1 ? 1 : (fill > ne ? ne : fill));
}

cudaError_t launch_rank3_closed(int ne, long long nipjp, const double* G, const double* W,
                                double* part, cudaStream_t s) {
  if (ne < 1 || ne > 28 || nipjp < 1) return cudaErrorInvalidValue;
  return launch_t<1, 1u, false>(ne, nipjp, 1, G, W, nullptr, nullptr, 0u, 0u, part, nullptr, s);
}

cudaError_t launch_rank3_open(int ne, long long nipjp, const double* G, const double* DA,
                              const double* DB, unsigned fa, unsigned fb, double* W, double* part,
                              double* ppart, cudaStream_t s) {
  if (ne < 1 || ne > 28 || nipjp < 1) return cudaErrorInvalidValue;
  const int n = rank3_split(ne, nipjp);
  const unsigned used = (fa ? 1u : 0u) | (fb ? 2u : 0u);
#define R3(U, F) launch_t<2, U, F>(ne, nipjp, n, G, W, DA, DB, fa, fb, part, ppart, s)
  if (n > 1 && ne <= kFormNE)
    return used == 3u ? R3(3u, true) : used == 2u ? R3(2u, true) : used == 1u ? R3(1u, true) : R3(0u, true);
  weights_open_kernel<<<wgrid(2LL * ne * ne * ne * ne), 256, 0, s>>>(ne, DA, DB, fa, fb, W);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  return used == 3u ? R3(3u, false) : used == 2u ? R3(2u, false) : used == 1u ? R3(1u, false) : R3(0u, false);
#undef R3
}

}  // namespace neoxc
