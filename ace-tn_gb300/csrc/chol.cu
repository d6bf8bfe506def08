// FP64 Cholesky factorisation and inverse factor on a cluster.
//
// The one-CTA cholesky_kernel<double> is bound by one SM's FP64 units (1.7 FMAs
// per cycle; q^3 / 3 of them with the inverse) and by one thread's chain through
// each diagonal block.  Here the rows (of the upper triangle W of G + shift I and
// of the identity E, eliminated together) are spread over a cluster in blocks of
// eight, block b on CTA b mod P.  Per block: the owner eliminates the diagonal
// block with one warp (lanes hold columns, reciprocals from FP32 seeds), then its
// eight rows at all columns, and writes the finished rows into every CTA's
// buffer; one cluster barrier later all CTAs subtract them from their rows below.
// Two buffers by parity, so that one barrier per block is enough.
//
// q = 66, 80, 160: 132, 153, 625 us as cholesky_kernel, 72, 86, 224 us here.
#include <cooperative_groups.h>

#include "engine.cuh"
#include "seeded.cuh"

namespace ctm {

namespace {

constexpr int kNb = 8;
constexpr int kCThreads = 256;
constexpr size_t kCSmem = 222 * 1024;

struct CholArgs {
  const double* G;
  int q, q8;        // q8: q rounded up to 8
  double shift_factor;
  double* Linv;     // q x q lower
  double* Lt;       // q x q upper, or null
  int* flags;
};

// Doubles per row: W, then E.
__host__ __device__ inline int chol_row(int q8) { return 2 * q8 + 2; }

inline size_t chol_smem(int64_t q8, int64_t P) {
  const int64_t blocks = q8 / kNb, local = (blocks + P - 1) / P;
  const size_t rs = size_t(chol_row(int(q8)));
  // own rows; two buffers of eight rows and their reciprocals; scaled multipliers
  return (size_t(local) * kNb * rs + 2 * (kNb * rs + kNb) + size_t(local) * kNb * kNb +
          size_t(local) * kNb + kNb * kNb) * sizeof(double);
}

__global__ void __launch_bounds__(kCThreads) cholesky_cluster_kernel(const CholArgs a) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const int P = int(cluster.num_blocks()), me = int(cluster.block_rank());
  const int q = a.q, q8 = a.q8, RS = chol_row(q8), blocks = q8 / kNb;
  const int local = (blocks + P - 1) / P;
  extern __shared__ __align__(16) double csm[];
  double* A = csm;                                   // local * 8 rows
  double* pan = A + size_t(local) * kNb * RS;        // [2][8 rows, then 8 reciprocals]
  const int PS = kNb * RS + kNb;
  double* S = pan + 2 * PS;                          // [local * 8][8]
  double* piv = S + size_t(local) * kNb * kNb;       // pivots of the own rows
  double* mul = piv + size_t(local) * kNb;           // [8][8]
  __shared__ double s_tr[kCThreads / 32];
  __shared__ int s_fail;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int kWarps = kCThreads / 32;
  auto row_of = [&](int l) { return ((l >> 3) * P + me) * kNb + (l & 7); };  // own row l
  double tr = 0.0;
  for (int i = tid; i < q; i += kCThreads) tr += a.G[size_t(i) * q + i];
  for (int o = 16; o > 0; o >>= 1) tr += __shfl_xor_sync(0xffffffffu, tr, o);
  if (lane == 0) s_tr[warp] = tr;
  if (tid == 0) s_fail = 0;
  for (int l = warp; l < local * kNb; l += kWarps) {
    const int r = row_of(l);
    double* row = A + size_t(l) * RS;
    for (int c = lane; c < q8; c += 32) {
      row[c] = r < q && c < q && c >= r ? a.G[size_t(r) * q + c] : 0.0;
      row[q8 + c] = r == c ? 1.0 : 0.0;
    }
  }
  __syncthreads();
  tr = 0.0;
  for (int w = 0; w < kWarps; ++w) tr += s_tr[w];
  const double shift = a.shift_factor * tr;
  for (int l = tid; l < local * kNb; l += kCThreads) {
    const int r = row_of(l);
    if (r < q) A[size_t(l) * RS + r] += shift;
  }
  if (P > 1) cluster.sync();
  else __syncthreads();
  // elimination inside diagonal block b, by one warp: lane v < 8 holds column v
  auto diagonal = [&](int b) {
    const int r0 = b * kNb;
    double* rows = A + size_t(b / P) * kNb * RS;
    double* buf = pan + (b & 1) * PS;
    const int v = lane & 7;
    double x[kNb];
#pragma unroll
    for (int t = 0; t < kNb; ++t) x[t] = rows[t * RS + r0 + v];
    bool fail = false;
#pragma unroll
    for (int t = 0; t < kNb; ++t) {
      const double d = __shfl_sync(0xffffffffu, x[t], t);
      const long long bits = __double_as_longlong(d);  // d > 0 (and no NaN)
      const bool ok = r0 + t < q && bits > 0 && bits <= 0x7ff0000000000000ll;
      fail = fail || (r0 + t < q && !ok);
      const double rd = ok ? positive_reciprocal(d) : 0.0;
      const double y = x[t] * rd;  // lane r: the multiplier of row r
      if (lane == t) {
        piv[(b / P) * kNb + t] = ok ? d : 0.0;
        buf[kNb * RS + t] = rd;
      }
      if (lane < kNb) mul[t * kNb + lane] = lane > t ? y : 0.0;
#pragma unroll
      for (int r = t + 1; r < kNb; ++r) {
        const double m = __shfl_sync(0xffffffffu, y, r);
        x[r] = fma(-m, x[t], x[r]);
      }
    }
    if (fail && lane == 0) s_fail = 1;
  };
  if (me == 0 && warp == 0) diagonal(0);
  __syncthreads();
  for (int b = 0; b < blocks; ++b) {
    const int r0 = b * kNb, owner = b % P;
    double* buf = pan + (b & 1) * PS;
    if (me == owner) {
      double* rows = A + size_t(b / P) * kNb * RS;
      // the eight rows at the columns of W from r0 on and of E below r0 + 8
      const int nw = (q8 - r0 + 31) / 32, ne = (r0 + kNb + 31) / 32;
      for (int ch = warp; ch < nw + ne; ch += kWarps) {
        const int c = ch < nw ? r0 + ch * 32 + lane : q8 + (ch - nw) * 32 + lane;
        const bool in = ch < nw ? c < q8 : c < q8 + r0 + kNb;
        double x[kNb];
#pragma unroll
        for (int t = 0; t < kNb; ++t)
          x[t] = in && (ch >= nw || r0 + t <= c) ? rows[t * RS + c] : 0.0;
#pragma unroll
        for (int t = 0; t < kNb; ++t)
#pragma unroll
          for (int r = t + 1; r < kNb; ++r) x[r] = fma(-mul[t * kNb + r], x[t], x[r]);
        if (in) {
#pragma unroll
          for (int t = 0; t < kNb; ++t)
            if (ch >= nw || r0 + t <= c) rows[t * RS + c] = x[t];
          for (int p = 0; p < P; ++p) {
            double* dst = P > 1 ? cluster.map_shared_rank(buf, p) : buf;
#pragma unroll
            for (int t = 0; t < kNb; ++t) dst[t * RS + c] = x[t];
          }
        }
      }
      if (P > 1 && warp == 0 && lane < kNb)  // (written by this warp above)
        for (int p = 0; p < P; ++p)
          if (p != me) cluster.map_shared_rank(buf, p)[kNb * RS + lane] = buf[kNb * RS + lane];
    }
    if (P > 1) cluster.sync();
    else __syncthreads();
    // own rows below the block: row -= sum_t (W[t][row] / d_t) pivot row t
    const int lb = (b + 1 - me + P - 1) / P;  // first own block above b, b * P + me > b
    const int l0 = max(lb, 0) * kNb;
    for (int i = l0 * kNb + tid; i < local * kNb * kNb; i += kCThreads) {
      const int l = i >> 3, t = i & 7, r = row_of(l);
      S[i] = r < q8 ? buf[t * RS + r] * buf[kNb * RS + t] : 0.0;
    }
    __syncthreads();
    // the next block's owner brings its diagonal block up to date first and
    // eliminates inside it with one warp while the others do the rest
    const bool next = b + 1 < blocks && (b + 1) % P == me;
    if (next) {
      const int l = (b + 1) / P * kNb + warp, c = r0 + kNb + (lane & 7);
      double* row = A + size_t(l) * RS;
      double y = row[c];
#pragma unroll
      for (int t = 0; t < kNb; ++t) y = fma(-S[l * kNb + t], buf[t * RS + c], y);
      if (lane < kNb) row[c] = y;
      __syncthreads();
      if (warp == 0) diagonal(b + 1);
    }
    const int nw = (q8 - r0 - kNb + 31) / 32, ne = (r0 + kNb + 31) / 32;
    const int w0 = next ? warp - 1 : warp, wn = next ? kWarps - 1 : kWarps;
    for (int ch = w0 < 0 ? nw + ne : w0; ch < nw + ne; ch += wn) {
      const bool w = ch < nw;
      const int c = w ? r0 + kNb + ch * 32 + lane : q8 + (ch - nw) * 32 + lane;
      const bool in = w ? c < q8 : c < q8 + r0 + kNb;
      double x[kNb];
#pragma unroll
      for (int t = 0; t < kNb; ++t) x[t] = in ? buf[t * RS + c] : 0.0;
      const int last = r0 + kNb + ch * 32 + 31;  // W: rows past the chunk's columns are done
      for (int l = l0; l < local * kNb; ++l) {
        const int r = row_of(l);
        if (r >= q8 || (w && r > last)) break;
        double* row = A + size_t(l) * RS;
        const bool done = next && ch == 0 && lane < kNb && (r >> 3) == b + 1;
        double y = in ? row[c] : 0.0;
#pragma unroll
        for (int t = 0; t < kNb; ++t) y = fma(-S[l * kNb + t], x[t], y);
        if (in && !done) row[c] = y;
      }
    }
    __syncthreads();
  }
  if (tid == 0 && s_fail) atomicOr(a.flags, 1);
  // L^-1 = diag(d)^-1/2 E, L^T = diag(d)^-1/2 W with sqrt(d) on its diagonal
  for (int l = warp; l < local * kNb; l += kWarps) {
    const int r = row_of(l);
    if (r >= q) continue;
    const double d = piv[l], sq = d > 0.0 ? sqrt(d) : 0.0, rs = d > 0.0 ? 1.0 / sq : 0.0;
    const double* row = A + size_t(l) * RS;
    for (int c = lane; c < q; c += 32) {
      a.Linv[size_t(r) * q + c] = c <= r ? row[q8 + c] * rs : 0.0;
      if (a.Lt != nullptr) a.Lt[size_t(r) * q + c] = c > r ? row[c] * rs : (c == r ? sq : 0.0);
    }
  }
  if (P > 1) cluster.sync();  // no CTA leaves while others may write its buffers
}

int chol_ctas(int64_t q) {
  const int64_t q8 = (q + kNb - 1) / kNb * kNb;
  for (int P : {4, 8, 16}) {
    if (P > max_cluster_ctas()) break;
    if (P < 16 && q8 / kNb > 3 * P) continue;  // at most three blocks of rows per CTA
    if (chol_smem(q8, P) <= kCSmem) return P;
  }
  for (int P : {16, 8})
    if (P <= max_cluster_ctas() && chol_smem(q8, P) <= kCSmem) return P;
  return 0;
}

}  // namespace

bool cholesky_cluster_fits(int64_t q) { return q <= 1024 && chol_ctas(q) > 0; }

void cholesky_cluster(Ctx& c, const double* G, int64_t q, double shift_factor, double* Linv,
                      double* Lt, int* flags) {
  const int P = chol_ctas(q);
  CholArgs a{};
  a.G = G;
  a.q = int(q);
  a.q8 = int((q + kNb - 1) / kNb * kNb);
  a.shift_factor = shift_factor;
  a.Linv = Linv;
  a.Lt = Lt;
  a.flags = flags;
  const size_t smem = chol_smem(a.q8, P);
  CTM_CUDA(cudaFuncSetAttribute(cholesky_cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
  CTM_CUDA(cudaFuncSetAttribute(cholesky_cluster_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  KernelTimer kt(c.stream, "cholesky_cluster_kernel", kUnitFlop, double(q) * q * q / 3.0);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(P));
  cfg.blockDim = dim3(kCThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = c.stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = unsigned(P);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  CTM_CUDA(cudaLaunchKernelEx(&cfg, cholesky_cluster_kernel, a));
  CTM_LAUNCH_CHECK();
}

}  // namespace ctm
