// FP64 Householder QR of a small tall matrix in the shared memory of a cluster.
//
// What bounds it: the latency of one column (an FP64 instruction issues once in
// 64 cycles per SM quarter, a cluster barrier with its remote stores takes
// about 1500 cycles), so a column costs one all-reduce and one pass over the
// rows.  Rows are spread over the CTAs and, inside a CTA, over four warps (one
// per SM quarter); lanes hold columns.  In column j every CTA needs
//   d[t] = sum_{i >= j} A[i][j] A[i][t]   (t >= j, one all-reduce) and row j;
// with alpha = -sign(A[j][j]) sqrt(d[j]) and v = A[:, j] - alpha e_j, the products
// v^T A[:, t] for the trailing columns are d[t] - alpha A[j][t].  The update of the
// rows and the sums of the next column's d are one pass.  Afterwards the strict
// upper triangle U of V^T V is formed and summed over the CTAs once, and Q = [I; 0] -
// V M with (diag(1 / beta) + U) M = V_1^T (the compact WY form; V_1: the first q rows
// of V): one triangular solve, its columns shared among the CTAs, and one product
// instead of q more all-reduces.
//
// 144 x 144: 909 us (1654 with the sums of d over all columns and the solve on every
// CTA).
// 80 x 22: 59 us (783 as householder_qr_kernel, two CTA reductions per column
// pair on one CTA).
#include <cooperative_groups.h>

#include <algorithm>

#include "engine.cuh"
#include "seeded.cuh"

namespace ctm {

namespace {

constexpr int kQrWarps = 4;
constexpr int kQrThreads = 32 * kQrWarps;
constexpr size_t kQrSmem = 224 * 1024;

struct QrArgs {
  double* Y;  // n x q, in: the matrix, out: Q
  double* R;  // q x q upper triangular, or null
  int n, q, nr;  // nr: rows per CTA
};

__host__ __device__ inline int qr_ld(int q) { return q | 1; }

inline size_t qr_smem(int64_t nr, int64_t q, int64_t P) {
  const size_t ld = size_t(qr_ld(int(q)));
  // rows; U and M; partial sums and row j by parity; warp sums; betas, diagonals
  return (size_t(nr) * ld + size_t(q) * ld + 2 * size_t(P + 1) * q + size_t(kQrWarps) * q +
          2 * size_t(q)) * sizeof(double);
}

template <int NC>  // column chunks of 32 lanes
__global__ void __launch_bounds__(kQrThreads) householder_cluster_kernel(const QrArgs a) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const int P = int(cluster.num_blocks()), me = int(cluster.block_rank());
  const int n = a.n, q = a.q, nr = a.nr, ld = qr_ld(q);
  extern __shared__ __align__(16) double qsm[];
  double* A = qsm;                        // nr x ld
  double* S = A + size_t(nr) * ld;        // q x ld: U above the diagonal, X^T on and below
  double* part = S + size_t(q) * ld;      // [2][P + 1][q]: partial sums by CTA, then row j
  double* red = part + 2 * size_t(P + 1) * q;  // [kQrWarps][q]
  double* betas = red + kQrWarps * q;
  double* diag = betas + q;               // R's diagonal
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int row0 = me * nr, rows = max(0, min(nr, n - row0));
  for (int i = warp; i < rows; i += kQrWarps)
    for (int t = lane; t < q; t += 32) A[i * ld + t] = a.Y[size_t(row0 + i) * q + t];
  auto sync_all = [&] {
    if (P > 1) cluster.sync();
    else __syncthreads();
  };
  sync_all();
  // more than 32 columns: U is formed at the end (one column chunk has no finished
  // chunks to skip, and its products with the earlier vectors come with the sums)
  constexpr bool kLate = NC > 1;
  double g[NC], acc[NC];
  double vj = 0.0;
  for (int j = 0; j <= q; ++j) {
    // update with column j - 1 (coefficients g, vectors in place) and the sums
    // of column j, in one pass over the rows >= j (row j - 1: its R entries)
#pragma unroll
    for (int c = 0; c < NC; ++c) acc[c] = 0.0;
    const int lo = max(0, j - 1 - row0);
    for (int i = lo + (warp - lo % kQrWarps + kQrWarps) % kQrWarps; i < rows; i += kQrWarps) {
      double* row = A + i * ld;
      double x[NC];
#pragma unroll
      for (int c = 0; c < NC; ++c)
        x[c] = (!kLate || 32 * c + 31 >= j) && lane + 32 * c < q ? row[lane + 32 * c] : 0.0;
      if (j > 0) {
        const bool pivot = row0 + i == j - 1;
        const double v = pivot ? vj : row[j - 1];
        __syncwarp();
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          const int t = lane + 32 * c;
          if (32 * c + 31 >= j && t >= j && t < q) {  // no FP64 issue slot for finished chunks
            x[c] = fma(-g[c], v, x[c]);
            row[t] = x[c];
          }
        }
        if (pivot) {
          if (lane == 0) row[j - 1] = vj;
          continue;
        }
      }
      if (j < q) {
        double xj = 0.0;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          const double s = __shfl_sync(0xffffffffu, x[c], j & 31);
          if (c == j >> 5) xj = s;
        }
#pragma unroll
        for (int c = 0; c < NC; ++c)
          if (!kLate || 32 * c + 31 >= j) acc[c] = fma(xj, x[c], acc[c]);
      }
    }
    if (j == q) break;
#pragma unroll
    for (int c = 0; c < NC; ++c)
      if ((!kLate || 32 * c + 31 >= j) && lane + 32 * c < q) red[warp * q + lane + 32 * c] = acc[c];
    __syncthreads();
    double* buf = part + (j & 1) * size_t(P + 1) * q;
    for (int t = (kLate ? j : 0) + tid; t < q; t += kQrThreads) {
      double s = red[t];
#pragma unroll
      for (int w = 1; w < kQrWarps; ++w) s += red[w * q + t];
      const bool owner = j >= row0 && j < row0 + rows;
      const double rj = owner ? A[(j - row0) * ld + t] : 0.0;
      for (int r = 0; r < P; ++r) {
        double* dst = P > 1 ? cluster.map_shared_rank(buf, r) : buf;
        dst[me * q + t] = s;
        if (owner) dst[P * q + t] = rj;
      }
    }
    sync_all();
    double d[NC], rj[NC];
    if (NC > 2) {  // each warp sums its share of the columns
      for (int t = j + tid; t < q; t += kQrThreads) {
        double s = buf[t];
        for (int r = 1; r < P; ++r) s += buf[r * q + t];
        red[t] = s;
      }
      __syncthreads();
    }
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const int t = lane + 32 * c;
      d[c] = 0.0;
      rj[c] = 0.0;
      if ((!kLate || t >= j) && t < q) {
        if (NC > 2) {
          d[c] = red[t];
        } else {
          d[c] = buf[t];
          for (int r = 1; r < P; ++r) d[c] += buf[r * q + t];
        }
        rj[c] = buf[P * q + t];
      }
    }
    if (NC > 2) __syncthreads();  // red is written again at the end of the next pass
    double dj = 0.0;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const double s = __shfl_sync(0xffffffffu, d[c], j & 31);
      if (c == j >> 5) dj = s;
    }
    const double ajj = buf[P * q + j];
    double alpha, beta;
    reflector(dj, ajj, alpha, beta);
    vj = ajj - alpha;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      g[c] = 0.0;
      if (!kLate || 32 * c + 31 >= j) {
        const double w = fma(-alpha, rj[c], d[c]);
        g[c] = beta * w;
        if (!kLate && warp == 0 && lane < j) S[lane * ld + j] = w;
      }
    }
    if (tid == 0) {
      betas[j] = beta;
      diag[j] = alpha;
    }
  }
  __syncthreads();
  // R, and V in place (zeros above its diagonal)
  for (int i = warp; i < min(rows, q - row0); i += kQrWarps) {
    const int gi = row0 + i;
    for (int t = lane; t < q; t += 32) {
      if (a.R != nullptr)
        a.R[size_t(gi) * q + t] = t > gi ? A[i * ld + t] : (t == gi ? diag[gi] : 0.0);
      if (t > gi) A[i * ld + t] = 0.0;
    }
  }
  sync_all();
  // U = the strict upper triangle of V^T V: every CTA's rows, then row t summed and
  // handed out by CTA t mod P
  if (kLate) {
    for (int t = warp; t < q; t += kQrWarps) {
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        if (32 * c + 31 <= t) continue;
        const int u = lane + 32 * c;
        double w = 0.0;
        if (u < q)
          for (int i = 0; i < rows; ++i) w = fma(A[i * ld + t], A[i * ld + u], w);
        if (u > t && u < q) S[t * ld + u] = w;
      }
    }
    sync_all();
    if (P > 1) {
      for (int t = me; t < q; t += P)
        for (int u = t + 1 + tid; u < q; u += kQrThreads) {
          double w = *cluster.map_shared_rank(S + t * ld + u, 0);
          for (int r = 1; r < P; ++r) w += *cluster.map_shared_rank(S + t * ld + u, r);
          for (int r = 0; r < P; ++r) *cluster.map_shared_rank(S + t * ld + u, r) = w;
        }
      cluster.sync();
    }
  }
  // (diag(1 / beta) + U) M = V_1^T with M[j][c] (c >= j) kept at S[c][j], from X = V_1^T
  auto row_of_v = [&](int r) {
    return (P > 1 ? cluster.map_shared_rank(A, r / nr) : A) + (r % nr) * ld;
  };
  if (P >= 4) {
    // a warp per column c, its lanes along j; the CTAs share the columns
    for (int col = me + P * warp; col < q; col += P * kQrWarps) {
      const double* src = row_of_v(col);
      double x[NC];
#pragma unroll
      for (int c = 0; c < NC; ++c) x[c] = lane + 32 * c <= col ? src[lane + 32 * c] : 0.0;
#pragma unroll
      for (int ck = NC - 1; ck >= 0; --ck) {
        for (int l = min(31, col - 32 * ck); l >= 0; --l) {
          const int k = 32 * ck + l;
          const double m = __shfl_sync(0xffffffffu, x[ck], l) * betas[k];
          if (lane == l) x[ck] = m;
#pragma unroll
          for (int c = 0; c <= ck; ++c) {
            const int j = lane + 32 * c;
            if (j < k) x[c] = fma(-S[j * ld + k], m, x[c]);
          }
        }
      }
      for (int r = 0; r < P; ++r) {
        double* dst = cluster.map_shared_rank(S, r) + col * ld;
#pragma unroll
        for (int c = 0; c < NC; ++c)
          if (lane + 32 * c <= col) dst[lane + 32 * c] = x[c];
      }
    }
    cluster.sync();
  } else {
    for (int r = warp; r < q; r += kQrWarps) {
      const double* src = row_of_v(r);
      for (int t = lane; t <= r; t += 32) S[r * ld + t] = src[t];
    }
    __syncthreads();
    for (int k = q - 1; k > 0; --k) {  // X[j][c] -= U[j][k] beta_k X[k][c], j < k <= c
      double m[NC];
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const int t = lane + 32 * c;
        m[c] = t >= k && t < q ? betas[k] * S[t * ld + k] : 0.0;
      }
      for (int j = warp; j < k; j += kQrWarps) {
        const double u = S[j * ld + k];
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          const int t = lane + 32 * c;
          if (t >= k && t < q) S[t * ld + j] = fma(-u, m[c], S[t * ld + j]);
        }
      }
      __syncthreads();
    }
    for (int r = warp; r < q; r += kQrWarps)
      for (int t = lane; t <= r; t += 32) S[r * ld + t] *= betas[t];
    __syncthreads();
  }
  // Q[i][c] = [i == c] - sum_{k <= c} V[i][k] M[k][c]
  for (int i = warp; i < rows; i += kQrWarps) {
    const int gi = row0 + i;
    double x[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) x[c] = lane + 32 * c == gi ? 1.0 : 0.0;
    const int kmax = min(q - 1, gi);
    for (int k = 0; k <= kmax; ++k) {
      const double v = A[i * ld + k];
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const int t = lane + 32 * c;
        if (k < 32 * c + 32 && t >= k && t < q) x[c] = fma(-v, S[t * ld + k], x[c]);
      }
    }
#pragma unroll
    for (int c = 0; c < NC; ++c)
      if (lane + 32 * c < q) a.Y[size_t(gi) * q + lane + 32 * c] = x[c];
  }
  if (P > 1) cluster.sync();  // remote reads of V are over
}

// Test hook's: 1 / x, then alpha and beta of (x, y).
__global__ void seeded_kernel(const double* x, const double* y, int64_t n, double* out) {
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x) {
    out[i] = positive_reciprocal(x[i]);
    reflector(x[i], y[i], out[n + i], out[2 * n + i]);
  }
}

}  // namespace

// CTAs of the cluster for an n x q matrix, 0 when it does not fit.
static int qr_ctas(int64_t n, int64_t q) {
  if (q > 160 || n > 1000000) return 0;
  int best = 0;
  double least = 0.0;
  const double nc = double((q + 31) / 32);
  for (int P : {1, 2, 4, 8, 16}) {
    if (P > max_cluster_ctas()) break;
    const int64_t nr = (n + P - 1) / P;
    if (qr_smem(nr, q, P) > kQrSmem) continue;
    // cycles: rows of a warp at 2 FMAs per chunk, sums over warps and CTAs,
    // barrier, reflector; then the solve and the product
    const double rows = double((nr + kQrWarps - 1) / kQrWarps);
    const double cost = double(q) * (rows * nc * 130.0 +
                                     (kQrWarps + P * (nc > 2.0 ? 2.0 : nc)) * 70.0 +
                                     (P > 1 ? 1800.0 : 200.0) + 1500.0) +
                        rows * nc * double(q) * 76.0;
    if (best == 0 || cost < least) {
      best = P;
      least = cost;
    }
  }
  return best;
}

bool householder_cluster_fits(int64_t n, int64_t q) { return qr_ctas(n, q) > 0; }

void householder_cluster(Ctx& c, double* Y, int64_t n, int64_t q, double* R) {
  const int P = qr_ctas(n, q);
  QrArgs a{};
  a.Y = Y;
  a.R = R;
  a.n = int(n);
  a.q = int(q);
  a.nr = int((n + P - 1) / P);
  const size_t smem = qr_smem(a.nr, q, P);
  auto launch = [&](auto kern) {
    CTM_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
    CTM_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    KernelTimer kt(c.stream, "householder_cluster_kernel", kUnitFlop, 4.0 * double(n) * q * q);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(unsigned(P));
    cfg.blockDim = dim3(kQrThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = c.stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = unsigned(P);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    CTM_CUDA(cudaLaunchKernelEx(&cfg, kern, a));
  };
  switch ((q + 31) / 32) {
    case 1: launch(householder_cluster_kernel<1>); break;
    case 2: launch(householder_cluster_kernel<2>); break;
    case 3: launch(householder_cluster_kernel<3>); break;
    case 4: launch(householder_cluster_kernel<4>); break;
    default: launch(householder_cluster_kernel<5>); break;
  }
  CTM_LAUNCH_CHECK();
}

}  // namespace ctm

// Test hook, not part of the plugin interface (no declaration in the public header): the
// functions of seeded.cuh on n pairs; out: n reciprocals, n alphas, n betas.
extern "C" int ctm_test_seeded(const double* x, const double* y, int64_t n, double* out,
                               void* stream) {
  ctm::seeded_kernel<<<ctm::grid_for(n, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(x, y, n,
                                                                                           out);
  return int(cudaGetLastError());
}
