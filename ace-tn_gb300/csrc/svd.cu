// FP64 thin SVD by one-sided (Hestenes) Jacobi rotations.
//
//  * jacobi_cluster_f64_kernel: all rows in the shared memory of one cluster
//    of up to 16 CTAs (up to about 320 x 320), from the rotations of an FP32
//    Jacobi when the matrix is square (144 x 144: 2.6 to 4.3 ms, 27 ms as
//    jacobi_sweeps_kernel; 80 x 80: 1.2 to 2.0 ms against 11 ms).
//  * From 32 columns to what the Householder cluster holds (149 square, L p^2 <= 4e6),
//    and for matrices more than six times as long as wide, a QR factorisation first: the
//    rows of the p x p factor R are rotated and the long singular vectors are
//    one product with Q.  R is graded even when the matrix is not, which is
//    what one-sided Jacobi needs: a 144 x 144 product of four enlarged corners
//    (values from 1 to 1e-17) takes ten FP32 and four FP64 sweeps from R, and
//    14 and 29 without the QR.  Householder in a cluster where it fits (any
//    rank), else a shifted Cholesky-QR3.
//  * jacobi_sweeps_kernel: rows in global memory, a cooperative grid with a
//    bounded grid barrier (Demmel & Veselic, SIAM J. Matrix Anal. Appl. 13
//    (1992) 1204): matrices beyond the cluster's shared memory, those on which
//    the Cholesky-QR fails its orthogonality check among them (numerically
//    rank-deficient ones; decided on the device, no synchronisation; in the
//    cluster form where they fit).
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>

#include "engine.cuh"
#include "seeded.cuh"

namespace ctm {

namespace {

constexpr int LT = 256;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ double block_sum(double v, double* sh) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) sh[w] = v;
  __syncthreads();
  double t = 0.0;
  for (int i = 0; i < int(blockDim.x >> 5); ++i) t += sh[i];
  return t;
}

// ------------------------------------------------------------- cluster Jacobi
//
// What bounds it: this part issues an FP64 warp instruction once in 64 cycles
// per SM quarter (measured: 1.7 lanes per cycle and SM with four warps or
// more), whatever the number of active lanes, so the count of FP64
// instructions of a round is its time.  Hence
//  * rotations as three shears (x -= h y; y += s x; x -= h y with
//    h = tan(theta / 2), s = sin(theta)): 3 FMAs per entry pair, not 4, and an
//    orthogonal map up to rounding for any h as long as s = 2 h / (1 + h^2)
//    holds in FP64, so that the angle itself may be an FP32 number;
//  * the angle and the convergence test in FP32 on mantissas and exponents
//    taken from the FP64 bit patterns by integer instructions (no FP64
//    division, square root or conversion; norms and dot products have to be
//    normal numbers, which svd_thin's scaling provides);
//  * squared row norms kept and updated (5 instructions) instead of two more
//    dot products per pair, and recomputed at the start of every sweep;
//  * two pairs per warp (kTP = 16 lanes each) where that fills the four SM
//    quarters: the scalar instructions then serve two pairs.
//
// The rows (padded with zero rows to 2 P m) form 2 P blocks of m; CTA k holds
// the blocks at tournament positions k and 2 P - 1 - k.  In each of the
// 2 P - 1 block rounds of a sweep a CTA rotates all m^2 pairs between its two
// blocks, m disjoint pairs at a time with a CTA barrier between them (in the
// first block round also the pairs inside each block), then writes its blocks
// into the next holders' second buffers (distributed shared memory; position
// 0 stays, the others advance by one) and one cluster barrier follows.  (A
// first form that moved two rows after every round of pairs spent about 2500
// cycles per round in the cluster barrier and its remote stores.)

__device__ __forceinline__ double twice(double x) {  // exact, normal x below 2^1023
  return __longlong_as_double(__double_as_longlong(x) + (1ll << 52));
}

__device__ __forceinline__ double negate(double x) {
  return __longlong_as_double(__double_as_longlong(x) ^ (long long)0x8000000000000000ull);
}

__device__ __forceinline__ double not_negative(double x) {
  return __double_as_longlong(x) < 0 ? 0.0 : x;
}

struct ClusterJacobi {
  double* W;        // p x L: rows to orthogonalise, in and out
  double* J;        // p x p: accumulated rotations, out (row j: of row j)
  const double* J0; // p x p: what is accumulated onto (null: the identity)
  double* norm2;    // p: squared norms of the final rows
  int p, L;
  int m;            // pairs per CTA
  int max_sweeps;
  float tol2;       // squared convergence tolerance
  int* flags;       // status word
  const int* skip;  // nothing to do when (*skip & 1) is not run_if
  int run_if;
};

// Doubles per row in shared memory: the row, its rotations, its squared norm and the first
// sweep's (an even number: block moves are 16-byte copies).
__host__ __device__ inline int jacobi_row(int p, int L) { return (L + p + 3) & ~1; }

// A row this much shorter than at first (squares) is what is left of a linear combination of
// the others, a rounding error 2^-53 of its first length and smaller by 2^-23 after each
// sweep: it becomes zero.  (Otherwise it is rotated until it underflows: with the input
// scaled to 2^440, more than 60 sweeps.)
constexpr double kCollapsed = 0x1p-150;

// One rotation of rows x and y (L entries, then p of the accumulated rotations,
// then the squared norm) by the kTP lanes of a group; returns whether it was
// applied.  Every lane of the group calls it.
template <int kTP>
__device__ __forceinline__ bool rotate_pair(double* x, double* y, int L, int p, int sub,
                                            unsigned gmask, float tol2) {
  const double al = x[L + p], be = y[L + p];
  double ga = 0.0;  // one chain: a dependent FMA issues as soon as an independent one
#pragma unroll 4
  for (int t = sub; t < L; t += kTP) ga = fma(x[t], y[t], ga);
#pragma unroll
  for (int o = kTP / 2; o > 0; o >>= 1) ga += __shfl_xor_sync(gmask, ga, o);
  float ma, mb, mg;
  int ea, eb, eg;
  if (!(split_f64(al, ma, ea) & split_f64(be, mb, eb) & split_f64(ga, mg, eg))) return false;
  {  // ga^2 > tol^2 al be
    const int ex = max(-120, min(120, 2 * eg - ea - eb));
    if (!(mg * mg * __int_as_float((ex + 127) << 23) > tol2 * (ma * mb))) return false;
  }
  const double de = be - al;
  float md;
  int ed;
  const bool dz = !split_f64(de, md, ed);  // equal norms: 45 degrees
  const bool neg = (__double_as_longlong(de) ^ __double_as_longlong(ga)) < 0;
  // zeta = de / (2 ga) = +-(md / mg) 2^(ed - eg - 1); t = tan(theta),
  // h = tan(theta / 2), both of zeta's sign
  const int ez = ed - eg - 1;
  double h;
  if (dz || ez < -60) {
    h = join_f64(0.41421357f, 0);
  } else if (ez < 30) {
    const float z = __fdividef(md, mg) * __int_as_float((ez + 127) << 23);
    const float t = __fdividef(1.f, z + sqrtf(fmaf(z, z, 1.f)));
    h = join_f64(__fdividef(t, 1.f + sqrtf(fmaf(t, t, 1.f))), 0);
  } else {  // t = 1 / (2 zeta), h = t / 2
    h = join_f64(__fdividef(mg, md), -ez - 2);
  }
  if (__double_as_longlong(h) == 0) return false;  // below the range of FP64
  if (!dz && neg) h = negate(h);
  // s = 2 h / (1 + h^2)
  const double d = fma(h, h, 1.0);
  float md1;
  int ed1;
  split_f64(d, md1, ed1);  // 1 <= d < 2
  const double s = twice(h) * mantissa_reciprocal(d, md1);
  const double mh = negate(h);
#pragma unroll 2
  for (int t = sub; t < L; t += kTP) {
    double u = x[t], v = y[t];
    u = fma(mh, v, u);
    v = fma(s, u, v);
    u = fma(mh, v, u);
    x[t] = u;
    y[t] = v;
  }
  double* xj = x + L;
  double* yj = y + L;
#pragma unroll 2
  for (int t = sub; t < p; t += kTP) {
    double u = xj[t], v = yj[t];
    u = fma(mh, v, u);
    v = fma(s, u, v);
    u = fma(mh, v, u);
    xj[t] = u;
    yj[t] = v;
  }
  // |x'|^2 = al + s (s de - 2 c ga), |y'|^2 = be - the same
  const double cs = fma(mh, s, 1.0);
  const double w = fma(negate(twice(cs)), ga, s * de);
  __syncwarp(gmask);  // every lane has read the norms
  if (sub == 0) {
    x[L + p] = not_negative(fma(s, w, al));
    y[L + p] = not_negative(fma(negate(s), w, be));
  }
  return true;
}

template <int kTP>
__global__ void __launch_bounds__(512) jacobi_cluster_f64_kernel(const ClusterJacobi a) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  if (a.skip != nullptr && (*a.skip & 1) != a.run_if) return;  // the whole cluster alike
  const int P = int(cluster.num_blocks()), k = int(cluster.block_rank());
  const int m = a.m, L = a.L, p = a.p;
  const int RS = jacobi_row(p, L);
  const int blk = m * RS;
  extern __shared__ __align__(16) double jsm[];
  __shared__ int s_rot[64];
  double* cur = jsm;            // top block, then bottom block
  double* nxt = jsm + 2 * blk;  // the blocks of the next round arrive here
  const int tid = threadIdx.x, nth = blockDim.x, lane = tid & 31, warp = tid >> 5;
  const int nwarps = nth >> 5;
  // block row q < 2 m of this CTA: its row of the matrix (the blocks are home)
  auto home = [&](int q) { return q < m ? k * m + q : (2 * P - 1 - k) * m + q - m; };
  for (int q = warp; q < 2 * m; q += nwarps) {
    double* s = cur + q * RS;
    const int row = home(q);
    for (int t = lane; t < L; t += 32) s[t] = row < p ? a.W[size_t(row) * L + t] : 0.0;
    for (int t = lane; t < p; t += 32)
      s[L + t] = a.J0 != nullptr && row < p ? a.J0[size_t(row) * p + t] : (t == row ? 1.0 : 0.0);
  }
  for (int i = tid; i < 64; i += nth) s_rot[i] = 0;
  if (P > 1) cluster.sync();
  else __syncthreads();
  const int g = tid / kTP, sub = tid % kTP;
  const unsigned gmask =
      kTP >= 32 ? 0xffffffffu : (((1u << kTP) - 1u) << (lane & ~(kTP - 1)));
  const int me = m + (m & 1);  // rows of a block, with a bye when odd
  int sweep = 0;
  for (; sweep < a.max_sweeps; ++sweep) {
    for (int q = warp; q < 2 * m; q += nwarps) {
      double* s = cur + q * RS;
      double v = 0.0;
      for (int t = lane; t < L; t += 32) v = fma(s[t], s[t], v);
      v = warp_sum(v);
      if (sweep > 0 && v < kCollapsed * s[L + p + 1]) {
        for (int t = lane; t < L; t += 32) s[t] = 0.0;
        v = 0.0;
      }
      __syncwarp();
      if (lane == 0) {
        s[L + p] = v;
        if (sweep == 0) s[L + p + 1] = v;
      }
    }
    __syncthreads();
    bool rotated = false;
    for (int t = 0; t < 2 * P - 1; ++t) {
      if (t == 0) {  // inside the blocks: circle method on me rows, me / 2 pairs each
        for (int r = 0; r < me - 1; ++r) {
          const int half = g < me / 2 ? 0 : 1, kk = g - half * (me / 2);
          const int i0 = kk == 0 ? 0 : (kk - 1 + r) % (me - 1) + 1;
          const int j0 = (me - 1 - kk - 1 + r) % (me - 1) + 1;
          if (g < me && i0 < m && j0 < m)
            rotated |= rotate_pair<kTP>(cur + half * blk + i0 * RS, cur + half * blk + j0 * RS, L,
                                        p, sub, gmask, a.tol2);
          __syncthreads();
        }
      }
      int j = g;
      for (int r = 0; r < m; ++r) {  // top row g against bottom row (g + r) mod m
        if (g < m)
          rotated |=
              rotate_pair<kTP>(cur + g * RS, cur + blk + j * RS, L, p, sub, gmask, a.tol2);
        if (++j == m) j = 0;
        __syncthreads();
      }
      if (P == 1) break;
      // position q -> q + 1 (2 P - 1 -> 1, 0 stays): top k is position k,
      // bottom k position 2 P - 1 - k
      double* dst_top = k == 0 ? nxt : k < P - 1 ? cluster.map_shared_rank(nxt, k + 1) : nxt + blk;
      double* dst_bot = k == 0 ? cluster.map_shared_rank(nxt, 1)
                               : cluster.map_shared_rank(nxt + blk, k - 1);
      const double2* st = reinterpret_cast<const double2*>(cur);
      const double2* sb = reinterpret_cast<const double2*>(cur + blk);
      for (int i = tid; i < blk / 2; i += nth) {
        reinterpret_cast<double2*>(dst_top)[i] = st[i];
        reinterpret_cast<double2*>(dst_bot)[i] = sb[i];
      }
      cluster.sync();
      double* tmp = cur;
      cur = nxt;
      nxt = tmp;
    }
    if (rotated) s_rot[sweep] = 1;
    int any = 0;
    if (P > 1) {
      cluster.sync();
      for (int q = 0; q < P; ++q) any |= *cluster.map_shared_rank(&s_rot[sweep], q);
    } else {
      __syncthreads();
      any = s_rot[sweep];
    }
    if (any == 0) break;  // every CTA reads the same words: all leave together
  }
  if (tid == 0 && k == 0 && sweep == a.max_sweeps) atomicOr(a.flags, 2);
  for (int q = warp; q < 2 * m; q += nwarps) {  // the blocks are home again
    const double* s = cur + q * RS;
    const int row = home(q);
    if (row >= p) continue;
    double v = 0.0;
    for (int t = lane; t < L; t += 32) {
      v = fma(s[t], s[t], v);
      a.W[size_t(row) * L + t] = s[t];
    }
    for (int t = lane; t < p; t += 32) a.J[size_t(row) * p + t] = s[L + t];
    v = warp_sum(v);
    if (lane == 0) a.norm2[row] = v;
  }
  if (P > 1) cluster.sync();  // no CTA leaves while others may read its shared memory
}

// Cluster shape for p rows of L entries: the number of CTAs and the lanes per
// pair with the smallest estimated sweep (FP64 instructions of the busiest SM
// quarter at 76 cycles; about 600 cycles of other work per round of pairs and
// 2500 per block move).  ctas = 0: does not fit.
struct JacobiShape {
  int ctas = 0, m = 0, tp = 0;
};

constexpr size_t kJacobiSmem = 226 * 1024;

size_t jacobi_smem(int64_t m, int64_t p, int64_t L) {
  return size_t(4 * m) * size_t(jacobi_row(int(p), int(L))) * sizeof(double);
}

JacobiShape jacobi_shape(int64_t p, int64_t L) {
  JacobiShape best;
  double least = 0.0;
  const int64_t h = (p + 1) / 2;
  for (int64_t P = 1; P <= max_cluster_ctas(); ++P) {
    const int64_t m = (h + P - 1) / P;
    if (P > 1 && (h + m - 1) / m != P) continue;  // a smaller cluster holds the same m
    if (m > 32 || L > 100000 || jacobi_smem(m, p, L) > kJacobiSmem) continue;
    for (int tp : {16, 32}) {
      const int64_t warps = ((m + (m & 1)) * tp + 31) / 32;
      if (warps > 16) continue;
      const int64_t el = (L + tp - 1) / tp, ep = (p + tp - 1) / tp;
      const int64_t instr = 4 * el + 3 * ep + (tp == 16 ? 4 : 5) + 11;
      const double round = 76.0 * double((warps + 3) / 4 * instr) + 600.0;
      const double cost = round * double((2 * P - 1) * m + m - 1) +
                          (P > 1 ? 2500.0 * double(2 * P) : 0.0);
      if (best.ctas == 0 || cost < least) {
        best.ctas = int(P);
        best.m = int(m);
        best.tp = tp;
        least = cost;
      }
    }
  }
  return best;
}

void jacobi_cluster(Ctx& c, const JacobiShape& sh, double* W, double* J, const double* J0,
                    double* norm2, int64_t p, int64_t L, double tol, const int* skip,
                    int run_if = 0) {
  ClusterJacobi a{};
  a.W = W;
  a.J = J;
  a.J0 = J0;
  a.norm2 = norm2;
  a.p = int(p);
  a.L = int(L);
  a.m = sh.m;
  a.max_sweeps = 60;
  a.tol2 = float(tol * tol);
  a.flags = status_flags(c);
  a.skip = skip;
  a.run_if = run_if;
  const size_t smem = jacobi_smem(sh.m, p, L);
  auto launch = [&](auto kern) {
    CTM_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
    CTM_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    KernelTimer kt(c.stream, "jacobi_cluster_f64_kernel", kUnitFlop, 0.0);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(unsigned(sh.ctas));
    cfg.blockDim = dim3(unsigned(((sh.m + (sh.m & 1)) * sh.tp + 31) / 32 * 32));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = c.stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = unsigned(sh.ctas);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    CTM_CUDA(cudaLaunchKernelEx(&cfg, kern, a));
  };
  if (sh.tp == 16) launch(jacobi_cluster_f64_kernel<16>);
  else launch(jacobi_cluster_f64_kernel<32>);
  CTM_LAUNCH_CHECK();
}

// ------------------------------------------------------------- grid Jacobi
struct JacobiArgs {
  double* W;      // p x L, row j = column j being orthogonalised
  double* J;      // p x p, row j = column j of the accumulated rotation
  int64_t p, L;
  int64_t pp;     // p rounded up to even
  double tol;
  int max_sweeps;
  unsigned* bar;  // [0] arrival count, [1] generation, [2] abort, [3..4] sweep flags
  int* flags;
  int64_t spin_limit;
  const int* only_if;  // run only when (*only_if & 1); null: always
};

// Bounded grid barrier.  Returns false when this CTA gave up waiting (the
// abort word is then set and the status flag records the timeout).
__device__ bool grid_sync(const JacobiArgs& a) {
  __syncthreads();
  __shared__ int ok;
  if (threadIdx.x == 0) {
    volatile unsigned* gen = a.bar + 1;
    volatile unsigned* abort_w = a.bar + 2;
    ok = 1;
    const unsigned g = *gen;
    __threadfence();
    const unsigned arrived = atomicAdd(a.bar, 1u);
    if (arrived == gridDim.x - 1) {
      atomicExch(a.bar, 0u);
      __threadfence();
      atomicAdd(const_cast<unsigned*>(gen), 1u);
    } else {
      int64_t it = 0;
      while (*gen == g) {
        if (*abort_w != 0u || ++it > a.spin_limit) {
          atomicExch(const_cast<unsigned*>(abort_w), 1u);
          atomicOr(a.flags, 2);
          ok = 0;
          break;
        }
        __nanosleep(64);
      }
    }
    __threadfence();
  }
  __syncthreads();
  return ok != 0;
}

__device__ __forceinline__ int64_t rr_pos(int64_t i, int64_t r, int64_t pp) {
  return i == 0 ? 0 : ((i - 1 + r) % (pp - 1)) + 1;
}

__global__ void __launch_bounds__(64) jacobi_sweeps_kernel(const JacobiArgs a) {
  if (a.only_if != nullptr && (*a.only_if & 1) == 0) return;  // the whole grid alike
  const int lane = threadIdx.x & 31;
  const int64_t warps_per_cta = blockDim.x >> 5;
  const int64_t gw = blockIdx.x * warps_per_cta + (threadIdx.x >> 5);
  const int64_t total_w = gridDim.x * warps_per_cta;
  const int64_t npairs = a.pp / 2;
  for (int sweep = 0; sweep < a.max_sweeps; ++sweep) {
    unsigned* rotated = a.bar + 3 + (sweep & 1);
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicExch(a.bar + 3 + ((sweep + 1) & 1), 0u);
    for (int64_t r = 0; r < a.pp - 1; ++r) {
      for (int64_t k = gw; k < npairs; k += total_w) {
        int64_t i = rr_pos(k, r, a.pp), j = rr_pos(a.pp - 1 - k, r, a.pp);
        if (i > j) { const int64_t t = i; i = j; j = t; }
        if (j >= a.p) continue;  // dummy partner
        double* wi = a.W + i * a.L;
        double* wj = a.W + j * a.L;
        double al = 0.0, be = 0.0, ga = 0.0;
        for (int64_t t = lane; t < a.L; t += 32) {
          const double x = wi[t], y = wj[t];
          al = fma(x, x, al);
          be = fma(y, y, be);
          ga = fma(x, y, ga);
        }
        al = warp_sum(al);
        be = warp_sum(be);
        ga = warp_sum(ga);
        if (al == 0.0 || be == 0.0 || !(fabs(ga) > a.tol * sqrt(al) * sqrt(be))) continue;
        const double zeta = (be - al) / (2.0 * ga);
        const double t = copysign(1.0, zeta) / (fabs(zeta) + sqrt(fma(zeta, zeta, 1.0)));
        const double cs = 1.0 / sqrt(fma(t, t, 1.0));
        const double sn = cs * t;
        for (int64_t u = lane; u < a.L; u += 32) {
          const double x = wi[u], y = wj[u];
          wi[u] = cs * x - sn * y;
          wj[u] = sn * x + cs * y;
        }
        double* ji = a.J + i * a.p;
        double* jj = a.J + j * a.p;
        for (int64_t u = lane; u < a.p; u += 32) {
          const double x = ji[u], y = jj[u];
          ji[u] = cs * x - sn * y;
          jj[u] = sn * x + cs * y;
        }
        if (lane == 0) atomicExch(rotated, 1u);
      }
      if (!grid_sync(a)) return;
    }
    const unsigned any = *(volatile unsigned*)rotated;
    if (!grid_sync(a)) return;
    if (any == 0u) return;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(a.flags, 2);
}

// Squared norms of the rows of W (p x L), one CTA per row.
__global__ void __launch_bounds__(LT) row_norms_kernel(const double* W, int64_t L, double* norm2,
                                                       const int* only_if) {
  if (only_if != nullptr && (*only_if & 1) == 0) return;
  __shared__ double sh[LT / 32];
  const double* w = W + int64_t(blockIdx.x) * L;
  double part = 0.0;
  for (int64_t t = threadIdx.x; t < L; t += blockDim.x) part = fma(w[t], w[t], part);
  part = block_sum(part, sh);
  if (threadIdx.x == 0) norm2[blockIdx.x] = part;
}

// The input is scaled by a power of two that puts its largest entry's exponent at kTop for
// the cluster form: squared norms stay below 2^1023 and the dot products of rows 2^-900 as
// long are still normal numbers.  The form in global memory compares subnormal ones too, and
// rows that collapse have to underflow there: 0.  (Exact, so the result has the same bits
// wherever none underflowed.)
constexpr int kTop = 440;

// Largest exponent field of the finite entries; *top zeroed where the grid has several CTAs.
__global__ void __launch_bounds__(1024) top_field_kernel(const double* X, int64_t n, int* top) {
  int e = 0;
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x) {
    const int f = int((unsigned long long)__double_as_longlong(X[i]) >> 52) & 0x7ff;
    if (f != 0x7ff) e = max(e, f);
  }
  for (int o = 16; o > 0; o >>= 1) e = max(e, __shfl_xor_sync(0xffffffffu, e, o));
  __shared__ int s_top;
  if (threadIdx.x == 0) s_top = 0;
  __syncthreads();
  if ((threadIdx.x & 31) == 0) atomicMax(&s_top, e);
  __syncthreads();
  if (threadIdx.x != 0) return;
  if (gridDim.x == 1) *top = s_top;
  else atomicMax(top, s_top);
}

__device__ __forceinline__ double pow2(int e) {
  return __longlong_as_double((long long)(e + 1023) << 52);
}

// x 2^e in two steps, the first of them exact where the second is not.
__device__ __forceinline__ double scaled(double x, int e) {
  return x * pow2(e / 2) * pow2(e - e / 2);
}

// Exponent of the scaling (even: the halves of the exponents that a square root sees stay).
__device__ __forceinline__ int scale_exponent(int top, int target) {
  return (target + 1023 - max(top, 1)) & ~1;
}

// dst[r][c] = X[r s0 + c s1] 2^e, rows x cols.
__global__ void __launch_bounds__(256) scaled_copy_kernel(const double* X, int64_t rows,
                                                          int64_t cols, int64_t s0, int64_t s1,
                                                          const int* top, int target, double* dst) {
  const int e = scale_exponent(*top, target);
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < rows * cols;
       i += int64_t(gridDim.x) * blockDim.x) {
    const int64_t r = i / cols, q = i - r * cols;
    dst[i] = scaled(X[r * s0 + q * s1], e);
  }
}

// Sorts the Jacobi result by descending row norm and writes the singular
// values and vectors, one CTA per row j: rank r of row j (strictly larger
// norms, ties by index; NaNs, whose bits are above an infinity's, come first and
// so have ranks of their own: every output is written), S[r] = |W_j| without the scaling, the short side's vectors
// Vs[t][r] = J_j[t] (p x p), the long side's Vl[t][r] = W_j[t] / S[r] (L x p).
__global__ void __launch_bounds__(LT) jacobi_finish_kernel(const double* W, const double* J,
                                                           const double* norm2, int64_t p,
                                                           int64_t L, double* Vs, double* S,
                                                           double* Vl, const int* top, int target,
                                                           const int* only_if) {
  if (only_if != nullptr && (*only_if & 1) == 0) return;
  const int64_t j = blockIdx.x;
  __shared__ int s_rank;
  const double nj2 = norm2[j];
  auto key = [](double v) { return __double_as_longlong(v) & 0x7fffffffffffffffll; };
  const long long kj = key(nj2);
  if (threadIdx.x == 0) s_rank = 0;
  __syncthreads();
  int cnt = 0;
  for (int64_t i = threadIdx.x; i < p; i += blockDim.x) {
    const long long ki = key(norm2[i]);
    if (i != j && (ki > kj || (ki == kj && i < j))) ++cnt;
  }
  if (cnt != 0) atomicAdd(&s_rank, cnt);
  __syncthreads();
  const int64_t rk = s_rank;
  const double sj = sqrt(nj2);
  const double inv = sj > 0.0 ? 1.0 / sj : 0.0;
  if (threadIdx.x == 0) S[rk] = scaled(sj, -scale_exponent(*top, target));
  for (int64_t t = threadIdx.x; t < p; t += blockDim.x) Vs[t * p + rk] = J[j * p + t];
  for (int64_t t = threadIdx.x; t < L; t += blockDim.x) Vl[t * p + rk] = W[j * L + t] * inv;
}

// Short side's vectors from the rows of a factor R, V (p x p), S sorted: where R has no full
// rank in exact arithmetic, the rotations shrink its last rows towards zero, and what is left
// of them, normalised, is a rounding error, or nothing.  These two kernels put vectors
// orthogonal to the others in such places.
//
// loose[r]: whether column r, of a value below 1e-8 of the largest, is not orthonormal to the
// others.  One CTA per column (2 us without small values).
__global__ void __launch_bounds__(LT) loose_columns_kernel(const double* V, const double* S, int p,
                                                           int* loose, const int* skip) {
  const int r = blockIdx.x, tid = threadIdx.x;
  if ((skip != nullptr && (*skip & 1) != 0) || !(S[r] < 1e-8 * S[0] || S[r] == 0.0)) {
    if (tid == 0) loose[r] = 0;
    return;
  }
  const double tol = 16.0 * 2.220446049250313e-16 * sqrt(double(p));
  extern __shared__ double s_col[];
  for (int t = tid; t < p; t += LT) s_col[t] = V[size_t(t) * p + r];
  __syncthreads();
  bool bad = false;
  for (int k = tid; k < p; k += LT) {
    double d = k == r ? -1.0 : 0.0;
    for (int t = 0; t < p; ++t) d = fma(s_col[t], V[size_t(t) * p + k], d);
    bad = bad || fabs(d) > tol;
  }
  bad = __syncthreads_or(bad);
  if (tid == 0) loose[r] = bad ? 1 : 0;
}

// The loose columns, orthogonalised twice against the others (from the unit vector e_t
// farthest from their span, whose squared distance is 1 minus the sum of squares of their
// entries t, where little of the column is left).  One CTA; returns at once without any.
__global__ void __launch_bounds__(LT) tighten_columns_kernel(double* V, int p, int* loose) {
  extern __shared__ double s_dot[];  // p coefficients, then p flags
  int* s_loose = reinterpret_cast<int*>(s_dot + p);
  __shared__ double sh[LT / 32];
  __shared__ int s_at;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  bool any = false;
  for (int k = tid; k < p; k += LT) {
    s_loose[k] = loose[k];
    any = any || s_loose[k] != 0;
  }
  if (!__syncthreads_or(any)) return;
  for (int r = 0; r < p; ++r) {
    if (s_loose[r] == 0) continue;
    // column r without its part in the span, to norm 1; its norm before that
    auto pass = [&] {
      __syncthreads();
      for (int k = warp; k < p; k += LT / 32) {
        double d = 0.0;
        if (s_loose[k] == 0)
          for (int t = lane; t < p; t += 32) d = fma(V[size_t(t) * p + k], V[size_t(t) * p + r], d);
        d = warp_sum(d);
        if (lane == 0) s_dot[k] = d;
      }
      __syncthreads();
      double part = 0.0;
      for (int t = tid; t < p; t += LT) {
        double v = V[size_t(t) * p + r];
        for (int k = 0; k < p; ++k)
          if (s_loose[k] == 0) v = fma(-s_dot[k], V[size_t(t) * p + k], v);
        V[size_t(t) * p + r] = v;
        part = fma(v, v, part);
      }
      const double norm = sqrt(block_sum(part, sh)), inv = norm > 0.0 ? 1.0 / norm : 0.0;
      for (int t = tid; t < p; t += LT) V[size_t(t) * p + r] *= inv;
      return norm;
    };
    if (!(pass() > 0.5)) {
      for (int t = warp; t < p; t += LT / 32) {
        double d = 0.0;
        for (int k = lane; k < p; k += 32)
          if (s_loose[k] == 0) d = fma(V[size_t(t) * p + k], V[size_t(t) * p + k], d);
        d = warp_sum(d);
        if (lane == 0) s_dot[t] = d;
      }
      __syncthreads();
      if (tid == 0) {
        s_at = 0;
        for (int t = 1; t < p; ++t)
          if (s_dot[t] < s_dot[s_at]) s_at = t;
      }
      __syncthreads();
      for (int t = tid; t < p; t += LT) V[size_t(t) * p + r] = t == s_at ? 1.0 : 0.0;
      pass();
    }
    pass();
    __syncthreads();
    if (tid == 0) s_loose[r] = 0;
    __syncthreads();
  }
}

__global__ void identity_kernel(double* X, int64_t p, const int* only_if) {
  if (only_if != nullptr && (*only_if & 1) == 0) return;
  for (int64_t idx = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; idx < p * p;
       idx += int64_t(gridDim.x) * blockDim.x)
    X[idx] = (idx / p == idx % p) ? 1.0 : 0.0;
}

void finish(Ctx& c, const double* W, const double* J, const double* norm2, int64_t p, int64_t L,
            double* Vs, double* S, double* Vl, const int* top, int target, const int* only_if) {
  KernelTimer kt(c.stream, "jacobi_finish_kernel", kUnitByte, 16.0 * double(p) * (p + L));
  jacobi_finish_kernel<<<unsigned(p), LT, 0, c.stream>>>(W, J, norm2, p, L, Vs, S, Vl, top, target, only_if);
  CTM_LAUNCH_CHECK();
}

// Jacobi with the rows in global memory; W and J are updated in place.
void jacobi_grid(Ctx& c, double* W, double* J, double* norm2, int64_t p, int64_t L,
                 const int* only_if) {
  Scope scope(c);
  unsigned* bar = c.alloc<unsigned>(8);
  if (c.sizing()) return;
  identity_kernel<<<grid_for(p * p, 256), 256, 0, c.stream>>>(J, p, only_if);
  CTM_LAUNCH_CHECK();
  CTM_CUDA(cudaMemsetAsync(bar, 0, 8 * sizeof(unsigned), c.stream));
  JacobiArgs a{};
  a.W = W;
  a.J = J;
  a.p = p;
  a.L = L;
  a.pp = p + (p & 1);
  a.tol = 2.220446049250313e-16 * std::sqrt(double(L));
  a.max_sweeps = 60;
  a.bar = bar;
  a.flags = status_flags(c);
  a.spin_limit = int64_t(20) * 1000 * 1000;  // ~1-2 s of 64 ns sleeps
  a.only_if = only_if;
  if (p > 1) {
    int dev = 0, sms = 0, per_sm = 0;
    CTM_CUDA(cudaGetDevice(&dev));
    CTM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int threads = 64;
    CTM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, jacobi_sweeps_kernel, threads, 0));
    const int64_t npairs = a.pp / 2;
    int64_t blocks = (npairs + 1) / 2;
    blocks = std::min<int64_t>(blocks, int64_t(sms) * std::max(per_sm, 1));
    blocks = std::min<int64_t>(blocks, sms);
    blocks = std::max<int64_t>(blocks, 1);
    void* args[] = {&a};
    KernelTimer kt(c.stream, "jacobi_sweeps_kernel", kUnitFlop, 0.0);
    CTM_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<void*>(jacobi_sweeps_kernel),
                                         dim3(unsigned(blocks)), dim3(threads), args, 0, c.stream));
    CTM_LAUNCH_CHECK();
  }
  row_norms_kernel<<<unsigned(p), LT, 0, c.stream>>>(W, L, norm2, only_if);
  CTM_LAUNCH_CHECK();
}

// FP32 copy of X (n entries) scaled by a power of two so that its largest entry
// is below 2 (one CTA; entries below the FP32 range become zeros; all of them when
// (*skip & 1): what follows then has nothing to do).
__global__ void __launch_bounds__(1024) scaled_f32_kernel(const double* X, int n, float* Y,
                                                          const int* skip) {
  if (skip != nullptr && (*skip & 1) != 0) {
    for (int i = threadIdx.x; i < n; i += blockDim.x) Y[i] = 0.f;
    return;
  }
  __shared__ int s_top;
  if (threadIdx.x == 0) s_top = 0;
  __syncthreads();
  int top = 0;  // the largest exponent of a finite entry
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const int e = int((unsigned long long)__double_as_longlong(X[i]) >> 52) & 0x7ff;
    if (e != 0x7ff) top = max(top, e);
  }
  for (int o = 16; o > 0; o >>= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, o));
  if ((threadIdx.x & 31) == 0) atomicMax(&s_top, top);
  __syncthreads();
  top = s_top;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(X[i]);
    const int e = (int(b >> 52) & 0x7ff) - top + 127;
    // truncation to 24 bits: this copy only steers the rotations
    Y[i] = e > 0 && e < 255
               ? __uint_as_float((unsigned(b >> 32) & 0x80000000u) | (unsigned(e) << 23) |
                                 (unsigned(b >> 29) & 0x7fffffu))
               : 0.f;
  }
}

// Preconditioned Jacobi on the rows of W (p x p, mostly a triangular factor), p in
// [kPreMin, kPreMax]: an FP32 Jacobi finds rotations T that make the rows
// orthogonal to about 1e-6, T is made orthogonal to FP64 accuracy by two Newton
// steps T <- (3 T - (T T^T) T) / 2 (its deviation of 1e-6 is squared twice), and
// the FP64 rotations start from T W and T: three or four sweeps instead of 9 to
// 20 (Drmac and Veselic's preconditioning, with an approximate SVD after the QR
// factor).  At p = 144 an FP64 sweep takes 0.5 ms, an FP32 one 0.1.
constexpr int64_t kPreMin = 16, kPreMax = 256;

void jacobi_square(Ctx& c, double* W, double* J, double* norm2, int64_t p, const int* skip) {
  const JacobiShape sh = jacobi_shape(p, p);
  const double tol = 2.220446049250313e-16 * std::sqrt(double(p));
  if (p < kPreMin || p > kPreMax) {
    if (!c.sizing()) jacobi_cluster(c, sh, W, J, nullptr, norm2, p, p, tol, skip);
    return;
  }
  Scope scope(c);
  const size_t pp = size_t(p) * p;
  float* Wf = c.alloc<float>(pp);
  float* Jf = c.alloc<float>(pp);
  float* nf = c.alloc<float>(p);
  double* T = c.alloc<double>(pp);
  double* T2 = c.alloc<double>(pp);
  double* G = c.alloc<double>(pp);
  int* unused = c.alloc<int>(1);  // an unfinished FP32 stage is not a failure
  if (!c.sizing()) {
    scaled_f32_kernel<<<1, 1024, 0, c.stream>>>(W, int(pp), Wf, skip);
    CTM_LAUNCH_CHECK();
  }
  // what is left after ten sweeps lies at the FP32 rounding level
  jacobi_rotations(c, Wf, p, Jf, nf, 10, unused);
  to_f64(c, Jf, T, p * p);
  const View t(T, {p, p}), t2(T2, {p, p}), g(G, {p, p}), w(W, {p, p});
  auto newton = [&](const View& from, const View& to) {
    einsum(c, "ik,jk->ij", from, from, g);
    if (!c.sizing())
      CTM_CUDA(cudaMemcpyAsync(to.p, from.p, pp * sizeof(double), cudaMemcpyDeviceToDevice,
                               c.stream));
    einsum(c, "ik,kj->ij", g, from, to, -0.5, 1.5);
  };
  newton(t, t2);
  newton(t2, t);
  einsum(c, "ik,kj->ij", t, w, t2);
  if (!c.sizing()) {
    CTM_CUDA(cudaMemcpyAsync(W, T2, pp * sizeof(double), cudaMemcpyDeviceToDevice, c.stream));
    jacobi_cluster(c, sh, W, J, T, norm2, p, p, tol, skip);
  }
}

}  // namespace

// CTAs of the largest cluster that this device runs at full shared memory (16
// where a GPC has that many free SMs, else 8, the portable size).
int max_cluster_ctas() {
  static const int n = [] {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(16);
    cfg.blockDim = dim3(512);
    cfg.dynamicSmemBytes = kJacobiSmem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 16;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    const auto kern = jacobi_cluster_f64_kernel<32>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kJacobiSmem)) !=
            cudaSuccess ||
        cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) !=
            cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) != cudaSuccess) {
      cudaGetLastError();
      return 8;
    }
    return clusters > 0 ? 16 : 8;
  }();
  return n;
}

void svd_thin(Ctx& c, const double* X, int64_t m, int64_t n, double* U, double* S, double* V) {
  CTM_REQUIRE(m >= 1 && n >= 1, CTM_ERR_INVALID, "svd_thin: empty matrix");
  const bool tall = m >= n;  // the rows rotated are the columns of X, else its rows
  const int64_t p = std::min(m, n), L = std::max(m, n);
  double* const Vs = tall ? V : U;  // singular vectors of the short side (p x p)
  double* const Vl = tall ? U : V;  // and of the long side (L x p)
  const double eps = 2.220446049250313e-16;
  Scope scope(c);
  double* W = c.alloc<double>(size_t(p) * L);
  double* J = c.alloc<double>(size_t(p) * p);
  double* norm2 = c.alloc<double>(p);
  int* top = c.alloc<int>(1);
  // dst = X (rows first) or X^T, scaled
  auto load = [&](double* dst, bool transposed, int target) {
    if (c.sizing()) return;
    KernelTimer kt(c.stream, "scaled_copy_kernel", kUnitByte, 16.0 * double(m) * n);
    scaled_copy_kernel<<<grid_for(m * n, 256), 256, 0, c.stream>>>(
        X, transposed ? n : m, transposed ? m : n, transposed ? 1 : n, transposed ? n : 1, top, target,
        dst);
    CTM_LAUNCH_CHECK();
  };
  const JacobiShape direct = jacobi_shape(p, L), square = jacobi_shape(p, p);
  const int target = direct.ctas > 0 ? kTop : 0;  // of W, which is rotated as it is
  auto load_w = [&] { load(W, tall, target); };   // W rows = columns of X (tall) or rows of X
  if (!c.sizing()) {
    const int ctas = int(std::min<int64_t>(sm_count_linalg(), (m * n + 32767) / 32768));
    if (ctas > 1) CTM_CUDA(cudaMemsetAsync(top, 0, sizeof(int), c.stream));
    top_field_kernel<<<ctas, 1024, 0, c.stream>>>(X, m * n, top);
    CTM_LAUNCH_CHECK();
  }
  // The one-cluster Householder QR up to the size where the Cholesky-QR (about
  // 20 launches and three one-SM factorisations) is faster; the latter only
  // where it saves long rows, as it takes well-conditioned input.  No QR for
  // small matrices: 22 x 80 takes 250 us in 8 sweeps, about what the QR and the
  // FP32 stage would.
  const bool house = householder_cluster_fits(L, p) && double(L) * p * p <= 4.0e6;
  const bool reduce = square.ctas > 0 && (L > 6 * p || direct.ctas == 0 ||
                                          (house && p >= 32 && p <= kPreMax));
  if (!reduce) {
    load_w();
    if (p == L && direct.ctas > 0) {
      jacobi_square(c, W, J, norm2, p, nullptr);
    } else if (direct.ctas > 0) {
      if (!c.sizing())
        jacobi_cluster(c, direct, W, J, nullptr, norm2, p, L, eps * std::sqrt(double(L)), nullptr);
    } else {
      jacobi_grid(c, W, J, norm2, p, L, nullptr);
    }
    if (!c.sizing()) finish(c, W, J, norm2, p, L, Vs, S, Vl, top, target, nullptr);
    return;
  }
  // long side = Y R.  The rows of R are rotated, R = J^T W: the short side's
  // vectors are the rows of W over their norms and the long side's Y J^T.
  // (Rows of R, not its columns: each QR factorisation is a step towards the
  // graded form; 12 sweeps instead of 20 on an ungraded 160-column matrix.)
  double* Y = c.alloc<double>(size_t(L) * p);
  double* R = c.alloc<double>(size_t(p) * p);
  double* W2 = c.alloc<double>(size_t(p) * p);
  double* Xs = c.alloc<double>(size_t(p) * p);
  int* failed = c.alloc<int>(1);
  int* loose = c.alloc<int>(p);
  load(Y, !tall, kTop);
  if (!house) orthonormalize_try(c, Y, L, p, R, failed);
  else if (!c.sizing()) householder_cluster(c, Y, L, p, R);
  const int* const flag = house ? nullptr : failed;
  if (!c.sizing())
    CTM_CUDA(cudaMemcpyAsync(W2, R, sizeof(double) * p * p, cudaMemcpyDeviceToDevice, c.stream));
  jacobi_square(c, W2, J, norm2, p, flag);
  if (!c.sizing()) {
    finish(c, W2, J, norm2, p, p, Xs, S, Vs, top, kTop, nullptr);
    KernelTimer kt(c.stream, "loose_columns_kernel", kUnitByte, 8.0 * double(p) * p);
    loose_columns_kernel<<<unsigned(p), LT, size_t(p) * sizeof(double), c.stream>>>(
        Vs, S, int(p), loose, flag);
    CTM_LAUNCH_CHECK();
    tighten_columns_kernel<<<1, LT, size_t(p) * (sizeof(double) + sizeof(int)), c.stream>>>(
        Vs, int(p), loose);
    CTM_LAUNCH_CHECK();
  }
  einsum(c, "ik,kj->ij", View(Y, {L, p}), View(Xs, {p, p}), View(Vl, {L, p}));
  if (house) return;
  // when the Cholesky-QR has failed: the whole matrix again, in a cluster where it fits (100
  // x 601 with values from 1 to 1e-15: 42 ms in global memory), else in global memory
  load_w();
  if (direct.ctas == 0) jacobi_grid(c, W, J, norm2, p, L, failed);
  else if (!c.sizing())
    jacobi_cluster(c, direct, W, J, nullptr, norm2, p, L, eps * std::sqrt(double(L)), failed, 1);
  if (!c.sizing()) finish(c, W, J, norm2, p, L, Vs, S, Vl, top, target, failed);
}

}  // namespace ctm
