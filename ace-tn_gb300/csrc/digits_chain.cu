// FMA chains for the outputs that the digit products mark.
//
// What bounds it: an FP64 warp instruction issues once in 64 cycles per SM quarter, and
// in the usual case, where few outputs are marked, the reading of their words and the
// latency of a launch.  So the marked outputs of 128 rows by one word are listed first
// and their terms spread over all threads of a CTA (32 lanes and fewer an output, sums
// joined in a fixed tree), the next words are fetched beside that work, and a block
// with more than a quarter marked is computed as a tile through shared memory.
#include <algorithm>

#include "digits.cuh"

namespace ctm {

namespace {

constexpr int kCThreads = 256;
constexpr int kCRows = 128;          // rows of a block of marks
constexpr int kDense = kCRows * 8;   // marked outputs from which a block is a tile
constexpr int kCK = 16;              // contracted indices per step of a tile

struct ChainOutputs {
  ChainArgs ch;
  Group GM, GN;         // output strides of rows and columns (m[].s1)
  Marks marks;
  int64_t columns, K, kchunk;  // kchunk: contracted indices per blockIdx.y
  double* C;
  double* part;         // gridDim.y > 1: sums of the ranges, [range][row][column]
  double alpha, beta;
};

// Word w of row r without bits beyond the columns (a product that gave up waiting, with
// the status flag set, leaves words unwritten).
__device__ __forceinline__ uint32_t marks_of(const ChainOutputs& a, int64_t w, int64_t r) {
  const int64_t live = min(int64_t(a.marks.per), a.columns - w * a.marks.per);
  const uint32_t mask = live >= 32 ? ~0u : live > 0 ? (1u << live) - 1u : 0u;
  return a.marks.word[w * a.marks.rows + r] & mask;
}

__device__ __forceinline__ void chain_store(const ChainOutputs& a, int64_t r, int64_t n, double v) {
  if (gridDim.y > 1) {
    a.part[(blockIdx.y * a.marks.rows + r) * a.columns + n] = v;
    return;
  }
  int64_t t, ro, co;
  decode(a.GM, r, t, ro);
  decode(a.GN, n, t, co);
  double* out = a.C + ro + co;
  v *= a.alpha;
  *out = a.beta != 0.0 ? fma(a.beta, *out, v) : v;
}

__device__ __forceinline__ void k_offsets(const ChainArgs& ch, int64_t k, int64_t& ka, int64_t& kb) {
  int64_t t0, t1;
  decode(ch.FK, k, t0, t1);
  ka = ch.swapped ? t1 : t0;
  kb = ch.swapped ? t0 : t1;
}

__global__ void __launch_bounds__(kCThreads, 4) chain_outputs_kernel(const ChainOutputs a) {
  __shared__ uint32_t s_mark[kCRows];
  __shared__ int s_first[kCRows / 32];
  __shared__ __align__(8) unsigned char s_buf[(kCK * (kCRows + 1) + kCK * 33) * sizeof(double)];
  __shared__ int64_t s_ro[kCRows], s_co[32], s_ka[kCK], s_kb[kCK];
  uint16_t* list = reinterpret_cast<uint16_t*>(s_buf);  // row * 32 + bit, at most kDense
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t rblocks = (a.marks.rows + kCRows - 1) / kCRows, items = rblocks * a.marks.words;
  const int64_t k0 = blockIdx.y * a.kchunk, k1 = min(a.K, k0 + a.kchunk);
  auto word_of = [&](int64_t item) -> uint32_t {
    const int64_t w = item / rblocks, r = (item - w * rblocks) * kCRows + tid;
    return tid < kCRows && item < items && r < a.marks.rows ? marks_of(a, w, r) : 0u;
  };
  uint32_t next = word_of(blockIdx.x);
  for (int64_t item = blockIdx.x; item < items; item += gridDim.x) {
    const uint32_t mark = next;
    next = word_of(item + gridDim.x);
    if (!__syncthreads_or(mark != 0u)) continue;
    const int64_t w = item / rblocks, r0 = (item - w * rblocks) * kCRows, n0 = w * a.marks.per;
    // places of the marked outputs in the list
    int at = __popc(mark);
    const int own = at;
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, at, o);
      if (lane >= o) at += v;
    }
    if (tid < kCRows) {
      s_mark[tid] = mark;
      if (lane == 31) s_first[warp] = at;
    }
    __syncthreads();
    int count = 0, base = 0;
#pragma unroll
    for (int i = 0; i < kCRows / 32; ++i) {
      if (i < warp) base += s_first[i];
      count += s_first[i];
    }
    if (count <= kDense) {
      at += base - own;
      for (uint32_t left = mark; left != 0u; left &= left - 1u)
        list[at++] = uint16_t(tid * 32 + __ffs(int(left)) - 1);
      __syncthreads();
      // lanes per output: all threads busy, a few terms each at least
      int g = 1;
      while (g < 32 && (count * g * 2 <= kCThreads || (k1 - k0) >= 1024) && 8 * g < k1 - k0) g *= 2;
      const int groups = kCThreads / g, sub = tid & (g - 1);
      for (int o0 = 0; o0 < count; o0 += groups) {
        const int o = o0 + tid / g;
        const int e = o < count ? list[o] : 0;
        double v = 0.0;
        if (o < count) {
          int64_t ao, bo, t, ka, kb;
          decode(a.ch.FM, r0 + (e >> 5), ao, t);
          decode(a.ch.FN, n0 + (e & 31), bo, t);
          const double* x = a.ch.a + ao;
          const double* y = a.ch.b + bo;
#pragma unroll 4
          for (int64_t k = k0 + sub; k < k1; k += g) {
            k_offsets(a.ch, k, ka, kb);
            v = fma(x[ka], y[kb], v);
          }
        }
        for (int s = g / 2; s > 0; s >>= 1) v += __shfl_xor_sync(0xffffffffu, v, s);
        if (o < count && sub == 0) chain_store(a, r0 + (e >> 5), n0 + (e & 31), v);
      }
      __syncthreads();
      continue;
    }
    // a tile of 128 x 32 outputs, 4 x 4 a thread
    double (*xs)[kCRows + 1] = reinterpret_cast<double (*)[kCRows + 1]>(s_buf);
    double (*ys)[33] = reinterpret_cast<double (*)[33]>(s_buf + kCK * (kCRows + 1) * sizeof(double));
    for (int i = tid; i < kCRows + 32; i += kCThreads) {
      int64_t o = -1, t;
      if (i < kCRows) {
        if (r0 + i < a.marks.rows) decode(a.ch.FM, r0 + i, o, t);
        s_ro[i] = o;
      } else {
        const int64_t n = n0 + i - kCRows;
        if (i - kCRows < a.marks.per && n < a.columns) decode(a.ch.FN, n, o, t);
        s_co[i - kCRows] = o;
      }
    }
    const int ty = tid >> 3, tx = tid & 7;
    double acc[4][4] = {};
    for (int64_t kb = k0; kb < k1; kb += kCK) {
      __syncthreads();
      if (tid < kCK) {
        int64_t ka = -1, kk = -1;
        if (kb + tid < k1) k_offsets(a.ch, kb + tid, ka, kk);
        s_ka[tid] = ka;
        s_kb[tid] = kk;
      }
      __syncthreads();
      for (int i = tid; i < kCK * kCRows; i += kCThreads) {
        const int k = i & (kCK - 1), r = i / kCK;
        xs[k][r] = s_ro[r] >= 0 && s_ka[k] >= 0 ? a.ch.a[s_ro[r] + s_ka[k]] : 0.0;
      }
      for (int i = tid; i < kCK * 32; i += kCThreads) {
        const int n = i & 31, k = i >> 5;
        ys[k][n] = s_co[n] >= 0 && s_kb[k] >= 0 ? a.ch.b[s_co[n] + s_kb[k]] : 0.0;
      }
      __syncthreads();
#pragma unroll 4
      for (int k = 0; k < kCK; ++k) {
        double x[4], y[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) x[i] = xs[k][ty + 32 * i];
#pragma unroll
        for (int j = 0; j < 4; ++j) y[j] = ys[k][tx + 8 * j];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = fma(x[i], y[j], acc[i][j]);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int r = ty + 32 * i, n = tx + 8 * j;
        if (s_mark[r] >> n & 1u) chain_store(a, r0 + r, n0 + n, acc[i][j]);
      }
    __syncthreads();
  }
}

// The ranges' sums of the marked outputs into C, one word a thread.
__global__ void __launch_bounds__(256) chain_sum_kernel(const ChainOutputs a, int ranges) {
  const int64_t total = a.marks.rows * a.marks.words;
  for (int64_t idx = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; idx < total;
       idx += int64_t(gridDim.x) * blockDim.x) {
    const int64_t w = idx / a.marks.rows, r = idx - w * a.marks.rows;
    for (uint32_t left = marks_of(a, w, r); left != 0u; left &= left - 1u) {
      const int64_t n = w * a.marks.per + __ffs(int(left)) - 1;
      double v = 0.0;
      for (int t = 0; t < ranges; ++t) v += a.part[(t * a.marks.rows + r) * a.columns + n];
      chain_store(a, r, n, v);
    }
  }
}

}  // namespace

void chain_outputs(Ctx& c, const GettArgs<double>& p, const ChainArgs& chain, const Group& GM,
                   const Group& GN, int64_t columns, const Marks& marks, int ranges, double* part) {
  if (c.sizing()) return;
  ChainOutputs a{};
  a.ch = chain;
  a.GM = GM;
  a.GN = GN;
  a.marks = marks;
  a.columns = columns;
  a.K = p.Kt;
  a.kchunk = (p.Kt + ranges - 1) / ranges;
  a.C = p.C;
  a.part = part;
  a.alpha = p.alpha;
  a.beta = p.beta;
  const int64_t items = (marks.rows + kCRows - 1) / kCRows * marks.words;
  const unsigned ctas = unsigned(std::min<int64_t>(items, 4 * sm_count_linalg()));
  {
    KernelTimer kt(c.stream, "chain_outputs_kernel", kUnitByte, 4.0 * double(marks.rows) * marks.words);
    chain_outputs_kernel<<<dim3(ctas, unsigned(ranges)), kCThreads, 0, c.stream>>>(a);
    CTM_LAUNCH_CHECK();
  }
  if (ranges > 1) {
    KernelTimer kt(c.stream, "chain_sum_kernel", kUnitByte, 4.0 * double(marks.rows) * marks.words);
    chain_sum_kernel<<<grid_for(marks.rows * marks.words, 256), 256, 0, c.stream>>>(a, ranges);
    CTM_LAUNCH_CHECK();
  }
}

}  // namespace ctm
