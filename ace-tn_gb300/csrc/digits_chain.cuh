// FMA chains for the outputs that the digit products mark, after the products (no pipeline
// waits for them): by the CTA that formed their neighbours, or in a kernel of their own.
//
// What bounds it: an FP64 warp instruction issues once in 64 cycles per SM quarter, and
// where few outputs are marked, as usual, the latency of their operands.  So all marked
// outputs of the CTA are listed first and their terms spread over its threads (g lanes an
// output, sums joined in a fixed tree).  When the list does not hold them the CTA goes
// block by block (128 rows by one word), and a block with more than a quarter marked is
// computed as a tile through shared memory.
#pragma once
#include "digits.cuh"

namespace ctm {

constexpr int kCRows = 128;          // rows of a block of marks
constexpr int kDense = kCRows * 8;   // marked outputs from which a block is a tile
constexpr int kCK = 16;              // contracted indices per step of a tile

// Shared memory: the list and a counter, or a tile's operands and offsets (32 KB at least).
constexpr size_t kChainTile = (size_t(kCK) * (kCRows + 1 + 33) + kCRows + 32 + 2 * kCK) * 8 +
                              (kCRows + 2) * 4;
constexpr size_t kChainSmem = 40 * 1024;
static_assert(kChainTile <= 32 * 1024 && kDense * 4 + 16 <= 32 * 1024, "chain_marked's buffer");

__device__ __forceinline__ void chain_store(const ChainOutputs& a, int64_t r, int64_t n, double v) {
  if (a.part != nullptr) {
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

// The outputs of list (block << 12 | row << 5 | bit), k0 <= k < k1.
template <int kThreads, class Where>
__device__ void chain_listed(const ChainOutputs& a, const uint32_t* list, int count, int64_t k0,
                             int64_t k1, Where&& where) {
  // a warp's lanes on one output where chains are long, else all threads busy and whole
  // sectors of four entries read
  int g = 4;
  while (g < 32 && (count * g * 2 <= kThreads || k1 - k0 >= 1024) && 8 * g < k1 - k0) g *= 2;
  const int sub = threadIdx.x & (g - 1), groups = kThreads / g;
  for (int o0 = 0; o0 < count; o0 += groups) {
    const int o = o0 + int(threadIdx.x) / g;
    int64_t r = 0, n = 0;
    double v = 0.0;
    if (o < count) {
      const uint32_t e = list[o];
      int64_t w, ao, bo, t, ka, kb;
      where(int(e >> 12), r, w);
      r += (e >> 5) & 127u;
      n = w * a.marks.per + (e & 31u);
      decode(a.ch.FM, r, ao, t);
      decode(a.ch.FN, n, bo, t);
      const double* x = a.ch.a + ao;
      const double* y = a.ch.b + bo;
#pragma unroll 4
      for (int64_t k = k0 + sub; k < k1; k += g) {
        k_offsets(a.ch, k, ka, kb);
        v = fma(x[ka], y[kb], v);
      }
    }
    for (int s = g / 2; s > 0; s >>= 1) v += __shfl_xor_sync(0xffffffffu, v, s);
    if (o < count && sub == 0) chain_store(a, r, n, v);
  }
}

// The marked outputs of the block at row r0, word w as a tile.
template <int kThreads>
__device__ void chain_tile(const ChainOutputs& a, uint8_t* buf, int64_t r0, int64_t w, int64_t k0,
                           int64_t k1) {
  double (*xs)[kCRows + 1] = reinterpret_cast<double (*)[kCRows + 1]>(buf);
  double (*ys)[33] = reinterpret_cast<double (*)[33]>(xs + kCK);
  int64_t* s_ro = reinterpret_cast<int64_t*>(ys + kCK);
  int64_t* s_co = s_ro + kCRows;
  int64_t* s_ka = s_co + 32;
  int64_t* s_kb = s_ka + kCK;
  uint32_t* s_mark = reinterpret_cast<uint32_t*>(s_kb + kCK);
  const int tid = threadIdx.x;
  const int64_t n0 = w * a.marks.per;
  for (int i = tid; i < kCRows + 32; i += kThreads) {
    int64_t o = -1, t;
    if (i < kCRows) {
      const bool in = r0 + i < a.marks.rows;
      if (in) decode(a.ch.FM, r0 + i, o, t);
      s_ro[i] = o;
      s_mark[i] = in ? a.marks.word[w * a.marks.rows + r0 + i] : 0u;
    } else {
      const int64_t n = n0 + i - kCRows;
      if (i - kCRows < a.marks.per && n < a.columns) decode(a.ch.FN, n, o, t);
      s_co[i - kCRows] = o;
    }
  }
  const int ty = tid >> 3, tx = tid & 7;  // the first 256 threads: 4 x 4 outputs each
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
    for (int i = tid; i < kCK * kCRows; i += kThreads) {
      const int k = i & (kCK - 1), r = i / kCK;
      xs[k][r] = s_ro[r] >= 0 && s_ka[k] >= 0 ? a.ch.a[s_ro[r] + s_ka[k]] : 0.0;
    }
    for (int i = tid; i < kCK * 32; i += kThreads) {
      const int n = i & 31, k = i >> 5;
      ys[k][n] = s_co[n] >= 0 && s_kb[k] >= 0 ? a.ch.b[s_co[n] + s_kb[k]] : 0.0;
    }
    __syncthreads();
    if (tid < 256) {
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
  }
  __syncthreads();
  if (tid < 256) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (s_mark[ty + 32 * i] >> (tx + 8 * j) & 1u)
          chain_store(a, r0 + ty + 32 * i, n0 + tx + 8 * j, acc[i][j]);
  }
}

// The marked outputs of this CTA's blocks; where(block, r0, w): their row and word.  All
// threads take part; their marks were written by this CTA, or before its launch.
template <int kThreads, class Where>
__device__ __noinline__ void chain_marked(const ChainOutputs& a, int blocks, Where where,
                                          uint8_t* buf, size_t bytes, int64_t k0, int64_t k1) {
  static_assert(kThreads >= 256, "chain_tile's outputs");
  int* s_count = reinterpret_cast<int*>(buf);
  uint32_t* list = reinterpret_cast<uint32_t*>(buf + 16);
  const int cap = int((bytes - 16) / 4);
  auto add = [&](int first, int last) {  // the marks of blocks first .. last - 1
    if (threadIdx.x == 0) *s_count = 0;
    __syncthreads();
    for (int b = first + int(threadIdx.x >> 5); b < last; b += kThreads / 32) {  // a warp each
      int64_t r, w;
      where(b, r, w);
      const int lane = threadIdx.x & 31;
      uint32_t left[kCRows / 32];
#pragma unroll
      for (int i = 0; i < kCRows / 32; ++i) {
        const int64_t row = r + 32 * i + lane;
        left[i] = row < a.marks.rows ? a.marks.word[w * a.marks.rows + row] : 0u;
      }
#pragma unroll
      for (int i = 0; i < kCRows / 32; ++i) {
        if (left[i] == 0u) continue;
        int at = atomicAdd(s_count, __popc(left[i]));
        for (uint32_t m = left[i]; m != 0u; m &= m - 1u, ++at)
          if (at < cap)
            list[at] = uint32_t(b) << 12 | uint32_t(32 * i + lane) << 5 | uint32_t(__ffs(int(m)) - 1);
      }
    }
    __syncthreads();
    const int n = *s_count;
    __syncthreads();
    return n;
  };
  const int count = add(0, blocks);
  if (count <= cap) {
    chain_listed<kThreads>(a, list, count, k0, k1, where);
    return;
  }
  for (int b = 0; b < blocks; ++b) {
    const int n = add(b, b + 1);
    if (n > kDense) {
      int64_t r, w;
      where(b, r, w);
      chain_tile<kThreads>(a, buf, r, w, k0, k1);
    } else {
      chain_listed<kThreads>(a, list, n, k0, k1, where);
    }
    __syncthreads();
  }
}

}  // namespace ctm
