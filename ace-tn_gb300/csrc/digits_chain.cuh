// FMA chains for the outputs that the digit products mark, after the products (no pipeline
// waits for them): by the CTA that formed their neighbours, or in a kernel of their own.
//
// What bounds it: an FP64 warp instruction issues once in 64 cycles per SM quarter, and
// where few outputs are marked, as usual, the latency of their operands.  So all marked
// outputs of the CTA are listed first, those whose digits may stand are struck off, and the
// others' terms spread over its threads (g lanes an output, sums joined in a fixed tree).
// When the list does not hold them the CTA takes fewer blocks (128 rows by one word) at a
// time.
#pragma once
#include "digits.cuh"

namespace ctm {

constexpr int kCRows = 128;          // rows of a block of marks

// Shared memory of the kernel of its own: the list and a counter, no more than leaves it
// room beside a CTA of digit_gemm_kernel (another stream's; 200 of 227 KB).
constexpr size_t kChainSmem = 20 * 1024;
static_assert(kCRows * 32 * 4 + 16 <= kChainSmem, "chain_marked's list holds a block");

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

// Bytes `byte` of four words.
__device__ __forceinline__ uint32_t plane(const uint4& v, int byte) {
  const uint32_t s = uint32_t(byte) | uint32_t(byte + 4) << 4;
  return __byte_perm(__byte_perm(v.x, v.y, s), __byte_perm(v.z, v.w, s), 0x5410);
}

// Classes of 32 entries of a row and a column, from the words at a and b (left: words up to
// the end of the row): adds to sum (units of 2^-14 of the scales) and any, false where one
// of the two has no digits.
__device__ __forceinline__ bool classes(const uint32_t* a, const uint32_t* b, int left, bool first,
                                        int& sum, uint32_t& any) {
  uint4 u = *reinterpret_cast<const uint4*>(a);
  const uint4 v = *reinterpret_cast<const uint4*>(b);
  if (first && (u.x == kBadCover || v.x == kBadCover)) return false;
  if (left < 4) {  // (not written beyond it)
    u.w = 0u;
    if (left < 3) u.z = 0u;
    if (left < 2) u.y = 0u;
  }
  const uint32_t la = plane(u, 0), lb = plane(v, 0), ma = plane(u, 1), mb = plane(v, 1);
  const uint32_t lm = (la & mb) | (ma & lb);
  if ((la & lb) != 0u) sum += kCoverSum;
  else sum += 6 * __popc(lm) + __popc(ma & mb & ~lm);  // 2^(14 - 11.2) and 1
  any |= plane(u, 2) & plane(v, 2);
  return true;
}

// Whether the digits of an output may stand (digits.cuh).
__device__ __forceinline__ bool covered(const uint32_t* a, const uint32_t* b, int groups) {
  uint32_t any = 0u;
  int sum = 0;
  for (int g = 0; g < groups; g += 4) {
    if (!classes(a + g, b + g, groups - g, g == 0, sum, any)) return false;
    if (sum >= kCoverSum) return true;
  }
  return any == 0u;
}

// The same by a warp or a CTA of kWarps.
template <int kWarps>
__device__ __forceinline__ bool covered_by(const uint32_t* a, const uint32_t* b, int groups) {
  uint32_t any = 0u;
  int sum = 0;
  bool bad = false;
  const int id = kWarps == 1 ? threadIdx.x & 31 : threadIdx.x;
  auto some = [](bool v) {
    return kWarps == 1 ? __any_sync(0xffffffffu, v) != 0 : __syncthreads_or(v) != 0;
  };
  for (int g0 = 0; g0 < groups; g0 += 512 * kWarps) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int g = g0 + 128 * kWarps * i + 4 * id;
      if (g < groups) bad |= !classes(a + g, b + g, groups - g, g == 0, sum, any);
    }
    if (some(bad)) return false;
    if (some(sum >= kCoverSum)) return true;
  }
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  // (summed over a warp only: the others' sums would make it easier to pass)
  return some(sum >= kCoverSum) || !some(any != 0u);
}

__device__ __forceinline__ bool covered(const Cover& c, int64_t rows, int64_t r, int64_t n) {
  const uint32_t* b = c.col + n * c.stride;
  if (c.phases == 0) return covered(c.row + r * c.stride, b, c.groups);
  if (b[0] == kBadCover) return false;
  uint32_t any = 0u;
  for (int i = 0; i < 2 * c.phases; ++i) {
    const uint32_t large = c.row[int64_t(2 * i) * rows + r];
    const uint32_t nonzero = c.row[int64_t(2 * i + 1) * rows + r];
    if ((large & ~nonzero) != 0u) return false;  // a row without digits
    const int first = (i >> 1) * c.per_phase, count = min(c.per_phase, c.blocks - first);
    for (int q = 0; q < count; ++q) {
      const int g = 2 * (first + q) + (i & 1);
      const uint32_t w = g < c.groups ? b[g] : 0u;
      if ((large >> (8 * q) & w & 0xffu) != 0u) return true;
      any |= nonzero >> (8 * q) & w >> 16 & 0xffu;
    }
  }
  return any == 0u;
}

__device__ __forceinline__ void k_offsets(const ChainArgs& ch, int64_t k, int64_t& ka, int64_t& kb) {
  int64_t t0, t1;
  decode(ch.FK, k, t0, t1);
  ka = ch.swapped ? t1 : t0;
  kb = ch.swapped ? t0 : t1;
}

// Outputs 0 .. count - 1, output(o, r, n): their row and column; k0 <= k < k1.  The threads
// id of `threads` (whole warps) share them.
template <class Output>
__device__ __forceinline__ void chain_each(const ChainOutputs& a, int count, int id, int threads,
                                           int64_t k0, int64_t k1, Output&& output) {
  // a warp's lanes on one output where chains are long, else all threads busy and whole
  // sectors of four entries read
  int g = 4;
  while (g < 32 && (int64_t(count) * g * 2 <= threads || k1 - k0 >= 1024) && 8 * g < k1 - k0) g *= 2;
  const int sub = id & (g - 1), groups = threads / g;
  for (int o0 = 0; o0 < count; o0 += groups) {
    if (o0 + (id & ~31) / g >= count) break;  // (the warp alike)
    const int o = o0 + id / g;
    int64_t r = 0, n = 0;
    double v = 0.0;
    if (o < count) {
      int64_t ao, bo, t, ka, kb;
      output(o, r, n);
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

// The outputs of list (block << 12 | row << 5 | bit) by the CTA.
template <int kThreads, class Where>
__device__ void chain_listed(const ChainOutputs& a, const uint32_t* list, int count, int64_t k0,
                             int64_t k1, Where&& where) {
  chain_each(a, count, threadIdx.x, kThreads, k0, k1, [&](int o, int64_t& r, int64_t& n) {
    const uint32_t e = list[o];
    int64_t w;
    where(int(e >> 12), r, w);
    r += (e >> 5) & 127u;
    n = w * a.marks.per + (e & 31u);
  });
}

// The marked outputs of this CTA's blocks; where(block, r0, w): their row and word.  All
// threads take part; their marks were written by this CTA, or before its launch.
template <int kThreads, class Where>
__device__ __noinline__ void chain_marked(const ChainOutputs& a, int blocks, Where where,
                                          uint8_t* buf, size_t bytes, int64_t k0, int64_t k1) {
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
      // (no bits beyond the columns: a product that gave up has not written its words)
      const uint32_t valid =
          low_bits(int(min(int64_t(a.marks.per), a.columns - w * a.marks.per)));
#pragma unroll
      for (int i = 0; i < kCRows / 32; ++i) {
        const int64_t row = r + 32 * i + lane;
        left[i] = row < a.marks.rows ? a.marks.word[w * a.marks.rows + row] & valid : 0u;
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
  auto keep = [&](int n) {  // strikes off what is covered
    if (a.cover.col == nullptr) return n;
    if (threadIdx.x == 0) *s_count = 0;
    // a warp each where rows are long (up to K = 5184 a thread each is faster, 8 against 36
    // us at 144 x 20736: most are covered within the first entries)
    constexpr int kWarps = kThreads / 32, kEach = 4;
    const bool by_warp = a.cover.phases == 0 && a.cover.groups > 1024;
    for (int i = 0; by_warp && i < n; i += kWarps * kEach) {
      uint32_t e[kEach];
      bool stays[kEach];
#pragma unroll
      for (int j = 0; j < kEach; ++j) {
        const int o = i + kWarps * j + int(threadIdx.x >> 5);
        e[j] = 0u;
        stays[j] = false;
        if (o >= n) continue;
        int64_t r, w;
        e[j] = list[o];
        where(int(e[j] >> 12), r, w);
        stays[j] = !covered_by<1>(a.cover.row + (r + ((e[j] >> 5) & 127u)) * a.cover.stride,
                                  a.cover.col + (w * a.marks.per + (e[j] & 31u)) * a.cover.stride,
                                  a.cover.groups);
      }
      __syncthreads();  // entries before i + kWarps kEach are read
      if ((threadIdx.x & 31) == 0) {
#pragma unroll
        for (int j = 0; j < kEach; ++j)
          if (stays[j]) list[atomicAdd(s_count, 1)] = e[j];
      }
    }
    for (int i = 0; !by_warp && i < n; i += kThreads) {
      const int o = i + int(threadIdx.x);
      uint32_t e = 0u;
      bool stays = false;
      if (o < n) {
        int64_t r, w;
        e = list[o];
        where(int(e >> 12), r, w);
        stays = !covered(a.cover, a.marks.rows, r + ((e >> 5) & 127u),
                         w * a.marks.per + (e & 31u));
      }
      __syncthreads();  // entries before i + kThreads are read
      if (stays) list[atomicAdd(s_count, 1)] = e;
    }
    __syncthreads();
    n = *s_count;
    __syncthreads();
    return n;
  };
  // n marked outputs of the blocks b0 .. b1 - 1, false when the list does not hold them
  auto listed = [&](int b0, int b1, int n) {
    if (n > cap) return false;
    n = keep(n);
    if (a.queue.entry == nullptr || n == 0) {
      chain_listed<kThreads>(a, list, n, k0, k1, where);
    } else {
      if (threadIdx.x == 0) {  // (a full queue's count grows no further)
        const int now = *reinterpret_cast<volatile int*>(a.queue.count);
        *s_count = now < a.queue.cap ? atomicAdd(a.queue.count, n) : now;
      }
      __syncthreads();
      const int at = *s_count, fit = min(n, max(0, a.queue.cap - at));
      for (int i = threadIdx.x; i < fit; i += kThreads) {
        int64_t r, w;
        where(int(list[i] >> 12), r, w);
        a.queue.entry[at + i] = make_uint2(uint32_t(r) + ((list[i] >> 5) & 127u),
                                           uint32_t(w) * a.marks.per + (list[i] & 31u));
      }
      chain_listed<kThreads>(a, list + fit, n - fit, k0, k1, where);
    }
    __syncthreads();
    return true;
  };
  const int count = add(0, blocks);
  if (count == 0 || (count <= cap && listed(0, blocks, count))) return;
  const int step = max(1, int(int64_t(blocks) * cap / (2 * int64_t(count))));
  for (int b0 = 0; b0 < blocks; b0 += step) {
    const int b1 = min(b0 + step, blocks);
    if (listed(b0, b1, add(b0, b1))) continue;
    for (int b = b0; b < b1; ++b) listed(b, b + 1, add(b, b + 1));  // (one always fits)
  }
}

}  // namespace ctm
