// Digit products of a long operand with a small one over a short contracted
// index: the site-tensor steps of the enlarged corners, the edge
// renormalization and the density matrices (K and the small side D^2 and D^2 d,
// the long side chi^2 D^2 and more).
//
// These are bound by memory and by the epilogue, not by the tensor cores: as
// digit_gemm_kernel products they wrote and re-read 16 bytes of digits per FP64
// entry and waited for one tile after another (746496 x 72 x 36: 0.28 ms of
// splitting and 1.07 ms of products, for 0.095 ms of FP64 traffic).  Here the
// long operand is read once as FP64: eight warps form the digits of a tile of 128
// rows straight in the shared memory that the MMAs read (32-byte swizzle, one
// block per 16 indices), the small operand's digits stay there for the whole
// kernel, and eight warps read the accumulators of one group of columns while
// the MMAs of the next run: 0.40 ms in one kernel.  K = 72 with 36 columns (two
// phases of the contracted index, one accumulator buffer) takes 0.72 ms, 1.16 ms
// as digit_gemm_kernel.  (Both before the splitting warps noted which entries are
// large, for the outputs far below their scales: 0.42 ms for the first.)
#include <algorithm>
#include <type_traits>

#include "digits.cuh"
#include "digits_chain.cuh"

namespace ctm {

namespace {

constexpr int kSThreads = 544;  // warps 0-7 split, warps 8-15 epilogue, warp 16 issues
constexpr int kTileM = 128;
constexpr uint32_t kABlock = kDigits * kTileM * 32;  // one block of 16 indices, all digits
constexpr int kMaxN = 128, kMaxK = 192, kMaxCols = 192;
constexpr size_t kStreamSmem = 217 * 1024;

struct StreamArgs {
  const double* x;      // the long operand
  Group FX, FK;         // its rows (s0) and the contracted index
  int k_is_s1;
  int64_t M;
  int N, K;
  Group GM, GN;         // output strides (s1)
  const int* eb;
  double* C;
  double alpha, beta;
  int blocks, per_phase, phases;  // blocks of 16 indices
  int passes;                     // groups of NT columns
  int nbuf;                       // digit buffers of the long operand
  int64_t tiles;
  int* status;
  int guard;                      // small outputs are marked too
  uint32_t* cover;                // of the long operand's rows (Cover::row)
  ChainOutputs out;               // word 2 * pass + half
};

__device__ __forceinline__ bool wait_warp(uint64_t* bar, uint32_t parity) {
  const bool ok = mbar_wait(bar, parity);
  __syncwarp();
  return __all_sync(0xffffffffu, ok);
}

// One output's eight accumulators as an integer in units of 2^-kUnit of the
// scales (the sum of K products below 1 fits in 63 bits), to nearest: the groups below
// kSmallGroups are under 2^22, converted by an FP32 addition each, the others by
// the conversion unit.  The rounding is 2^-58, 2^-57 and 2^-56 at most (K <= 36, 80, 192),
// with a deviation of 2^-59.8 to 2^-57.8 beside the dropped digit products' sqrt(K)
// 2^-62.2, and 60 instructions per output fewer than 96 bits need: the epilogue's
// instructions bound these products.
template <int kSmallGroups, int kUnit>
__device__ __forceinline__ long long fixed_point(const float (&f)[kDigits]) {
  int g[kDigits];
#pragma unroll
  for (int s = 0; s < kDigits; ++s)
    g[s] = s < kSmallGroups ? int_small(f[s]) : __float2int_rn(f[s]);
  // group s weighs 2^(-12 - 8 s)
  long long t;
  if (kSmallGroups == kDigits) {
    t = (long long)(g[2] * 256 + g[3]) * (1 << (kUnit - 36));
    t += (long long)(g[4] * 256 + g[5]) * (1 << (kUnit - 52));
    t += (g[6] * 256 + g[7] + (1 << (67 - kUnit))) >> (68 - kUnit);
  } else {
    t = (long long)g[2] * (1 << (kUnit - 28));
    t += (long long)g[3] * (1 << (kUnit - 36));
    t += (long long)g[4] * (1 << (kUnit - 44));
    t += (long long)g[5] * (1 << (kUnit - 52));
    t += ((long long)g[6] * 256 + g[7] + (1 << (67 - kUnit))) >> (68 - kUnit);
  }
  const uint32_t top = uint32_t(g[0] * 256 + g[1]) << (kUnit - 52);
  return (long long)((unsigned long long)t + ((unsigned long long)top << 32));
}

// Outside the normal range, and zeros.
__device__ __noinline__ double rare_value(long long t, int er, int ec, int unit) {
  return round_96(t >> 32, uint32_t(t), row_exponent(er) + row_exponent(ec) - 2 * 1023 - unit);
}

// kMode 0: K <= 36, all groups below 2^22 (7 2^14 K); 1: K <= 80, the first four
// (3 2^14 K); 2: K <= 192, the first two.
template <int NT, int kMode>
__global__ void __launch_bounds__(kSThreads, 1)
    digit_stream_kernel(const __grid_constant__ CUtensorMap tB,
                        const __grid_constant__ StreamArgs p) {
  extern __shared__ uint8_t dyn_smem[];
  uint8_t* base = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(dyn_smem) + 1023) & ~uintptr_t(1023));
  constexpr uint32_t kBBlock = uint32_t(kDigits) * NT * 32;
  constexpr int kT = 512 / (kDigits * NT);  // accumulator buffers in tensor memory
  const uint32_t a_bytes = uint32_t(p.per_phase) * kABlock;
  uint8_t* sA = base;
  uint8_t* sB = base + size_t(p.nbuf) * a_bytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sB + size_t(p.passes) * p.blocks * kBBlock);
  uint64_t* a_full = bars;           // [2]
  uint64_t* a_empty = bars + 2;      // [2]
  uint64_t* t_full = bars + 4;       // [4]
  uint64_t* t_empty = bars + 8;      // [4]
  uint64_t* b_full = bars + 12;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(bars + 13);
  __shared__ int s_fail, s_split_fail[2];
  __shared__ int s_half[2][kTileM];
  __shared__ int64_t s_ko[kMaxK];
  __shared__ int64_t s_cn[kMaxCols];
  __shared__ int s_eb[kMaxCols];
  __shared__ uint32_t s_bad[kMaxCols / 8];  // columns without digits, by pass and half
  __shared__ int s_er[8][kTileM];  // tiles in flight: two digit buffers, up to four accumulators

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    s_fail = 0;
    s_split_fail[0] = s_split_fail[1] = 0;
    for (int i = 0; i < 2; ++i) {
      mbar_init(&a_full[i], 8);
      mbar_init(&a_empty[i], 1);
    }
    for (int i = 0; i < 4; ++i) {
      mbar_init(&t_full[i], 1);
      mbar_init(&t_empty[i], 8);
    }
    mbar_init(b_full, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int k = threadIdx.x; k < p.K; k += kSThreads) {
    int64_t o0, o1;
    decode(p.FK, k, o0, o1);
    s_ko[k] = p.k_is_s1 ? o1 : o0;
  }
  for (int n = threadIdx.x; n < p.passes * NT; n += kSThreads) {
    int64_t t, off = -1;
    int e = 0;
    if (n < p.N) {
      decode(p.GN, n, t, off);
      e = p.eb[n];
    }
    s_cn[n] = off;
    s_eb[n] = e;
  }
  if (warp < 2 * p.passes) {  // (16 warps and more: at most 12 words)
    const int n = warp * (NT / 2) + lane;
    const bool bad = lane < NT / 2 && n < p.N && p.eb[n] == kBadField;
    const uint32_t mask = __ballot_sync(0xffffffffu, bad);
    if (lane == 0) s_bad[warp] = mask;
  }
  if (warp == 16) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_holder)),
                 "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_holder;
  const int refills = p.phases == 1 ? 1 : p.passes * p.phases;  // digit buffers per tile

  if (warp < 8) {
    // ---------------- digits of the long operand: two threads per row, each every
    // other group of eight indices
    constexpr int kGroups = 3;
    const int row = threadIdx.x & (kTileM - 1), half = threadIdx.x >> 7;
    uint32_t fill = 0;
    int ring = 0;
    bool ok = true;
    for (int64_t tile = blockIdx.x; tile < p.tiles && ok; tile += gridDim.x, ring = (ring + 1) & 7) {
      const int64_t m = tile * kTileM + row;
      const bool valid = m < p.M;
      int64_t xo = 0, t;
      if (valid) decode(p.FX, m, xo, t);
      const double* x = p.x + xo;
      // entries, then digit words: group `half` of block q of a phase (five blocks'
      // worth for K = 72 spills)
      unsigned long long u[kGroups][8];
      auto load = [&](int first, int count) {
#pragma unroll
        for (int q = 0; q < kGroups; ++q)
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int k = (first + q) * 16 + half * 8 + i;
            u[q][i] = valid && q < count && k < p.K
                          ? (unsigned long long)__double_as_longlong(x[s_ko[k]])
                          : 0ull;
          }
      };
      // phase ph's entries into words, and which of them are large or nonzero
      auto words = [&](int e, int ph, int count, bool note) {
        const int E = row_exponent(e);
        uint32_t large = 0u, nonzero = 0u;
#pragma unroll
        for (int q = 0; q < kGroups; ++q) {
          if (q >= count) continue;
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            nonzero |= (u[q][i] << 1 != 0ull ? 1u : 0u) << (8 * q + i);
            u[q][i] = digit_word(__longlong_as_double((long long)u[q][i]), E);
            large |= (large_digit(u[q][i]) ? 1u : 0u) << (8 * q + i);
          }
        }
        if (note && valid) {
          uint32_t* c = p.cover + int64_t(4 * ph + 2 * half) * p.M + m;
          c[0] = e == kBadField ? 1u : large;
          c[p.M] = e == kBadField ? 0u : nonzero;
        }
      };
      int e = 0;
      if (p.phases == 1) {
        load(0, p.blocks);
#pragma unroll
        for (int q = 0; q < kGroups; ++q)
#pragma unroll
          for (int i = 0; i < 8; ++i) e = max(e, int(u[q][i] >> 52) & 0x7ff);
      } else if (valid) {
#pragma unroll 8
        for (int k = half; k < p.K; k += 2) e = max(e, exponent_field(x[s_ko[k]]));
      }
      s_half[half][row] = e;
      asm volatile("bar.sync 2, 256;" ::: "memory");  // the eight splitting warps
      e = max(e, s_half[half ^ 1][row]);
      if (p.phases == 1) words(e, 0, p.blocks, true);
      for (int f = 0; f < refills; ++f, ++fill) {
        const int first = (f % p.phases) * p.per_phase;
        const int count = min(p.per_phase, p.blocks - first);
        if (p.phases > 1) {
          load(first, count);
          words(e, f % p.phases, count, f < p.phases);
        }
        const int b = int(fill) % p.nbuf;
        ok = ok && wait_warp(&a_empty[b], ((fill / uint32_t(p.nbuf)) & 1u) ^ 1u);
        if (!ok) continue;  // (all eight warps still meet at the next tile's barrier)
        if (f == 0 && half == 0) s_er[ring][row] = e;
        uint8_t* dst = sA + size_t(b) * a_bytes + row * 32 + ((half ^ ((row >> 2) & 1)) << 4);
#pragma unroll
        for (int q = 0; q < kGroups; ++q) {
          if (q < count)
            put_digits(u[q], [&](int d, uint4 w) {
              *reinterpret_cast<uint4*>(dst + q * kABlock + d * (kTileM * 32)) = w;
            });
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(&a_full[b]);
      }
      // a warp that gave up tells the others before they meet again
      if (!ok && lane == 0) s_split_fail[ring & 1] = 1;
      asm volatile("bar.sync 2, 256;" ::: "memory");
      if (s_split_fail[ring & 1]) ok = false;
    }
    if (!ok && lane == 0) atomicOr(&s_fail, 1);
  } else if (warp == 16) {
    if (lane == 0) {
      // ---------------- the small operand, then the MMAs
      const uint32_t bytes = uint32_t(p.passes) * p.blocks * kBBlock;
      mbar_expect_tx(b_full, bytes);
      for (int ps = 0; ps < p.passes; ++ps)
        for (int kb = 0; kb < p.blocks; ++kb)
          tma_load_3d(sB + size_t(ps * p.blocks + kb) * kBBlock, &tB, kb * 16, ps * NT, 0, b_full);
      bool ok = mbar_wait(b_full, 0);
      uint32_t use = 0, acc = 0;
      for (int64_t tile = blockIdx.x; tile < p.tiles && ok; tile += gridDim.x) {
        for (int ps = 0; ps < p.passes && ok; ++ps, ++acc) {
          const int tb = int(acc) % kT;
          ok = mbar_wait_spin(&t_empty[tb], ((acc / kT) & 1u) ^ 1u);
          const uint32_t dst = tmem + uint32_t(tb * kDigits * NT);
          for (int ph = 0; ph < p.phases && ok; ++ph) {
            const bool fresh = p.phases > 1 || ps == 0;
            const int b = int(use) % p.nbuf;
            if (fresh) ok = mbar_wait_spin(&a_full[b], (use / uint32_t(p.nbuf)) & 1u);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int first = ph * p.per_phase, count = min(p.per_phase, p.blocks - first);
            for (int kb = 0; kb < count; ++kb) {
              const uint64_t da = smem_desc(sA + size_t(b) * a_bytes + size_t(kb) * kABlock, 16);
              const uint64_t db =
                  smem_desc(sB + size_t(ps * p.blocks + first + kb) * kBBlock, 16);
#pragma unroll
              for (int i = 0; i < kDigits; ++i) {
                constexpr int kGroup = 256 / NT;
#pragma unroll
                for (int j = 0; j < kDigits - i; j += kGroup) {
                  const int cnt = min(kGroup, kDigits - i - j);
                  mma_bf16(dst + uint32_t((i + j) * NT), da + uint64_t((i * kTileM * 32) >> 4),
                           db + uint64_t((j * NT * 32) >> 4), idesc_bf16(kTileM, cnt * NT),
                           (ph == 0 && kb == 0 && i == 0) ? 0u : 1u);
                }
              }
            }
            if (p.phases > 1 || ps == p.passes - 1) {
              mma_commit(&a_empty[b]);
              ++use;
            }
          }
          if (ok) mma_commit(&t_full[tb]);
        }
      }
      if (!ok) {
        atomicOr(&s_fail, 1);
        (void)mbar_wait(b_full, 0);  // no copy in flight when the CTA leaves
      }
    }
    __syncwarp();
  } else {
    // ---------------- epilogue
    constexpr int kHalf = NT / 2;
    constexpr int kSmallGroups = kMode == 0 ? 8 : kMode == 1 ? 4 : 2;
    constexpr int kUnit = kMode == 0 ? 57 : kMode == 1 ? 56 : 55;
    const unsigned long long small = p.guard ? 1ull << (kUnit - kCoverBits) : 0ull;
    const bool scaled = !(p.alpha == 1.0 && p.beta == 0.0);
    const int lane_base = (warp & 3) * 32, half = (warp - 8) >> 2;
    const int row = lane_base + lane;
    uint32_t acc = 0;
    int ring = 0;
    bool ok = true;
    for (int64_t tile = blockIdx.x; tile < p.tiles && ok; tile += gridDim.x, ring = (ring + 1) & 7) {
      const int64_t m = tile * kTileM + row;
      const bool valid = m < p.M;
      int64_t ro = 0, t;
      if (valid) decode(p.GM, m, t, ro);
      double* out = p.C + ro;
      for (int ps = 0; ps < p.passes; ++ps, ++acc) {
        const int tb = int(acc) % kT;
        ok = wait_warp(&t_full[tb], (acc / kT) & 1u);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const int er = s_er[ring][row];
        // (er + 1) + (ec + 1) - 2 1023 - unit + 1023
        const int ebase = max(er, 1) + 2 - 1023 - kUnit;
        const uint32_t ta = tmem + (uint32_t(lane_base) << 16) +
                            uint32_t(tb * kDigits * NT + half * kHalf);
        const int n0 = ps * NT + half * kHalf;
        // marked: the chain's, stored after the products
        uint32_t mark = s_bad[2 * ps + half];
        if (er == kBadField) mark = low_bits(min(kHalf, p.N - n0));
        // one copy of the body (the roles' code together has to stay in the
        // instruction cache: unrolled, a third of the cycles waited for it)
#pragma unroll 1
        for (int c = 0; c < kHalf && n0 + c < p.N; c += 4) {  // the warp alike
          float f[kDigits][4];
#pragma unroll
          for (int s = 0; s < kDigits; ++s) tmem_ld4(ta + uint32_t(s * NT + c), f[s]);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int s = 0; s < kDigits; ++s)
#pragma unroll
            for (int j = 0; j < 4; ++j) asm volatile("" : "+f"(f[s][j]));
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int64_t off = s_cn[n0 + c + j];
            const float g[kDigits] = {f[0][j], f[1][j], f[2][j], f[3][j],
                                      f[4][j], f[5][j], f[6][j], f[7][j]};
            const long long fx = fixed_point<kSmallGroups, kUnit>(g);
            if (valid && off >= 0) {
              const int ec = s_eb[n0 + c + j];
              const unsigned long long mag = (unsigned long long)(fx < 0 ? -fx : fx);
              if (mag < small) mark |= 1u << (c + j);
              const int lz = __clzll((long long)mag);
              const unsigned long long nm = mag << (lz & 63);
              // 53 bits, to nearest even
              const unsigned long long r = (nm + 0x3ff + ((nm >> 11) & 1)) >> 11;
              // exponent field of the leading bit (bit 63 - lz of fx); a carry out of
              // the rounding leaves r = 0 in 53 bits and goes through the rare path
              const int ef = ebase + max(ec, 1) + (63 - lz);
              double v;
              if (nm < 0xfffffffffffffc00ull && unsigned(ef - 1) < 2044u && mag != 0)
                v = __longlong_as_double(
                    (long long)((((unsigned long long)unsigned(ef - 1)) << 52) + r) |
                    (fx & (long long)0x8000000000000000ull));
              else
                v = rare_value(fx, er, ec, kUnit);
              if (scaled) {
                v *= p.alpha;
                if (p.beta != 0.0) v = (mark >> (c + j) & 1u) ? out[off] : fma(p.beta, out[off], v);
              }
              out[off] = v;
            }
          }
          __syncwarp();
        }
        if (valid) p.out.marks.word[(2 * ps + half) * p.M + m] = mark;
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        if (lane == 0) mbar_arrive(&t_empty[tb]);
      }
    }
    if (!ok && lane == 0) atomicOr(&s_fail, 1);
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (threadIdx.x == 0 && s_fail) atomicOr(p.status, 2);
  if (warp == 16) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u)
                 : "memory");
  }
  if (s_fail == 0) {
    const int words = 2 * p.passes;
    const int mine = int((p.tiles - blockIdx.x + gridDim.x - 1) / gridDim.x);
    auto where = [&](int b, int64_t& r, int64_t& w) {
      const int t = b / words;
      r = (blockIdx.x + int64_t(t) * gridDim.x) * kTileM;
      w = b - t * words;
    };
    chain_marked<kSThreads>(p.out, mine * words, where, base,
                            size_t(p.nbuf) * a_bytes, 0, p.K);
  }
}

// Columns per pass, blocks per phase and digit buffers; false: does not fit.
struct StreamPlan {
  int nt = 0, passes = 0, blocks = 0, per_phase = 0, phases = 0, nbuf = 0;
  size_t smem = 0;
};

bool stream_plan(int64_t N, int64_t K, StreamPlan& pl) {
  if (N > kMaxN || K > kMaxK || N < 1 || K < 1) return false;
  pl.blocks = int((K + 15) / 16);
  const bool one_phase = pl.blocks <= 3;
  // one phase: columns in groups of 32, two accumulator buffers; else all
  // columns at once where they fit, as every group needs the digits again
  pl.nt = N <= 16 ? 16 : N <= 32 || one_phase ? 32 : N <= 48 || (N > 64 && N <= 96) ? 48 : 64;
  pl.passes = int((N + pl.nt - 1) / pl.nt);
  const size_t b = size_t(pl.passes) * pl.blocks * kDigits * pl.nt * 32;
  // blocks per phase and buffers (two buffers of two blocks instead of one of three
  // took 8 % longer at K = 72)
  struct Try {
    int per, nbuf;
  };
  const Try tries[] = {{3, 2}, {3, 1}, {2, 2}, {2, 1}, {1, 2}, {1, 1}};
  for (const Try& t : tries) {
    const int per = std::min(t.per, pl.blocks);
    const size_t smem = 1024 + size_t(t.nbuf) * per * kABlock + b + 256;
    if (smem > kStreamSmem) continue;
    pl.per_phase = per;
    pl.phases = (pl.blocks + per - 1) / per;
    pl.nbuf = t.nbuf;
    pl.smem = smem;
    return true;
  }
  return false;
}

}  // namespace

bool stream_fits(const GettArgs<double>& p, bool& swap) {
  swap = p.Nt > p.Mt;
  const int64_t M = swap ? p.Nt : p.Mt, N = swap ? p.Mt : p.Nt;
  StreamPlan pl;
  return p.bext == 1 && M >= 8192 && stream_plan(N, p.Kt, pl);
}

void stream_contract(Ctx& c, const GettArgs<double>& p, bool swap) {
  Scope scope(c);
  const Digits db = operand_digits(c, p, swap);
  StreamPlan pl;
  StreamArgs a{};
  a.M = swap ? p.Nt : p.Mt;
  a.N = int(swap ? p.Mt : p.Nt);
  a.K = int(p.Kt);
  stream_plan(a.N, a.K, pl);
  Marks marks{};
  marks.rows = a.M;
  marks.per = pl.nt / 2;
  marks.words = 2 * pl.passes;
  marks.word = c.alloc<uint32_t>(size_t(marks.rows) * marks.words);
  a.cover = c.alloc<uint32_t>(size_t(4 * pl.phases) * size_t(a.M));
  if (c.sizing()) return;
  a.x = swap ? p.B : p.A;
  a.FX = swap ? p.N : p.M;
  a.FK = p.K;
  a.k_is_s1 = swap ? 1 : 0;
  a.GM = a.FX;
  a.GN = swap ? p.M : p.N;
  a.eb = db.exps;
  a.C = p.C;
  a.alpha = p.alpha;
  a.beta = p.beta;
  a.blocks = pl.blocks;
  a.per_phase = pl.per_phase;
  a.phases = pl.phases;
  a.passes = pl.passes;
  a.nbuf = pl.nbuf;
  a.tiles = (a.M + kTileM - 1) / kTileM;
  a.status = status_flags(c);
  a.guard = p.beside_scales ? 0 : 1;
  a.out = chain_outputs(p, swap, marks);
  a.out.cover = Cover{a.cover, p.beta != 0.0 ? nullptr : db.cover, cover_stride(p.Kt),
                      int((p.Kt + 7) / 8), pl.phases, pl.per_phase, pl.blocks};
  const int64_t Kp = (p.Kt + 7) / 8 * 8;
  CUtensorMap tB;
  {
    const cuuint64_t dims[3] = {cuuint64_t(Kp), cuuint64_t(a.N), cuuint64_t(kDigits)};
    const cuuint64_t strides[2] = {cuuint64_t(Kp) * 2, cuuint64_t(a.N) * cuuint64_t(Kp) * 2};
    const cuuint32_t box[3] = {16, cuuint32_t(pl.nt), cuuint32_t(kDigits)};
    const cuuint32_t estr[3] = {1, 1, 1};
    const CUresult res = encode_tiled()(
        &tB, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, db.dig, dims, strides, box, estr,
        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_32B,
        CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    CTM_REQUIRE(res == CUDA_SUCCESS, CTM_ERR_CUDA,
                "cuTensorMapEncodeTiled failed with code " + std::to_string(int(res)));
  }
  const unsigned grid = unsigned(std::min<int64_t>(a.tiles, sm_count_linalg()));
  auto launch = [&](auto kern) {
    CTM_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(pl.smem)));
    const double flops = 2.0 * double(a.M) * a.N * a.K;
    KernelTimer timer(c.stream, kTagGettF64, flops);
    KernelTimer kt(c.stream, "digit_stream_kernel", kUnitFlop, flops);
    kern<<<grid, kSThreads, pl.smem, c.stream>>>(tB, a);
  };
  auto pick = [&](auto nt) {
    constexpr int n = decltype(nt)::value;
    if (a.K <= 36) launch(digit_stream_kernel<n, 0>);
    else if (a.K <= 80) launch(digit_stream_kernel<n, 1>);
    else launch(digit_stream_kernel<n, 2>);
  };
  if (pl.nt == 16) pick(std::integral_constant<int, 16>());
  else if (pl.nt == 32) pick(std::integral_constant<int, 32>());
  else if (pl.nt == 48) pick(std::integral_constant<int, 48>());
  else pick(std::integral_constant<int, 64>());
  CTM_LAUNCH_CHECK();
}

}  // namespace ctm
