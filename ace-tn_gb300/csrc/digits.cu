// FP64 contractions as exact digit products on the tensor cores.
//
// GB300's FP64 units deliver 1.1 TFLOP/s and its BF16 tensor cores 1945, so an
// FP64 product is formed from BF16 products that carry no rounding error
// (error-free splitting after Ozaki, Ogita, Oishi and Rump, Numer. Algorithms
// 59 (2012) 95):
//
//  * every row of an operand (its entries over the contracted index) is scaled
//    by a power of two to |x| < 1, rounded to 62 fractional bits and written in
//    eight balanced base-256 digits, each in [-128, 127] (the top one in
//    [-64, 64]) and so exact in BF16;
//  * the 36 products of digit i of A with digit j of B, i + j <= 7, accumulate
//    in eight FP32 accumulators by s = i + j.  A digit product is an integer of
//    at most 2^14 (2^13 with a top digit, 2^12 with two), so the partial sums
//    of the groups s <= 5 over up to 192 contracted indices are integers below
//    2^24: exact in FP32, in any order.  (Groups 6 and 7 reach 2^24.2 and
//    2^24.4 when all digits are extreme; an error of one there is 2^-60 of the
//    scales.)
//  * after every 192 indices the accumulators go from tensor memory into a
//    96-bit integer per output, and the last step rounds that integer to FP64
//    once.
//
// What is dropped is the digit products with i + j >= 8, at most 7 K 2^14 /
// 2^76 of the product of the two rows' scales and about sqrt(K) 2^-60 of it on
// data without sign structure, against K 2^-53 (sqrt(K) 2^-54) of the entries'
// products for a chain of FMAs: on random operands the result is 10 to 100
// times closer to the exact one than the FMA chain's.
//
// That is the error beside the two rows' scales.  Outputs whose terms all lie far
// below them (a row graded one way along the contracted index, the column the
// other; digits.cuh), and those on a row or column with an infinity or a NaN,
// which has no digits, are marked and formed by the FMA chain after the products
// (digits_chain.cuh).
#include <cuda_bf16.h>

#include <algorithm>

#include "digits.cuh"
#include "digits_chain.cuh"

namespace ctm {

namespace {

// ------------------------------------------------------------- splitting
struct SplitSide {
  const double* x;
  Group R;         // rows: R.m[].s0 is this operand's stride
  Group K;
  int k_is_s1;     // the contracted group's stride of this operand is s1 (second operand)
  int64_t rows;
  int kfast;       // the contracted index has unit stride (else rows are read fastest)
  int* exps;       // rows: the largest exponent field
  bf16* dig;       // [digit][row][Kp]
  uint32_t* cover;
};

struct SplitArgs {
  SplitSide s[2];
  int64_t K, Kp;
  int rb, kc;            // rows per CTA; Kp
  int64_t blocks0;       // CTAs of side 0
};

// Loads the CTA's rows into shared memory (row stride kc + 1); walks whichever
// index has unit stride across the lanes.
__device__ void load_block(const SplitSide& s, const SplitArgs& a, int64_t r0, double* sx,
                           int64_t* s_ro, int64_t* s_ko) {
  const int tid = threadIdx.x, nth = blockDim.x, lane = tid & 31, warp = tid >> 5;
  const int nwarps = nth >> 5;
  const int nr = int(min(int64_t(a.rb), s.rows - r0)), nk = int(a.K);
  for (int i = tid; i < nr + nk; i += nth) {
    int64_t o0, o1;
    if (i < nr) {
      decode(s.R, r0 + i, o0, o1);
      s_ro[i] = o0;
    } else {
      decode(s.K, i - nr, o0, o1);
      s_ko[i - nr] = s.k_is_s1 ? o1 : o0;
    }
  }
  __syncthreads();
  const int ld = a.kc + 1;
  if (s.kfast) {
    for (int r = warp; r < nr; r += nwarps) {
      const double* xr = s.x + s_ro[r];
#pragma unroll 4
      for (int k = lane; k < nk; k += 32) sx[r * ld + k] = xr[s_ko[k]];
    }
  } else {
    const int rblocks = (nr + 31) / 32;
#pragma unroll 4
    for (int q = warp; q < nk * rblocks; q += nwarps) {
      const int k = q / rblocks, r = (q - k * rblocks) * 32 + lane;
      if (r < nr) sx[r * ld + k] = s.x[s_ro[r] + s_ko[k]];
    }
  }
  __syncthreads();
}

// Largest exponent field of each row of the block.  Four lanes per row.
__device__ void row_exponents(const SplitArgs& a, int nr, int nk, const double* sx, int* s_e) {
  const int ld = a.kc + 1;
  for (int q = threadIdx.x; q < a.rb * 4; q += blockDim.x) {
    const int r = q >> 2;
    int e = 0;
    if (r < nr)
      for (int k = q & 3; k < nk; k += 4) e = max(e, exponent_field(sx[r * ld + k]));
    e = max(e, __shfl_xor_sync(0xffffffffu, e, 1));
    e = max(e, __shfl_xor_sync(0xffffffffu, e, 2));
    if ((q & 3) == 0) s_e[r] = e;
  }
  __syncthreads();
}

__global__ void __launch_bounds__(256) split_digits_kernel(const SplitArgs a) {
  extern __shared__ __align__(16) double sx[];
  __shared__ int64_t s_ro[128], s_ko[256];
  __shared__ int s_e[128];
  const bool second = int64_t(blockIdx.x) >= a.blocks0;
  const SplitSide& s = a.s[second ? 1 : 0];
  const int64_t b = second ? int64_t(blockIdx.x) - a.blocks0 : int64_t(blockIdx.x);
  const int64_t r0 = b * a.rb;
  load_block(s, a, r0, sx, s_ro, s_ko);
  const int nr = int(min(int64_t(a.rb), s.rows - r0)), nk = int(a.K);
  row_exponents(a, nr, nk, sx, s_e);
  for (int r = threadIdx.x; r < nr; r += blockDim.x) s.exps[r0 + r] = s_e[r];
  const int ld = a.kc + 1;
  // 16-byte groups of 8 digits; two lanes cover 32 contiguous bytes of a row
  const int ng = a.kc / 8, ng2 = (ng + 1) / 2;
  const int64_t plane = s.rows * a.Kp;
  for (int q = threadIdx.x; q < ng2 * a.rb * 2; q += blockDim.x) {
    const int pair = q / (a.rb * 2), rest = q - pair * (a.rb * 2);
    const int r = rest >> 1, g = pair * 2 + (rest & 1);
    if (r >= nr || g >= ng) continue;
    double x[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int k = g * 8 + i;
      x[i] = k < nk ? sx[r * ld + k] : 0.0;
    }
    write_digits(x, s_e[r], s.dig + (r0 + r) * a.Kp + g * 8, plane,
                 s.cover + (r0 + r) * cover_stride(a.K) + g);
  }
}

// Rows of more than 256 entries: the warps read along whichever index has unit
// stride.  One contracted mode (kMulti false): 5184 x 5184 by rows, exponents 39 us
// and digits 94 us (147 + 229 us through blocks in shared memory).  Several: their
// offsets are tabled in shared memory, or stepped: 36 and 72 rows of 746496 entries,
// exponents 93 + 97 us and digits 142 + 276 us (555 and 892 us through the blocks).
struct LongRows {
  const double* x;
  Group R, Kg;      // strides in s0
  int64_t rows, K, Kp;
  int64_t kc;       // contracted indices per CTA of the exponent kernels
  int* exps;        // zeroed when kc < K
  bf16* dig;
  uint32_t* cover;
};

__device__ __forceinline__ int64_t k_offset(const LongRows& a, int64_t k) {
  int64_t o0, o1;
  decode(a.Kg, k, o0, o1);
  return o0;
}

__device__ __forceinline__ void put_field(const LongRows& a, int64_t r, int e) {
  if (a.kc < a.K) atomicMax(a.exps + r, e);
  else a.exps[r] = e;
}

// The largest exponent field of x[offset of k], k = k0 + first, + step, .. < k1 (all
// threads of the CTA take part; live: this thread has a row).
template <bool kMulti>
__device__ __forceinline__ int largest_field(const LongRows& a, const double* x, bool live,
                                             int64_t k0, int64_t k1, int first, int step) {
  int e = 0;
  if (!kMulti) {
    const int64_t ks = a.Kg.m[0].s0;
    if (live) {
#pragma unroll 8
      for (int64_t k = k0 + first; k < k1; k += step) e = max(e, exponent_field(x[k * ks]));
    }
  } else {
    constexpr int kTable = 512;
    __shared__ int64_t s_ko[kTable];
    for (int64_t kb = k0; kb < k1; kb += kTable) {
      const int n = int(min(int64_t(kTable), k1 - kb));
      __syncthreads();
      for (int i = threadIdx.x; i < n; i += blockDim.x) s_ko[i] = k_offset(a, kb + i);
      __syncthreads();
      if (live) {
#pragma unroll 8
        for (int i = first; i < n; i += step) e = max(e, exponent_field(x[s_ko[i]]));
      }
    }
  }
  return e;
}

// Contracted index of unit stride: one warp per row.
template <bool kMulti>
__global__ void __launch_bounds__(256) long_exponents_k_kernel(const LongRows a) {
  const int lane = threadIdx.x & 31;
  const int64_t r = blockIdx.x * int64_t(8) + (threadIdx.x >> 5);
  const bool live = r < a.rows;
  int64_t ro = 0, t;
  if (live) decode(a.R, r, ro, t);
  const int64_t k0 = blockIdx.y * a.kc, k1 = min(k0 + a.kc, a.K);
  int e = largest_field<kMulti>(a, a.x + ro, live, k0, k1, lane, 32);
  for (int o = 16; o > 0; o >>= 1) e = max(e, __shfl_xor_sync(0xffffffffu, e, o));
  if (lane == 0 && live) put_field(a, r, e);
}

// Otherwise 32 rows per CTA, its warps share the contracted index.
template <bool kMulti>
__global__ void __launch_bounds__(512) long_exponents_r_kernel(const LongRows a) {
  __shared__ int s_e[16][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t r = blockIdx.x * int64_t(32) + lane;
  const int64_t k0 = blockIdx.y * a.kc, k1 = min(k0 + a.kc, a.K);
  const bool live = r < a.rows;
  int64_t ro = 0, t;
  if (live) decode(a.R, r, ro, t);
  int e = largest_field<kMulti>(a, a.x + ro, live, k0, k1, warp, 16);
  s_e[warp][lane] = e;
  __syncthreads();
  if (warp == 0 && live) {
    for (int w = 1; w < 16; ++w) e = max(e, s_e[w][lane]);
    put_field(a, r, e);
  }
}

// kfast: a warp takes 8 rows x 32 indices, four lanes of eight per row, straight
// from memory.  Else a CTA takes 32 rows x 64 indices through shared memory; two
// lanes write 32 contiguous bytes of a row.
template <bool kfast, bool kMulti>
__global__ void __launch_bounds__(256) long_split_kernel(const LongRows a) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t plane = a.rows * a.Kp;
  if (kfast) {
    const int64_t kblocks = (a.Kp + 31) / 32;
    const int64_t w = blockIdx.x * int64_t(8) + warp;
    // several modes: neighbouring warps take neighbouring rows, whose runs of the
    // innermost mode often share their sectors
    const int64_t rblocks = (a.rows + 7) / 8;
    const int64_t rb = kMulti ? w % rblocks : w / kblocks;
    const int64_t kb = kMulti ? w / rblocks : w % kblocks;
    const int64_t r = rb * 8 + (lane >> 2), k0 = kb * 32 + (lane & 3) * 8;
    if (r >= a.rows || k0 >= a.Kp) return;
    int64_t ro, t;
    decode(a.R, r, ro, t);
    double x[8];
    if (!kMulti) {
      const int64_t ks = a.Kg.m[0].s0;
#pragma unroll
      for (int i = 0; i < 8; ++i) x[i] = k0 + i < a.K ? a.x[ro + (k0 + i) * ks] : 0.0;
    } else {
      // offsets within the innermost mode are steps; a new decode where it wraps
      const Mode in = a.Kg.m[a.Kg.n - 1];
      const uint32_t ext = uint32_t(in.ext);
      const int64_t st = in.s0;
      uint32_t left = 0;
      int64_t off = 0;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (left == 0 && k0 + i < a.K) {
          off = ro + k_offset(a, k0 + i);
          left = ext - uint32_t(k0 + i) % ext;
        }
        x[i] = k0 + i < a.K ? a.x[off] : 0.0;
        off += st;
        --left;
      }
    }
    write_digits(x, a.exps[r], a.dig + r * a.Kp + k0, plane,
                 a.cover + r * cover_stride(a.K) + k0 / 8);
  } else {
    __shared__ double sx[32][65];
    __shared__ int64_t s_ko[64];
    const int64_t rblocks = (a.rows + 31) / 32;
    const int64_t r0 = int64_t(blockIdx.x) % rblocks * 32, kb = int64_t(blockIdx.x) / rblocks * 64;
    if (kMulti) {
      if (threadIdx.x < 64 && kb + threadIdx.x < a.K)
        s_ko[threadIdx.x] = k_offset(a, kb + threadIdx.x);
      __syncthreads();
    }
    {
      const int64_t r = r0 + lane;
      int64_t ro = 0, t;
      if (r < a.rows) decode(a.R, r, ro, t);
      const int64_t ks = kMulti ? 0 : a.Kg.m[0].s0;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int64_t k = kb + warp + 8 * i;
        const bool ok = r < a.rows && k < a.K;
        sx[lane][warp + 8 * i] = ok ? a.x[ro + (kMulti ? s_ko[warp + 8 * i] : k * ks)] : 0.0;
      }
    }
    __syncthreads();
    const int rl = (warp & 1) * 16 + (lane >> 1), g = (warp >> 1) * 2 + (lane & 1);
    const int64_t r = r0 + rl, k0 = kb + g * 8;
    if (r >= a.rows || k0 >= a.Kp) return;
    double x[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = sx[rl][g * 8 + i];
    write_digits(x, a.exps[r], a.dig + r * a.Kp + k0, plane,
                 a.cover + r * cover_stride(a.K) + k0 / 8);
  }
}

// ------------------------------------------------------------- products
constexpr int kM = 128;             // rows per tile (tensor-memory lanes)
constexpr int kStageK = 32;         // contracted indices per stage (64-byte rows)
constexpr int kStages = 2;
constexpr int kChunkStages = 6;     // stages between two reads of the accumulators
constexpr int kDThreads = 384;      // producer, MMA issuer, two idle warps, eight epilogue warps
constexpr uint32_t kABytes = kDigits * kM * kStageK * 2;

struct DigitArgs {
  int64_t M, N, K;      // rows, columns, contracted
  Group GM, GN;         // output strides of rows and columns (m[].s1)
  const int* ea;
  const int* eb;
  double* C;            // C, or the split-K partials
  int64_t ldm, ldn;     // partial sums: strides of rows and columns (split > 1)
  int64_t part_stride;
  double alpha, beta;
  int m_tiles, n_tiles, tiles, n_fast;
  int split;            // K ranges
  int stages_per_split; // multiple of kChunkStages
  int stages_total;
  int* status;
  uint32_t* marks;      // split 1: word 2 * column tile + half of row m at word * M + m
  int* queued;          // ChainQueue::count, or null
  int guard;            // small outputs are marked too
};

// round_96 as a call: inlined once per column it made 30 KB of code that every tile's
// epilogue fetched anew (41 x 3 tiles of K = 144, one a CTA: 20.5 us, 19.5 as a call).
static __device__ __noinline__ double rounded(long long hi, uint32_t lo, int e) {
  return round_96(hi, lo, e);
}

// Tiles of 128 rows x ntile columns, persistent over blockIdx.x.  The eight
// accumulators of a tile fill tensor memory (8 x 64 columns).  One stage holds
// 32 contracted indices of all eight digits of both operands (64 + 32 KB, two
// stages), loaded by two TMA copies; for digit i of A the digits j = 0..7-i of
// B are adjacent rows of one operand whose products fall into adjacent
// accumulators, so 12 MMAs of up to 256 columns do the 36 products of 16
// indices.  Warp 0 lane 0 loads, warp 1 lane 0 issues, warps 4-11 read tensor
// memory (warp w: lanes 32 (w % 4).., half (w - 4) / 4 of the columns).
template <int kHalf>
__global__ void __launch_bounds__(kDThreads, 1)
    digit_gemm_kernel(const __grid_constant__ CUtensorMap tA,
                      const __grid_constant__ CUtensorMap tB,
                      const DigitArgs p) {
  extern __shared__ uint8_t dyn_smem[];
  uint8_t* base = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(dyn_smem) + 1023) & ~uintptr_t(1023));
  constexpr int NT = 2 * kHalf;
  constexpr uint32_t b_bytes = uint32_t(kDigits) * NT * kStageK * 2;
  constexpr uint32_t stage_bytes = kABytes + b_bytes;
  uint64_t* full = reinterpret_cast<uint64_t*>(base + size_t(kStages) * stage_bytes);
  uint64_t* empty = full + kStages;
  uint64_t* tfull = empty + kStages;
  uint64_t* tempty = tfull + 1;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(tempty + 1);
  __shared__ int s_fail, s_epi_fail[2];
  __shared__ int64_t s_cn[2][NT];
  __shared__ int s_eb[2][NT];
  __shared__ uint32_t s_bad[2][2];  // columns without digits, by half

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    if (blockIdx.x == 0 && p.queued != nullptr) *p.queued = 0;
    s_fail = 0;
    s_epi_fail[0] = s_epi_fail[1] = 0;
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(tfull, 1);
    mbar_init(tempty, 8);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
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
  const int work = p.tiles * p.split;
  // item -> tile origin and stage range
  auto item = [&](int it, int& m0, int& n0, int& s0, int& s1, int& sp) {
    sp = it / p.tiles;
    const int t = it - sp * p.tiles;
    int mt, nt;
    if (p.n_fast) {
      mt = t / p.n_tiles;
      nt = t - mt * p.n_tiles;
    } else {
      nt = t / p.m_tiles;
      mt = t - nt * p.m_tiles;
    }
    m0 = mt * kM;
    n0 = nt * NT;
    s0 = sp * p.stages_per_split;
    s1 = min(p.stages_total, s0 + p.stages_per_split);
  };
  int issued = 0;
  if (threadIdx.x == 0) {
    // ---------------- TMA producer
    int g = 0;
    bool fail = false;
    for (int it = blockIdx.x; it < work && !fail; it += gridDim.x) {
      int m0, n0, s0, s1, sp;
      item(it, m0, n0, s0, s1, sp);
      for (int s = s0; s < s1; ++s, ++g) {
        const int st = g % kStages;
        if (!mbar_wait_spin(&empty[st], ((g / kStages) & 1) ^ 1)) {
          atomicOr(&s_fail, 1);
          fail = true;
          break;
        }
        uint8_t* sm = base + size_t(st) * stage_bytes;
        mbar_expect_tx(&full[st], stage_bytes);
        tma_load_3d(sm, &tA, s * kStageK, m0, 0, &full[st]);
        tma_load_3d(sm + kABytes, &tB, s * kStageK, n0, 0, &full[st]);
        issued = g + 1;
      }
    }
  } else if (threadIdx.x == 32) {
    // ---------------- MMA issuer
    int g = 0, chunk = 0;
    bool fail = false;
    for (int it = blockIdx.x; it < work && !fail; it += gridDim.x) {
      int m0, n0, s0, s1, sp;
      item(it, m0, n0, s0, s1, sp);
      for (int s = s0; s < s1; ++s, ++g) {
        const bool first = (s - s0) % kChunkStages == 0;
        if (first && !mbar_wait_spin(tempty, (chunk & 1) ^ 1)) {
          atomicOr(&s_fail, 1);
          fail = true;
          break;
        }
        const int st = g % kStages;
        if (!mbar_wait_spin(&full[st], (g / kStages) & 1)) {
          atomicOr(&s_fail, 1);
          fail = true;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint64_t da = smem_desc(base + size_t(st) * stage_bytes, kStageK);
        const uint64_t db = smem_desc(base + size_t(st) * stage_bytes + kABytes, kStageK);
        const int steps = p.K - int64_t(s) * kStageK > 16 ? 2 : 1;
        for (int kk = 0; kk < steps; ++kk) {
#pragma unroll
          for (int i = 0; i < kDigits; ++i) {
            constexpr int kGroup = 256 / NT;  // digits of B per MMA
#pragma unroll
            for (int j = 0; j < kDigits - i; j += kGroup) {
              const int cnt = min(kGroup, kDigits - i - j);
              mma_bf16(tmem + uint32_t((i + j) * NT),
                       da + uint64_t((i * kM * kStageK * 2 + kk * 32) >> 4),
                       db + uint64_t((j * NT * kStageK * 2 + kk * 32) >> 4),
                       idesc_bf16(kM, cnt * NT), (first && kk == 0 && i == 0) ? 0u : 1u);
            }
          }
        }
        mma_commit(&empty[st]);
        if ((s - s0) % kChunkStages == kChunkStages - 1 || s == s1 - 1) {
          mma_commit(tfull);
          ++chunk;
        }
      }
    }
  } else if (warp >= 4) {
    // ---------------- epilogue
    const int etid = threadIdx.x - 128;
    const int lane_base = (warp & 3) * 32, half = (warp - 4) >> 2;
    const uint32_t trow = tmem + (uint32_t(lane_base) << 16) + uint32_t(half * kHalf);
    int chunk = 0, par = 0;
    for (int it = blockIdx.x; it < work; it += gridDim.x, par ^= 1) {
      int m0, n0, s0, s1, sp;
      item(it, m0, n0, s0, s1, sp);
      if (warp < 6) {  // warp 4 + h: columns of half h
        const int64_t n = int64_t(n0) + (warp - 4) * kHalf + lane;
        const bool bad = lane < kHalf && n < p.N && p.eb[n] == kBadField;
        const uint32_t mask = __ballot_sync(0xffffffffu, bad);
        if (lane == 0) s_bad[par][warp - 4] = mask;
      }
      for (int c = etid; c < NT; c += 256) {
        const int64_t n = int64_t(n0) + c;
        int64_t off = -1, t;
        int e = 0;
        if (n < p.N) {
          if (p.split > 1) off = n * p.ldn;
          else decode(p.GN, n, t, off);
          e = p.eb[n];
        }
        s_cn[par][c] = off;
        s_eb[par][c] = e;
      }
      const int64_t row = int64_t(m0) + lane_base + lane;
      int64_t ro = 0, t0;
      int er = 0;
      if (row < p.M) {
        if (p.split > 1) ro = row * p.ldm + sp * p.part_stride;
        else decode(p.GM, row, t0, ro);
        er = p.ea[row];
      }
      long long hi[kHalf];
      uint32_t lo[kHalf];
#pragma unroll
      for (int j = 0; j < kHalf; ++j) {
        hi[j] = 0;
        lo[j] = 0u;
      }
      const int chunks = (s1 - s0 + kChunkStages - 1) / kChunkStages;
      bool lost = false;
      for (int ch = 0; ch < chunks; ++ch, ++chunk) {
        bool ok = mbar_wait(tfull, chunk & 1);
        __syncwarp();
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) {
          lost = true;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int c = 0; c < kHalf; c += 4) {
          float f[kDigits][4];
#pragma unroll
          for (int s = 0; s < kDigits; ++s) tmem_ld4(trow + uint32_t(s * NT + c), f[s]);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          // the loaded registers are valid only after the wait
#pragma unroll
          for (int s = 0; s < kDigits; ++s)
#pragma unroll
            for (int j = 0; j < 4; ++j) asm volatile("" : "+f"(f[s][j]));
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float v[kDigits] = {f[0][j], f[1][j], f[2][j], f[3][j],
                                      f[4][j], f[5][j], f[6][j], f[7][j]};
            add_groups(v, hi[c + j], lo[c + j]);
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        if (lane == 0) mbar_arrive(tempty);
      }
      // all eight warps arrive and decide together (a flag per parity: a warp
      // already at the next item cannot change this one's)
      if (lost && lane == 0) s_epi_fail[par] = 1;
      asm volatile("bar.sync 1, 256;" ::: "memory");
      if (s_epi_fail[par]) {
        if (etid == 0) atomicOr(&s_fail, 1);
        break;
      }
      if (row < p.M) {
        double* out = p.C + ro;
        // marked: the chain's, stored after the products
        uint32_t mark = s_bad[par][half];
        if (er == kBadField) mark = low_bits(min(kHalf, int(p.N) - n0 - half * kHalf));
#pragma unroll
        for (int c = 0; c < kHalf; ++c) {
          const int64_t off = s_cn[par][half * kHalf + c];
          const int e = s_eb[par][half * kHalf + c];
          if (off < 0) continue;
          // units of 2^-68 of the scales (digit s of the product: 2^(-12 - 8 s))
          constexpr long long kSmall = 1ll << (68 - kCoverBits - 32);
          if (p.guard && hi[c] < kSmall && hi[c] >= -kSmall) mark |= 1u << c;
          double v = rounded(hi[c], lo[c], row_exponent(er) + row_exponent(e) - 2 * 1023 - 68);
          if (p.split == 1 && !(p.alpha == 1.0 && p.beta == 0.0)) {
            v *= p.alpha;
            if (p.beta != 0.0) v = (mark >> c & 1u) ? out[off] : fma(p.beta, out[off], v);
          }
          out[off] = v;
        }
        if (p.split == 1) p.marks[int64_t(n0 / kHalf + half) * p.M + row] = mark;
      }
    }
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  // on failure: let in-flight copies land before the CTA's memory goes away
  if (threadIdx.x == 0 && s_fail) {
    for (int i = max(0, issued - kStages); i < issued; ++i)
      (void)mbar_wait(&full[i % kStages], (i / kStages) & 1);
    atomicOr(p.status, 2);
  }
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u)
                 : "memory");
  }
}

// Sums the K ranges' partial outputs (in the order of gett_splitk_reduce) into C, eight
// rows by one word a CTA.  kChain: the marked ones follow at once; else they are left to
// chain_outputs_kernel.
struct ReduceArgs {
  GettArgs<double> p;   // part and splitk set
  const int* ea;        // of the rows and columns of p
  const int* eb;
  ChainOutputs out;
};

template <bool kChain>
__global__ void __launch_bounds__(256) digit_reduce_kernel(const __grid_constant__ ReduceArgs a) {
  __shared__ uint32_t list[256];
  __shared__ int s_count;
  const GettArgs<double>& p = a.p;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t words = (p.Nt + 31) / 32, total = (p.Mt + 7) / 8 * words, plane = p.Mt * p.Nt;
  for (int64_t idx = blockIdx.x; idx < total; idx += gridDim.x) {
    const int64_t r0 = idx / words * 8, w = idx - r0 / 8 * words, m = r0 + warp, n = w * 32 + lane;
    if (kChain) {
      if (threadIdx.x == 0) s_count = 0;
      __syncthreads();
    }
    bool mark = false, small = false;
    double sum = 0.0;
    if (m < p.Mt && n < p.Nt) {
      const double* pt = p.part + m * p.Nt + n;
      double s0 = 0.0, s1 = 0.0, m0 = 0.0, m1 = 0.0;
      int t = 0;
      for (; t + 1 < p.splitk; t += 2) {
        const double v0 = pt[t * plane], v1 = pt[(t + 1) * plane];
        s0 += v0;
        s1 += v1;
        m0 += fabs(v0);
        m1 += fabs(v1);
      }
      if (t < p.splitk) {
        s0 += pt[t * plane];
        m0 += fabs(pt[t * plane]);
      }
      sum = s0 + s1;
      const int ea = a.ea[m], eb = a.eb[n];
      mark = ea == kBadField || eb == kBadField;
      // (|sums| with a field below the scales' by kCoverBits)
      small = !mark && !p.beside_scales &&
              exponent_field(m0 + m1) < row_exponent(ea) + row_exponent(eb) - 1023 - kCoverBits;
    }
    const Cover& cv = a.out.cover;
    if (kChain) {  // a warp each
      for (uint32_t left = __ballot_sync(0xffffffffu, small); left != 0u; left &= left - 1u) {
        const int l = __ffs(int(left)) - 1;
        const bool ok =
            covered_by<1>(cv.row + m * cv.stride, cv.col + (w * 32 + l) * cv.stride, cv.groups);
        if (lane == l) mark = !ok;
      }
    } else {  // long rows: the CTA each
      if (threadIdx.x == 0) s_count = 0;
      __syncthreads();
      if (small) list[atomicAdd(&s_count, 1)] = threadIdx.x;
      __syncthreads();
      for (int i = 0; i < s_count; ++i) {
        const uint32_t t = list[i];
        const bool ok = covered_by<8>(cv.row + (r0 + (t >> 5)) * cv.stride,
                                      cv.col + (w * 32 + (t & 31u)) * cv.stride, cv.groups);
        if (threadIdx.x == t) mark = !ok;
      }
      __syncthreads();
    }
    if (m < p.Mt && n < p.Nt) {
      if (!mark) {
        int64_t am, cm, bn, cn;
        decode(p.M, m, am, cm);
        decode(p.N, n, bn, cn);
        double* c = p.C + cm + cn;
        const double v = p.alpha * sum;
        *c = p.beta != 0.0 ? fma(p.beta, *c, v) : v;
      }
    }
    if (kChain) {
      if (mark) list[atomicAdd(&s_count, 1)] = threadIdx.x;
      __syncthreads();
      auto where = [&](int, int64_t& r, int64_t& word) {
        r = r0;
        word = w;
      };
      chain_listed<256>(a.out, list, s_count, 0, a.out.K, where);
      __syncthreads();
    } else {
      const uint32_t word = __ballot_sync(0xffffffffu, mark);
      if (lane == 0 && m < p.Mt) a.out.marks.word[w * p.Mt + m] = word;
    }
  }
}

// Contracted indices from which the marked outputs of a product in K ranges are summed in
// ranges too (746496 terms of one output take a CTA 190 us).
constexpr int64_t kLongChain = 16384;

// The marked outputs, over blockIdx.y's range of the contracted index where part is set.
// (At the end of digit_gemm_kernel itself this code cost 64 us of 405 at 5184 x 5184 x 144
// with nothing marked; as a kernel 4 us.)
__global__ void __launch_bounds__(256) chain_outputs_kernel(
    const __grid_constant__ ChainOutputs a, int64_t kchunk) {
  __shared__ __align__(16) uint8_t buf[kChainSmem];
  const int64_t rblocks = (a.marks.rows + kCRows - 1) / kCRows, items = rblocks * a.marks.words;
  const int mine = int((items - blockIdx.x + gridDim.x - 1) / gridDim.x);
  auto where = [&](int b, int64_t& r, int64_t& w) {
    const uint32_t it = blockIdx.x + uint32_t(b) * gridDim.x, rb = uint32_t(rblocks);  // < 2^32
    const uint32_t q = it / rb;
    w = q;
    r = int64_t(it - q * rb) * kCRows;
  };
  const int64_t k0 = blockIdx.y * kchunk;
  chain_marked<256>(a, mine, where, buf, sizeof(buf), k0, min(a.K, k0 + kchunk));
}

// The queued outputs.  (Where the kernel that finds them forms them too, the CTA that has
// a row or column of many takes as long as all others together.)
__global__ void __launch_bounds__(256) chain_queue_kernel(const __grid_constant__ ChainOutputs a) {
  const int count = min(*a.queue.count, a.queue.cap);
  // neighbouring outputs go to different SMs
  const int id = ((threadIdx.x >> 5) * gridDim.x + blockIdx.x) * 32 + (threadIdx.x & 31);
  chain_each(a, count, id, gridDim.x * 256, 0, a.K, [&](int o, int64_t& r, int64_t& n) {
    const uint2 e = a.queue.entry[o];
    r = e.x;
    n = e.y;
  });
}

// The ranges' sums of the marked outputs into C.
__global__ void __launch_bounds__(256) chain_sum_kernel(ChainOutputs a, int ranges) {
  const double* part = a.part;
  a.part = nullptr;
  const int64_t total = a.marks.rows * a.marks.words;
  for (int64_t idx = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; idx < total;
       idx += int64_t(gridDim.x) * blockDim.x) {
    const int64_t w = idx / a.marks.rows, r = idx - w * a.marks.rows;
    for (uint32_t left = a.marks.word[idx]; left != 0u; left &= left - 1u) {
      const int64_t n = w * a.marks.per + __ffs(int(left)) - 1;
      double v = 0.0;
      for (int t = 0; t < ranges; ++t) v += part[(t * a.marks.rows + r) * a.columns + n];
      chain_store(a, r, n, v);
    }
  }
}

void digit_map(CUtensorMap* map, const bf16* dig, int64_t rows, int64_t Kp, uint32_t box_rows) {
  const cuuint64_t dims[3] = {cuuint64_t(Kp), cuuint64_t(rows), cuuint64_t(kDigits)};
  const cuuint64_t strides[2] = {cuuint64_t(Kp) * 2, cuuint64_t(rows) * cuuint64_t(Kp) * 2};
  const cuuint32_t box[3] = {uint32_t(kStageK), box_rows, uint32_t(kDigits)};
  const cuuint32_t estr[3] = {1, 1, 1};
  const CUresult res = encode_tiled()(
      map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<bf16*>(dig), dims, strides, box, estr,
      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B,
      CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  CTM_REQUIRE(res == CUDA_SUCCESS, CTM_ERR_CUDA,
              "cuTensorMapEncodeTiled failed with code " + std::to_string(int(res)));
}

// Cycles of one stage of a tile of ntile columns: 36 products of 32 indices
// at 4096 multiply-adds per cycle, or its bytes at about 45 per cycle and SM.
double stage_cycles(int ntile) {
  return std::max(36.0 * ntile, (65536.0 + 512.0 * ntile) / 45.0);
}

int best_ntile(int64_t n) {
  int best = 64;
  double least = 1e300;
  for (int t : {64, 48, 32, 16}) {
    const double cost = double((n + t - 1) / t) * stage_cycles(t);
    if (cost < least) {
      least = cost;
      best = t;
    }
  }
  return best;
}

Digits alloc_digits(Ctx& c, int64_t rows, int64_t K) {
  Digits d;
  d.rows = rows;
  d.K = K;
  d.dig = c.alloc<bf16>(size_t(kDigits) * rows * ((K + 7) / 8 * 8));
  d.exps = c.alloc<int>(size_t(rows));
  d.cover = c.alloc<uint32_t>(size_t(rows) * size_t(cover_stride(K)));
  return d;
}

// The contracted modes as one operand sees them (strides in s0): neighbours joined
// where they are contiguous in it.
Group joined(const Group& k, bool second) {
  Group g{};
  for (int i = 0; i < k.n; ++i) {
    const Mode m{k.m[i].ext, second ? k.m[i].s1 : k.m[i].s0, 0};
    if (g.n > 0 && g.m[g.n - 1].s0 == m.ext * m.s0) {
      g.m[g.n - 1].ext *= m.ext;
      g.m[g.n - 1].s0 = m.s0;
    } else {
      g.m[g.n++] = m;
    }
  }
  return g;
}

// Exponents and digits of those of the two sides that are wanted.
void split_sides(Ctx& c, const SplitSide* side, int want0, int want1, int64_t K, int64_t Kp) {
  if (c.sizing()) return;
  int want[2] = {want0, want1};
  for (int i = 0; i < 2; ++i) {
    const SplitSide& s = side[i];
    if (!want[i] || K <= 256) continue;
    want[i] = 0;
    // the modes of this operand alone, joined where they are contiguous in it
    LongRows a{s.x, s.R, joined(s.K, s.k_is_s1 != 0), s.rows, K, Kp, K, s.exps, s.dig, s.cover};
    const bool multi = a.Kg.n > 1;
    // enough CTAs of the exponent kernels to cover the SMs twice
    const int64_t rb = s.kfast ? 8 : 32, rblocks = (s.rows + rb - 1) / rb;
    const int64_t least = s.kfast ? 512 : 256, want_ctas = 2 * sm_count_linalg();
    if (rblocks < want_ctas) a.kc = std::min(K, std::max(least, K * rblocks / want_ctas));
    const int64_t chunks = (K + a.kc - 1) / a.kc;
    CTM_REQUIRE(chunks <= 65535, CTM_ERR_UNSUPPORTED, "einsum: grid too large");
    if (chunks > 1)
      CTM_CUDA(cudaMemsetAsync(s.exps, 0, sizeof(int) * size_t(s.rows), c.stream));
    {
      KernelTimer kt(c.stream, "long_exponents_kernel", kUnitByte, 8.0 * double(s.rows) * K);
      const dim3 grid(unsigned(rblocks), unsigned(chunks), 1);
      if (s.kfast) {
        if (multi) long_exponents_k_kernel<true><<<grid, 256, 0, c.stream>>>(a);
        else long_exponents_k_kernel<false><<<grid, 256, 0, c.stream>>>(a);
      } else {
        if (multi) long_exponents_r_kernel<true><<<grid, 512, 0, c.stream>>>(a);
        else long_exponents_r_kernel<false><<<grid, 512, 0, c.stream>>>(a);
      }
      CTM_LAUNCH_CHECK();
    }
    KernelTimer kt(c.stream, "long_split_kernel", kUnitByte, 24.0 * double(s.rows) * K);
    const int64_t ctas = s.kfast ? ((s.rows + 7) / 8 * ((Kp + 31) / 32) + 7) / 8
                                 : (s.rows + 31) / 32 * ((Kp + 63) / 64);
    CTM_REQUIRE(ctas < (int64_t(1) << 31), CTM_ERR_UNSUPPORTED, "einsum: grid too large");
    if (s.kfast) {
      if (multi) long_split_kernel<true, true><<<unsigned(ctas), 256, 0, c.stream>>>(a);
      else long_split_kernel<true, false><<<unsigned(ctas), 256, 0, c.stream>>>(a);
    } else {
      if (multi) long_split_kernel<false, true><<<unsigned(ctas), 256, 0, c.stream>>>(a);
      else long_split_kernel<false, false><<<unsigned(ctas), 256, 0, c.stream>>>(a);
    }
    CTM_LAUNCH_CHECK();
  }
  if (!want[0] && !want[1]) return;
  SplitArgs sa{};
  sa.s[0] = side[0];
  sa.s[1] = side[1];
  sa.K = K;
  sa.Kp = Kp;
  sa.kc = int(Kp);
  sa.rb = sa.kc <= 64 ? 128 : sa.kc <= 128 ? 64 : 32;
  auto blocks_of = [&](int i) {
    return want[i] ? (side[i].rows + sa.rb - 1) / sa.rb : int64_t(0);
  };
  sa.blocks0 = blocks_of(0);
  const int64_t blocks = sa.blocks0 + blocks_of(1);
  const size_t ssm = size_t(sa.rb) * (sa.kc + 1) * sizeof(double);
  const double entries = ((want[0] ? side[0].rows : 0) + (want[1] ? side[1].rows : 0)) * double(K);
  CTM_CUDA(cudaFuncSetAttribute(split_digits_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(ssm)));
  KernelTimer kt(c.stream, "split_digits_kernel", kUnitByte, 24.0 * entries);
  split_digits_kernel<<<unsigned(blocks), 256, ssm, c.stream>>>(sa);
  CTM_LAUNCH_CHECK();
}

bool unit_stride(const Group& g, bool second) {
  return g.n > 0 && (second ? g.m[g.n - 1].s1 : g.m[g.n - 1].s0) == 1;
}

}  // namespace

// From about 2e7 multiply-adds on the digit form is the faster one, whole calls: 256^3
// takes 49 us in the FP64 GETT, 272^3 72 us in digits and 68 to 80 in the GETT, 400^3
// (6.4e7) 78 against 200; 5184 x 5184 x 144 takes 0.33 ms against 11 ms.
bool digits_pay(int64_t rows, int64_t columns, int64_t K) {
  return double(rows) * double(columns) * double(K) >= 2.0e7 && K >= 16 &&
         std::min(rows, columns) >= 16;
}

bool digits_pay(const GettArgs<double>& p) {
  return p.bext == 1 && digits_pay(p.Mt, p.Nt, p.Kt);
}

Digits digit_rows(Ctx& c, const View& x, int row_dim) {
  CTM_REQUIRE(x.nd == 2, CTM_ERR_INVALID, "digit_rows: expects a 2-D view");
  const int kd = 1 - row_dim;
  Digits d = alloc_digits(c, x.shape[row_dim], x.shape[kd]);
  SplitSide s{};
  s.x = x.p;
  s.R.n = 1;
  s.R.m[0] = Mode{x.shape[row_dim], x.stride[row_dim], 0};
  s.K.n = 1;
  s.K.m[0] = Mode{x.shape[kd], x.stride[kd], 0};
  s.rows = d.rows;
  s.kfast = x.stride[kd] == 1 && x.stride[row_dim] != 1 ? 1 : 0;
  s.exps = d.exps;
  s.dig = d.dig;
  s.cover = d.cover;
  const SplitSide side[2] = {s, s};
  split_sides(c, side, 1, 0, d.K, (d.K + 7) / 8 * 8);
  return d;
}

Digits operand_digits(Ctx& c, const GettArgs<double>& p, bool first) {
  const Digits d = alloc_digits(c, first ? p.Mt : p.Nt, p.Kt);
  SplitSide s{};
  s.x = first ? p.A : p.B;
  s.R = first ? p.M : p.N;
  s.K = p.K;
  s.k_is_s1 = first ? 0 : 1;
  s.rows = d.rows;
  s.kfast = unit_stride(p.K, !first) && !unit_stride(s.R, false) ? 1 : 0;
  s.exps = d.exps;
  s.dig = d.dig;
  s.cover = d.cover;
  const SplitSide side[2] = {s, s};
  split_sides(c, side, 1, 0, d.K, (d.K + 7) / 8 * 8);
  return d;
}

namespace {

// The digits take twice their operand's bytes.  Beyond this many bytes for one operand
// the contraction is done in parts, so that the workspace of any size grows by two
// gigabytes at most (16384 x 16384 x 272 in five parts: each still fills the SMs, and
// the small operand's digits are formed again in under 0.1 of a part's time).
constexpr double kMaxDigitBytes = 1e9;

// p as two contractions over halves of the outermost mode of its rows (0), columns (1)
// or contracted indices (2); the second half of the latter adds to the first's result.
bool halves(const GettArgs<double>& p, int which, GettArgs<double>& lo, GettArgs<double>& hi) {
  lo = hi = p;
  const Group& g = which == 0 ? p.M : which == 1 ? p.N : p.K;
  if (g.n == 0 || g.m[0].ext < 2) return false;
  const Mode m = g.m[0];
  const int64_t e1 = m.ext / 2, off0 = e1 * m.s0, off1 = e1 * m.s1;
  auto cut = [&](GettArgs<double>& q, int64_t ext) {
    Group& h = which == 0 ? q.M : which == 1 ? q.N : q.K;
    int64_t& total = which == 0 ? q.Mt : which == 1 ? q.Nt : q.Kt;
    total = total / m.ext * ext;
    h.m[0].ext = ext;
    if (ext == 1) {  // no modes of one entry
      for (int i = 0; i + 1 < h.n; ++i) h.m[i] = h.m[i + 1];
      --h.n;
    }
  };
  cut(lo, e1);
  cut(hi, m.ext - e1);
  if (which == 0) {
    hi.A += off0;
    hi.C += off1;
  } else if (which == 1) {
    hi.B += off0;
    hi.C += off1;
  } else {
    hi.A += off0;
    hi.B += off1;
    hi.beta = 1.0;
  }
  return true;
}

}  // namespace

void digit_contract(Ctx& c, const GettArgs<double>& p, const Digits* pre_a, const Digits* pre_b) {
  bool stream_swap = false;
  if (pre_a == nullptr && pre_b == nullptr) {
    if (stream_fits(p, stream_swap)) {
      stream_contract(c, p, stream_swap);
      return;
    }
    const int64_t most = std::max(p.Mt, p.Nt);
    GettArgs<double> lo, hi;
    if (16.0 * double(most) * double(p.Kt) > kMaxDigitBytes &&
        ((most > 512 && halves(p, p.Mt >= p.Nt ? 0 : 1, lo, hi)) || halves(p, 2, lo, hi))) {
      digit_contract(c, lo);
      digit_contract(c, hi);
      return;
    }
  }
  const int64_t K = p.Kt, Kp = (K + 7) / 8 * 8;
  const int sms = sm_count_linalg();
  // which operand's rows lie on the tensor-memory lanes: fewer waves of tiles,
  // and when equal the one whose rows are contiguous in C (a warp stores one
  // column of 32 rows)
  auto waves = [&](int64_t m, int64_t n) {
    const int nt = best_ntile(n);
    const int64_t tiles = (m + kM - 1) / kM * ((n + nt - 1) / nt);
    return double((tiles + sms - 1) / sms) * stage_cycles(nt);
  };
  const double w0 = waves(p.Mt, p.Nt), w1 = waves(p.Nt, p.Mt);
  const bool swap = w1 < 0.98 * w0 || (w1 <= 1.02 * w0 && unit_stride(p.M, true) < unit_stride(p.N, true));
  const int64_t M = swap ? p.Nt : p.Mt, N = swap ? p.Mt : p.Nt;
  const int nt = best_ntile(N);
  Scope scope(c);
  const Digits* pre_m = swap ? pre_b : pre_a;
  const Digits* pre_n = swap ? pre_a : pre_b;
  const bool ready_a = pre_m != nullptr, ready_b = pre_n != nullptr;
  const Digits da = ready_a ? *pre_m : alloc_digits(c, M, K);
  const Digits db = ready_b ? *pre_n : alloc_digits(c, N, K);
  const int64_t m_tiles = (M + kM - 1) / kM, n_tiles = (N + nt - 1) / nt;
  const int64_t tiles = m_tiles * n_tiles;
  const int64_t stages = (K + kStageK - 1) / kStageK;
  // K ranges when the tiles leave most SMs idle; at least one read of the
  // accumulators' worth of stages each
  int64_t split = 1;
  if (tiles * 2 <= sms) split = std::min<int64_t>(sms / tiles, stages / kChunkStages);
  split = std::max<int64_t>(split, 1);
  int64_t per = (stages + split - 1) / split;
  per = (per + kChunkStages - 1) / kChunkStages * kChunkStages;
  split = (stages + per - 1) / per;
  double* part = split > 1 ? c.alloc<double>(size_t(split) * p.Mt * p.Nt) : nullptr;
  Marks marks{};
  marks.rows = split > 1 ? p.Mt : M;
  marks.per = split > 1 ? 32 : nt / 2;
  marks.words = int(split > 1 ? (p.Nt + 31) / 32 : 2 * n_tiles);
  marks.word = c.alloc<uint32_t>(size_t(marks.rows) * marks.words);
  ChainQueue queue{};
  // Room for half of the outputs, 32 MB at most; a launch less where there are few of them
  // (272 x 272 x 272: 78 us with a queue, 72 formed where they are found; 68 to 80 as FMAs).
  if (split == 1 && M * N > int64_t(1) << 18) {
    queue.cap = int(std::min(int64_t(1) << 22, M * N / 2));
    queue.entry = c.alloc<uint2>(size_t(queue.cap));
    queue.count = c.alloc<int>(1);
  }
  if (c.sizing()) return;
  CTM_REQUIRE(tiles * split < (int64_t(1) << 31), CTM_ERR_UNSUPPORTED, "einsum: grid too large");

  SplitSide side[2];
  auto fill = [&](SplitSide& s, bool first, int64_t rows, const Digits& d) {
    s.x = first ? p.A : p.B;
    s.R = first ? p.M : p.N;
    s.K = p.K;
    s.k_is_s1 = first ? 0 : 1;
    s.rows = rows;
    s.kfast = unit_stride(p.K, !first) && !unit_stride(s.R, false) ? 1 : 0;
    s.exps = d.exps;
    s.dig = d.dig;
    s.cover = d.cover;
  };
  fill(side[0], !swap, M, da);
  fill(side[1], swap, N, db);
  split_sides(c, side, ready_a ? 0 : 1, ready_b ? 0 : 1, K, Kp);

  DigitArgs d{};
  d.M = M;
  d.N = N;
  d.K = K;
  d.GM = swap ? p.N : p.M;
  d.GN = swap ? p.M : p.N;
  d.ea = da.exps;
  d.eb = db.exps;
  d.C = split > 1 ? part : p.C;
  d.ldm = swap ? 1 : p.Nt;
  d.ldn = swap ? p.Nt : 1;
  d.part_stride = p.Mt * p.Nt;
  d.alpha = p.alpha;
  d.beta = p.beta;
  d.m_tiles = int(m_tiles);
  d.n_tiles = int(n_tiles);
  d.tiles = int(tiles);
  d.n_fast = N <= M ? 1 : 0;
  d.split = int(split);
  d.stages_per_split = int(per);
  d.stages_total = int(stages);
  d.status = status_flags(c);
  d.marks = marks.word;
  d.queued = queue.count;
  d.guard = split == 1 && !p.beside_scales ? 1 : 0;
  CUtensorMap tA, tB;
  digit_map(&tA, da.dig, M, Kp, kM);
  digit_map(&tB, db.dig, N, Kp, uint32_t(nt));
  const size_t smem = 1024 + size_t(kStages) * (kABytes + size_t(kDigits) * nt * kStageK * 2) + 128;
  const unsigned grid = unsigned(std::min<int64_t>(tiles * split, sms));
  auto launch = [&](auto kern) {
    CTM_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
    const double flops = 2.0 * double(M) * N * K;
    KernelTimer timer(c.stream, kTagGettF64, flops);
    KernelTimer kt(c.stream, "digit_gemm_kernel", kUnitFlop, flops);
    kern<<<grid, kDThreads, smem, c.stream>>>(tA, tB, d);
  };
  if (nt == 64) launch(digit_gemm_kernel<32>);
  else if (nt == 48) launch(digit_gemm_kernel<24>);
  else if (nt == 32) launch(digit_gemm_kernel<16>);
  else launch(digit_gemm_kernel<8>);
  CTM_LAUNCH_CHECK();
  ChainOutputs out = chain_outputs(p, split == 1 && swap, marks);
  const bool as_d = split == 1 || !swap;  // the outputs' rows are da's
  out.cover = Cover{as_d ? da.cover : db.cover, as_d ? db.cover : da.cover, cover_stride(K),
                    int(Kp / 8), 0, 0, 0};
  const bool ranges = split > 1 && K > kLongChain;
  if (split > 1) {
    ReduceArgs r{p, swap ? db.exps : da.exps, swap ? da.exps : db.exps, out};
    r.p.splitk = int(split);
    r.p.part = part;
    KernelTimer kt(c.stream, "digit_reduce_kernel", kUnitByte, 8.0 * (split + 1.0) * p.Mt * p.Nt);
    const int ctas = grid_for((p.Mt + 7) / 8 * marks.words, 1);
    if (ranges) digit_reduce_kernel<false><<<ctas, 256, 0, c.stream>>>(r);
    else digit_reduce_kernel<true><<<ctas, 256, 0, c.stream>>>(r);
    CTM_LAUNCH_CHECK();
    if (!ranges) return;
    out.part = part;
  }
  if (split > 1 || p.beta != 0.0) out.cover.col = nullptr;  // marks are final
  out.queue = queue;
  const int64_t blocks = (marks.rows + kCRows - 1) / kCRows * marks.words;
  KernelTimer kt(c.stream, "chain_outputs_kernel", kUnitByte, 4.0 * double(marks.rows) * marks.words);
  chain_outputs_kernel<<<dim3(unsigned(std::min<int64_t>(blocks, 4 * sms)),
                              unsigned(ranges ? split : 1)),
                         256, 0, c.stream>>>(out, ranges ? (K + split - 1) / split : K);
  CTM_LAUNCH_CHECK();
  if (queue.cap > 0) {
    chain_queue_kernel<<<unsigned(4 * sms), 256, 0, c.stream>>>(out);
    CTM_LAUNCH_CHECK();
  }
  if (ranges) {
    chain_sum_kernel<<<grid_for(marks.rows * marks.words, 256), 256, 0, c.stream>>>(out, int(split));
    CTM_LAUNCH_CHECK();
  }
}

}  // namespace ctm
