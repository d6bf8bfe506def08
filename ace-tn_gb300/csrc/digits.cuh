// Pieces shared by the FP64 digit-product kernels (digits.cu says how they work).
#pragma once
#include <cuda_bf16.h>

#include "gett.cuh"
#include "tcgen05.cuh"

namespace ctm {

using bf16 = __nv_bfloat16;

constexpr int kDigits = 8;
// A row's scale is kept as the largest exponent field of its entries: |x| <
// 2^(row_exponent(field) - 1023).  Field 2047: a non-finite entry, no digits.
constexpr int kBadField = 2047;
__device__ __forceinline__ int row_exponent(int field) { return max(field, 1) + 1; }

__device__ __forceinline__ int exponent_field(double x) {
  return int((unsigned long long)__double_as_longlong(x) >> 52) & 0x7ff;
}

// Which outputs the digits may form.  Their error is relative to the product sA sB of the
// row's and the column's scales, an FMA chain's to S = sum_k |a_k b_k|: where the large
// entries of a row meet the small ones of a column (or zeros), S is far below sA sB and the
// digits would lose what the chain keeps.  So an output is left to the chain unless
// S >= 2^-8.4 sA sB is known: from |C| <= S, from the K ranges' |sums|, or from classes of
// the entries, large (above 2^-4.2 of the scale) and medium (above 2^-7): one k with two
// large ones, 8 with a large and a medium one or 48 with two medium ones.  With that the
// dropped digit products' deviation, sqrt(K) 2^-62.2 sA sB, is at most sqrt(K) 2^-53.8 S.
// Where no k has two nonzero entries, zero is exact.
// (Environments at D = 6, chi = 144: 1.4 % of the outputs of 5184 x 5184 x 144 are below
// 2^-8, 0.05 to 0.1 % fail the classes; none of the products over 36, 72 or 5184 does.)
//
// A word tells of eight consecutive entries: bits 0-7 large (|top digit| >= 4), 8-15
// medium (>= 1), 16-23 nonzero.
constexpr int kCoverBits = 8;      // |C| >= 2^-8 sA sB: no look at the entries
constexpr int kCoverSum = 48;      // units of 2^-14
constexpr uint32_t kBadCover = 1;  // first word of a row without digits
__host__ __device__ inline int64_t cover_stride(int64_t K) { return (K + 31) / 32 * 4; }

__device__ __forceinline__ bool large_digit(unsigned long long u) {
  return uint32_t(u >> 56) - 125u > 6u;
}

// Digit b (0..7, 0 the least significant) of the biased word w as BF16 bits in
// the upper half: the byte minus 128, exact.
__device__ __forceinline__ uint32_t digit_f32(uint32_t w, int byte) {
  const uint32_t u = __byte_perm(w, 0x4B000000u, 0x7650u | uint32_t(byte));
  return __float_as_uint(__uint_as_float(u) - 8388736.f);  // 2^23 + 128
}

// x 2^62 / 2^(E - 1023) rounded to an integer, biased so that byte j minus 128 is
// the balanced digit of weight 256^j.
__device__ __forceinline__ unsigned long long digit_word(double x, int E) {
  const long long bits = __double_as_longlong(x);
  const int ex = int((unsigned long long)bits >> 52) & 0x7ff;
  const long long mant = (bits & 0xfffffffffffffll) | (ex != 0 ? 0x10000000000000ll : 0ll);
  const int sh = max(ex, 1) - E + 10;  // x = mant 2^(ex - 1075), so mant 2^sh; sh <= 9
  long long t;
  if (sh >= 0) t = mant << sh;
  else if (sh >= -54) t = (mant + (1ll << (-sh - 1))) >> -sh;
  else t = 0;
  if (bits < 0) t = -t;
  return ((unsigned long long)t + 0x0080808080808080ull) ^ 0x8000000000000000ull;
}

// The eight digits of eight consecutive entries: put(d, 16 bytes) for each digit.
template <class Put>
__device__ __forceinline__ void put_digits(const unsigned long long (&u)[8], Put&& put) {
#pragma unroll
  for (int d = 0; d < kDigits; ++d) {  // digit 0 is the top byte
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t f0 = digit_f32(uint32_t(d < 4 ? u[2 * i] >> 32 : u[2 * i]), 3 - (d & 3));
      const uint32_t f1 =
          digit_f32(uint32_t(d < 4 ? u[2 * i + 1] >> 32 : u[2 * i + 1]), 3 - (d & 3));
      w[i] = __byte_perm(f0, f1, 0x7632);
    }
    put(d, make_uint4(w[0], w[1], w[2], w[3]));
  }
}

__device__ __forceinline__ void write_digits(const double (&x)[8], int field, bf16* dst,
                                             int64_t plane, uint32_t* cover) {
  unsigned long long u[8];
  const int E = row_exponent(field);
  uint32_t c = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    u[i] = digit_word(x[i], E);
    c |= (large_digit(u[i]) ? 1u : 0u) << i | (uint32_t(u[i] >> 56) != 128u ? 0x100u : 0u) << i |
         (x[i] != 0.0 ? 0x10000u : 0u) << i;
  }
  *cover = field == kBadField ? kBadCover : c;
  put_digits(u, [&](int d, uint4 w) { *reinterpret_cast<uint4*>(dst + int64_t(d) * plane) = w; });
}

// (hi 2^32 + lo) 2^e rounded to nearest even.
__device__ __forceinline__ double round_96(long long hi, uint32_t lo, int e) {
  const bool neg = hi < 0;
  if (neg) {
    lo = 0u - lo;
    hi = ~hi + (lo == 0u ? 1 : 0);
  }
  if (hi == 0 && lo == 0u) return 0.0;
  const int lz = hi != 0 ? __clzll(hi) : 64 + __clz(int(lo));
  unsigned long long m;
  uint32_t rest = 0u;
  if (lz >= 64) {
    m = (unsigned long long)lo << (lz - 32);
  } else if (lz >= 32) {
    m = ((unsigned long long)hi << lz) | ((unsigned long long)lo << (lz - 32));
  } else {
    m = ((unsigned long long)hi << lz) | (((unsigned long long)lo << lz) >> 32);
    rest = lo << lz;
  }
  unsigned long long r = m >> 11;  // 53 bits
  const uint32_t low = uint32_t(m) & 0x7ffu;
  if (low > 0x400u || (low == 0x400u && (rest != 0u || (r & 1ull) != 0ull))) ++r;
  const int ef = 95 - lz + e + 1023;  // exponent field of the leading bit
  double v;
  if (ef >= 1 && ef < 2046)
    v = __longlong_as_double((long long)(((unsigned long long)(ef - 1) << 52) + r));
  else  // overflow and gradual underflow
    v = scalbn(double((long long)r), ef - 1023 - 52);
  return neg ? -v : v;
}

// The operands themselves, for rows and columns without digits.
struct ChainArgs {
  const double* a;
  const double* b;
  Group FM, FN, FK;     // FM.m[].s0, FN.m[].s0, FK: (first, second operand) strides
  int swapped;          // the row operand is the contraction's second one
};

inline ChainArgs chain_args(const GettArgs<double>& p, bool swap) {
  ChainArgs c{};
  c.a = swap ? p.B : p.A;
  c.b = swap ? p.A : p.B;
  c.FM = swap ? p.N : p.M;
  c.FN = swap ? p.M : p.N;
  c.FK = p.K;
  c.swapped = swap ? 1 : 0;
  return c;
}

// Outputs that the products leave to the FMA chain (digits_chain.cuh): bit b of
// word[w * rows + r] is the one of row r and column w * per + b.  Every word is
// written by the kernel that forms the outputs.  Marked ones are not to be relied on
// (with beta = 0 they may be stored like the others) unless Cover says so.
struct Marks {
  uint32_t* word;
  int64_t rows;
  int words, per;
};

__device__ __forceinline__ uint32_t low_bits(int n) {
  return n >= 32 ? ~0u : n > 0 ? (1u << n) - 1u : 0u;
}

// Whether a candidate's digits may stand: words of rows and columns (null: they may not).
struct Cover {
  const uint32_t* row;
  const uint32_t* col;
  int64_t stride;
  int groups;           // words of a row
  // rows of the streaming kernel: [4 phase + 2 half + {large, nonzero}][row], bits 8 q of
  // its block q of 16 entries; phases 0: as the columns
  int phases, per_phase, blocks;
};

// Marked outputs (row, column) for a kernel of their own; cap entries, others are formed
// where they are found.  count is zeroed before.
struct ChainQueue {
  uint2* entry;         // null: no queue
  int* count;
  int cap;
};

struct ChainOutputs {
  ChainArgs ch;
  Cover cover;
  ChainQueue queue;
  Group GM, GN;         // output strides of rows and columns (m[].s1)
  Marks marks;
  int64_t columns, K;
  double* C;
  double* part;         // not null: sums of K ranges, [blockIdx.y][row][column]
  double alpha, beta;
};

inline ChainOutputs chain_outputs(const GettArgs<double>& p, bool swap, const Marks& marks) {
  ChainOutputs o{};
  o.ch = chain_args(p, swap);
  o.GM = swap ? p.N : p.M;
  o.GN = swap ? p.M : p.N;
  o.marks = marks;
  o.columns = swap ? p.Mt : p.Nt;
  o.K = p.Kt;
  o.C = p.C;
  o.alpha = p.alpha;
  o.beta = p.beta;
  return o;
}

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int x, int y, int z,
                                            uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ void tmem_ld4(uint32_t taddr, float (&v)[4]) {
  uint32_t r[4];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr));
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = __uint_as_float(r[i]);
}

// Integer value of f, |f| < 2^22 (an FP32 addition; the conversion unit does
// 16 values per cycle and SM, these adders 128).
__device__ __forceinline__ int int_small(float f) {
  return __float_as_int(f + 12582912.f) - 0x4B400000;
}
// The same for |f| < 2^25: multiples of 8 and the rest.
__device__ __forceinline__ int int_wide(float f) {
  const float t = f + 100663296.f;  // 1.5 2^26: unit 8
  const float r = f - (t - 100663296.f);
  return 8 * (__float_as_int(t) - 0x4CC00000) + int_small(r);
}

// Adds one output's eight accumulators to the integer hi 2^32 + lo, in units of
// 2^-68 of the two scales.
__device__ __forceinline__ void add_groups(const float (&f)[kDigits], long long& hi, uint32_t& lo) {
  const int g01 = int_small(f[0]) * 256 + int_small(f[1]);
  const int g23 = int_wide(f[2]) * 256 + int_wide(f[3]);
  long long l = (long long)int_wide(f[4]) * 16777216 + lo;
  l += (long long)__float2int_rn(f[5]) * 65536;
  l += (long long)__float2int_rn(f[6]) * 256;
  l += __float2int_rn(f[7]);
  lo = uint32_t(l);
  hi += (long long)g01 * 65536 + g23 + (l >> 32);
}

// Contractions of a long operand with a small one over a short index
// (digits_stream.cu): swap says that the long operand is the second one.
bool stream_fits(const GettArgs<double>& p, bool& swap);
void stream_contract(Ctx& c, const GettArgs<double>& p, bool swap);
// Exponents and digits of the rows of one operand (first or second).
Digits operand_digits(Ctx& c, const GettArgs<double>& p, bool first);

}  // namespace ctm
