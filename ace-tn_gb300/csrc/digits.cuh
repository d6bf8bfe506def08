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

__device__ __forceinline__ void write_digits(const double (&x)[8], int E, bf16* dst,
                                             int64_t plane) {
  unsigned long long u[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) u[i] = digit_word(x[i], E);
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
// written by the kernel that forms the outputs; marked ones are not stored.
struct Marks {
  uint32_t* word;
  int64_t rows;
  int words, per;
};

__device__ __forceinline__ uint32_t low_bits(int n) {
  return n >= 32 ? ~0u : n > 0 ? (1u << n) - 1u : 0u;
}

struct ChainOutputs {
  ChainArgs ch;
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
