// Index groups of a two-operand contraction: shared by the GETT kernels and the
// digit products.
#pragma once
#include "engine.cuh"

namespace ctm {

constexpr int kMaxModes = 4;

struct Mode {
  int64_t ext;
  int64_t s0;  // stride in the first operand of the pair
  int64_t s1;  // stride in the second operand of the pair
};

struct Group {
  int n;
  Mode m[kMaxModes];
};

template <class T>
struct GettArgs {
  const T* A;
  const T* B;
  T* C;
  Group M, N, K;  // M: (A, C) strides, N: (B, C), K: (A, B)
  int64_t Mt, Nt, Kt;
  int64_t bext, bsa, bsb, bsc;
  T alpha, beta;
  int splitk;
  int64_t kchunk;
  T* part;
  int kfa, kfb;  // tile loaders walk K fastest (K is the unit-stride mode of A / B)
  int swap_xy;   // grid x runs over column tiles (more than 65535 of them)
  int beside_scales;  // outputs need only be exact beside their row's and column's largest entries
  int sym;       // A and B are one operand (a Gram matrix): tiles above the diagonal are mirrored
};

// Group index -> the two operands' offsets.  Decoded in 32-bit arithmetic
// (every group's extent is below 2^31, checked on the host): a 64-bit
// division by a run-time divisor is a long software sequence, and the tile
// loaders decode 16 K indices per step.
__device__ __forceinline__ void decode(const Group& g, int64_t idx, int64_t& o0, int64_t& o1) {
  o0 = 0;
  o1 = 0;
  uint32_t rem = uint32_t(idx);
#pragma unroll
  for (int j = kMaxModes - 1; j >= 0; --j) {
    if (j < g.n) {
      const uint32_t e = uint32_t(g.m[j].ext);
      const uint32_t q = rem / e;
      const int64_t r = int64_t(rem - q * e);
      rem = q;
      o0 += r * g.m[j].s0;
      o1 += r * g.m[j].s1;
    }
  }
}

// C = alpha A B + beta C by exact digit products on the tensor cores (no batch
// mode), and whether that is the faster form for this contraction.
bool digits_pay(const GettArgs<double>& p);
void digit_contract(Ctx& c, const GettArgs<double>& p, const Digits* pre_a = nullptr,
                    const Digits* pre_b = nullptr);
// One FP32 contraction (p.splitk and p.kchunk set).
void gett_f32(Ctx& c, GettArgs<float>& p);

}  // namespace ctm
