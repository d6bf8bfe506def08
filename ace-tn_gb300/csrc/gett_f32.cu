// FP32 strided contraction (the GETT kernel of the mixed path and of its site
// density matrices).
//
// A CTA computes a tile of 16 kM x 16 kN outputs, kM x kN per thread in paired
// FMAs (fma.rn.f32x2 on two rows, each half rounded as an FMA); every output is
// one chain of FMAs over its K range in order, whatever the tile.  K is staged 16
// or 32 indices at a time by cp.async with three or two steps in flight behind the
// one computed.  With 64 x 64 tiles of 4 x 4 outputs a thread and one step of
// register prefetch the shared-memory loads cost twice the FMAs' time and a CTA
// alone on its SM waited 1.5 us a step:
//   5184^2 over K = 144                 452 -> 205 us (38 TFLOP/s)
//   16384^2 over K = 256               8340 -> 3090 us (44 TFLOP/s)
//   272 x 272 over K = 16384, 7 ranges  229 -> 121 us
#include "engine.cuh"
#include "gett.cuh"

#include <algorithm>

namespace ctm {

namespace {

constexpr int kThreads = 256;

// shared memory of one stage: kK rows of A, then of B, all 16-byte aligned
template <int kM, int kN, int kK>
struct Tile {
  static constexpr int bm = 16 * kM, bn = 16 * kN;
  static constexpr int lda = bm + 4, ldb = bn + 4;
  static constexpr int stages = kK == 16 ? 4 : 3;
  static constexpr int stage = kK * (lda + ldb);  // floats; a multiple of 4
  static constexpr size_t smem = size_t(stages) * stage * sizeof(float);
};

__device__ __forceinline__ unsigned long long pack2(float x, float y) {
  return ((unsigned long long)__float_as_uint(y) << 32) | __float_as_uint(x);
}

__device__ __forceinline__ unsigned long long fma_f32x2(unsigned long long a, unsigned long long b,
                                                        unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

// 4 kV bytes of global memory into shared memory; zeros where !ok (src is not read)
template <int kV>
__device__ __forceinline__ void copy(uint32_t dst, const float* src, bool ok) {
  const int n = ok ? 4 * kV : 0;
  if constexpr (kV == 4)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n)
                 : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(dst), "l"(src),
                 "n"(4 * kV), "r"(n)
                 : "memory");
}

// kK K indices (offsets ks) of 16 kT rows (offsets rows) into dst[k * ld + row], kV
// consecutive rows a copy.  Rows beyond the operand (-1) are left as they are (zero),
// K indices beyond the range become zeros.
template <int kT, int kV, int kK>
__device__ __forceinline__ void stage_rows(uint32_t dst, int ld, const float* x,
                                           const int64_t* rows, const int64_t* ks) {
  constexpr int per = 16 * kT / kV;  // copies per K index
#pragma unroll
  for (int e = 0; e < (per * kK + kThreads - 1) / kThreads; ++e) {
    const int idx = int(threadIdx.x) + e * kThreads;
    if (per * kK % kThreads != 0 && idx >= per * kK) break;
    const int kk = idx / per, r = idx % per * kV;
    const int64_t ro = rows[r], ko = ks[kk];
    if (ro >= 0) copy<kV>(dst + 4u * uint32_t(kk * ld + r), ko >= 0 ? x + ro + ko : x, ko >= 0);
  }
}

// The same with neighbouring threads on consecutive K indices.
template <int kT, int kK>
__device__ __forceinline__ void stage_k(uint32_t dst, int ld, const float* x, const int64_t* rows,
                                        const int64_t* ks) {
  constexpr int rows_at_once = kThreads / kK;
  const int kk = int(threadIdx.x) % kK, r0 = int(threadIdx.x) / kK;
  const int64_t ko = ks[kk];
#pragma unroll
  for (int i = 0; i < 16 * kT / rows_at_once; ++i) {
    const int r = r0 + rows_at_once * i;
    const int64_t ro = rows[r];
    if (ro >= 0) copy<1>(dst + 4u * uint32_t(kk * ld + r), ko >= 0 ? x + ro + ko : x, ko >= 0);
  }
}

template <int kT, int kK>
__device__ __forceinline__ void stage(int form, uint32_t dst, int ld, const float* x,
                                      const int64_t* rows, const int64_t* ks) {
  if (form == 0) stage_k<kT, kK>(dst, ld, x, rows, ks);
  else if (form == 4) stage_rows<kT, 4, kK>(dst, ld, x, rows, ks);
  else if (form == 2) stage_rows<kT, 2, kK>(dst, ld, x, rows, ks);
  else stage_rows<kT, 1, kK>(dst, ld, x, rows, ks);
}

template <int kM, int kN, int kK>
__global__ void __launch_bounds__(kThreads, kM == 8 || kK == 32 ? 2 : 3)
    gett_f32_kernel(const GettArgs<float> p, int form_a, int form_b) {
  using Tl = Tile<kM, kN, kK>;
  constexpr int kStages = Tl::stages;
  __shared__ int64_t sAm[Tl::bm], sCm[Tl::bm], sBn[Tl::bn], sCn[Tl::bn];
  __shared__ int64_t sAk[2 * kStages][kK], sBk[2 * kStages][kK];
  extern __shared__ __align__(16) float gsm[];
  const int tid = threadIdx.x;
  const int64_t m0 = int64_t(p.swap_xy ? blockIdx.y : blockIdx.x) * Tl::bm;
  const int64_t n0 = int64_t(p.swap_xy ? blockIdx.x : blockIdx.y) * Tl::bn;
  const int64_t batch = blockIdx.z % p.bext, split = blockIdx.z / p.bext;
  const float* A = p.A + batch * p.bsa;
  const float* B = p.B + batch * p.bsb;
  for (int t = tid; t < Tl::bm + Tl::bn; t += kThreads) {
    if (t < Tl::bm) {
      if (m0 + t < p.Mt) decode(p.M, m0 + t, sAm[t], sCm[t]);
      else { sAm[t] = -1; sCm[t] = -1; }
    } else {
      const int u = t - Tl::bm;
      if (n0 + u < p.Nt) decode(p.N, n0 + u, sBn[u], sCn[u]);
      else { sBn[u] = -1; sCn[u] = -1; }
    }
  }
  const int64_t kb = split * p.kchunk;
  const int64_t ke = min(kb + p.kchunk, p.Kt);
  const int nsteps = ke > kb ? int((ke - kb + kK - 1) / kK) : 0;
  auto decode_k = [&](int step, int kk) {
    const int slot = step % (2 * kStages);
    const int64_t k = kb + int64_t(step) * kK + kk;
    if (step < nsteps && k < ke) decode(p.K, k, sAk[slot][kk], sBk[slot][kk]);
    else { sAk[slot][kk] = -1; sBk[slot][kk] = -1; }
  };
  if (tid < kStages * kK) decode_k(tid / kK, tid % kK);
  // rows beyond the operands stay zero in every stage
  if (m0 + Tl::bm > p.Mt || n0 + Tl::bn > p.Nt)
    for (int t = tid; t < kStages * Tl::stage; t += kThreads) gsm[t] = 0.f;
  const uint32_t base = uint32_t(__cvta_generic_to_shared(gsm));
  auto load = [&](int step) {
    if (step < nsteps) {
      const int slot = step % (2 * kStages);
      const uint32_t dst = base + uint32_t(step % kStages) * (Tl::stage * 4u);
      stage<kM, kK>(form_a, dst, Tl::lda, A, sAm, sAk[slot]);
      stage<kN, kK>(form_b, dst + 4u * kK * Tl::lda, Tl::ldb, B, sBn, sBk[slot]);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // rows 4 hi + {0..3} (+ 64), columns lo + 16 j; a warp without rows only copies
  const int lo = tid & 15, hi = tid >> 4;
  const bool work = m0 + 8 * (tid >> 5) < p.Mt;
  unsigned long long acc[kM / 2][kN];
#pragma unroll
  for (int i = 0; i < kM / 2; ++i)
#pragma unroll
    for (int j = 0; j < kN; ++j) acc[i][j] = 0ull;
  __syncthreads();
  for (int s = 0; s < kStages - 1; ++s) load(s);
  for (int st = 0; st < nsteps; ++st) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
    __syncthreads();  // step st is in; every read of the buffer refilled next is done
    load(st + kStages - 1);
    // the offsets of the step after that, by a different warp each time
    if ((tid >> 5) == (st & 7) && (tid & 31) < kK) decode_k(st + kStages, tid & 31);
    const float* as = gsm + (st % kStages) * Tl::stage + 4 * hi;
    const float* bs = gsm + (st % kStages) * Tl::stage + kK * Tl::lda + lo;
    if (!work) continue;
#pragma unroll
    for (int kk = 0; kk < kK; ++kk) {
      unsigned long long a[kM / 2];
#pragma unroll
      for (int i = 0; i < kM / 4; ++i) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(as + kk * Tl::lda + 64 * i);
        a[2 * i] = v.x;
        a[2 * i + 1] = v.y;
      }
#pragma unroll
      for (int j = 0; j < kN; ++j) {
        const float b = bs[kk * Tl::ldb + 16 * j];
        const unsigned long long bb = pack2(b, b);
#pragma unroll
        for (int i = 0; i < kM / 2; ++i) acc[i][j] = fma_f32x2(a[i], bb, acc[i][j]);
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
  for (int i = 0; i < kM; ++i) {
    const int mi = 64 * (i / 4) + 4 * hi + (i & 3);
    const int64_t m = m0 + mi;
    if (m >= p.Mt) continue;
#pragma unroll
    for (int j = 0; j < kN; ++j) {
      const int nj = lo + 16 * j;
      const int64_t n = n0 + nj;
      if (n >= p.Nt) continue;
      const unsigned long long w = acc[i / 2][j];
      const float x = __uint_as_float((i & 1) ? unsigned(w >> 32) : unsigned(w));
      if (p.splitk > 1) {
        p.part[((split * p.bext + batch) * p.Mt + m) * p.Nt + n] = x;
      } else {
        float* c = p.C + batch * p.bsc + sCm[mi] + sCn[nj];
        const float v = p.alpha * x;
        *c = (p.beta != 0.f) ? fmaf(p.beta, *c, v) : v;
      }
    }
  }
}

template <int kM, int kN, int kK>
void launch_k(Ctx& c, GettArgs<float>& p, int form_a, int form_b) {
  using Tl = Tile<kM, kN, kK>;
  const int64_t mb = (p.Mt + Tl::bm - 1) / Tl::bm, nb = (p.Nt + Tl::bn - 1) / Tl::bn;
  p.swap_xy = nb > 65535 ? 1 : 0;
  const dim3 grid(unsigned(p.swap_xy ? nb : mb), unsigned(p.swap_xy ? mb : nb),
                  unsigned(p.bext * p.splitk));
  CTM_REQUIRE(grid.y <= 65535 && p.bext * p.splitk <= 65535 && grid.x <= 0x7fffffffLL,
              CTM_ERR_UNSUPPORTED, "einsum: grid too large");
  CTM_CUDA(cudaFuncSetAttribute(gett_f32_kernel<kM, kN, kK>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, int(Tl::smem)));
  gett_f32_kernel<kM, kN, kK><<<grid, kThreads, Tl::smem, c.stream>>>(p, form_a, form_b);
  CTM_LAUNCH_CHECK();
}

// 32 K indices a step halve the barriers of the small tiles where K is long (272 x 272
// over K = 16384 in 7 ranges: 148 -> 121 us); a short K would be padded (746496 x 72
// over K = 36: 320 -> 424 us) and the large tiles lose their second CTA's overlap
// (5184^2 over K = 144: 202 -> 231 us).
template <int kM, int kN>
void launch(Ctx& c, GettArgs<float>& p, int form_a, int form_b) {
  if constexpr (kM == 4) {
    if (std::min(p.kchunk, p.Kt) >= 256) return launch_k<kM, kN, 32>(c, p, form_a, form_b);
  }
  launch_k<kM, kN, 16>(c, p, form_a, form_b);
}

// How an operand's tiles are copied: 0 along K, else along the rows, 4, 2 or 1 of them
// at once (they must be neighbours in memory, and every start aligned).
int copy_form(const float* x, int64_t batch_stride, int64_t bext, const Group& rows,
              const Group& k, bool first, int kfast) {
  if (kfast) return 0;
  if (rows.n == 0 || rows.m[rows.n - 1].s0 != 1) return 1;
  for (int v : {4, 2}) {
    bool ok = reinterpret_cast<uintptr_t>(x) % (4 * v) == 0 && rows.m[rows.n - 1].ext % v == 0 &&
              (bext == 1 || batch_stride % v == 0);
    for (int i = 0; i + 1 < rows.n; ++i) ok = ok && rows.m[i].s0 % v == 0;
    for (int i = 0; i < k.n; ++i) ok = ok && (first ? k.m[i].s0 : k.m[i].s1) % v == 0;
    if (ok) return v;
  }
  return 1;
}

}  // namespace

void gett_f32(Ctx& c, GettArgs<float>& p) {
  const int64_t sms = sm_count_linalg();
  const int fa = copy_form(p.A, p.bsa, p.bext, p.M, p.K, true, p.kfa);
  const int fb = copy_form(p.B, p.bsb, p.bext, p.N, p.K, false, p.kfb);
  // The tile with the least estimated time.  What bounds a K step is the shared memory's
  // 128 bytes a cycle: kM + kN words a thread and index (the FMAs of 8 x 8 outputs take
  // as long), and the copies' writes.  A CTA alone on its SM takes about 1.45 times
  // that.  The estimates pick the measured best of 272 x 272 in 7 ranges (64 x 80: 148
  // us; 64 x 48: 149, 64 x 32: 168, 64 x 64: 178, 128 x 96: 223), 36 x 72 in 76 ranges
  // (64 x 48: 538 us; 64 x 16: 577, 64 x 80: 705) and 16384 x 272 over K = 272
  // (128 x 96: 85 us; 64 x 96: 102).
  int bm = 4, bn = 4;
  double least = 0.0;
  const double steps = double(std::min(p.kchunk, p.Kt)) / 16.0;
  auto consider = [&](int km, int kn) {
    const int64_t tiles = (p.Mt + 16 * km - 1) / (16 * km) * ((p.Nt + 16 * kn - 1) / (16 * kn));
    const double r = double((tiles * p.bext * p.splitk + sms - 1) / sms);
    const double busy = 128.0 * (km + kn) + 16.0 * (km * (fa == 4 ? 1 : 2) + kn * (fb == 4 ? 1 : 2));
    const double cost = steps * std::max(1.45, r) * busy + r * (1500.0 + 16.0 * km * kn);
    if (least == 0.0 || cost < least) {
      least = cost;
      bm = km;
      bn = kn;
    }
  };
  for (int kn : {8, 6, 5}) consider(8, kn);
  for (int kn : {6, 5, 4, 3, 2}) consider(4, kn);
  if (bm == 8) {
    if (bn == 8) launch<8, 8>(c, p, fa, fb);
    else if (bn == 6) launch<8, 6>(c, p, fa, fb);
    else launch<8, 5>(c, p, fa, fb);
  } else {
    switch (bn) {
      case 6: launch<4, 6>(c, p, fa, fb); break;
      case 5: launch<4, 5>(c, p, fa, fb); break;
      case 4: launch<4, 4>(c, p, fa, fb); break;
      case 3: launch<4, 3>(c, p, fa, fb); break;
      default: launch<4, 2>(c, p, fa, fb); break;
    }
  }
}

}  // namespace ctm
