// float32 linear layer on the 5th-generation tensor cores, with float32's accuracy.
//
//   out[m, n] = act( sum_k a[m, k] * w[n, k] + bias[n] ) (+ residual[m, n])
//
// A float32 number is the sum of three bfloat16 terms (8 bits of mantissa each, formed by rounding and
// exact subtraction), so a product of two is six products of terms - high x high and the five others
// whose size is above 2^-24 of it; the three left out are below 2^-26.  Products of bfloat16 numbers are
// exact in the tensor cores; what they lose is in the sum, which they cut off below the last bit instead
// of rounding it: over 1,024 products in one accumulator that is 1.0e-6 of the result (an FMA chain:
// 5.7e-7).  So the summed index is cut into chunks of 64: a chunk starts from zero with its small products
// and ends with its high x high ones, then goes through float32 additions with rounding, four chunks to a
// segment and the segments one after the other.  Off float64 by
// 6.6e-8 (k = 1,024) and 7.6e-8 (4,096) of the result, FMA chains by 3.3e-7 and 6.6e-7.
//
// The order of the sums is fixed by k alone: not by the number of rows, the tile an output lies in or how
// many blocks share the segments.  So a row's bits are the same in every batch.  A result that is not
// finite is computed again as a chain of FMAs, since the terms of an infinity are not numbers.
//
// A tile is 128 features (the weights are the operand of 128 rows) x NR rows of `a`, NR = 16 .. 128.
//   warps 0..7    fetch both operands as float32 a chunk or two ahead (registers), cut them into terms and
//                 store these in the 128-byte swizzled operand layout (ring of stages);
//   warps 8..11   add up chunks and segments in tensor memory (registers for 128 columns a thread do not
//                 exist beside eight fetching warps, and spills find little first-level cache beside 200 KB
//                 of shared memory) and finish the tile: a lane owns a feature, a column is a row of `a`,
//                 so loads and stores are 128 contiguous bytes a warp;
//   warp 12       issues the MMAs.
// With few tiles the segments of a tile, or its single chunks, are shared out between blocks: their sums go to scratch
// and a second kernel adds them in the same order.
//
// Operands below 2^-109 have a third term below bfloat16's range: a product is off by 2^-134 of the other operand at
// most, where a chain would keep their digits.
//
// 1,024 x 4,096 x 1,024: 223 us as FMA chains (linear_simt.cu) -> 68; 1,024 x 1,024 x 4,096: 317 -> 82; 64 x
// 4,096 x 1,024: 29 -> 16; 8 x 1,024 x 4,096: 19 -> 11; 1 x 768 x 768 5.1 -> 5.6 (8.3 with whole segments a block).  A
// chunk of a 128 x 128 tile takes 1.8 us: 24 MMAs that read 8 KB of shared memory each (1.5 us alone) beside the
// stores of terms.
#include "tcgen05.cuh"

namespace hs {

constexpr int LF_BM = 128, LF_BK = 64;
constexpr int LF_SEG = 4;                 // chunks of 64 a segment holds (1 << 2)
constexpr int LF_CONV = 8, LF_SUM = 4;    // warps
constexpr int LF_THREADS = 32 * (LF_CONV + LF_SUM + 1);
constexpr int LF_A_TERM = LF_BM * LF_BK * 2;

template <int NR>
struct LfShape {
  static constexpr int B_TERM = NR * LF_BK * 2;
  static constexpr int STAGE = 3 * (LF_A_TERM + B_TERM);
  static constexpr int STAGES = NR >= 128 ? 2 : (NR == 16 ? 4 : 3);
  static constexpr int SMEM = STAGES * STAGE + 1024;
  static constexpr int TMEM = 4 * NR;     // two chunks, the segment's sum, the segments' sum
  static constexpr int AHEAD = NR >= 128 ? 1 : 2;       // chunks fetched ahead
};

struct LfParams {
  float* out;
  const float *a, *w, *bias, *residual;
  float* partial;                  // [segments][M][N] when segments are shared out
  int* status;
  int M, N, K, act;
  float2 act_ab;
  int tiles_m, parts, splits, kb_per_split, part_shift, items;   // a part: 1 << part_shift chunks summed up in scratch
};

__device__ __forceinline__ void lf_tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
// W columns of a lane: 16 or 32
template <int W>
__device__ __forceinline__ void lf_tmem_ld(uint32_t taddr, uint32_t (&r)[W]) {
  if constexpr (W == 32) tmem_ld32(taddr, r);
  else lf_tmem_ld16(taddr, r);
}
template <int W>
__device__ __forceinline__ void lf_tmem_st(uint32_t taddr, const uint64_t (&v)[W / 2]) {
  uint32_t r[W];
#pragma unroll
  for (int j = 0; j < W / 2; ++j) asm("mov.b64 {%0, %1}, %2;" : "=r"(r[2 * j]), "=r"(r[2 * j + 1]) : "l"(v[j]));
  if constexpr (W == 32)
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, "
        "%22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]),
          "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]),
          "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]),
          "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]),
          "r"(r[31])
        : "memory");
  else
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]),
          "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]),
          "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void lf_tmem_st_wait() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 lf_ldg_w(const float* p) {      // weights: read once a tile
  float4 v;
  asm("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ uint64_t lf_pair(float x, float y) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ uint64_t lf_pair(uint32_t x, uint32_t y) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(x), "r"(y));
  return r;
}
// two sums with rounding, side by side
__device__ __forceinline__ uint64_t lf_add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// the next bfloat16 term of two numbers; what it leaves stays behind (exact)
__device__ __forceinline__ uint32_t lf_term(uint64_t& xy) {
  float x, y;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(xy));
  const __nv_bfloat162 b = __floats2bfloat162_rn(x, y);
  const uint32_t u = *(const uint32_t*)&b;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(xy) : "l"(xy), "l"(lf_pair(u << 16, u & 0xffff0000u)));
  return u;
}
__device__ __forceinline__ void lf_store_terms(uint32_t dst, uint32_t term_bytes, float4 v) {
  uint64_t xy = lf_pair(v.x, v.y), zw = lf_pair(v.z, v.w);
#pragma unroll
  for (int t = 0; t < 3; ++t) {
    const uint32_t lo = lf_term(xy), hi = lf_term(zw);
    asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(dst + t * term_bytes), "r"(lo), "r"(hi) : "memory");
  }
}
// A result that is not finite is formed again as a chain of FMAs (the terms of an infinity are not numbers).
// Where a row of `a` or a feature's weights hold no number, which a warp sees by a look along them, so does the
// result; else the chain, its numbers eight pieces ahead, until it holds none.  (us for 8 x 1,024 x 4,096 with a row of
// NaNs, 12 without: 294 as chains of single loads; 1,024 rows of NaNs, 83 without: 18,800.)
__device__ __forceinline__ bool lf_finite(float x) { return fabsf(x) <= 3.402823466e38f; }
// whether a row holds something that is no number; the whole warp asks for the same row
__device__ __forceinline__ bool lf_row_nan(const float* __restrict__ row, int K) {
  for (int k0 = 0; k0 < K; k0 += 512) {
    bool nan = false;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int k = k0 + j * 128 + (threadIdx.x & 31) * 4;
      const float4 x = k < K ? *(const float4*)(row + k) : make_float4(0.f, 0.f, 0.f, 0.f);
      nan = nan || x.x != x.x || x.y != x.y || x.z != x.z || x.w != x.w;
    }
    if (__any_sync(0xffffffffu, nan)) return true;
  }
  return false;
}
// the chain of a row (the same for the whole warp) and the lane's weights; lanes that want none come along
template <int AHEAD>
__device__ __forceinline__ float lf_chain(const float* __restrict__ x, const float* __restrict__ y, int K, bool wanted) {
  float sum = 0.f;
  for (int k0 = 0; k0 < K; k0 += 4 * AHEAD) {
    const int lane = threadIdx.x & 31;
    const float mine = lane < 4 * AHEAD && k0 + lane < K ? x[k0 + lane] : 0.f;
    float4 v[AHEAD];
#pragma unroll
    for (int j = 0; j < AHEAD; ++j)
      if (k0 + 4 * j < K) v[j] = *(const float4*)(y + k0 + 4 * j);
#pragma unroll
    for (int j = 0; j < AHEAD; ++j)
      if (k0 + 4 * j < K) {
        sum = fmaf(__shfl_sync(0xffffffffu, mine, 4 * j), v[j].x, sum);
        sum = fmaf(__shfl_sync(0xffffffffu, mine, 4 * j + 1), v[j].y, sum);
        sum = fmaf(__shfl_sync(0xffffffffu, mine, 4 * j + 2), v[j].z, sum);
        sum = fmaf(__shfl_sync(0xffffffffu, mine, 4 * j + 3), v[j].w, sum);
      }
    if (__all_sync(0xffffffffu, !wanted || sum != sum)) break;
  }
  return sum;
}
// The sums of a warp's lanes (feature n each, -1: none) with row m, those that are not finite formed again.  nans:
// lanes whose weights are known to hold no number.
template <int AHEAD>
__device__ __forceinline__ float lf_again(const LfParams& p, float sum, int m, int n, unsigned& nans) {
  const float nan = __int_as_float(0x7fffffff);
  const int lane = threadIdx.x & 31;
  unsigned odd = __ballot_sync(0xffffffffu, n >= 0 && !lf_finite(sum));
  if (odd >> lane & 1 & nans >> lane) sum = nan;
  odd &= ~nans;
  if (odd == 0) return sum;
  if (lf_row_nan(p.a + (size_t)m * p.K, p.K)) return odd >> lane & 1 ? nan : sum;
  if (__popc(odd) <= 4) {
    for (unsigned rest = odd; rest; rest &= rest - 1) {
      const int l = __ffs(rest) - 1, f = __shfl_sync(0xffffffffu, n, l);
      if (!lf_row_nan(p.w + (size_t)f * p.K, p.K)) continue;
      nans |= 1u << l;
      odd &= ~(1u << l);
      if (lane == l) sum = nan;
    }
  }
  const float chain = lf_chain<AHEAD>(p.a + (size_t)m * p.K, p.w + (size_t)max(n, 0) * p.K, p.K, odd >> lane & 1);
  return odd >> lane & 1 ? chain : sum;
}
// Rows m0 .. m0 + n - 1 of a tile some of whose sums are not finite, finished (up to sixteen); the lane's feature is f.
// (Few registers: what a called function needs the kernel keeps free, and its fetching warps have none to spare.)
__device__ __noinline__ unsigned lf_odd_rows(const LfParams& p, uint32_t taddr, int m0, int n, int f, unsigned nans) {
  // rows of NaNs are most often that from their first number on
  float first = 0.f;
  if ((threadIdx.x & 31) < min(n, 16)) first = p.a[(size_t)(m0 + (threadIdx.x & 31)) * p.K];
  const unsigned gone = __ballot_sync(0xffffffffu, first != first);
#pragma unroll 1
  for (int j = 0; j < min(n, 16); ++j) {
    uint32_t c;
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(c) : "r"(taddr + j) : "memory");
    tmem_ld_wait();
    float v = __uint_as_float(c);
    if (!(gone >> j & 1)) v = lf_again<4>(p, v, m0 + j, f < p.N ? f : -1, nans);
    if (f < p.N) {
      v = apply_act(v + (p.bias ? p.bias[f] : 0.f), p.act, p.act_ab);
      const size_t at = (size_t)(m0 + j) * p.N + f;
      if (p.residual) v += p.residual[at];
      p.out[at] = v;
    }
    __syncwarp();
  }
  return nans;
}

// where an item lies: tiles of rows run fastest (blocks that run together share the weights), then the
// shares of a tile's segments, then tiles of features
struct LfItem {
  int m0, f0, kb0, kb1;
};
template <int NR>
__device__ __forceinline__ LfItem lf_item(const LfParams& p, int w) {
  LfItem r;
  const int s = w / p.tiles_m, f = s / p.splits;
  r.m0 = (w - s * p.tiles_m) * NR;
  r.f0 = f * LF_BM;
  r.kb0 = (s - f * p.splits) * p.kb_per_split;
  r.kb1 = min(r.kb0 + p.kb_per_split, (p.K + LF_BK - 1) / LF_BK);
  return r;
}

template <int NR, bool SPLIT>
__global__ void __launch_bounds__(LF_THREADS, 1) linear_f32_tc_kernel(const __grid_constant__ LfParams p) {
  using S = LfShape<NR>;
  extern __shared__ uint8_t lf_smem[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)lf_smem + 1023) & ~(uintptr_t)1023);
  __shared__ uint64_t full_bar[S::STAGES], empty_bar[S::STAGES], acc_full[2], acc_empty[2], drain_bar;
  __shared__ uint32_t tmem_slot;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  pdl_trigger();
  if (threadIdx.x == 0) {
    for (int s = 0; s < S::STAGES; ++s) {
      mbar_init(&full_bar[s], LF_CONV);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], LF_SUM);
    }
    mbar_init(&drain_bar, 1);
    fence_barrier_init();
  }
  if (warp == LF_CONV + LF_SUM) {
    tmem_alloc(&tmem_slot, S::TMEM);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;

  if (warp == LF_CONV + LF_SUM) {
    constexpr uint32_t idesc = make_idesc(LF_BM, NR);
    constexpr uint64_t TA = LF_A_TERM >> 4, TB = S::B_TERM >> 4;
    pdl_wait();                      // (the limit of the waits is not for the kernel before)
    uint32_t limit = HS_SPIN_LIMIT;
    int s = 0, round = 0, cc = 0;
    for (int w = blockIdx.x; w < p.items; w += gridDim.x) {
      const LfItem it = lf_item<NR>(p, w);
      for (int kb = it.kb0; kb < it.kb1; ++kb, ++cc) {
        const int b = cc & 1;
        if (cc > 1) mbar_wait_warp(&acc_empty[b], ((cc >> 1) - 1) & 1, p.status, limit);
        mbar_wait_warp(&full_bar[s], round & 1, p.status, limit);
        tc_fence_after();
        const uint32_t acc = tmem + b * NR, base = smem_u32(smem + s * S::STAGE);
        const uint64_t da = make_smem_desc(base), db = make_smem_desc(base + 3 * LF_A_TERM);
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < LF_BK / 16; ++k) {         // small products
            umma_bf16(acc, da + 2 * k, db + 2 * k + 2 * TB, idesc, k > 0 ? 1u : 0u);
            umma_bf16(acc, da + 2 * k + 2 * TA, db + 2 * k, idesc, 1u);
            umma_bf16(acc, da + 2 * k + TA, db + 2 * k + TB, idesc, 1u);
            umma_bf16(acc, da + 2 * k, db + 2 * k + TB, idesc, 1u);
            umma_bf16(acc, da + 2 * k + TA, db + 2 * k, idesc, 1u);
          }
#pragma unroll
          for (int k = 0; k < LF_BK / 16; ++k) umma_bf16(acc, da + 2 * k, db + 2 * k, idesc, 1u);
          umma_commit(&empty_bar[s]);
          umma_commit(&acc_full[b]);
        }
        __syncwarp();
        if (++s == S::STAGES) { s = 0; ++round; }
      }
    }
    umma_drain(&drain_bar, limit, p.status);
  } else if (warp < LF_CONV) {
    // ---- operands: four numbers a piece, 16 pieces a row of a step, 16 rows a pass
    constexpr int PA = LF_BM / 16, PB = NR / 16, AHEAD = S::AHEAD;
    const int c4 = threadIdx.x & 15, r = threadIdx.x >> 4;
    const uint32_t place = r * 128 + (((c4 >> 1) ^ (r & 7)) << 4) + (c4 & 1) * 8;   // rows r + 16 i: + 2048 i
    const size_t pass = (size_t)16 * p.K;                 // numbers from one pass's row to the next's
    float4 va[AHEAD][PA], vb[AHEAD][PB];
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    // the step to fetch next, ahead of the one that is cut into terms
    int lw = blockIdx.x, lkb = 0, lend = 0, left_w = 0, left_a = 0;   // left: rows from this thread's on
    const float *src_w = p.w, *src_a = p.a;
    auto open_item = [&] {
      left_w = left_a = 0;
      if (lw >= p.items) return;
      const LfItem li = lf_item<NR>(p, lw);
      lkb = li.kb0;
      lend = li.kb1;
      left_w = p.N - li.f0 - r;
      left_a = p.M - li.m0 - r;
      src_w = p.w + (size_t)(li.f0 + r) * p.K + lkb * LF_BK + c4 * 4;
      src_a = p.a + (size_t)(li.m0 + r) * p.K + lkb * LF_BK + c4 * 4;
    };
    auto advance = [&] {
      src_w += LF_BK;
      src_a += LF_BK;
      if (++lkb == lend) {
        lw += gridDim.x;
        open_item();
      }
    };
    auto fetch_w = [&](float4 (&v)[PA]) {
      const int left = lkb * LF_BK + c4 * 4 < p.K ? left_w : 0;
      if (left > 16 * (PA - 1)) {
#pragma unroll
        for (int i = 0; i < PA; ++i) v[i] = lf_ldg_w(src_w + i * pass);
      } else {
#pragma unroll
        for (int i = 0; i < PA; ++i) v[i] = 16 * i < left ? lf_ldg_w(src_w + i * pass) : zero;
      }
    };
    auto fetch_a = [&](float4 (&v)[PB]) {
      const int left = lkb * LF_BK + c4 * 4 < p.K ? left_a : 0;
      if (left > 16 * (PB - 1)) {
#pragma unroll
        for (int i = 0; i < PB; ++i) v[i] = *(const float4*)(src_a + i * pass);
      } else {
#pragma unroll
        for (int i = 0; i < PB; ++i) v[i] = 16 * i < left ? *(const float4*)(src_a + i * pass) : zero;
      }
    };
    open_item();
    // the weights do not change during a step: the first are on their way before the kernel before ends
    fetch_w(va[0]);
    pdl_wait();
    fetch_a(vb[0]);
    advance();
    if (AHEAD == 2) {
      fetch_w(va[AHEAD - 1]);
      fetch_a(vb[AHEAD - 1]);
      advance();
    }
    int steps = 0;
    for (int w = blockIdx.x; w < p.items; w += gridDim.x) {
      const LfItem it = lf_item<NR>(p, w);
      steps += it.kb1 - it.kb0;
    }
    int s = 0, round = 0;
    bool ok = true;
    for (int i0 = 0; i0 < steps && ok; i0 += AHEAD) {
#pragma unroll
      for (int d = 0; d < AHEAD; ++d) {
        if (i0 + d >= steps) break;
        if (round > 0 && !mbar_wait(&empty_bar[s], (round - 1) & 1, p.status)) ok = false;
        if (!ok) break;
        const uint32_t dst = smem_u32(smem + s * S::STAGE) + place;
#pragma unroll
        for (int i = 0; i < PA; ++i) lf_store_terms(dst + i * 2048, LF_A_TERM, va[d][i]);
        fetch_w(va[d]);
#pragma unroll
        for (int i = 0; i < PB; ++i) lf_store_terms(dst + 3 * LF_A_TERM + i * 2048, S::B_TERM, vb[d][i]);
        fetch_a(vb[d]);
        advance();
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(&full_bar[s]);
        if (++s == S::STAGES) { s = 0; ++round; }
      }
    }
  } else {
    // ---- chunks added up: warp w owns lanes 32 (w % 4) .. of the accumulators = features
    pdl_wait();
    const int q = warp & 3;
    const uint32_t lanes = tmem + ((uint32_t)(q * 32) << 16), seg = lanes + 2 * NR, total = lanes + 3 * NR;
    int cc = 0;
    bool ok = true;
    for (int w = blockIdx.x; w < p.items && ok; w += gridDim.x) {
      const LfItem it = lf_item<NR>(p, w);
      const int f = it.f0 + q * 32 + lane, n = min(NR, p.M - it.m0);
      for (int kb = it.kb0; kb < it.kb1; ++kb, ++cc) {
        const int b = cc & 1;
        const int part = SPLIT ? (1 << p.part_shift) - 1 : LF_SEG - 1;
        const bool opens = (kb & part) == 0, last = kb + 1 == it.kb1, ends = last || ((kb + 1) & part) == 0;
        ok = mbar_wait(&acc_full[b], (cc >> 1) & 1, p.status);
        if (!ok) break;
        tc_fence_after();
        const bool fold = !SPLIT && ends && kb - it.kb0 >= LF_SEG;      // onto the segments before
        const uint32_t dst_cols = !SPLIT && ends ? total : seg;
        constexpr int W = NR >= 32 ? 32 : 16;
        for (int j0 = 0; j0 < n; j0 += W) {
          uint32_t c[W], g[W];
          uint64_t v[W / 2];
          lf_tmem_ld<W>(lanes + b * NR + j0, c);
          if (!opens) lf_tmem_ld<W>(seg + j0, g);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < W / 2; ++j) v[j] = lf_pair(c[2 * j], c[2 * j + 1]);
          if (!opens) {
#pragma unroll
            for (int j = 0; j < W / 2; ++j) v[j] = lf_add2(lf_pair(g[2 * j], g[2 * j + 1]), v[j]);
          }
          if (fold) {
            lf_tmem_ld<W>(total + j0, g);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < W / 2; ++j) v[j] = lf_add2(lf_pair(g[2 * j], g[2 * j + 1]), v[j]);
          }
          lf_tmem_st<W>(dst_cols + j0, v);
        }
        lf_tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&acc_empty[b]);
        if (SPLIT ? !ends : !last) continue;
        // the sums of a segment (SPLIT) or of the tile, sixteen rows of `a` at a time
        const float bias = !SPLIT && p.bias && f < p.N ? p.bias[f] : 0.f;
        float* dst = SPLIT ? p.partial + ((size_t)(kb >> p.part_shift) * p.M + it.m0) * p.N + f
                           : p.out + (size_t)it.m0 * p.N + f;
        unsigned nans = 0;                       // lanes whose weights hold no number
#pragma unroll 1
        for (int j0 = 0; j0 < n; j0 += 16) {
          uint32_t c[16];
          lf_tmem_ld16((SPLIT ? seg : total) + j0, c);
          tmem_ld_wait();
          if (!SPLIT) {
            bool finite = true;
#pragma unroll
            for (int j = 0; j < 16; ++j) finite = finite && lf_finite(__uint_as_float(c[j]));
            if (__any_sync(0xffffffffu, !finite && f < p.N)) {
              nans = lf_odd_rows(p, total + j0, it.m0 + j0, n - j0, f, nans);
              continue;
            }
          }
          if (f < p.N) {
            float v[16], res[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              v[j] = __uint_as_float(c[j]);
              if (!SPLIT) res[j] = (p.residual && j0 + j < n) ? p.residual[(size_t)(it.m0 + j0 + j) * p.N + f] : 0.f;
            }
            if (!SPLIT) {
#pragma unroll
              for (int j = 0; j < 16; ++j) v[j] += bias;
              if (p.act == HS_ACT_GELU_TANH) {
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] = gelu_tanh(v[j]);
              } else if (p.act != HS_ACT_NONE) {
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] = apply_act(v[j], p.act, p.act_ab);
              }
              if (p.residual) {
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] += res[j];
              }
            }
#pragma unroll
            for (int j = 0; j < 16; ++j)
              if (j0 + j < n) dst[(size_t)(j0 + j) * p.N] = v[j];
          }
          __syncwarp();
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == LF_CONV + LF_SUM) {
    tc_fence_after();
    tmem_dealloc(tmem, S::TMEM);
  }
}

// the segments' sums added in order, bias, activation, residual
__global__ void __launch_bounds__(128) linear_f32_tc_sum_kernel(const __grid_constant__ LfParams p) {
  pdl_trigger();
  pdl_wait();
  const long long size = (long long)p.M * p.N, at = (long long)blockIdx.x * 128 + threadIdx.x;
  const long long i = at < size ? at : size - 1;         // (whole warps come to the end)
  const float* src = p.partial + i;
  float sum = 0.f;
  if (p.part_shift) {                                    // segments
    for (int c0 = 0; c0 < p.parts; c0 += 8) {
      float v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (c0 + j < p.parts) v[j] = src[(c0 + j) * size];
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (c0 + j < p.parts) sum = c0 + j ? sum + v[j] : v[j];
    }
  } else {                                               // chunks, four to a segment
    for (int c0 = 0; c0 < p.parts; c0 += 16) {
      float v[16];
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (c0 + j < p.parts) v[j] = src[(c0 + j) * size];
#pragma unroll
      for (int j = 0; j < 16; j += LF_SEG) {
        if (c0 + j >= p.parts) break;
#pragma unroll
        for (int k = 1; k < LF_SEG; ++k)
          if (c0 + j + k < p.parts) v[j] += v[j + k];
        sum = c0 + j ? sum + v[j] : v[j];
      }
    }
  }
  const int m = (int)(i / p.N), n = (int)(i - (long long)m * p.N);
  if (__any_sync(0xffffffffu, !lf_finite(sum))) {
    unsigned nans = 0;
    const int last = __shfl_sync(0xffffffffu, m, 31);      // (a warp's outputs lie in one row, or in rows one by one)
    for (int row = __shfl_sync(0xffffffffu, m, 0); row <= last; ++row)
      sum = lf_again<8>(p, sum, row, m == row ? n : -1, nans);
  }
  if (at >= size) return;
  float y = apply_act(sum + (p.bias ? p.bias[n] : 0.f), p.act, p.act_ab);
  if (p.residual) y += p.residual[i];
  p.out[i] = y;
}

struct LfPlan {
  int nr, splits, kb_per_split, part_shift, parts, tiles_m, items;
};
static bool plan_lf(int M, int N, int K, int force_nr, LfPlan& pl) {
  // One chunk of 64 is a launch's beginning and end and little else: 4,096 x 1,024 x 16 22.9 us, 9.9 on the CUDA cores, x 64
  // 22.9 and 21.9 (1,024 x 1,024 x 128: 10.9 and 13.6).  And a sum of up to eight products is no closer to float64 here.
  if (K % 4 || M <= 0 || N <= 0 || K <= LF_BK) return false;
  const int sms = hs_sm_count(), ft = (N + LF_BM - 1) / LF_BM;
  const int num_kb = (K + LF_BK - 1) / LF_BK;
  // us a chunk takes by rows of the tile, and a tile's beginning and end, measured (148 SMs, 1,024 rows: 16
  // rows a tile 268 us for 14 rounds of 16 chunks, 32 147 for 7, 64 76 for 3 and 84 for one of 64, 128 68
  // for 2).  A tile's segments, or its single chunks, are shared out through scratch where tiles are few; that costs the second launch
  // and their way to the L2 and back.
  const int sizes[4] = {16, 32, 64, 128};
  const double step[4] = {0.95, 1.06, 1.26, 1.8};
  double best = -1.0;
  for (int i = 0; i < 4; ++i) {
    const int nr = sizes[i];
    if (force_nr ? nr != force_nr : (nr > 16 && nr / 2 >= M)) continue;
    const long long mt = (M + nr - 1) / nr, tiles = mt * ft;
    if (tiles > (1 << 30) / num_kb) continue;
    // whole tiles; segments and chunks that fill one round; single chunks, as many as there are
    for (int form = 0; form < 4; ++form) {
      const int unit = form == 1 ? LF_SEG : 1, parts = (num_kb + unit - 1) / unit;
      int splits = form == 0 ? 1 : form == 3 ? parts : (int)(sms / tiles < parts ? sms / tiles : parts);
      if (form && splits < 2) continue;
      const int per = form ? (parts + splits - 1) / splits * unit : num_kb;
      splits = (num_kb + per - 1) / per;
      const double rounds = (double)((tiles * splits + sms - 1) / sms);
      double cost = form == 3 ? rounds * (step[i] + 0.4) + 4.0 : rounds * (per * step[i] + 4.0);
      // (the adding kernel has eight segments or sixteen chunks on their way at a time)
      if (form) cost += 3.0 + 8.0 * parts * (double)M * N / 3e6 + 1.5 * (unit == 1 ? (parts + 15) / 16 : (parts + 7) / 8);
      if (best < 0 || cost < best) {
        best = cost;
        pl.nr = nr; pl.splits = form ? splits : 1; pl.kb_per_split = per;
        pl.part_shift = unit == 1 ? 0 : 2; pl.parts = parts;
        pl.tiles_m = (int)mt; pl.items = (int)(tiles * splits);
      }
    }
  }
  return best >= 0;
}

template <int NR, bool SPLIT>
static int launch_lf(const LfParams& p, cudaStream_t st) {
  auto kern = linear_f32_tc_kernel<NR, SPLIT>;
  constexpr int smem = LfShape<NR>::SMEM;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return (int)e;
  const int sms = hs_sm_count();
  e = hs_launch(kern, dim3(p.items < sms ? p.items : sms), dim3(LF_THREADS), (size_t)smem, st,
                hs_pdl_enabled(), p);
  if (e != cudaSuccess) return (int)e;
  if (SPLIT) {
    const long long size = (long long)p.M * p.N;
    e = hs_launch(linear_f32_tc_sum_kernel, dim3((unsigned)((size + 127) / 128)), dim3(128), 0, st,
                  hs_pdl_enabled(), p);
  }
  return e == cudaSuccess ? HS_OK : (int)e;
}

}  // namespace hs

// Floats of scratch a launch needs (0: none); HS_ERR_UNSUPPORTED for shapes it does not take.
HS_EXPORT int hs_linear_f32_tc_scratch(int M, int N, int K, int rows, long long* floats) {
  hs::LfPlan pl;
  if (!hs::plan_lf(M, N, K, rows, pl)) return HS_ERR_UNSUPPORTED;
  *floats = pl.splits > 1 ? (long long)pl.parts * M * N : 0;
  return HS_OK;
}

// rows: of `a` a tile takes (16, 32, 64, 128; 0: decided here).  Refuses (HS_ERR_UNSUPPORTED) by N, K and
// alignment alone, never by M: a row's bits do not depend on its batch.
HS_EXPORT int hs_linear_f32_tc(float* out, const float* a, const float* w, const float* bias,
                               const float* residual, int M, int N, int K, int act, float act_a,
                               float act_b, int rows, float* scratch, int* status, void* stream) {
  using namespace hs;
  if (!out || !a || !w || !status) return HS_ERR_ARGUMENT;
  if (M <= 0 || N <= 0) return HS_OK;
  if (act < HS_ACT_NONE || act > HS_ACT_LAST) return HS_ERR_UNSUPPORTED;
  if (((uintptr_t)a | (uintptr_t)w) & 15) return HS_ERR_UNSUPPORTED;
  LfPlan pl;
  if (!plan_lf(M, N, K, rows, pl)) return HS_ERR_UNSUPPORTED;
  if (pl.splits > 1 && !scratch) return HS_ERR_ARGUMENT;
  LfParams p;
  p.out = out; p.a = a; p.w = w; p.bias = bias; p.residual = residual; p.partial = scratch; p.status = status;
  p.M = M; p.N = N; p.K = K; p.act = act; p.act_ab = make_float2(act_a, act_b);
  p.tiles_m = pl.tiles_m; p.parts = pl.parts; p.splits = pl.splits;
  p.kb_per_split = pl.kb_per_split; p.part_shift = pl.part_shift; p.items = pl.items;
  cudaStream_t st = (cudaStream_t)stream;
#define HS_LF(NR) (pl.splits > 1 ? launch_lf<NR, true>(p, st) : launch_lf<NR, false>(p, st))
  switch (pl.nr) {
    case 16: return HS_LF(16);
    case 32: return HS_LF(32);
    case 64: return HS_LF(64);
    default: return HS_LF(128);
  }
#undef HS_LF
}
