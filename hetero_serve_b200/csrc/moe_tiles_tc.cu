// Tiles of the routed feed-forward on the 5th-generation tensor cores (tcgen05): the pairs of a step
// sorted by expert (moe.cu), tiles of one expert's rows.
//
// The weight tile is the operand of 128 rows (output features) and the pairs are the columns:
// D[feature, pair] in tensor memory, so a tile takes as many pairs as the expert's segment leaves it
// (16 .. 128 or 256, in steps of 16) and short segments cost no padded MMAs.
//
//   gate/up   D_gate and D_up [128 x n], n <= 256 pairs: one copy of the gathered rows serves both
//             products, and a thread finds gate and up of a feature in its own lane: the activation
//             needs no exchange.  Rows of the step's tokens are gathered by cp.async (a TMA copy of
//             few rows costs what one of 128 does).
//   down      two accumulators D [128 x n], n <= 256 pairs: the epilogue of one tile runs under the
//             products of the next; the activated rows lie in expert order: TMA.
//
// Persistent blocks, one an SM: eight warps drain the accumulator, four gather rows (gate/up), one issues
// TMA copies, one MMAs.  The ring holds as many stages of 64 over the summed index as the step's widest
// tile leaves room for (three to six).  2,048 tokens, 32 experts of 512, four a token, weights from DRAM (100 MB): gate
// and up 32 us, down 16, against 93 and 56 with 64 x 64 tiles on mma.sync; 64 tokens 30 us in all against
// 67 (a kernel for few pairs a tile is not needed).  The floor is the weights: 15 us.
//
// Every wait is bounded (tcgen05.cuh); a wait that runs out sets the status bit, its warp leaves, and the issuing
// warp goes on with waits that look once, then waits for the MMAs it has issued.
#include "tcgen05.cuh"
#include "moe_tiles_tc.cuh"

namespace hs {

constexpr int MT_BM = 128;            // features of a tile
constexpr int MT_BK = 64;             // 128 bytes: a swizzle row
constexpr int MT_EPI_WARPS = 8, MT_LOAD_WARPS = 4;
constexpr int MT_MAX_STAGES = 6;
constexpr int MT_RING = 204 * 1024;
constexpr int MT_SMEM = MT_RING + 1024;

struct MtParams {
  void* out;                          // [pairs, N] rows in expert order
  const __nv_bfloat16* a;             // GATHER: the tokens' rows
  const int* tiles;
  const int* row_token;
  int* status;
  int N, K, f_tiles, act;
  float limit;
};

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}

// 1 / d and n / d for 1 <= d <= 2^126: an approximate value and one correction by its remainder (Markstein's
// theorem), without the branch of the division, which keeps sixteen chains from running side by side (2,048
// tokens, 32 experts: 106 us with it, 94 so).  Checked over all floats g: silu and the clamped gate are those
// of expert_act, but for the last bit of one.
__device__ __forceinline__ float near_reciprocal(float d) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
  return r;
}
__device__ __forceinline__ float reciprocal(float d) {
  const float r = near_reciprocal(d);
  return fmaf(fmaf(-r, d, 1.0f), r, r);
}
__device__ __forceinline__ float quotient(float n, float d) {
  const float r = near_reciprocal(d), q = n * r;
  return fabsf(q) <= 3.402823466e38f ? fmaf(fmaf(-q, d, n), r, q) : q;
}
// what the gate's exponential is formed of, and below which its sum with 1 may leave quotient's range
template <int ACT>
__device__ __forceinline__ float gate_argument(float g, float limit) { return ACT == 1 ? g : 1.702f * fminf(g, limit); }
constexpr float GATE_LOW = -87.f;
// expert_act for gate arguments from GATE_LOW up
template <int ACT>
__device__ __forceinline__ float expert_act_near(float g, float u, float limit) {
  const float d = 1.0f + expf(-gate_argument<ACT>(g, limit));
  if (ACT == 1) return quotient(g, d) * u;
  return fminf(g, limit) * reciprocal(d) * (fminf(fmaxf(u, -limit), limit) + 1.0f);
}
template <int ACT>
__device__ __noinline__ float expert_act_low(float g, float u, float limit) { return expert_act<ACT>(g, u, limit); }
// sixteen features' activations; one branch for all of them
template <int ACT, bool GATED>
__device__ __forceinline__ void expert_acts(float (&v)[16], const uint32_t (&u)[16], float limit) {
  float least[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) least[j] = fminf(v[j], v[j + 8]);
#pragma unroll
  for (int n = 4; n; n >>= 1)
#pragma unroll
    for (int j = 0; j < n; ++j) least[j] = fminf(least[j], least[j + n]);
  const bool low = gate_argument<ACT>(least[0], limit) < GATE_LOW;
  if (ACT == 2) {
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = expert_act<ACT>(v[j], v[j], limit);
  } else if (low) {
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = expert_act_low<ACT>(v[j], GATED ? __uint_as_float(u[j]) : v[j], limit);
  } else {
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = expert_act_near<ACT>(v[j], GATED ? __uint_as_float(u[j]) : v[j], limit);
  }
}

// NB weight matrices against the same rows (2: gate and up).  ACT: rows leave activated in bfloat16,
// else as float32 sums.  GATHER: rows of `a` through row_token, else rows of map_a in order.
template <int NB, bool GATHER, bool ACT>
__global__ void __launch_bounds__(32 * (MT_EPI_WARPS + (GATHER ? MT_LOAD_WARPS : 0) + 2), 1)
moe_tiles_tc_kernel(const __grid_constant__ CUtensorMap map_w0,
                    const __grid_constant__ CUtensorMap map_w1,
                    const __grid_constant__ CUtensorMap map_a32,
                    const __grid_constant__ CUtensorMap map_a128, const MtParams p) {
  constexpr int W_BYTES = MT_BM * MT_BK * 2;
  constexpr int NACC = NB == 2 ? 1 : 2;
  constexpr int TMA_WARP = MT_EPI_WARPS + (GATHER ? MT_LOAD_WARPS : 0), MMA_WARP = TMA_WARP + 1;
  extern __shared__ uint8_t mt_smem[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)mt_smem + 1023) & ~(uintptr_t)1023);
  __shared__ uint64_t full_bar[MT_MAX_STAGES], empty_bar[MT_MAX_STAGES], acc_full[2], acc_empty[2], drain_bar;
  __shared__ uint32_t tmem_slot;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  pdl_trigger();
  if (threadIdx.x == 0) {
    for (int s = 0; s < MT_MAX_STAGES; ++s) {
      mbar_init(&full_bar[s], GATHER ? 1 + 32 * MT_LOAD_WARPS : 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&acc_full[a], 1);
      mbar_init(&acc_empty[a], MT_EPI_WARPS);
    }
    mbar_init(&drain_bar, 1);
    fence_barrier_init();
  }
  if (warp == MMA_WARP) {
    tmem_alloc(&tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  pdl_wait();
  const int n_items = p.tiles[0] * p.f_tiles;
  const int stage_bytes = NB * W_BYTES + (GATHER ? p.tiles[1] : (p.tiles[1] + 127) & ~127) * MT_BK * 2;
  const int stages = min(MT_MAX_STAGES, MT_RING / stage_bytes);
  const int num_kb = (p.K + MT_BK - 1) / MT_BK;

  if (warp == TMA_WARP) {
    if (lane == 0) {
      bool ok = true;
      int s = 0, round = 0;
      for (int w = blockIdx.x; w < n_items && ok; w += gridDim.x) {
        const int tile = w / p.f_tiles, f0 = (w - tile * p.f_tiles) * MT_BM;
        const int e = p.tiles[2 + 3 * tile], row0 = p.tiles[3 + 3 * tile], rows = p.tiles[4 + 3 * tile];
        // rows a copy brings: one box of 32, or boxes of 128
        const int boxes = rows <= 32 ? 1 : (rows + 127) / 128;
        const uint32_t bytes = NB * W_BYTES + (GATHER ? 0 : boxes * (rows <= 32 ? 32 : 128) * MT_BK * 2);
        for (int kb = 0; kb < num_kb; ++kb) {
          if (round > 0) ok = mbar_wait(&empty_bar[s], (round - 1) & 1, p.status);
          if (!ok) break;
          uint8_t* dst = smem + s * stage_bytes;
          mbar_expect_tx(&full_bar[s], bytes);
          tma_load_2d(dst, &map_w0, &full_bar[s], kb * MT_BK, e * p.N + f0);
          if (NB == 2) tma_load_2d(dst + W_BYTES, &map_w1, &full_bar[s], kb * MT_BK, e * p.N + f0);
          if (!GATHER) {
            uint8_t* rows_dst = dst + NB * W_BYTES;
            if (rows <= 32)
              tma_load_2d(rows_dst, &map_a32, &full_bar[s], kb * MT_BK, row0);
            else
              for (int b = 0; b < boxes; ++b)
                tma_load_2d(rows_dst + b * 128 * MT_BK * 2, &map_a128, &full_bar[s], kb * MT_BK,
                            row0 + b * 128);
          }
          if (++s == stages) { s = 0; ++round; }
        }
      }
    }
  } else if (warp == MMA_WARP) {
    uint32_t limit = HS_SPIN_LIMIT;
    int s = 0, round = 0, wi = 0;
    for (int w = blockIdx.x; w < n_items; w += gridDim.x, ++wi) {
      const int rows = p.tiles[4 + 3 * (w / p.f_tiles)];
      const uint32_t idesc = make_idesc(MT_BM, (rows + 15) & ~15);
      const int acc = wi % NACC, acc_round = wi / NACC;
      if (acc_round > 0) mbar_wait_warp(&acc_empty[acc], (acc_round - 1) & 1, p.status, limit);
      tc_fence_after();
      const uint32_t d = tmem + acc * 256;
      for (int kb = 0; kb < num_kb; ++kb) {
        mbar_wait_warp(&full_bar[s], round & 1, p.status, limit);
        if (GATHER) fence_proxy_async();     // rows the loading threads' copies wrote
        tc_fence_after();
        const uint32_t base = smem_u32(smem + s * stage_bytes);
        const uint64_t wdesc = make_smem_desc(base), bdesc = make_smem_desc(base + NB * W_BYTES);
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < MT_BK / 16; ++k) {
            const uint32_t more = (kb > 0 || k > 0) ? 1u : 0u;
            umma_bf16(d, wdesc + 2 * k, bdesc + 2 * k, idesc, more);
            if (NB == 2) umma_bf16(d + 256, wdesc + (W_BYTES >> 4) + 2 * k, bdesc + 2 * k, idesc, more);
          }
          umma_commit(&empty_bar[s]);
        }
        __syncwarp();
        if (++s == stages) { s = 0; ++round; }
      }
      if (elect_one()) umma_commit(&acc_full[acc]);
      __syncwarp();
    }
    umma_drain(&drain_bar, limit, p.status);
  } else if (GATHER && warp >= MT_EPI_WARPS) {
    // a piece of 16 bytes is column c of its row, rows r0, r0 + 16, ..; a row beyond the segment, and
    // numbers beyond K, are zeros.  Each thread's copies arrive at the stage's barrier when they have
    // landed, so every stage of the ring can be in flight.
    constexpr int STEP = MT_LOAD_WARPS * 4, MAX_ROWS = MT_PAIRS / STEP;
    const int t = threadIdx.x - MT_EPI_WARPS * 32;
    const int c = t & 7, r0 = t >> 3;
    const uint32_t dst0 = smem_u32(smem) + NB * W_BYTES + r0 * 128 + ((c ^ (r0 & 7)) << 4);
    bool ok = true;
    int s = 0, round = 0;
    for (int w = blockIdx.x; w < n_items && ok; w += gridDim.x) {
      const int tile = w / p.f_tiles;
      const int row0 = p.tiles[3 + 3 * tile], rows = p.tiles[4 + 3 * tile], cols = (rows + 15) & ~15;
      const __nv_bfloat16* src[MAX_ROWS];
#pragma unroll
      for (int i = 0; i < MAX_ROWS; ++i) {
        const int r = r0 + i * STEP;
        src[i] = r < rows ? p.a + (size_t)p.row_token[row0 + r] * p.K : nullptr;
      }
      for (int kb = 0; kb < num_kb; ++kb) {
        if (round > 0) ok = mbar_wait(&empty_bar[s], (round - 1) & 1, p.status);
        if (!ok) break;
        const int k = kb * MT_BK + c * 8;
        const uint32_t dst = dst0 + s * stage_bytes;
#pragma unroll
        for (int i = 0; i < MAX_ROWS; ++i)
          if (i * STEP < cols) {
            const bool have = src[i] != nullptr && k < p.K;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + i * STEP * 128),
                         "l"(have ? src[i] + k : p.a), "r"(have ? 16 : 0) : "memory");
          }
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&full_bar[s]))
                     : "memory");
        if (++s == stages) { s = 0; ++round; }
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else {
    // ---- epilogue: warp w owns lanes 32 (w % 4) .. of the accumulator, 16 pairs at a time, the two
    // warps of a quarter in turn
    const int q = warp & 3, half = warp >> 2;
    int wi = 0;
    for (int w = blockIdx.x; w < n_items; w += gridDim.x, ++wi) {
      const int tile = w / p.f_tiles, f = (w - tile * p.f_tiles) * MT_BM + q * 32 + lane;
      const int row0 = p.tiles[3 + 3 * tile], rows = p.tiles[4 + 3 * tile];
      const int acc = wi % NACC;
      if (!mbar_wait(&acc_full[acc], (wi / NACC) & 1, p.status)) break;
      tc_fence_after();
      const uint32_t t_addr = tmem + acc * 256 + ((uint32_t)(q * 32) << 16);
      for (int c0 = half * 16; c0 < rows; c0 += 32) {
        uint32_t g[16], u[16];
        tmem_ld16(t_addr + c0, g);
        if (NB == 2) tmem_ld16(t_addr + 256 + c0, u);
        tmem_ld_wait();
        float v[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(g[j]);
        if (ACT) {
          if (p.act == 0) expert_acts<0, NB == 2>(v, u, p.limit);
          else if (p.act == 1) expert_acts<1, NB == 2>(v, u, p.limit);
          else expert_acts<2, NB == 2>(v, u, p.limit);
        }
        const int n = f < p.N ? rows - c0 : 0;
        const size_t at = (size_t)(row0 + c0) * p.N + f;
        if (n >= 16) {
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (ACT) ((__nv_bfloat16*)p.out)[at + (size_t)j * p.N] = __float2bfloat16_rn(v[j]);
            else ((float*)p.out)[at + (size_t)j * p.N] = v[j];
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (j < n) {
              if (ACT) ((__nv_bfloat16*)p.out)[at + (size_t)j * p.N] = __float2bfloat16_rn(v[j]);
              else ((float*)p.out)[at + (size_t)j * p.N] = v[j];
            }
        }
        __syncwarp();
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[acc]);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == MMA_WARP) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// a [rows, K] bfloat16 matrix, boxes of [box_rows x 64], 128-byte swizzle
static int mt_map(CUtensorMap* map, const void* base, long long rows, int K, int box_rows) {
  typedef CUresult (*Encode)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                             const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                             CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                             CUtensorMapFloatOOBfill);
  static const Encode enc = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      f = nullptr;
    return (Encode)f;
  }();
  if (!enc) return HS_ERR_UNSUPPORTED;
  cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)K * 2};
  cuuint32_t box[2] = {(cuuint32_t)MT_BK, (cuuint32_t)box_rows}, elem[2] = {1, 1};
  const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides,
                         box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? HS_OK : HS_ERR_UNSUPPORTED;
}

template <int NB, bool GATHER, bool ACT>
static int mt_launch(const CUtensorMap& w0, const CUtensorMap& w1, const CUtensorMap& a32,
                     const CUtensorMap& a128, const MtParams& p, long long items, cudaStream_t st) {
  auto kern = moe_tiles_tc_kernel<NB, GATHER, ACT>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, MT_SMEM);
  if (e != cudaSuccess) return (int)e;
  const int sms = hs_sm_count();
  e = hs_launch(kern, dim3(items < sms ? (unsigned)items : sms),
                dim3(32 * (MT_EPI_WARPS + (GATHER ? MT_LOAD_WARPS : 0) + 2)), (size_t)MT_SMEM, st,
                hs_pdl_enabled(), w0, w1, a32, a128, p);
  return e == cudaSuccess ? HS_OK : (int)e;
}

int moe_tiles_tc(__nv_bfloat16* act_rows, float* down_rows, const __nv_bfloat16* h,
                 const __nv_bfloat16* w_gate, const __nv_bfloat16* w_up, const __nv_bfloat16* w_down,
                 const int* tiles, int max_tiles, const int* row_token, int pairs, int width, int ff, int E, float limit, int act,
                 int* status, cudaStream_t st) {
  for (const void* q : {(const void*)h, (const void*)w_gate, (const void*)w_up, (const void*)w_down,
                        (const void*)act_rows})
    if ((uintptr_t)q & 15) return HS_ERR_UNSUPPORTED;
  CUtensorMap up, gate, down, a32, a128;
  if (int e = mt_map(&up, w_up, (long long)E * ff, width, MT_BM)) return e;
  gate = up;
  if (w_gate)
    if (int e = mt_map(&gate, w_gate, (long long)E * ff, width, MT_BM)) return e;
  if (int e = mt_map(&down, w_down, (long long)E * width, ff, MT_BM)) return e;
  if (int e = mt_map(&a32, act_rows, pairs, ff, 32)) return e;
  if (int e = mt_map(&a128, act_rows, pairs, ff, 128)) return e;
  MtParams p;
  p.out = act_rows; p.a = h; p.tiles = tiles; p.row_token = row_token; p.status = status;
  p.N = ff; p.K = width; p.f_tiles = (ff + MT_BM - 1) / MT_BM; p.act = act; p.limit = limit;
  const long long up_items = (long long)max_tiles * p.f_tiles;
  if (int e = w_gate ? mt_launch<2, true, true>(gate, up, a32, a128, p, up_items, st)
                     : mt_launch<1, true, true>(up, up, a32, a128, p, up_items, st))
    return e;
  p.out = down_rows; p.a = nullptr;
  p.N = width; p.K = ff; p.f_tiles = (width + MT_BM - 1) / MT_BM;
  return mt_launch<1, false, false>(down, down, a32, a128, p, (long long)max_tiles * p.f_tiles, st);
}

}  // namespace hs
