// A float32-accumulating linear layer on the CUDA cores (FFMA), for shapes and operands that the
// tensor-core kernels refuse (linear_f32_tc.cu, linear_tcgen05.cu) and where they are switched off.
//
//   out[m, n] = act( sum_k a[m, k] * w[n, k] + bias[n] ) (+ residual[m, n])
//
// `w` is [N, K] with K contiguous (Conv1D weights, stored [in, out], are transposed once when
// they are bound; the tied head uses the token table as it is).  Reference call sites:
// `h @ attn_w + attn_b`, `x + (attn @ proj_w + proj_b)`, `gelu(x @ fc_w + fc_b) @ fcp_w + fcp_b`,
// `ln_f(x) @ wte.T` (heteroserve/model/torch_engine.py:77-79,86-87,122,139).
//
// Every output element is one chain of fused multiply-adds over k = 0..K-1 in index order,
// whatever M is and wherever the row sits in its tile: a row's result does not depend on
// the batch it is computed in.  No tensor cores, no TF32, no split over K.
#include "tcgen05.cuh"

namespace hs {

// four consecutive elements of a row in one load (the rows are 16-byte / 8-byte aligned there)
__device__ __forceinline__ void ls_load4(const float* p, float (&v)[4]) {
  const float4 x = *(const float4*)p;
  v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
}
__device__ __forceinline__ void ls_load4(const __nv_bfloat16* p, float (&v)[4]) {
  const uint2 x = *(const uint2*)p;
  v[0] = __uint_as_float(x.x << 16); v[1] = __uint_as_float(x.x & 0xffff0000u);
  v[2] = __uint_as_float(x.y << 16); v[3] = __uint_as_float(x.y & 0xffff0000u);
}

__device__ __forceinline__ void ls_store4(float* p, const float (&v)[4]) {
  *(float4*)p = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void ls_store4(__nv_bfloat16* p, const float (&v)[4]) {
  const __nv_bfloat162 a = __floats2bfloat162_rn(v[0], v[1]), b = __floats2bfloat162_rn(v[2], v[3]);
  *(uint2*)p = make_uint2(*(const uint32_t*)&a, *(const uint32_t*)&b);
}

// Where lanes read 16 bytes each and share addresses, a warp's read takes two wavefronts of shared
// memory when the lanes of a pair (2i, 2i + 1) or all but every eighth agree, and four otherwise
// (counted: lane % 8 -> four, (lane >> 1) & 7 -> two).  So eight columns go to lane bits 1-3 and
// four rows to bits 0 and 4.
__device__ __forceinline__ int ls_col(int lane) { return (lane >> 1) & 7; }
__device__ __forceinline__ int ls_row(int lane) { return (lane & 1) | ((lane >> 3) & 2); }

// Two fused multiply-adds in one instruction, each rounded as fmaf rounds (fma.rn.f32x2): half as
// many issue slots go to the products.
__device__ __forceinline__ void fma2(uint64_t& acc, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ uint64_t twice(float a) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(a));
  return r;
}

// ---- many rows (prompts): tiles of 64 x 64 outputs (H = 2) or 32 x 32 (H = 1) -----------------
// A CTA is two warps, a thread owns a patch of 8 x 8 (4 x 4) outputs; several CTAs share an SM, so
// the tiles of a layer spread evenly (1,024 x 1,024 outputs are 64 tiles of 128 x 128, which left
// 84 of 148 SMs idle) and one CTA's products cover another's loads and barriers.  Both operands are kept k-major ([k][row]), a
// row's column XORed with a multiple of four that depends on k, so that neither the 4-byte stores
// nor the 16-byte reads meet a bank conflict.  32-bit operands are scattered there by 4-byte
// cp.async copies through a ring of LT_STAGES stages of 8 k (fetched through registers, one stage
// ahead, the L2's latency was exposed in every stage); bfloat16 ones go through registers.
// Measured (float32, one B200, before -> now; the form before fetched 128 x 128 tiles through
// registers and used single FMAs): 2,048 x 4,096 x 1,024 485 -> 384 us (44.8 TFLOP/s, FMA pipe 62 %
// busy, shared-memory pipe 62 %), 1,024 x 1,024 x 4,096 632 -> 316 us, 256 x 1,024 x 4,096 660 -> 163.
constexpr int LT_BK = 8, LT_THREADS = 64, LT_STAGES = 4;

__device__ __forceinline__ int lt_swizzle(int k) { return (k & 7) << 2; }

// LOAD: 2 (32-bit operands): asynchronous copies; 1: K is a multiple of 4 and both matrices start on
// an 8-byte (32-bit: 16-byte) boundary, so a thread's four k of a row come in one load; 0: any.
template <typename TI, typename TO, int H, int LOAD>
__global__ void __launch_bounds__(LT_THREADS)
linear_simt_tile_kernel(TO* out, const TI* __restrict__ a, const TI* __restrict__ w,
                        const float* __restrict__ bias, const float* residual, int M, int N, int K,
                        int act, float2 ab) {
  constexpr int LT_BM = 32 * H, LT_BN = 32 * H, P = 4 * H;
  constexpr int BUFS = LOAD == 2 ? LT_STAGES : 2;
  __shared__ __align__(16) float As[BUFS][LT_BK][LT_BM];
  __shared__ __align__(16) float Ws[BUFS][LT_BK][LT_BN];
  const int tid = threadIdx.x, lane = tid & 31;
  const int tx = ls_col(lane), ty = ls_row(lane) | ((tid >> 5) << 2);
  const int m0 = blockIdx.y * LT_BM, n0 = blockIdx.x * LT_BN;
  uint64_t acc[P][P / 2];
#pragma unroll
  for (int i = 0; i < P; ++i)
#pragma unroll
    for (int j = 0; j < P / 2; ++j) acc[i][j] = 0;

  auto products = [&](int buf) {
#pragma unroll
    for (int kk = 0; kk < LT_BK; ++kk) {
      // rows ty*4..+3 and columns tx*4..+3 of each half
      const int sx = lt_swizzle(kk);
      float av[P];
      uint64_t wv[P / 2];
#pragma unroll
      for (int u = 0; u < H; ++u) {
        const float4 x = *(const float4*)&As[buf][kk][32 * u + ((ty * 4) ^ sx)];
        const ulonglong2 y = *(const ulonglong2*)&Ws[buf][kk][32 * u + ((tx * 4) ^ sx)];
        av[4 * u] = x.x; av[4 * u + 1] = x.y; av[4 * u + 2] = x.z; av[4 * u + 3] = x.w;
        wv[2 * u] = y.x; wv[2 * u + 1] = y.y;
      }
#pragma unroll
      for (int i = 0; i < P; ++i) {
        const uint64_t a2 = twice(av[i]);
#pragma unroll
        for (int j = 0; j < P / 2; ++j) fma2(acc[i][j], a2, wv[j]);
      }
    }
  };
  // rows past the last one repeat it (their outputs are never stored); k past the end is zero
  if constexpr (LOAD == 2) {
    // a warp copies the eight k of four rows at a time: thread -> k, rows lr + 8 i
    const int lk = tid & 7, lr = tid >> 3;
    const int n_kt = (K + LT_BK - 1) / LT_BK;
    uint32_t sa[2];
    sa[0] = (uint32_t)__cvta_generic_to_shared(&As[0][lk][0]);
    sa[1] = (uint32_t)__cvta_generic_to_shared(&Ws[0][lk][0]);
    int row_a[4 * H], row_w[4 * H];                       // offsets of the rows from the tile's first
#pragma unroll
    for (int i = 0; i < 4 * H; ++i) {
      row_a[i] = min(lr + 8 * i, M - 1 - m0) * K;
      row_w[i] = min(lr + 8 * i, N - 1 - n0) * K;
    }
    const TI* a_t = a + (size_t)m0 * K;
    const TI* w_t = w + (size_t)n0 * K;
    auto issue = [&](int kt) {
      if (kt < n_kt) {
        const int gk = kt * LT_BK + lk;
        const int n = gk < K ? 4 : 0;
        const int ck = gk < K ? gk : 0;
        const uint32_t to = (uint32_t)((kt % LT_STAGES) * LT_BK * LT_BM * 4);
#pragma unroll
        for (int i = 0; i < 4 * H; ++i) {
          const uint32_t col = (uint32_t)((((lr + 8 * i) & 31) ^ lt_swizzle(lk)) + (i >= 4 ? 32 : 0)) * 4;
          asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(sa[0] + to + col),
                       "l"(a_t + row_a[i] + ck), "r"(n) : "memory");
          asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(sa[1] + to + col),
                       "l"(w_t + row_w[i] + ck), "r"(n) : "memory");
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int s = 0; s < LT_STAGES - 1; ++s) issue(s);
#pragma unroll 1
    for (int kt = 0; kt < n_kt; ++kt) {
      asm volatile("cp.async.wait_group %0;" ::"n"(LT_STAGES - 2) : "memory");
      __syncthreads();               // stage kt has landed; stage kt - 1 is free for every thread
      issue(kt + LT_STAGES - 1);
      products(kt % LT_STAGES);
    }
  } else {
    // thread -> row lr of each half, four consecutive k of the 8
    const int lr = tid >> 1, lk = (tid & 1) * 4;
    const TI *ap[H], *wp[H];
    float ra[H][4], rw[H][4];
#pragma unroll
    for (int i = 0; i < H; ++i) {
      ap[i] = a + (size_t)min(m0 + lr + 32 * i, M - 1) * K;
      wp[i] = w + (size_t)min(n0 + lr + 32 * i, N - 1) * K;
    }
    auto fetch = [&](int k0) {
      const int gk = k0 + lk;
#pragma unroll
      for (int i = 0; i < H; ++i) {
        if (LOAD == 1) {
#pragma unroll
          for (int j = 0; j < 4; ++j) ra[i][j] = rw[i][j] = 0.f;
          if (gk < K) {                                   // K % 4 == 0: all four or none
            ls_load4(ap[i] + gk, ra[i]);
            ls_load4(wp[i] + gk, rw[i]);
          }
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            ra[i][j] = gk + j < K ? to_f(ap[i][gk + j]) : 0.f;
            rw[i][j] = gk + j < K ? to_f(wp[i][gk + j]) : 0.f;
          }
        }
      }
    };
    auto stash = [&](int buf) {
#pragma unroll
      for (int i = 0; i < H; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          As[buf][lk + j][(lr ^ lt_swizzle(lk + j)) + 32 * i] = ra[i][j];
          Ws[buf][lk + j][(lr ^ lt_swizzle(lk + j)) + 32 * i] = rw[i][j];
        }
    };
    fetch(0);
    stash(0);
    __syncthreads();
    int buf = 0;
#pragma unroll 1
    for (int k0 = 0; k0 < K; k0 += LT_BK) {
      const bool more = k0 + LT_BK < K;
      if (more) fetch(k0 + LT_BK);                        // in flight during the products below
      products(buf);
      if (more) {
        stash(buf ^ 1);
        __syncthreads();
        buf ^= 1;
      }
    }
  }
  // four neighbouring columns a store where every row of the outputs allows it
  const bool wide = N % 4 == 0 && !((uintptr_t)out & (4 * sizeof(TO) - 1)) && !((uintptr_t)residual & 15);
#pragma unroll
  for (int i = 0; i < P; ++i) {
    const int gm = m0 + 32 * (i >> 2) + ty * 4 + (i & 3);
    if (gm >= M) continue;
    if (wide) {
#pragma unroll
      for (int u = 0; u < H; ++u) {
        const int gn = n0 + 32 * u + tx * 4;
        if (gn >= N) continue;
        const size_t at = (size_t)gm * N + gn;
        float v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          v[j] = __uint_as_float((uint32_t)(acc[i][2 * u + (j >> 1)] >> ((j & 1) * 32)));
          if (bias) v[j] += bias[gn + j];
          v[j] = apply_act(v[j], act, ab);
        }
        if (residual) {
          const float4 r = *(const float4*)(residual + at);
          v[0] += r.x; v[1] += r.y; v[2] += r.z; v[3] += r.w;
        }
        ls_store4(out + at, v);
      }
      continue;
    }
#pragma unroll
    for (int j = 0; j < P; ++j) {
      const int gn = n0 + 32 * (j >> 2) + tx * 4 + (j & 3);
      if (gn >= N) continue;
      float v = __uint_as_float((uint32_t)(acc[i][j >> 1] >> ((j & 1) * 32)));
      if (bias) v += bias[gn];
      v = apply_act(v, act, ab);
      if (residual) v += residual[(size_t)gm * N + gn];
      out[(size_t)gm * N + gn] = from_f<TO>(v);
    }
  }
}

// ---- bfloat16, many large tiles: 128 x 128 outputs, an 8 x 8 patch per thread ------------------
// The same chains again.  bfloat16 operands reach the tiles above through registers, one stage of 8 k
// ahead, and their two warps wait for the L2 in every stage; eight warps on a tile twice as wide share
// one such wait, two tiles an SM.  The wider tile pays where it fills the device (see the launch).
constexpr int LB_BM = 128, LB_BN = 128, LB_BK = 8, LB_THREADS = 256;

// VEC: K is a multiple of 4 and both matrices start on a 16-byte boundary, so a thread's four
// k of a row come in one load (with one 4-byte load per element the load pipe, 16 sectors an
// instruction, took as long as the products).
template <typename TI, typename TO, bool VEC>
__global__ void __launch_bounds__(LB_THREADS)
linear_simt_big_kernel(TO* out, const TI* __restrict__ a, const TI* __restrict__ w,
                       const float* __restrict__ bias, const float* residual, int M, int N, int K,
                       int act, float2 ab) {
  __shared__ __align__(16) float As[2][LB_BK][LB_BM];
  __shared__ __align__(16) float Ws[2][LB_BK][LB_BN];
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;                 // 16 x 16 threads, 8 x 8 outputs each
  const int m0 = blockIdx.y * LB_BM, n0 = blockIdx.x * LB_BN;
  // loader: thread -> (row 0..127, 4 consecutive k of the 8)
  const int lr = tid >> 1, lk = (tid & 1) * 4;
  float acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
  float ra[4], rw[4];
  auto fetch = [&](int k0) {
    const int gm = m0 + lr, gn = n0 + lr;
    if (VEC) {
      const int gk = k0 + lk;                             // K % 4 == 0: all four or none
#pragma unroll
      for (int j = 0; j < 4; ++j) ra[j] = rw[j] = 0.f;
      if (gm < M && gk < K) ls_load4(a + (size_t)gm * K + gk, ra);
      if (gn < N && gk < K) ls_load4(w + (size_t)gn * K + gk, rw);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int gk = k0 + lk + j;
        ra[j] = (gm < M && gk < K) ? to_f(a[(size_t)gm * K + gk]) : 0.f;
        rw[j] = (gn < N && gk < K) ? to_f(w[(size_t)gn * K + gk]) : 0.f;
      }
    }
  };
  auto stash = [&](int buf) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      As[buf][lk + j][lr] = ra[j];
      Ws[buf][lk + j][lr] = rw[j];
    }
  };
  fetch(0);
  stash(0);
  __syncthreads();
  int buf = 0;
  for (int k0 = 0; k0 < K; k0 += LB_BK) {
    const bool more = k0 + LB_BK < K;
    if (more) fetch(k0 + LB_BK);                          // in flight during the products below
#pragma unroll
    for (int kk = 0; kk < LB_BK; ++kk) {
      // rows ty*4..+3 and 64+ty*4..+3, columns tx*4..+3 and 64+tx*4..+3: 16-byte reads, no
      // bank conflicts
      const float4 a0 = *(const float4*)&As[buf][kk][ty * 4];
      const float4 a1 = *(const float4*)&As[buf][kk][64 + ty * 4];
      const float4 w0 = *(const float4*)&Ws[buf][kk][tx * 4];
      const float4 w1 = *(const float4*)&Ws[buf][kk][64 + tx * 4];
      const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
      const float wv[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(av[i], wv[j], acc[i][j]);
    }
    if (more) {
      stash(buf ^ 1);
      __syncthreads();
      buf ^= 1;
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int gm = m0 + (i < 4 ? ty * 4 + i : 64 + ty * 4 + (i - 4));
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int gn = n0 + (j < 4 ? tx * 4 + j : 64 + tx * 4 + (j - 4));
      if (gn >= N) continue;
      float v = acc[i][j];
      if (bias) v += bias[gn];
      v = apply_act(v, act, ab);
      if (residual) v += residual[(size_t)gm * N + gn];
      out[(size_t)gm * N + gn] = from_f<TO>(v);
    }
  }
}

// ---- few rows (decode): the same chains, laid out for a weight stream -------------------------
// An output is one chain of K dependent FMAs, so no layout is through before 4 K cycles (2.1 us
// at K = 1,024); what a layout can do is to keep that chain fed.  A CTA owns F features.  Lane
// (f, g) of a consumer warp runs the chains of RPT rows (g, g + G, ...) for feature f.  One more
// warp fetches: weight and activation rows arrive in stages of BK k through a ring of 16-byte
// cp.async copies that arrive on an mbarrier (the copies' addresses and issue slots, in the
// consumers' own instruction stream, took longer than the chain).  Rows are padded by 16 bytes
// against bank conflicts; the operands of the next 16 (8) k are read from shared memory while this
// set's chains run.  Measured (float32, M x N x K, before -> now): 8 x 1,024 x 4,096 53.5 -> 19.3 us,
// 8 x 3,072 x 1,024 17.9 -> 11.2, 64 x 4,096 x 1,024 45.9 -> 28.3, 8 x 50,257 x 1,024 146 -> 88.
template <typename TI, int RPT, int F, int WARPS>
struct LfShape {
  static constexpr int G = 32 / F * WARPS;                   // row groups
  static constexpr int ROWS = G * RPT;
  static constexpr int BK = ROWS <= 16 ? 128 : 64;           // k per stage
  static constexpr int VEC = 16 / (int)sizeof(TI);           // elements per 16 bytes
  static constexpr int LD = BK + VEC;                        // row stride in shared memory
  static constexpr int STAGE = (F + ROWS) * LD;              // elements per stage
  static constexpr int STAGES = sizeof(TI) * STAGE * 6 <= 56 * 1024 ? 6 : 4;
  static constexpr size_t SMEM = (size_t)STAGES * STAGE * sizeof(TI);
};

// K is a multiple of 16 bytes and both matrices start on a 16-byte boundary.
template <typename TI, typename TO, int RPT, int F, int WARPS>
__global__ void __launch_bounds__(WARPS * 32 + 32)
linear_simt_few_rows_kernel(TO* out, const TI* __restrict__ a, const TI* __restrict__ w,
                            const float* __restrict__ bias, const float* residual, int M, int N,
                            int K, int act, float2 ab, int* status) {
  using S = LfShape<TI, RPT, F, WARPS>;
  constexpr int BK = S::BK;
  extern __shared__ __align__(16) uint8_t lf_smem[];
  __shared__ uint64_t full[S::STAGES], empty[S::STAGES];
  TI* ring = (TI*)lf_smem;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = blockIdx.x * F;
  const int num_kt = (K + BK - 1) / BK;
  if (threadIdx.x == 0) {
    for (int s = 0; s < S::STAGES; ++s) {
      mbar_init(&full[s], 32);
      mbar_init(&empty[s], WARPS);
    }
    fence_barrier_init();
  }
  __syncthreads();
  if (warp == WARPS) {
    // the copying warp: RPI rows a trip, a lane per 16-byte piece.  Trips past the last row and pieces
    // past the end of K are left out: what their places hold reaches no output.  (Copies of the last
    // row in their stead went to one line of the L2 from every block: float32, 9 x 20,000 x 256 took
    // 66 us and takes 18, 33 x 4,096 x 1,024 82 and 27.  Asking per row instead of per trip: 48 x
    // 1,024 x 4,096 55 us with the copies, 69 with the questions, 43 so.)  A trip's last row may
    // stand in for the next ones.
    constexpr int CPR = BK / S::VEC;                         // pieces per row of a stage
    constexpr int RPI = 32 / CPR;
    const int crow = lane / CPR, ck = (lane % CPR) * S::VEC;
    const uint32_t ring_at = smem_u32(ring) + (uint32_t)(crow * S::LD + ck) * (uint32_t)sizeof(TI);
    for (int kt = 0; kt < num_kt; ++kt) {
      const int s = kt % S::STAGES;
      if (kt >= S::STAGES && !mbar_wait(&empty[s], ((kt / S::STAGES) - 1) & 1, status)) break;
      const int gk = kt * BK + ck;
      if (gk < K) {
        uint32_t to = ring_at + (uint32_t)(s * S::STAGE) * (uint32_t)sizeof(TI);
#pragma unroll
        for (int row = 0; row < F; row += RPI) {
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to),
                       "l"(w + (size_t)min(n0 + row + crow, N - 1) * K + gk) : "memory");
          to += RPI * S::LD * (uint32_t)sizeof(TI);
        }
        if (M >= S::ROWS) {
#pragma unroll 8
          for (int row = 0; row < S::ROWS; row += RPI) {
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to),
                         "l"(a + (size_t)(row + crow) * K + gk) : "memory");
            to += RPI * S::LD * (uint32_t)sizeof(TI);
          }
        } else {
#pragma unroll 8
          for (int row = 0; row < M; row += RPI) {
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to),
                         "l"(a + (size_t)min(row + crow, M - 1) * K + gk) : "memory");
            to += RPI * S::LD * (uint32_t)sizeof(TI);
          }
        }
      }
      asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&full[s]))
                   : "memory");
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    return;
  }
  const int f = F == 8 ? ls_col(lane) : lane >> 1;         // (F is 8 or 16)
  const int g = warp * (32 / F) + (F == 8 ? ls_row(lane) : lane & 1);
  float acc[RPT];
#pragma unroll
  for (int r = 0; r < RPT; ++r) acc[r] = 0.f;
  constexpr int U = RPT > 2 ? 8 : 16;                        // k per register set
  struct Set { float w[U], x[RPT][U]; };
  for (int kt = 0; kt < num_kt; ++kt) {
    const int st = kt % S::STAGES;
    if (!mbar_wait(&full[st], (kt / S::STAGES) & 1, status)) return;
    const TI* sw = ring + (size_t)st * S::STAGE + f * S::LD;
    const TI* sa = ring + (size_t)st * S::STAGE + (F + g) * S::LD;
    auto read = [&](int k, Set& s) {
#pragma unroll
      for (int q = 0; q < U; q += 4) {
        ls_load4(sw + k + q, *(float(*)[4])&s.w[q]);
#pragma unroll
        for (int r = 0; r < RPT; ++r)
          ls_load4(sa + r * S::G * S::LD + k + q, *(float(*)[4])&s.x[r][q]);
      }
    };
    auto products = [&](const Set& s, int n) {
      if (n >= U) {
#pragma unroll
        for (int q = 0; q < U; ++q)
#pragma unroll
          for (int r = 0; r < RPT; ++r) acc[r] = fmaf(s.x[r][q], s.w[q], acc[r]);
      } else {                                               // the end of K: no product past it
#pragma unroll
        for (int q = 0; q < U; ++q)
          if (q < n) {
#pragma unroll
            for (int r = 0; r < RPT; ++r) acc[r] = fmaf(s.x[r][q], s.w[q], acc[r]);
          }
      }
    };
    const int kmax = min(BK, K - kt * BK);                   // a multiple of 4
    Set s0, s1;
    read(0, s0);
    if (kmax == BK) {
#pragma unroll
      for (int k = 0; k < BK; k += 2 * U) {
        read(k + U, s1);
        products(s0, U);
        if (k + 2 * U < BK) read(k + 2 * U, s0);
        products(s1, U);
      }
    } else {
      for (int k = 0; k < kmax; k += U) {
        products(s0, kmax - k);
        if (k + U < kmax) read(k + U, s0);
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[st]);
  }
  const int gn = n0 + f;
  if (gn >= N) return;
#pragma unroll
  for (int r = 0; r < RPT; ++r) {
    const int gm = g + S::G * r;
    if (gm >= M) continue;
    float v = acc[r];
    if (bias) v += bias[gn];
    v = apply_act(v, act, ab);
    if (residual) v += residual[(size_t)gm * N + gn];
    out[(size_t)gm * N + gn] = from_f<TO>(v);
  }
}

template <typename TI, typename TO, int RPT, int F, int WARPS>
static int launch_few_rows_as(void* out, const void* a, const void* w, const float* bias,
                              const float* residual, int M, int N, int K, int act, float2 ab,
                              int* status, cudaStream_t st) {
  using S = LfShape<TI, RPT, F, WARPS>;
  auto* k = linear_simt_few_rows_kernel<TI, TO, RPT, F, WARPS>;
  static cudaError_t state = cudaErrorUnknown;
  if (state != cudaSuccess)
    state = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM);
  if (state != cudaSuccess) return (int)state;
  k<<<(N + F - 1) / F, WARPS * 32 + 32, S::SMEM, st>>>(
      (TO*)out, (const TI*)a, (const TI*)w, bias, residual, M, N, K, act, ab, status);
  return HS_OK;
}

template <typename TI, typename TO>
static int launch_few_rows(void* out, const void* a, const void* w, const float* bias,
                           const float* residual, int M, int N, int K, int act, float2 ab,
                           int* status, cudaStream_t st) {
  if (M <= 4) return launch_few_rows_as<TI, TO, 1, 8, 1>(out, a, w, bias, residual, M, N, K, act, ab, status, st);
  if (M <= 8) return launch_few_rows_as<TI, TO, 2, 8, 1>(out, a, w, bias, residual, M, N, K, act, ab, status, st);
  if (M <= 16) return launch_few_rows_as<TI, TO, 2, 8, 2>(out, a, w, bias, residual, M, N, K, act, ab, status, st);
  // 16 features a CTA where that still gives every SM one, else 8 (64 rows of 1,024 features: 64
  // CTAs took 62 us at k = 4,096)
  const bool wide = (N + 15) / 16 >= hs_sm_count();
  if (M <= 32) return wide ? launch_few_rows_as<TI, TO, 4, 16, 4>(out, a, w, bias, residual, M, N, K, act, ab, status, st)
                           : launch_few_rows_as<TI, TO, 2, 8, 4>(out, a, w, bias, residual, M, N, K, act, ab, status, st);
  return wide ? launch_few_rows_as<TI, TO, 8, 16, 4>(out, a, w, bias, residual, M, N, K, act, ab, status, st)
              : launch_few_rows_as<TI, TO, 4, 8, 4>(out, a, w, bias, residual, M, N, K, act, ab, status, st);
}

}  // namespace hs

HS_EXPORT int hs_linear_simt(void* out, const void* a, const void* w, const float* bias,
                             const float* residual, int M, int N, int K, int act, float act_a,
                             float act_b, int in_dtype, int out_dtype, int* status, void* stream) {
  const float2 ab = make_float2(act_a, act_b);
  if (!out || !a || !w || !status) return HS_ERR_ARGUMENT;
  if (M <= 0 || N <= 0) return HS_OK;
  if (K <= 0) return HS_ERR_ARGUMENT;
  if (act < HS_ACT_NONE || act > HS_ACT_LAST) return HS_ERR_UNSUPPORTED;
  cudaStream_t st = (cudaStream_t)stream;
  using bf16 = __nv_bfloat16;
  // few rows: the weight-stream kernel (rows and pointers that 16-byte copies can take)
  const int vec = in_dtype == HS_DT_F32 ? 4 : 8;
  // (float32, us, few-rows kernel against tiles: 32 x 4,096 x 1,024 20 and 44, 32 x
  // 50,257 x 768 114 and 141, 64 x 4,096 x 1,024 34 and 46; but 64 x 6,400 x 768 50 and 40, 64 x 50,257
  // x 768 287 and 153)
  const bool few = M <= 32 || (M <= 64 && (N + 15) / 16 <= 2 * hs_sm_count());
  if (few && K % vec == 0 && !((uintptr_t)a & 15) && !((uintptr_t)w & 15)) {
    int rc = HS_ERR_UNSUPPORTED;
    if (in_dtype == HS_DT_F32 && out_dtype == HS_DT_F32)
      rc = hs::launch_few_rows<float, float>(out, a, w, bias, residual, M, N, K, act, ab, status, st);
    else if (in_dtype == HS_DT_BF16 && out_dtype == HS_DT_BF16)
      rc = hs::launch_few_rows<bf16, bf16>(out, a, w, bias, residual, M, N, K, act, ab, status, st);
    else if (in_dtype == HS_DT_BF16 && out_dtype == HS_DT_F32)
      rc = hs::launch_few_rows<bf16, float>(out, a, w, bias, residual, M, N, K, act, ab, status, st);
    if (rc != HS_OK) return rc;
    HS_LAUNCH_CHECK();
    return HS_OK;
  }
  const long long big = (long long)((N + 127) / 128) * ((M + 127) / 128);
  const bool vec4 = K % 4 == 0 && !((uintptr_t)a & 7) && !((uintptr_t)w & 7);
  // bfloat16, us, 64 x 64 against 128 x 128 tiles.  Loads of four: the last round of two tiles an SM is
  // mostly full (1,024 x 4,096 x 1,028, 256 tiles, 263 and 229; 1,024 x 8,192 x 1,028, 512, 546 and 459;
  // but 300 x 8,192 x 1,028, 192, 209 and 226; 300 x 16,384 x 516, 384, 185 and 235).  Single loads: one
  // round of a tile an SM, mostly full (2,048 x 1,024 x 1,023, 128 tiles, 233 and 186; but 2,048 x 4,096
  // x 1,022, 512, 470 and 547)
  const long long sms = hs_sm_count();
  const bool fills = vec4 ? big > sms && (big % (2 * sms) == 0 || 10 * (big % (2 * sms)) >= 14 * sms)
                          : 4 * big >= 3 * sms && big <= sms;
  if (in_dtype == HS_DT_BF16 && M >= 256 && fills && (M + 127) / 128 <= 65535) {
    const dim3 grid((N + 127) / 128, (M + 127) / 128);
#define HS_LB_LAUNCH(TO, VEC)                                                                  \
  hs::linear_simt_big_kernel<bf16, TO, VEC><<<grid, hs::LB_THREADS, 0, st>>>(                  \
      (TO*)out, (const bf16*)a, (const bf16*)w, bias, residual, M, N, K, act, ab)
    if (out_dtype == HS_DT_F32 && vec4) HS_LB_LAUNCH(float, true);
    else if (out_dtype == HS_DT_F32) HS_LB_LAUNCH(float, false);
    else if (out_dtype == HS_DT_BF16 && vec4) HS_LB_LAUNCH(bf16, true);
    else if (out_dtype == HS_DT_BF16) HS_LB_LAUNCH(bf16, false);
    else return HS_ERR_UNSUPPORTED;
#undef HS_LB_LAUNCH
    HS_LAUNCH_CHECK();
    return HS_OK;
  }
  // the large tile where it gives every SM about four (below that an SM has too few warps to hide
  // its own latencies)
  const long long large = (long long)((N + 63) / 64) * ((M + 63) / 64);
  const int side = large >= 4ll * hs_sm_count() ? 64 : 32;
  const dim3 grid((N + side - 1) / side, (M + side - 1) / side);
  if (grid.y > 65535) return HS_ERR_UNSUPPORTED;
#define HS_LT_LAUNCH(TI, TO, LOAD)                                                             \
  do {                                                                                         \
    if (side == 64)                                                                            \
      hs::linear_simt_tile_kernel<TI, TO, 2, LOAD><<<grid, hs::LT_THREADS, 0, st>>>(           \
          (TO*)out, (const TI*)a, (const TI*)w, bias, residual, M, N, K, act, ab);             \
    else                                                                                       \
      hs::linear_simt_tile_kernel<TI, TO, 1, LOAD><<<grid, hs::LT_THREADS, 0, st>>>(           \
          (TO*)out, (const TI*)a, (const TI*)w, bias, residual, M, N, K, act, ab);             \
  } while (0)
  if (in_dtype == HS_DT_F32 && out_dtype == HS_DT_F32) {
    if (64ll * K < (1ll << 31)) HS_LT_LAUNCH(float, float, 2);      // (32-bit offsets in a tile)
    else HS_LT_LAUNCH(float, float, 0);
  } else if (in_dtype == HS_DT_BF16 && out_dtype == HS_DT_BF16) {
    if (vec4) HS_LT_LAUNCH(bf16, bf16, 1);
    else HS_LT_LAUNCH(bf16, bf16, 0);
  } else if (in_dtype == HS_DT_BF16 && out_dtype == HS_DT_F32) {
    if (vec4) HS_LT_LAUNCH(bf16, float, 1);
    else HS_LT_LAUNCH(bf16, float, 0);
  } else {
    return HS_ERR_UNSUPPORTED;
  }
#undef HS_LT_LAUNCH
  HS_LAUNCH_CHECK();
  return HS_OK;
}
