// Gated delta rule with one decay per head and key channel, as a recurrent mixer.
//
// A token's row of the fused input projection holds  [q | k | v | b | a | g]:
//   q, k: kv_heads x D     v: heads x V     b: heads     a: ra numbers     g: rg numbers.
// Four kernels:
//   prepare    per token: causal short convolution over time (taps weights per channel, the
//              last one on the current token; inputs before a portion's start come from the
//              request's state) and silu on q, k, v; q and k to unit length per head
//              (x / sqrt(sum x^2 + 1e-6)), q also times D^-1/2; beta = sigmoid(b);
//              decay = exp(-exp(A_log[h]) * softplus(W_a2 a + dt_bias))   [heads x D]
//   conv state per request: keeps the last taps-1 inputs of q, k, v
//   recurrence per request and head, token after token on the float32 state S [D x V]:
//                 S <- decay * S (row-wise);  u = beta (v - S^T k);  S <- S + k u^T;  o = S^T q
//   finish     per token and head: o / sqrt(mean(o^2) + eps) * w * sigmoid(W_g2 g)
// Everything here is float32 whatever the model's matrix type is.  The two small matrices W_a2
// and W_g2 are held with the summed index slowest ([ra, heads x D] and [rg, heads x V]) so that
// neighbouring threads read neighbouring weights.
//
// State of a slot: [heads x D x V | (taps-1) x channels] floats.
#include "tcgen05.cuh"

#include <type_traits>

namespace hs {

__device__ __forceinline__ float sigmoidf_(float z) { return 1.0f / (1.0f + expf(-z)); }
__device__ __forceinline__ float softplusf_(float z) { return z > 20.f ? z : log1pf(expf(z)); }

struct DeltaShape {
  int heads, kv_heads, D, V, taps, ra, rg;
  int stride;                    // floats in a projection row
  int b_off, a_off, g_off;       // columns of b, a, g (q, k, v start at 0)
  int state_stride;              // floats in a slot
};

__device__ __forceinline__ int channels(const DeltaShape& s) {
  return 2 * s.kv_heads * s.D + s.heads * s.V;
}

// Three blocks a token (blockIdx.y): 0 convolves q and k and makes them unit vectors, 1 convolves
// v and forms beta, 2 forms the decay.  They share nothing.
template <bool FOUR>
__global__ void __launch_bounds__(256)
delta_prepare_kernel(float* __restrict__ qn, float* __restrict__ kn, float* __restrict__ vv,
                     float* __restrict__ beta, float* __restrict__ decay,
                     const float* __restrict__ proj, const float* __restrict__ conv_w,
                     const float* __restrict__ a2, const float* __restrict__ dt_bias,
                     const float* __restrict__ A_log, const float* __restrict__ state,
                     const int* __restrict__ tok_req, const int* __restrict__ req_start,
                     const int* __restrict__ req_slot, DeltaShape s,
                     const float* __restrict__ z_a) {
  extern __shared__ float s_c[];                 // [2 * kv_heads * D] q and k after conv and silu
  pdl_trigger();
  pdl_wait();
  const int t = blockIdx.x;
  const int r = tok_req[t];
  if (r < 0) return;
  const int C = channels(s);
  const int QK = s.kv_heads * s.D;
  const float* row = proj + (size_t)t * s.stride;
  if (blockIdx.y == 2) {
    const int HD = s.heads * s.D;
    for (int i = threadIdx.x; i < HD; i += blockDim.x) {
      float z = 0.f;
      if (z_a) {                                   // W_a2 a was formed as a matrix product
        z = z_a[(size_t)t * HD + i];
      } else {
#pragma unroll 8
        for (int k = 0; k < s.ra; ++k) z = fmaf(a2[(size_t)k * HD + i], row[s.a_off + k], z);
      }
      z += dt_bias[i];
      decay[(size_t)t * HD + i] = expf(-expf(A_log[i / s.D]) * softplusf_(z));
    }
    return;
  }
  const int first = req_start[r];
  const int l = t - first;
  const float* cst = state + (size_t)req_slot[r] * s.state_stride + (size_t)s.heads * s.D * s.V;
  const int hist = s.taps - 1;
  // FOUR (prompts through four taps with more than two channels a thread): four channels c, c + 256, ...
  // at a time where every input is of this portion; the loads of all are on their way before the first
  // sum.  Everything else channel by channel: the other form's registers cost more than it gives.  us,
  // channel by channel against four: 1,024 tokens of 3,072 channels and 4 taps 30.7 and 25.8, of 512
  // channels 11.3 and 13.1; 64 single tokens of 3,072 10.7 and 11.7.
  auto conv = [&](int c0, int end, auto put) {
    if (FOUR && l >= 3) {
      constexpr int U = 4;
      const int step = blockDim.x;
      for (int c = c0; c < end; c += U * step) {
        float in[U][4];
        float4 w[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int cc = min(c + u * step, end - 1);
#pragma unroll
          for (int j = 0; j < 4; ++j) in[u][j] = proj[(size_t)(t - 3 + j) * s.stride + cc];
          w[u] = make_float4(conv_w[4 * (size_t)cc], conv_w[4 * (size_t)cc + 1],
                             conv_w[4 * (size_t)cc + 2], conv_w[4 * (size_t)cc + 3]);
        }
        float acc[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          acc[u] = fmaf(w[u].x, in[u][0], 0.f);
          acc[u] = fmaf(w[u].y, in[u][1], acc[u]);
          acc[u] = fmaf(w[u].z, in[u][2], acc[u]);
          acc[u] = fmaf(w[u].w, in[u][3], acc[u]);
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (c + u * step < end) put(c + u * step, acc[u] * sigmoidf_(acc[u]));
      }
      return;
    }
    for (int c = c0; c < end; c += blockDim.x) {
      float acc = 0.f;
#pragma unroll 4
      for (int j = 0; j < s.taps; ++j) {
        const int local = l - (hist - j);
        const float in = local >= 0 ? proj[(size_t)(first + local) * s.stride + c]
                                    : cst[(size_t)(local + hist) * C + c];
        acc = fmaf(conv_w[(size_t)c * s.taps + j], in, acc);
      }
      put(c, acc * sigmoidf_(acc));
    }
  };
  if (blockIdx.y == 1) {
    const int HV = s.heads * s.V;
    conv(2 * QK + threadIdx.x, 2 * QK + HV,
         [&](int c, float x) { vv[(size_t)t * HV + c - 2 * QK] = x; });
    for (int h = threadIdx.x; h < s.heads; h += blockDim.x)
      beta[(size_t)t * s.heads + h] = sigmoidf_(row[s.b_off + h]);
    return;
  }
  conv(threadIdx.x, 2 * QK, [&](int c, float x) { s_c[c] = x; });
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (int vec = warp; vec < 2 * s.kv_heads; vec += nw) {       // q heads, then k heads
    const float* src = s_c + (size_t)vec * s.D;
    float ss = 0.f;
    for (int d = lane; d < s.D; d += 32) ss = fmaf(src[d], src[d], ss);
    ss = warp_sum(ss);
    float inv = 1.0f / sqrtf(ss + 1e-6f);
    const bool is_q = vec < s.kv_heads;
    if (is_q) inv *= 1.0f / sqrtf((float)s.D);
    float* dst = is_q ? qn + (size_t)t * QK + (size_t)vec * s.D
                      : kn + (size_t)t * QK + (size_t)(vec - s.kv_heads) * s.D;
    for (int d = lane; d < s.D; d += 32) dst[d] = src[d] * inv;
  }
}

// The same for prompts through four taps with heads of 32 to 128 key channels: a warp takes eight tokens of
// one head's q or k, of 128 value channels or of 128 decays, lane l the channels l, l + 32, .. (the sums of the
// kernel above, in its order: the same bits).  The eleven inputs of a channel are fetched once and slide
// through registers, where a block a token reads every input four times.  Eight tokens that are not one
// request's, or reach behind its portion, are taken one by one.  2,048 tokens of 3,072
// channels and 1,024 decays: 39.6 us in blocks of a token, 29.8 so; exponentials and quotients issue for half of it.
constexpr int DP_TOK = 8;

__global__ void __launch_bounds__(128)
delta_prepare_rows_kernel(float* __restrict__ qn, float* __restrict__ kn, float* __restrict__ vv,
                          float* __restrict__ beta, float* __restrict__ decay,
                          const float* __restrict__ proj, const float* __restrict__ conv_w,
                          const float* __restrict__ a2, const float* __restrict__ dt_bias,
                          const float* __restrict__ A_log, const float* __restrict__ state,
                          const int* __restrict__ tok_req, const int* __restrict__ req_start,
                          const int* __restrict__ req_slot, DeltaShape s,
                          const float* __restrict__ z_a, int n_tokens) {
  pdl_trigger();
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const int t0 = blockIdx.x * DP_TOK;
  const int QK = s.kv_heads * s.D, HV = s.heads * s.V, HD = s.heads * s.D, C = channels(s);
  const int v_groups = (HV + 127) / 128;
  int g = blockIdx.y * 4 + (threadIdx.x >> 5);
  const int mine = lane < DP_TOK && t0 + lane < n_tokens ? tok_req[t0 + lane] : -1;
  const int here = min(DP_TOK, n_tokens - t0);
  const unsigned live = __ballot_sync(0xffffffffu, mine >= 0);
  if (g >= 2 * s.kv_heads + v_groups) {            // ---- decays
    g -= 2 * s.kv_heads + v_groups;
    for (int j = 0; j < 4; ++j) {
      const int i = g * 128 + 32 * j + lane;
      if (i >= HD) return;
      const float bias = dt_bias[i], rate = -expf(A_log[i / s.D]);
      float z[DP_TOK];
#pragma unroll
      for (int u = 0; u < DP_TOK; ++u) {
        z[u] = 0.f;
        if (u < here && z_a) z[u] = z_a[(size_t)(t0 + u) * HD + i];
      }
      if (!z_a)
        for (int u = 0; u < here; ++u)
#pragma unroll 8
          for (int k = 0; k < s.ra; ++k)
            z[u] = fmaf(a2[(size_t)k * HD + i], proj[(size_t)(t0 + u) * s.stride + s.a_off + k], z[u]);
#pragma unroll
      for (int u = 0; u < DP_TOK; ++u)
        if (live >> u & 1)
          decay[(size_t)(t0 + u) * HD + i] = expf(rate * softplusf_(z[u] + bias));
    }
    return;
  }
  const bool is_v = g >= 2 * s.kv_heads;
  const int c0 = is_v ? 2 * QK + (g - 2 * s.kv_heads) * 128 : g * s.D;
  const int nc = is_v ? min(128, 2 * QK + HV - c0) : s.D;
  float w[4][4];                                   // [channel][tap]
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int k = 0; k < 4; ++k) w[j][k] = 32 * j + lane < nc ? conv_w[4 * (size_t)(c0 + 32 * j + lane) + k] : 0.f;
  // what becomes of a token's convolved channels
  auto finish = [&](int t, float (&x)[4]) {
    if (is_v) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (32 * j + lane < nc) vv[(size_t)t * HV + c0 - 2 * QK + 32 * j + lane] = x[j];
      return;
    }
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (32 * j + lane < nc) ss = fmaf(x[j], x[j], ss);
    ss = warp_sum(ss);
    float inv = 1.0f / sqrtf(ss + 1e-6f);
    const bool is_q = g < s.kv_heads;
    if (is_q) inv *= 1.0f / sqrtf((float)s.D);
    float* dst = (is_q ? qn : kn) + (size_t)t * QK + (size_t)(is_q ? g : g - s.kv_heads) * s.D;
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (32 * j + lane < nc) dst[32 * j + lane] = x[j] * inv;
  };
  const int r0 = __shfl_sync(0xffffffffu, mine, 0);
  const bool one = __all_sync(0xffffffffu, lane >= DP_TOK || mine == r0) && r0 >= 0;
  if (one && t0 - req_start[r0] >= 3) {
    float in[DP_TOK + 3][4];
#pragma unroll
    for (int m = 0; m < DP_TOK + 3; ++m)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        in[m][j] = 32 * j + lane < nc ? proj[(size_t)(t0 - 3 + m) * s.stride + c0 + 32 * j + lane] : 0.f;
#pragma unroll
    for (int u = 0; u < DP_TOK; ++u) {
      float x[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float acc = fmaf(w[j][0], in[u][j], 0.f);
#pragma unroll
        for (int k = 1; k < 4; ++k) acc = fmaf(w[j][k], in[u + k][j], acc);
        x[j] = acc * sigmoidf_(acc);
      }
      finish(t0 + u, x);
    }
  } else {
    for (int u = 0; u < here; ++u) {
      const int t = t0 + u, r = __shfl_sync(0xffffffffu, mine, u);
      if (r < 0) continue;
      const int first = req_start[r], l = t - first;
      const float* cst = state + (size_t)req_slot[r] * s.state_stride + (size_t)s.heads * s.D * s.V;
      float x[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int c = c0 + 32 * j + lane;
        float acc = 0.f;
        if (32 * j + lane < nc) {
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int local = l - (3 - k);
            const float in = local >= 0 ? proj[(size_t)(first + local) * s.stride + c]
                                        : cst[(size_t)(local + 3) * C + c];
            acc = fmaf(w[j][k], in, acc);
          }
        }
        x[j] = acc * sigmoidf_(acc);
      }
      finish(t, x);
    }
  }
  if (g == 2 * s.kv_heads)
    for (int i = lane; i < here * s.heads; i += 32) {
      const int u = i / s.heads, h = i - u * s.heads;
      if (tok_req[t0 + u] >= 0)
        beta[(size_t)(t0 + u) * s.heads + h] = sigmoidf_(proj[(size_t)(t0 + u) * s.stride + s.b_off + h]);
    }
}

__global__ void delta_conv_state_kernel(float* __restrict__ state, const float* __restrict__ proj,
                                        const int* __restrict__ req_start,
                                        const int* __restrict__ req_len,
                                        const int* __restrict__ req_slot, DeltaShape s) {
  pdl_trigger();
  pdl_wait();
  const int r = blockIdx.y;
  const int n = req_len[r];
  if (n <= 0) return;
  const int C = channels(s);
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= C) return;
  const int hist = s.taps - 1;
  float* cst = state + (size_t)req_slot[r] * s.state_stride + (size_t)s.heads * s.D * s.V;
  const int first = req_start[r];
  // slot i receives the input at local index n - hist + i; an index below zero is an older
  // input, found at n + i of the old state, which lies ahead of every slot written so far
  for (int i = 0; i < hist; ++i) {
    const int local = n - hist + i;
    cst[(size_t)i * C + c] = local >= 0 ? proj[(size_t)(first + local) * s.stride + c]
                                        : cst[(size_t)(n + i) * C + c];
  }
}

constexpr int DR_DP = 16;         // state rows a thread keeps
constexpr int DR_STAGES = 3;      // chunks of tokens in shared memory
constexpr int DR_THREADS = 64;   // few warps a block: the shared-memory pipe of an SM bounds a block's step from token to token

__device__ __forceinline__ void cp_async4(float* dst, const float* src) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(sa), "l"(src));
}
__device__ __forceinline__ void cp_async16(float* dst, const float* src) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sa), "l"(src));
}

// Thread (col, part) keeps DP rows of column col of S: the four rows 4*part + 4*KS*j .. + 3 for
// j = 0 .. DP/4 - 1, so that the KS neighbouring lanes of a column read neighbouring 16-byte
// pieces of a row in shared memory (no bank conflict); they sum their shares with a butterfly.
// The tokens' q, k, decay
// rows (padded with zeros to KS*DP), v columns and betas come through shared memory a chunk of
// CH tokens at a time, fetched asynchronously two chunks ahead: the latency of fetching them is
// off the token-to-token chain.
__global__ void __launch_bounds__(DR_THREADS)
delta_recurrence_kernel(float* __restrict__ o, float* __restrict__ state,
                        const float* __restrict__ qn, const float* __restrict__ kn,
                        const float* __restrict__ vv, const float* __restrict__ beta,
                        const float* __restrict__ decay, const int* __restrict__ req_start,
                        const int* __restrict__ req_len, const int* __restrict__ req_slot,
                        DeltaShape s, int KS, int CH, int vec, int long_from) {
  extern __shared__ __align__(16) float sm[];
  const int r = blockIdx.x, h = blockIdx.y;
  const int n = req_len[r];
  if (n <= 0 || n >= long_from) return;            // long portions: delta_blocks_kernel
  const int Dp = KS * DR_DP;
  const int cols = DR_THREADS / KS;
  const int per_buf = (3 * CH * Dp + CH * cols + CH + 3) & ~3;      // buffers 16-byte aligned
  const int part = threadIdx.x % KS;
  const int lc = threadIdx.x / KS;
  const int col0 = blockIdx.z * cols;
  const int col = col0 + lc;
  const bool col_ok = col < s.V;
  const int kh = h / (s.heads / s.kv_heads);
  const int d0 = part * 4;                       // row of st[i]: d0 + 4*KS*(i/4) + i%4
  const int dj = 4 * KS;
  float* S = state + (size_t)req_slot[r] * s.state_stride + (size_t)h * s.D * s.V;
  float st[DR_DP];
#pragma unroll
  for (int i = 0; i < DR_DP; ++i) {
    const int d = d0 + dj * (i >> 2) + (i & 3);
    st[i] = (col_ok && d < s.D) ? S[(size_t)d * s.V + col] : 0.f;
  }
  const int QK = s.kv_heads * s.D, HV = s.heads * s.V, HD = s.heads * s.D;
  const int first = req_start[r];
  for (int i = threadIdx.x; i < DR_STAGES * per_buf; i += DR_THREADS) sm[i] = 0.f;   // padding stays 0
  __syncthreads();
  auto fetch = [&](int buf, int c0) {
    float* b_k = sm + buf * per_buf;
    float* b_q = b_k + CH * Dp;
    float* b_g = b_q + CH * Dp;
    float* b_v = b_g + CH * Dp;
    float* b_b = b_v + CH * cols;
    const int nc = min(CH, n - c0);
    if (vec) {
      const int D4 = s.D >> 2;
      for (int i = threadIdx.x; i < nc * D4; i += DR_THREADS) {
        const int tt = i / D4, d = (i - tt * D4) * 4;
        const size_t row = first + c0 + tt;
        cp_async16(b_k + tt * Dp + d, kn + row * QK + kh * s.D + d);
        cp_async16(b_q + tt * Dp + d, qn + row * QK + kh * s.D + d);
        cp_async16(b_g + tt * Dp + d, decay + row * HD + h * s.D + d);
      }
    } else {
      for (int i = threadIdx.x; i < nc * s.D; i += DR_THREADS) {
        const int tt = i / s.D, d = i - tt * s.D;
        const size_t row = first + c0 + tt;
        cp_async4(b_k + tt * Dp + d, kn + row * QK + kh * s.D + d);
        cp_async4(b_q + tt * Dp + d, qn + row * QK + kh * s.D + d);
        cp_async4(b_g + tt * Dp + d, decay + row * HD + h * s.D + d);
      }
    }
    for (int i = threadIdx.x; i < nc * cols; i += DR_THREADS) {
      const int tt = i / cols, cc = i - tt * cols;
      if (col0 + cc < s.V)
        cp_async4(b_v + i, vv + (size_t)(first + c0 + tt) * HV + h * s.V + col0 + cc);
    }
    if (threadIdx.x < nc)
      cp_async4(b_b + threadIdx.x, beta + (size_t)(first + c0 + threadIdx.x) * s.heads + h);
    asm volatile("cp.async.commit_group;");
  };
  // three buffers: while a chunk is worked on, the two behind it are on their way (a fetch
  // takes longer than a chunk of tokens does).  Every turn commits a group, an empty one at
  // the end, so that "all but the newest two have landed" always names the chunk of this turn.
  fetch(0, 0);
  if (CH < n) fetch(1, CH); else asm volatile("cp.async.commit_group;");
  int buf = 0;
  for (int c0 = 0; c0 < n; c0 += CH, buf = (buf + 1) % DR_STAGES) {
    const int nc = min(CH, n - c0);
    if (c0 + 2 * CH < n) fetch((buf + 2) % DR_STAGES, c0 + 2 * CH);
    else asm volatile("cp.async.commit_group;");
    asm volatile("cp.async.wait_group 2;");
    __syncthreads();
    const float* b_k = sm + buf * per_buf;
    const float* b_q = b_k + CH * Dp;
    const float* b_g = b_q + CH * Dp;
    const float* b_v = b_g + CH * Dp;
    const float* b_b = b_v + CH * cols;
    // Two register sets alternate: while a token is worked on, the rows of the next one are
    // already on their way from shared memory.  The sum over a column's lanes for a token's
    // output (needed only by the store) rides along with the next token's sum for its dot
    // product, stage by stage, so the chain from token to token holds one butterfly, not two.
    struct Rows { float k[DR_DP], q[DR_DP], g[DR_DP], v, b; };
    auto read = [&](int tt, Rows& r) {
      const float4* k4 = (const float4*)(b_k + tt * Dp + d0);
      const float4* q4 = (const float4*)(b_q + tt * Dp + d0);
      const float4* g4 = (const float4*)(b_g + tt * Dp + d0);
#pragma unroll
      for (int j = 0; j < DR_DP / 4; ++j) {
        const float4 a = k4[j * KS], b = q4[j * KS], c = g4[j * KS];
        r.k[4 * j] = a.x; r.k[4 * j + 1] = a.y; r.k[4 * j + 2] = a.z; r.k[4 * j + 3] = a.w;
        r.q[4 * j] = b.x; r.q[4 * j + 1] = b.y; r.q[4 * j + 2] = b.z; r.q[4 * j + 3] = b.w;
        r.g[4 * j] = c.x; r.g[4 * j + 1] = c.y; r.g[4 * j + 2] = c.z; r.g[4 * j + 3] = c.w;
      }
      r.v = b_v[tt * cols + lc];
      r.b = b_b[tt];
    };
    float pend = 0.f;               // the token before: its output, not yet summed over the lanes
    int pend_tt = -1;
    auto work = [&](int tt, const Rows& r, Rows& next) {
      if (tt + 1 < nc) read(tt + 1, next);
      float dot0 = 0.f, dot1 = 0.f;
#pragma unroll
      for (int j = 0; j < DR_DP; j += 2) {
        st[j] *= r.g[j];
        st[j + 1] *= r.g[j + 1];
        dot0 = fmaf(st[j], r.k[j], dot0);
        dot1 = fmaf(st[j + 1], r.k[j + 1], dot1);
      }
      float dot = dot0 + dot1;
      for (int off = 1; off < KS; off <<= 1) {
        const float d2 = __shfl_xor_sync(0xffffffffu, dot, off);
        const float p2 = __shfl_xor_sync(0xffffffffu, pend, off);
        dot += d2;
        pend += p2;
      }
      if (pend_tt >= 0 && part == 0 && col_ok)
        o[(size_t)(first + c0 + pend_tt) * HV + h * s.V + col] = pend;
      const float u = r.b * (r.v - dot);
      float out0 = 0.f, out1 = 0.f;
#pragma unroll
      for (int j = 0; j < DR_DP; j += 2) {
        st[j] = fmaf(r.k[j], u, st[j]);
        st[j + 1] = fmaf(r.k[j + 1], u, st[j + 1]);
        out0 = fmaf(st[j], r.q[j], out0);
        out1 = fmaf(st[j + 1], r.q[j + 1], out1);
      }
      pend = out0 + out1;
      pend_tt = tt;
    };
    Rows ra, rb;
    read(0, ra);
    for (int tt = 0; tt < nc; tt += 2) {
      work(tt, ra, rb);
      if (tt + 1 < nc) work(tt + 1, rb, ra);
    }
    for (int off = 1; off < KS; off <<= 1) pend += __shfl_xor_sync(0xffffffffu, pend, off);
    if (part == 0 && col_ok) o[(size_t)(first + c0 + pend_tt) * HV + h * s.V + col] = pend;
    __syncthreads();                              // this buffer is fetched into again next turn
  }
#pragma unroll
  for (int i = 0; i < DR_DP; ++i) {
    const int d = d0 + dj * (i >> 2) + (i & 3);
    if (col_ok && d < s.D) S[(size_t)d * s.V + col] = st[i];
  }
}

// ---- portions: four tokens at a time ----------------------------------------------------------
// Token after token, the chain above is bounded by its latencies: a token's dot product with the
// state, the butterfly over a column's lanes, the update (0.4 us a token, one warp a scheduler).
// Four tokens i = 0..3 that start from the state S need only S itself:
//     a_i = S^T K'_i,   K'_i = k_i g_0 .. g_i                 (g: decays, per row)
//     u_i = beta_i (v_i - a_i - sum_{j<i} c_ij u_j),           c_ij  = sum k_i k_j g_j+1 .. g_i
//     o_i = S^T Q'_i + sum_{j<=i} e_ij u_j,  Q'_i = q_i g_0 .. g_i,  e_ij = sum q_i k_j g_j+1 .. g_i
//     S <- g_0 .. g_3 S + sum_j K"_j u_j,                      K"_j  = k_j g_j+1 .. g_3
// so four butterflies overlap and the chain is paid once in four tokens.  The decays enter as
// products of at most four factors below one (no quotients, nothing can overflow).  What does not
// depend on the state (K', Q', K", the decay of all four, c, e, beta) is formed beforehand for all
// tokens in parallel; a head's blocks lie one behind the other, so that a stage of the recurrence
// is one bulk copy.  All of it is float32, packed two rows an instruction.  Measured (2 x 1,024
// tokens, 8 heads of 128 x 128): 412 us token after token, 16 + 155 us so.
//
// The form is chosen per request, from its own number of tokens, so that its sums do not depend on
// its neighbours: each kernel leaves the other's requests alone.
constexpr int DB_TOK = 4, DB_COEF = 32;
constexpr int DB_STAGE_BLOCKS = 2, DB_STAGES = 4;
constexpr int DB_WARPS = 4;                       // that work; one more fetches
__host__ __device__ constexpr int db_floats(int D) { return 13 * D + DB_COEF; }

// blocks of four tokens of a request of n tokens (long_from > 0)
__device__ __forceinline__ int db_blocks(int n, int long_from) {
  return n >= long_from ? (n + DB_TOK - 1) / DB_TOK : 0;
}
// The long request of number i, or (by_block) the one that block number i belongs to: its row, or -1
// where there are fewer; `before`: blocks of the long requests before it.  By a whole warp, 32
// requests at a time (one after the other, a block of a step of 64 requests spent 8 us on this).
__device__ __forceinline__ int db_request(const int* __restrict__ req_len, int n_requests,
                                          int long_from, int i, bool by_block, int* before) {
  const int lane = threadIdx.x & 31;
  int seen = 0;                                    // long requests, or blocks, before these 32
  *before = 0;
  for (int r0 = 0; r0 < n_requests; r0 += 32) {
    const int nb = r0 + lane < n_requests ? db_blocks(req_len[r0 + lane], long_from) : 0;
    int incl = nb;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += u;
    }
    const unsigned many = __ballot_sync(0xffffffffu, nb > 0);
    const int at = seen + (by_block ? incl - nb : __popc(many & ((1u << lane) - 1u)));
    const unsigned hit = __ballot_sync(0xffffffffu, nb > 0 && i >= at && i < at + (by_block ? nb : 1));
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    if (hit) {
      const int who = __ffs(hit) - 1;
      *before += __shfl_sync(0xffffffffu, incl - nb, who);
      return r0 + who;
    }
    seen += by_block ? total : __popc(many);
    *before += total;
  }
  return -1;
}

__global__ void __launch_bounds__(128)
delta_blocks_prepare_kernel(float* __restrict__ blocks, const float* __restrict__ qn,
                            const float* __restrict__ kn, const float* __restrict__ beta,
                            const float* __restrict__ decay, const int* __restrict__ req_start,
                            const int* __restrict__ req_len, int n_requests, int cap_blocks,
                            DeltaShape s, int long_from) {
  __shared__ float red[4][16];
  pdl_trigger();
  pdl_wait();
  const int h = blockIdx.y;
  int before;                                      // the request this block of tokens belongs to
  const int r = db_request(req_len, n_requests, long_from, blockIdx.x, true, &before);
  if (r < 0) return;
  const int blk = blockIdx.x - before;
  const int n = min(DB_TOK, req_len[r] - blk * DB_TOK);       // tokens that exist
  const int t0 = req_start[r] + blk * DB_TOK;
  const int kh = h / (s.heads / s.kv_heads);
  const int QK = s.kv_heads * s.D, HD = s.heads * s.D, D = s.D;
  float* out = blocks + ((size_t)h * cap_blocks + blockIdx.x) * db_floats(D);
  float c[6] = {}, e[10] = {};
  for (int d = threadIdx.x; d < D; d += 128) {
    float k[4], q[4], g[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const bool on = i < n;
      k[i] = on ? kn[(size_t)(t0 + i) * QK + kh * D + d] : 0.f;
      q[i] = on ? qn[(size_t)(t0 + i) * QK + kh * D + d] : 0.f;
      g[i] = on ? decay[(size_t)(t0 + i) * HD + h * D + d] : 1.f;
    }
    float all = 1.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      all *= g[i];
      out[i * D + d] = k[i] * all;
      out[(4 + i) * D + d] = q[i] * all;
      float rest = 1.f;
#pragma unroll
      for (int m = i + 1; m < 4; ++m) rest *= g[m];
      out[(8 + i) * D + d] = k[i] * rest;
    }
    out[12 * D + d] = all;
    int ci = 0, ei = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j <= i; ++j) {
        float f = k[j];
#pragma unroll
        for (int m = j + 1; m <= i; ++m) f *= g[m];
        e[ei] = fmaf(q[i], f, e[ei]);
        ++ei;
        if (j < i) {
          c[ci] = fmaf(k[i], f, c[ci]);
          ++ci;
        }
      }
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const float v = warp_sum(i < 6 ? c[i < 6 ? i : 0] : e[i < 6 ? 0 : i - 6]);
    if (lane == 0) red[warp][i] = v;
  }
  __syncthreads();
  // [c: 10 20 21 30 31 32, - -][beta, - - - -][e: four rows of four, zero above the diagonal]
  if (threadIdx.x < DB_COEF) {
    const int i = threadIdx.x;
    int from = -1;
    if (i < 6) from = i;
    else if (i >= 16 && (i & 3) <= ((i - 16) >> 2)) {
      const int row = (i - 16) >> 2;
      from = 6 + row * (row + 1) / 2 + (i & 3);
    }
    float v = 0.f;
    if (from >= 0) v = (red[0][from] + red[1][from]) + (red[2][from] + red[3][from]);
    else if (i >= 8 && i < 12 && i - 8 < n) v = beta[(size_t)(t0 + i - 8) * s.heads + h];
    out[13 * D + i] = v;
  }
}

__device__ __forceinline__ void db_fma(uint64_t& acc, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ uint64_t db_mul(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t db_add(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t db_pair(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float db_fold(uint64_t a) {
  return __uint_as_float((uint32_t)a) + __uint_as_float((uint32_t)(a >> 32));
}

// KS = D / 16 lanes hold a column of S, 16 rows each (rows 4 part + 4 KS j .. + 3, j < 4).  The
// parts lie on lane bits 1 up, so that a 16-byte read of a row by a warp takes two wavefronts of
// shared memory (on bits 0 up it took four).  There is about one warp a scheduler, so what a phase
// reads from shared memory is read a phase ahead, into registers (225 -> 155 us; with 8 rows a lane
// and twice the warps 170: shared memory, busy for half of the time, then serves every row twice as
// often).
template <int KS>
__global__ void __launch_bounds__(DB_WARPS * 32 + 32)
delta_blocks_kernel(float* __restrict__ o, float* __restrict__ state,
                    const float* __restrict__ blocks, const float* __restrict__ vv,
                    const int* __restrict__ req_start, const int* __restrict__ req_len,
                    const int* __restrict__ req_slot, int n_requests, int cap_blocks, DeltaShape s,
                    int long_from, int* status) {
  constexpr int NJ = 4, D = 4 * NJ * KS, SZ = db_floats(D);
  constexpr int COLS = 32 / KS, CTA_COLS = DB_WARPS * COLS;      // of a warp, of the block
  constexpr int ST_TOK = DB_STAGE_BLOCKS * DB_TOK;             // tokens of a stage
  extern __shared__ __align__(16) float sm[];                  // [stages][blocks of a stage][SZ]
  __shared__ float s_v[DB_STAGES][ST_TOK][CTA_COLS];
  __shared__ uint64_t full[DB_STAGES], empty[DB_STAGES];
  pdl_trigger();
  pdl_wait();
  const int h = blockIdx.y;
  int before;                                      // (there may be fewer long requests than blocks)
  const int r = db_request(req_len, n_requests, long_from, blockIdx.x, false, &before);
  if (r < 0) return;
  const int n = req_len[r];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nb = (n + DB_TOK - 1) / DB_TOK, n_stages = (nb + DB_STAGE_BLOCKS - 1) / DB_STAGE_BLOCKS;
  const int first = req_start[r], HV = s.heads * s.V, col0 = blockIdx.z * CTA_COLS;
  if (threadIdx.x == 0) {
    for (int i = 0; i < DB_STAGES; ++i) {
      mbar_init(&full[i], 1 + 32);
      mbar_init(&empty[i], DB_WARPS);
    }
    fence_barrier_init();
  }
  __syncthreads();
  if (warp == DB_WARPS) {
    // the fetching warp: lane 0 copies the blocks of a stage, all lanes the stage's values
    const float* src = blocks + ((size_t)h * cap_blocks + before) * SZ;
    const float* vsrc = vv + (size_t)first * HV + h * s.V;
    int i = 0;
    for (; i < n_stages; ++i) {
      const int st = i % DB_STAGES;
      if (i >= DB_STAGES && !mbar_wait(&empty[st], ((i / DB_STAGES) - 1) & 1, status)) break;
      if (lane == 0) {
        const int here = min(DB_STAGE_BLOCKS, nb - i * DB_STAGE_BLOCKS);
        const uint32_t bytes = (uint32_t)(here * SZ * 4);
        mbar_expect_tx(&full[st], bytes);
        asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                smem_u32(sm + (size_t)st * DB_STAGE_BLOCKS * SZ)),
            "l"(src + (size_t)i * DB_STAGE_BLOCKS * SZ), "r"(bytes), "r"(smem_u32(&full[st]))
            : "memory");
      }
      for (int e = lane; e < ST_TOK * CTA_COLS; e += 32) {
        const int t = min(i * ST_TOK + e / CTA_COLS, n - 1), c = min(col0 + e % CTA_COLS, s.V - 1);
        cp_async4(&s_v[st][0][0] + e, vsrc + (size_t)t * HV + c);
      }
      asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&full[st]))
                   : "memory");
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    // the block stays until what it fetched has landed, also where the working warps gave up
    for (int k = max(0, i - DB_STAGES); k < i; ++k)
      mbar_wait(&full[k % DB_STAGES], (k / DB_STAGES) & 1, status);
    return;
  }
  const int part = (lane >> 1) & (KS - 1);
  const int lc = warp * COLS + ((lane & 1) | ((lane >> 1) / KS) << 1);
  const int col = col0 + lc;
  const bool col_ok = col < s.V;
  const int tok = 2 * (part & 1) + ((part >> 1) & 1);          // the token of a block this lane stores
  const bool stores = part < 4 && col_ok;
  float* ocol = o + (size_t)(first + tok) * HV + h * s.V + col;
  float* S = state + (size_t)req_slot[r] * s.state_stride + (size_t)h * D * s.V + col;
  uint64_t st[2 * NJ];
#pragma unroll
  for (int j = 0; j < 2 * NJ; ++j) {
    const int d = 4 * part + 4 * KS * (j >> 1) + 2 * (j & 1);
    st[j] = col_ok ? db_pair(S[(size_t)d * s.V], S[(size_t)(d + 1) * s.V]) : 0;
  }
  struct Four { ulonglong2 p[4][NJ]; };            // this lane's rows of four vectors
  auto read4 = [&](const float* x, int vec, Four& f) {
#pragma unroll
    for (int t = 0; t < 4; ++t)
#pragma unroll
      for (int j = 0; j < NJ; ++j)
        f.p[t][j] = *(const ulonglong2*)(x + (vec + t) * D + 4 * part + 4 * KS * j);
  };
  Four fk, fq, fw;
  if (!mbar_wait(&full[0], 0, status)) return;
  read4(sm, 0, fk);
  for (int blk = 0; blk < nb; ++blk) {
    const int i = blk / DB_STAGE_BLOCKS, sg = i % DB_STAGES, in = blk % DB_STAGE_BLOCKS;
    const float* x = sm + (size_t)(sg * DB_STAGE_BLOCKS + in) * SZ;
    read4(x, 4, fq);
    uint64_t aw[4][2] = {}, ow[4][2] = {};
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
#pragma unroll
      for (int t = 0; t < 4; ++t) db_fma(aw[t][0], st[2 * j], fk.p[t][j].x);
#pragma unroll
      for (int t = 0; t < 4; ++t) db_fma(aw[t][1], st[2 * j + 1], fk.p[t][j].y);
    }
    float a[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) a[t] = db_fold(db_add(aw[t][0], aw[t][1]));
    ulonglong2 g[NJ];
#pragma unroll
    for (int j = 0; j < NJ; ++j) g[j] = *(const ulonglong2*)(x + 12 * D + 4 * part + 4 * KS * j);
    const float4* cf = (const float4*)(x + 13 * D);
    const float4 c0 = cf[0], c1 = cf[1], be = cf[2], ev = cf[4 + tok];
    const float* vt = &s_v[sg][in * DB_TOK][lc];
    const float v0 = vt[0], v1 = vt[CTA_COLS], v2 = vt[2 * CTA_COLS], v3 = vt[3 * CTA_COLS];
    // the sums over a column's lanes of what the u need, between the products for the outputs
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if ((2 << j) <= KS) {
#pragma unroll
        for (int t = 0; t < 4; ++t) a[t] += __shfl_xor_sync(0xffffffffu, a[t], 2 << j);
      }
#pragma unroll
      for (int t = 0; t < 4; ++t) db_fma(ow[t][0], st[2 * j], fq.p[t][j].x);
#pragma unroll
      for (int t = 0; t < 4; ++t) db_fma(ow[t][1], st[2 * j + 1], fq.p[t][j].y);
    }
    read4(x, 8, fw);
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      st[2 * j] = db_mul(st[2 * j], g[j].x);
      st[2 * j + 1] = db_mul(st[2 * j + 1], g[j].y);
    }
    if (blk + 1 < nb) {                            // the next block's K'
      const int i2 = (blk + 1) / DB_STAGE_BLOCKS, sg2 = i2 % DB_STAGES;
      if (i2 != i && !mbar_wait(&full[sg2], (i2 / DB_STAGES) & 1, status)) return;
      read4(sm + (size_t)(sg2 * DB_STAGE_BLOCKS + (blk + 1) % DB_STAGE_BLOCKS) * SZ, 0, fk);
    }
    // (a token past the end leaves the state alone: its zero beta and key would make NaN of an
    // infinity)
    const int here = n - blk * DB_TOK;
    float u[4];
    u[0] = be.x * (v0 - a[0]);
    u[1] = here > 1 ? be.y * ((v1 - a[1]) - c0.x * u[0]) : 0.f;
    u[2] = here > 2 ? be.z * ((v2 - a[2]) - c0.y * u[0] - c0.z * u[1]) : 0.f;
    u[3] = here > 3 ? be.w * ((v3 - a[3]) - c0.w * u[0] - c1.x * u[1] - c1.y * u[2]) : 0.f;
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const uint64_t u2 = db_pair(u[t], u[t]);
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        db_fma(st[2 * j], fw.p[t][j].x, u2);
        db_fma(st[2 * j + 1], fw.p[t][j].y, u2);
      }
    }
    // the four outputs' sums: two exchanges leave every lane one token's share, then they add up
    float ob[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) ob[t] = db_fold(db_add(ow[t][0], ow[t][1]));
    const bool hi = part & 1, hi2 = part & 2;
    float w0 = hi ? ob[2] : ob[0], w1 = hi ? ob[3] : ob[1];
    w0 += __shfl_xor_sync(0xffffffffu, hi ? ob[0] : ob[2], 2);
    w1 += __shfl_xor_sync(0xffffffffu, hi ? ob[1] : ob[3], 2);
    float out = hi2 ? w1 : w0;
    out += __shfl_xor_sync(0xffffffffu, hi2 ? w0 : w1, 4);
#pragma unroll
    for (int off = 8; off <= KS; off <<= 1) out += __shfl_xor_sync(0xffffffffu, out, off);
    // (a later token's u is left out, not multiplied by the zero above the diagonal: it may be an
    // infinity or a NaN that the token must not see)
    out += ev.x * u[0] + ev.y * (tok > 0 ? u[1] : 0.f) + ev.z * (tok > 1 ? u[2] : 0.f) +
           ev.w * (tok > 2 ? u[3] : 0.f);
    if (stores && tok < here) ocol[(size_t)blk * DB_TOK * HV] = out;
    if (in == DB_STAGE_BLOCKS - 1) {
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[sg]);
    }
  }
  if (col_ok) {
#pragma unroll
    for (int j = 0; j < 2 * NJ; ++j) {
      const int d = 4 * part + 4 * KS * (j >> 1) + 2 * (j & 1);
      S[(size_t)d * s.V] = __uint_as_float((uint32_t)st[j]);
      S[(size_t)(d + 1) * s.V] = __uint_as_float((uint32_t)(st[j] >> 32));
    }
  }
}

// The gated norm of a head's outputs where W_g2 g was formed as a matrix product and a head has 32 to 256 values, a multiple of 32: a
// warp a token and head, its sums those of the four warps of a block below (the same bits).  2,048 tokens, 8
// heads of 128: 21 us in blocks a token and head, 9.7 so.
template <typename TO>
__global__ void __launch_bounds__(256)
delta_finish_rows_kernel(TO* __restrict__ out, const float* __restrict__ o,
                         const float* __restrict__ norm_w, const int* __restrict__ tok_req, float eps,
                         DeltaShape s, const float* __restrict__ z_g, int n_tokens) {
  pdl_trigger();
  pdl_wait();
  const int i = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int t = i / s.heads, h = i - t * s.heads;
  if (t >= n_tokens || tok_req[t] < 0) return;
  const size_t at = ((size_t)t * s.heads + h) * s.V;
  constexpr int N = 8;
  float x[N], z[N];
#pragma unroll
  for (int j = 0; j < N; ++j) {
    const int e = 32 * j + lane;
    x[j] = e < s.V ? o[at + e] : 0.f;
    z[j] = e < s.V ? z_g[at + e] : 0.f;
  }
  float tot = 0.f;
#pragma unroll
  for (int w = 0; w < 4; ++w) tot += warp_sum(fmaf(x[w + 4], x[w + 4], fmaf(x[w], x[w], 0.f)));
  const float inv = 1.0f / sqrtf(tot / (float)s.V + eps);
#pragma unroll
  for (int j = 0; j < N; ++j) {
    const int e = 32 * j + lane;
    if (e < s.V) out[at + e] = from_f<TO>(x[j] * inv * norm_w[e] * sigmoidf_(z[j]));
  }
}

// One block per token and head: the head's root mean square by a block reduction, then one
// thread per output forms its gate (a sum over the rg inputs, several loads in flight).
template <typename TO>
__global__ void __launch_bounds__(128)
delta_finish_kernel(TO* __restrict__ out, const float* __restrict__ o,
                    const float* __restrict__ proj, const float* __restrict__ g2,
                    const float* __restrict__ norm_w, const int* __restrict__ tok_req,
                    float eps, DeltaShape s, const float* __restrict__ z_g) {
  __shared__ float red[4];
  extern __shared__ float s_gin[];                  // [rg]
  pdl_trigger();
  pdl_wait();
  const int t = blockIdx.x, h = blockIdx.y;
  if (tok_req[t] < 0) return;
  const int HV = s.heads * s.V;
  const float* gin = proj + (size_t)t * s.stride + s.g_off;
  for (int k = threadIdx.x; k < s.rg; k += blockDim.x) s_gin[k] = gin[k];
  const float* src = o + (size_t)t * HV + (size_t)h * s.V;
  float ss = 0.f;
  for (int e = threadIdx.x; e < s.V; e += blockDim.x) ss = fmaf(src[e], src[e], ss);
  ss = warp_sum(ss);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
  __syncthreads();
  float tot = 0.f;
  for (int i = 0; i < (int)(blockDim.x >> 5); ++i) tot += red[i];
  const float inv = 1.0f / sqrtf(tot / (float)s.V + eps);
  for (int e = threadIdx.x; e < s.V; e += blockDim.x) {
    const float* gcol = g2 + (size_t)h * s.V + e;
    float z = 0.f;
    if (z_g) {                                     // W_g2 g was formed as a matrix product
      z = z_g[(size_t)t * HV + h * s.V + e];
    } else {
#pragma unroll 8
      for (int k = 0; k < s.rg; ++k) z = fmaf(gcol[(size_t)k * HV], s_gin[k], z);
    }
    out[(size_t)t * HV + h * s.V + e] = from_f<TO>(src[e] * inv * norm_w[e] * sigmoidf_(z));
  }
}

}  // namespace hs

static int delta_shape(hs::DeltaShape* s, int heads, int kv_heads, int D, int V, int taps, int ra,
                       int rg) {
  if (heads <= 0 || kv_heads <= 0 || heads % kv_heads || D <= 0 || V <= 0 || taps < 1 ||
      ra <= 0 || rg <= 0)
    return HS_ERR_UNSUPPORTED;
  s->heads = heads; s->kv_heads = kv_heads; s->D = D; s->V = V; s->taps = taps;
  s->ra = ra; s->rg = rg;
  const int C = 2 * kv_heads * D + heads * V;
  s->b_off = C;
  s->a_off = C + heads;
  s->g_off = C + heads + ra;
  s->stride = C + heads + ra + rg;
  s->state_stride = heads * D * V + (taps - 1) * C;
  return HS_OK;
}

// rows_form: a warp over several tokens or a head (1) or a block a token (0); -1: decided here.
HS_EXPORT int hs_delta_prepare(float* qn, float* kn, float* vv, float* beta, float* decay,
                               const float* proj, const float* conv_w, const float* a2,
                               const float* dt_bias, const float* A_log, float* state,
                               const int* tok_req, const int* req_start, const int* req_len,
                               const int* req_slot, int n_tokens, int n_requests, int heads,
                               int kv_heads, int D, int V, int taps, int ra, int rg,
                               const float* z_a, int rows_form, void* stream) {
  if (!qn || !kn || !vv || !beta || !decay || !proj || !conv_w || !a2 || !dt_bias || !A_log ||
      !state || !tok_req || !req_start || !req_len || !req_slot)
    return HS_ERR_ARGUMENT;
  hs::DeltaShape s;
  int rc = delta_shape(&s, heads, kv_heads, D, V, taps, ra, rg);
  if (rc) return rc;
  if (n_tokens <= 0 || n_requests <= 0) return HS_OK;
  const int C = 2 * kv_heads * D + heads * V;
  const size_t smem = (size_t)2 * kv_heads * D * sizeof(float);
  if (smem > 200 * 1024) return HS_ERR_UNSUPPORTED;
  cudaStream_t st = (cudaStream_t)stream;
  const int widest = 2 * kv_heads * D > heads * V ? 2 * kv_heads * D : heads * V;
  const bool four = taps == 4 && widest > 512 && n_tokens >= 512 && n_tokens >= 8 * n_requests;
  const bool pdl = hs_pdl_enabled();
  cudaError_t e;
  // Eight tokens a warp where there is work for many warps and few of the eights straddle portions: us, a block a
  // token against eight tokens a warp, 8 heads of 128 (W_a2 a handed in): 768 tokens 18.6 and 20.5, 1,536 30.1 and
  // 26.2, in portions of 64 31.1 and 28.4, of 16 32.9 and 33.8; 4 heads, 1,536 20.2 and 20.7, 4,096 45.5 and 28.2;
  // heads of 64 gain later (16 of them, 1,536 tokens 32.9 and 33.5, 4,096 91.7 and 71.8), heads of 32 not at all (64
  // of them, 4,096 190 and 209).  Where the warps form W_a2 a themselves: 8 heads of 128, 2,048 tokens 104 and 108,
  // 4,096 249 and 181; 16 heads, 512 tokens 66 and 97, 768 114 and 103, 1,536 236 and 158.
  const long long size = (long long)n_tokens * heads * D;
  bool rows = four && size >= (heads * D >= 2048 ? 3LL << 19 : 9LL << 18);
  if (z_a)
    rows = four && D >= 64 && n_tokens >= 32LL * n_requests &&
           size * D >= (n_tokens >= 128LL * n_requests ? 128LL : 160LL) << 20;
  if (rows_form >= 0) rows = rows_form && taps == 4;
  if (rows && D % 32 == 0 && D <= 128) {
    const int groups = 2 * kv_heads + (heads * V + 127) / 128 + (heads * D + 127) / 128;
    e = hs_launch(hs::delta_prepare_rows_kernel, dim3((n_tokens + hs::DP_TOK - 1) / hs::DP_TOK, (groups + 3) / 4),
                  dim3(128), 0, st, pdl, qn, kn, vv, beta, decay, proj, conv_w, a2, dt_bias, A_log,
                  (const float*)state, tok_req, req_start, req_slot, s, z_a, n_tokens);
  } else {
    auto* prepare = four ? hs::delta_prepare_kernel<true> : hs::delta_prepare_kernel<false>;
    if (smem > 48 * 1024)
      cudaFuncSetAttribute(prepare, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    e = hs_launch(prepare, dim3(n_tokens, 3), dim3(256), smem, st, pdl, qn, kn, vv, beta, decay, proj, conv_w, a2,
                  dt_bias, A_log, (const float*)state, tok_req, req_start, req_slot, s, z_a);
  }
  if (e != cudaSuccess) return (int)e;
  if (taps > 1) {
    dim3 grid((C + 127) / 128, n_requests);
    e = hs_launch(hs::delta_conv_state_kernel, grid, dim3(128), 0, st, pdl, state, proj, req_start, req_len,
                  req_slot, s);
    if (e != cudaSuccess) return (int)e;
  }
  return HS_OK;
}

// requests of long_from tokens or more that n_tokens tokens of n_requests requests can hold, and the
// blocks of four tokens these can bring
static int delta_most_long(int n_tokens, int n_requests, int long_from) {
  const int most = n_tokens / long_from;
  return n_requests < most ? n_requests : most;
}
static int delta_blocks_cap(int n_tokens, int n_requests, int long_from) {
  return n_tokens / hs::DB_TOK + delta_most_long(n_tokens, n_requests, long_from);
}

// Floats the blocks of n_tokens tokens of n_requests requests take when those of long_from tokens or
// more go four tokens at a time, or 0 when none can, by their number or by their size.
HS_EXPORT int hs_delta_blocks_scratch(int n_tokens, int n_requests, int heads, int D, int long_from,
                                      long long* floats) {
  if (!floats || long_from <= 0) return HS_ERR_ARGUMENT;
  *floats = (D == 64 || D == 128 || D == 256) && n_tokens >= long_from
                ? (long long)heads * delta_blocks_cap(n_tokens, n_requests, long_from) *
                      hs::db_floats(D)
                : 0;
  return HS_OK;
}

// `blocks` (hs_delta_blocks_scratch floats, 16-byte aligned; null: token after token): requests of
// long_from tokens or more go four tokens at a time.  `has_short` 0: there are no others.
HS_EXPORT int hs_delta_recurrence(float* o, float* state, const float* qn, const float* kn,
                                  const float* vv, const float* beta, const float* decay,
                                  const int* req_start, const int* req_len, const int* req_slot,
                                  int n_requests, int heads, int kv_heads, int D, int V, int taps,
                                  int ra, int rg, int n_tokens, int long_from, int has_short,
                                  float* blocks, int* status, void* stream) {
  if (!o || !state || !qn || !kn || !vv || !beta || !decay || !req_start || !req_len || !req_slot)
    return HS_ERR_ARGUMENT;
  hs::DeltaShape s;
  int rc = delta_shape(&s, heads, kv_heads, D, V, taps, ra, rg);
  if (rc) return rc;
  if (D > hs::DR_DP * 32) return HS_ERR_UNSUPPORTED;   // a column's parts are lanes of one warp
  if (n_requests <= 0) return HS_OK;
  int KS = 1;
  while (KS * hs::DR_DP < D) KS <<= 1;
  const int cols = hs::DR_THREADS / KS;
  const int Dp = KS * hs::DR_DP;
  int CH = 1024 / Dp;                               // tokens a chunk: 3 * CH * Dp <= 3072 floats
  CH = CH < 2 ? 2 : (CH > 16 ? 16 : CH);
  const size_t smem = hs::DR_STAGES * (size_t)((3 * CH * Dp + CH * cols + CH + 3) & ~3) * sizeof(float);
  // 16-byte copies need rows of q, k and the decay that start on 16-byte boundaries
  const int vec = D % 4 == 0 && !((uintptr_t)qn & 15) && !((uintptr_t)kn & 15) &&
                  !((uintptr_t)decay & 15);
  dim3 grid(n_requests, heads, (V + cols - 1) / cols);
  cudaStream_t st = (cudaStream_t)stream;
  const bool with_blocks = blocks && n_tokens >= long_from;
  if (with_blocks && ((D != 64 && D != 128 && D != 256) || ((uintptr_t)blocks & 15) || !status ||
                      long_from <= 0))
    return HS_ERR_ARGUMENT;
  if (has_short || !with_blocks) {
    hs::delta_recurrence_kernel<<<grid, hs::DR_THREADS, smem, st>>>(
        o, state, qn, kn, vv, beta, decay, req_start, req_len, req_slot, s, KS, CH, vec,
        with_blocks ? long_from : 0x7fffffff);
    HS_LAUNCH_CHECK();
  }
  if (!with_blocks) return HS_OK;
  const int most = delta_most_long(n_tokens, n_requests, long_from);
  const int cap = delta_blocks_cap(n_tokens, n_requests, long_from);
  cudaError_t e = hs_launch(hs::delta_blocks_prepare_kernel, dim3(cap, heads), dim3(128), 0, st,
                            hs_pdl_enabled(), blocks, qn, kn, beta, decay, req_start, req_len, n_requests, cap,
                            s, long_from);
  if (e != cudaSuccess) return (int)e;
  const size_t block_smem =
      (size_t)hs::DB_STAGES * hs::DB_STAGE_BLOCKS * hs::db_floats(D) * sizeof(float);
#define HS_DB(KS)                                                                                 \
  do {                                                                                            \
    const int block_cols = hs::DB_WARPS * (32 / KS);                                              \
    e = cudaFuncSetAttribute(hs::delta_blocks_kernel<KS>,                                         \
                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)block_smem);       \
    if (e == cudaSuccess)                                                                         \
      e = hs_launch(hs::delta_blocks_kernel<KS>,                                                  \
                    dim3(most, heads, (V + block_cols - 1) / block_cols),                         \
                    dim3(hs::DB_WARPS * 32 + 32), block_smem, st, hs_pdl_enabled(), o, state,     \
                    (const float*)blocks, vv, req_start, req_len, req_slot, n_requests, cap, s,   \
                    long_from, status);                                                           \
  } while (0)
  if (D == 64) HS_DB(4);
  else if (D == 128) HS_DB(8);
  else HS_DB(16);
#undef HS_DB
  if (e != cudaSuccess) return (int)e;
  HS_LAUNCH_CHECK();
  return HS_OK;
}

// rows_form: a warp over several tokens or a head (1) or a block a token (0); -1: decided here.
HS_EXPORT int hs_delta_finish(void* out, const float* o, const float* proj, const float* g2,
                              const float* norm_w, const int* tok_req, int n_tokens, float eps,
                              int heads, int kv_heads, int D, int V, int taps, int ra, int rg,
                              int out_dtype, const float* z_g, int rows_form, void* stream) {
  if (!out || !o || !proj || !g2 || !norm_w || !tok_req) return HS_ERR_ARGUMENT;
  hs::DeltaShape s;
  int rc = delta_shape(&s, heads, kv_heads, D, V, taps, ra, rg);
  if (rc) return rc;
  if (n_tokens <= 0) return HS_OK;
  cudaStream_t st = (cudaStream_t)stream;
  const bool pdl = hs_pdl_enabled();
  cudaError_t e;
  auto go = [&](auto* dst) {
    using TO = std::remove_pointer_t<decltype(dst)>;
    if (z_g && rows_form != 0 && V % 32 == 0 && V <= 256)
      e = hs_launch(hs::delta_finish_rows_kernel<TO>, dim3(((long long)n_tokens * heads + 7) / 8), dim3(256), 0,
                    st, pdl, dst, o, norm_w, tok_req, eps, s, z_g, n_tokens);
    else
      e = hs_launch(hs::delta_finish_kernel<TO>, dim3(n_tokens, heads), dim3(128), rg * sizeof(float), st, pdl,
                    dst, o, proj, g2, norm_w, tok_req, eps, s, z_g);
  };
  if (out_dtype == HS_DT_F32) go((float*)out);
  else if (out_dtype == HS_DT_BF16) go((__nv_bfloat16*)out);
  else return HS_ERR_UNSUPPORTED;
  return e == cudaSuccess ? HS_OK : (int)e;
}

