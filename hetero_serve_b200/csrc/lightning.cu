// Linear attention with a constant decay per head (lightning attention), as a recurrence on a
// float32 state S [dim, vdim] per head and request:
//
//     q, k, v = act(projection columns)        act = silu, applied here in float32
//     S <- decay_h * S + k v^T ;   o = S^T q    token after token
//
// The state lives in the request's state slot ([heads, dim, vdim] floats) and is carried from
// step to step.  One block per (request, head, group of value columns): a thread keeps 16 rows
// of one column of S in registers, the P = ceil(dim / 16) (rounded up to a power of two) parts
// of a column are neighbouring lanes of one warp and fold their shares of o by a butterfly.
// The tokens' rows are staged through shared memory 16 tokens at a time, two buffers in turn:
// for steps of many tokens the activations are applied by a pass of their own into compact rows
// and the recurrence fetches the next portion by cp.async while it walks the current one.  A
// token's arithmetic is the same chain whatever the batch or the cut of the prompt: results are
// bit-equal across both.
//
// Retention is the same recurrence with q and k turned by the token's position on their first
// rot_dims numbers (number i pairs with i + rot_dims/2) and k scaled: with a table of
// frequencies the rows are turned where they are activated (in the pass of its own, or while
// they are staged), by the same expression in both places.
#include "lightning.cuh"
#include "tcgen05.cuh"

namespace hs {

constexpr int LA_THREADS = 128;
constexpr int LA_ROWS = 16;          // state rows a thread keeps
constexpr int LA_PART = LA_ROWS + 4; // floats between two parts' rows of a token in shared memory:
                                     // the parts of a column read 16-byte pieces from distinct banks
constexpr int LA_TOK = 16;           // tokens staged at a time (8 when dim is above 128)

__device__ __forceinline__ void la_cp16(void* smem_dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem_dst)), "l"(src)
               : "memory");
}

// dst[t, :] = act(q | k | v columns of proj[t]) as one compact row of 2 H D + H V floats
__global__ void lightning_act_kernel(float* __restrict__ dst, const float* __restrict__ proj,
                                     int n_tokens, int stride, int q_off, int k_off, int v_off,
                                     int hd, int hv, int act, int D,
                                     const int* __restrict__ tok_pos,
                                     const float* __restrict__ freq, int rot_dims,
                                     float k_scale) {
  pdl_trigger();
  pdl_wait();
  const int row_len = 2 * hd + hv;
  for (int t = blockIdx.x; t < n_tokens; t += gridDim.x) {
    const float* row = proj + (size_t)t * stride;
    float* out = dst + (size_t)t * row_len;
    const int pos = rot_dims > 0 ? tok_pos[t] : 0;
    for (int c = threadIdx.x; c < row_len; c += blockDim.x) {
      if (c < 2 * hd) {
        const bool is_q = c < hd;
        const int e = is_q ? c : c - hd, d = e % D;
        out[c] = la_entry(row + (is_q ? q_off : k_off) + (e - d), d, act, rot_dims, freq, pos,
                          is_q ? 1.0f : k_scale);
      } else {
        out[c] = la_act(row[v_off + c - 2 * hd], act);
      }
    }
  }
}

// One token on a thread's 16 state rows: s <- decay s + k v, and the thread's share of o = S^T q
// as four partial sums folded pairwise (the same order wherever the token stands).
__device__ __forceinline__ float la_token(float (&s)[LA_ROWS], const float* kp, const float* qp,
                                          float vt, float dh) {
  float part_sum[LA_ROWS / 4];
#pragma unroll
  for (int i4 = 0; i4 < LA_ROWS / 4; ++i4) {
    const float4 k4 = *(const float4*)(kp + 4 * i4), q4 = *(const float4*)(qp + 4 * i4);
    s[4 * i4 + 0] = fmaf(k4.x, vt, dh * s[4 * i4 + 0]);
    s[4 * i4 + 1] = fmaf(k4.y, vt, dh * s[4 * i4 + 1]);
    s[4 * i4 + 2] = fmaf(k4.z, vt, dh * s[4 * i4 + 2]);
    s[4 * i4 + 3] = fmaf(k4.w, vt, dh * s[4 * i4 + 3]);
    float a = s[4 * i4 + 0] * q4.x;
    a = fmaf(s[4 * i4 + 1], q4.y, a);
    a = fmaf(s[4 * i4 + 2], q4.z, a);
    part_sum[i4] = fmaf(s[4 * i4 + 3], q4.w, a);
  }
  return (part_sum[0] + part_sum[1]) + (part_sum[2] + part_sum[3]);
}

// A portion of up to ntok tokens of request rows (from token `tok` on) into one buffer (q [ntok][Dp],
// k [ntok][Dp], v [ntok][cols]).  `bulk`: the rows are activated already and 16-byte aligned,
// and go in by cp.async (the walk over the portion before runs meanwhile); otherwise plain loads
// with the activation applied on the way.
__device__ __forceinline__ void la_stage(float* s_q, const float* __restrict__ proj, int tok,
                                         int here, int stride, int q_off, int k_off, int v_off,
                                         int h, int D, int V, int Dp, int cols, int v0, int ntok,
                                         int act, int bulk, const int* __restrict__ tok_pos,
                                         const float* __restrict__ freq, int rot_dims,
                                         float k_scale) {
  float* s_k = s_q + ntok * Dp;
  float* s_v = s_k + ntok * Dp;
  if (bulk) {
    const int dq = D / 4, cq = cols / 4;
    for (int e = threadIdx.x; e < here * dq; e += LA_THREADS) {
      const int tt = e / dq, c = e - tt * dq;
      const float* row = proj + (size_t)(tok + tt) * stride + (size_t)h * D + 4 * c;
      const int at = tt * Dp + (4 * c) / LA_ROWS * LA_PART + (4 * c) % LA_ROWS;
      la_cp16(s_q + at, row + q_off);
      la_cp16(s_k + at, row + k_off);
    }
    for (int e = threadIdx.x; e < here * cq; e += LA_THREADS) {
      const int tt = e / cq, c = e - tt * cq;
      if (v0 + 4 * c < V)
        la_cp16(s_v + tt * cols + 4 * c,
                proj + (size_t)(tok + tt) * stride + v_off + (size_t)h * V + v0 + 4 * c);
    }
  } else {
#pragma unroll 4
    for (int e = threadIdx.x; e < here * D; e += LA_THREADS) {
      const int tt = e / D, d = e - tt * D;
      const float* row = proj + (size_t)(tok + tt) * stride + (size_t)h * D;
      const int at = tt * Dp + d / LA_ROWS * LA_PART + d % LA_ROWS;
      const int pos = rot_dims > 0 ? tok_pos[tok + tt] : 0;
      s_q[at] = la_entry(row + q_off, d, act, rot_dims, freq, pos, 1.0f);
      s_k[at] = la_entry(row + k_off, d, act, rot_dims, freq, pos, k_scale);
    }
    for (int e = threadIdx.x; e < here * cols; e += LA_THREADS) {
      const int tt = e / cols, c = e - tt * cols;
      if (v0 + c < V)
        s_v[e] = la_act(proj[(size_t)(tok + tt) * stride + v_off + (size_t)h * V + v0 + c], act);
    }
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}

__global__ void __launch_bounds__(LA_THREADS, 1)
lightning_kernel(float* __restrict__ o, float* __restrict__ state, const float* __restrict__ proj,
                 const float* __restrict__ decay, const int* __restrict__ req_start,
                 const int* __restrict__ req_len, const int* __restrict__ req_slot, int stride,
                 int q_off, int k_off, int v_off, int H, int D, int V, int P, int act, int ntok,
                 int bulk, const int* __restrict__ tok_pos, const float* __restrict__ freq,
                 int rot_dims, float k_scale, int most) {
  extern __shared__ __align__(16) float smem[];
  pdl_trigger();
  pdl_wait();
  const int Dp = P * LA_PART;                       // a token's q (or k) row: P parts, padded
  const int cols = LA_THREADS / P;                  // value columns of this block
  const int per_buf = ntok * (2 * Dp + cols);       // a buffer: q [ntok][Dp], k [ntok][Dp], v [ntok][cols]
  const int r = blockIdx.z, h = blockIdx.y;
  const int n = req_len[r];
  if (n <= 0 || n > most) return;
  const int t0 = req_start[r];
  const int slot = req_slot[r];
  const int part = threadIdx.x % P, col = threadIdx.x / P;
  const int v0 = blockIdx.x * cols;
  const int v = v0 + col;
  const bool col_ok = v < V;
  const float dh = decay[h];
  float* S = state + ((size_t)slot * H + h) * D * V;
  float s[LA_ROWS];
#pragma unroll
  for (int i = 0; i < LA_ROWS; ++i) {
    const int d = part * LA_ROWS + i;
    s[i] = (col_ok && d < D) ? S[(size_t)d * V + v] : 0.f;
  }
  if (D != P * LA_ROWS || V % cols) {               // rows or columns past the sizes read as zero
    for (int e = threadIdx.x; e < 2 * per_buf; e += LA_THREADS) smem[e] = 0.f;
    __syncthreads();
  }
  la_stage(smem, proj, t0, min(ntok, n), stride, q_off, k_off, v_off, h, D, V, Dp, cols, v0, ntok,
           act, bulk, tok_pos, freq, rot_dims, k_scale);
  int buf = 0;
  for (int base = 0; base < n; base += ntok, buf ^= 1) {
    const int here = min(ntok, n - base);
    if (base + ntok < n) {
      la_stage(smem + (buf ^ 1) * per_buf, proj, t0 + base + ntok, min(ntok, n - base - ntok), stride,
               q_off, k_off, v_off, h, D, V, Dp, cols, v0, ntok, act, bulk, tok_pos, freq, rot_dims,
               k_scale);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    const float* s_q = smem + buf * per_buf;
    const float* s_k = s_q + ntok * Dp;
    const float* s_v = s_k + ntok * Dp;
    int tt = 0;
    for (; tt + 4 <= here; tt += 4) {               // four tokens: their sums and folds overlap
      float acc[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        acc[u] = la_token(s, s_k + (tt + u) * Dp + part * LA_PART,
                          s_q + (tt + u) * Dp + part * LA_PART, s_v[(tt + u) * cols + col], dh);
      for (int off = 1; off < P; off <<= 1) {
#pragma unroll
        for (int u = 0; u < 4; ++u) acc[u] += __shfl_xor_sync(0xffffffffu, acc[u], off);
      }
      if (part == 0 && col_ok) {
#pragma unroll
        for (int u = 0; u < 4; ++u)
          o[(size_t)(t0 + base + tt + u) * H * V + (size_t)h * V + v] = acc[u];
      }
    }
    for (; tt < here; ++tt) {
      float acc = la_token(s, s_k + tt * Dp + part * LA_PART, s_q + tt * Dp + part * LA_PART,
                           s_v[tt * cols + col], dh);
      for (int off = 1; off < P; off <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
      if (part == 0 && col_ok) o[(size_t)(t0 + base + tt) * H * V + (size_t)h * V + v] = acc;
    }
    __syncthreads();                                // this buffer is staged into again next turn
  }
#pragma unroll
  for (int i = 0; i < LA_ROWS; ++i) {
    const int d = part * LA_ROWS + i;
    if (col_ok && d < D) S[(size_t)d * V + v] = s[i];
  }
}

// ---- steps of many tokens, heads of 64, 128 or 256 --------------------------------------------
// The same chain of operations per token (the same bits), laid out for a stream of tokens.  The
// kernel above spends 108 instructions a token and warp and waits for shared memory in front of most
// of them (0.24 us a token at one warp a scheduler).  Here
//   * the rows pass through `lightning_rows_kernel`, which activates, turns and scales them (an angle
//     is formed once per token, not once per head and entry) and leaves them in the order in which
//     they are used: per head and token, 16-byte piece j of every part side by side, and inside a part
//     entries i and i + 4 neighbours, so that a part's four partial sums are two packed pairs;
//     values per head and group of columns;
//   * a warp of the recurrence only fetches: a stage of LS_TOK tokens is two bulk copies;
//   * state, products and sums are packed two an instruction (fma.rn.f32x2, each half rounded as
//     fmaf rounds), four tokens at a time, the rows of the next four read ahead; the parts lie on
//     lane bits 1 up (a 16-byte read by a warp: two wavefronts of shared memory, four on bits 0 up);
//   * the four tokens' sums over the parts are exchanged so that a lane finishes one of them (the
//     butterfly's tree, a third of its shuffles).
// Measured (2 x 1,024 tokens, 8 heads of 128 x 128): the recurrence 249 -> 70-99 us; about one working
// warp a scheduler waits on its chain (shared-memory pipe 38 % busy: eight 16-byte reads a token and
// warp).
constexpr int LS_TOK = 8, LS_STAGES = 4, LS_WARPS = 4;

__host__ __device__ constexpr int ls_cols(int D) { return LS_WARPS * 32 * LA_ROWS / D; }

// q | k of token t and head h: rows + ((h * n_tokens + t) * 2 D); value column c of head h: group
// c / cols: vals + (((h * groups + c / cols) * n_tokens + t) * cols + c % cols), columns past V zero.
// A block takes one token and `per` heads: all of them where there are tokens enough, fewer where the
// blocks would leave SMs idle (the whole operation, 128 tokens of 32 heads of 128: 71 us with one
// block a token, 28 so).
__global__ void __launch_bounds__(256)
lightning_rows_kernel(float* __restrict__ rows, float* __restrict__ vals,
                      const float* __restrict__ proj, int n_tokens, int stride, int q_off, int k_off,
                      int v_off, int H, int D, int V, int act, const int* __restrict__ tok_pos,
                      const float* __restrict__ freq, int rot_dims, float k_scale, int per,
                      const int* __restrict__ req_start, const int* __restrict__ req_len,
                      int n_requests, int most) {
  pdl_trigger();
  pdl_wait();
  __shared__ float s_c[128], s_s[128];
  const int h0 = blockIdx.y * per, nh = min(per, H - h0);
  const int t = blockIdx.x, half = rot_dims >> 1;
  if (most < n_tokens) {                                  // rows of a request that goes in chunks
    bool left_out = false;
    for (int r = threadIdx.x; r < n_requests; r += blockDim.x)
      left_out = left_out || (req_len[r] > most && t >= req_start[r] && t < req_start[r] + req_len[r]);
    if (__syncthreads_or(left_out)) return;
  }
  const int pos = rot_dims > 0 ? tok_pos[t] : 0;
  for (int i = threadIdx.x; i < half; i += blockDim.x) pair_angle(pos, freq[i], &s_c[i], &s_s[i]);
  __syncthreads();
  const float* row = proj + (size_t)t * stride;
  const int P4 = D / 4;                                   // floats of a piece over all parts
  for (int x = threadIdx.x; x < 2 * nh * D; x += blockDim.x) {
    const int hh = x / (2 * D), y = x - hh * 2 * D, h = h0 + hh;
    const bool is_q = y < D;
    const int z = is_q ? y : y - D;
    const int j = z / P4, part = (z - j * P4) >> 2, e = z & 3;
    const int at = 4 * j + e;                             // place inside the part
    const int i = (at & 8) + ((at & 7) >> 1) + ((at & 1) << 2);
    const int d = part * LA_ROWS + i;
    const float* vec = row + (is_q ? q_off : k_off) + h * D;
    float own = la_act(vec[d], act);
    if (d < rot_dims) {                                   // as la_entry
      const bool low = d < half;
      const float partner = la_act(vec[low ? d + half : d - half], act);
      const int f = low ? d : d - half;
      const float cross = __fmul_rn(partner, s_s[f]);
      own = fmaf(own, s_c[f], low ? -cross : cross);
    }
    rows[((size_t)h * n_tokens + t) * 2 * D + y] = __fmul_rn(own, is_q ? 1.0f : k_scale);
  }
  const int cols = ls_cols(D), groups = (V + cols - 1) / cols;
  for (int x = threadIdx.x; x < nh * groups * cols; x += blockDim.x) {
    const int hh = x / (groups * cols), c = x - hh * groups * cols, g = c / cols, h = h0 + hh;
    vals[(((size_t)h * groups + g) * n_tokens + t) * cols + (c - g * cols)] =
        c < V ? la_act(row[v_off + h * V + c], act) : 0.f;
  }
}

__device__ __forceinline__ uint64_t ls_fma(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t ls_mul(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t ls_pair(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float ls_lo(uint64_t a) { return __uint_as_float((uint32_t)a); }
__device__ __forceinline__ float ls_hi(uint64_t a) { return __uint_as_float((uint32_t)(a >> 32)); }

template <int P>                                          // parts of a column: D / 16
__global__ void __launch_bounds__(LS_WARPS * 32 + 32, 1)
lightning_stream_kernel(float* __restrict__ o, float* __restrict__ state,
                        const float* __restrict__ rows, const float* __restrict__ vals,
                        const float* __restrict__ decay, const int* __restrict__ req_start,
                        const int* __restrict__ req_len, const int* __restrict__ req_slot,
                        int n_tokens, int H, int V, int most, int* status) {
  constexpr int D = P * LA_ROWS, COLS = 32 / P, CTA_COLS = LS_WARPS * COLS;
  extern __shared__ __align__(16) float smem[];           // [stages][LS_TOK][q | k], then the values
  __shared__ uint64_t full[LS_STAGES], empty[LS_STAGES];
  float* s_v = smem + LS_STAGES * LS_TOK * 2 * D;         // [stages][LS_TOK][CTA_COLS]
  const int r = blockIdx.z, h = blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < LS_STAGES; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], LS_WARPS);
    }
    fence_barrier_init();
  }
  __syncthreads();
  pdl_trigger();
  pdl_wait();
  const int n = req_len[r];
  if (n <= 0 || n > most) return;
  const int t0 = req_start[r], n_stages = (n + LS_TOK - 1) / LS_TOK;
  if (warp == LS_WARPS) {
    if (lane == 0) {
      const float* src = rows + ((size_t)h * n_tokens + t0) * 2 * D;
      const float* vsrc = vals + (((size_t)h * gridDim.x + blockIdx.x) * n_tokens + t0) * CTA_COLS;
      int i = 0;
      for (; i < n_stages; ++i) {
        const int st = i % LS_STAGES;
        if (i >= LS_STAGES && !mbar_wait(&empty[st], ((i / LS_STAGES) - 1) & 1, status)) break;
        const int here = min(LS_TOK, n - i * LS_TOK);
        const uint32_t rb = (uint32_t)(here * 2 * D * 4), vb = (uint32_t)(here * CTA_COLS * 4);
        mbar_expect_tx(&full[st], rb + vb);
        asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                smem_u32(smem + (size_t)st * LS_TOK * 2 * D)),
            "l"(src + (size_t)i * LS_TOK * 2 * D), "r"(rb), "r"(smem_u32(&full[st]))
            : "memory");
        asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                smem_u32(s_v + (size_t)st * LS_TOK * CTA_COLS)),
            "l"(vsrc + (size_t)i * LS_TOK * CTA_COLS), "r"(vb), "r"(smem_u32(&full[st]))
            : "memory");
      }
      // the block stays until what it fetched has landed, also where the working warps gave up
      for (int k = max(0, i - LS_STAGES); k < i; ++k)
        mbar_wait(&full[k % LS_STAGES], (k / LS_STAGES) & 1, status);
    }
    return;
  }
  const int part = (lane >> 1) & (P - 1);
  const int lc = warp * COLS + ((lane & 1) | ((lane >> 1) / P) << 1);
  const int v = blockIdx.x * CTA_COLS + lc;
  const bool col_ok = v < V;
  const int tok = 2 * (part & 1) + ((part >> 1) & 1);     // the token of four this lane finishes
  const bool stores = part < 4 && col_ok;
  const uint64_t dh = ls_pair(decay[h], decay[h]);
  float* S = state + (((size_t)req_slot[r] * H + h) * D + part * LA_ROWS) * V + v;
  uint64_t s[8];                                          // rows (i, i + 4), then (8 + i, 12 + i)
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int d = (i & 4) * 2 + (i & 3);
    s[i] = col_ok ? ls_pair(S[(size_t)d * V], S[(size_t)(d + 4) * V]) : 0;
  }
  float* ocol = o + (size_t)(t0 + tok) * H * V + (size_t)h * V + v;

  struct Rows { ulonglong2 q[4], k[4]; float v; };
  auto read = [&](const float* x, const float* xv, int tt, Rows& f) {
    const float* at = x + (size_t)tt * 2 * D + 4 * part;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      f.q[j] = *(const ulonglong2*)(at + 4 * P * j);
      f.k[j] = *(const ulonglong2*)(at + D + 4 * P * j);
    }
    f.v = xv[tt * CTA_COLS + lc];
  };
  auto token = [&](const Rows& f) {
    const uint64_t vt = ls_pair(f.v, f.v);
    uint64_t sum[2];
#pragma unroll
    for (int g = 0; g < 2; ++g) {                         // quads 0 and 1, quads 2 and 3
      const uint64_t k[4] = {f.k[2 * g].x, f.k[2 * g].y, f.k[2 * g + 1].x, f.k[2 * g + 1].y};
      const uint64_t q[4] = {f.q[2 * g].x, f.q[2 * g].y, f.q[2 * g + 1].x, f.q[2 * g + 1].y};
#pragma unroll
      for (int e = 0; e < 4; ++e) s[4 * g + e] = ls_fma(k[e], vt, ls_mul(dh, s[4 * g + e]));
      uint64_t a = ls_mul(s[4 * g], q[0]);
#pragma unroll
      for (int e = 1; e < 4; ++e) a = ls_fma(s[4 * g + e], q[e], a);
      sum[g] = a;
    }
    return (ls_lo(sum[0]) + ls_hi(sum[0])) + (ls_lo(sum[1]) + ls_hi(sum[1]));
  };
  const bool hi = part & 1, hi2 = part & 2;
  for (int i = 0; i < n_stages; ++i) {
    const int st = i % LS_STAGES;
    if (!mbar_wait(&full[st], (i / LS_STAGES) & 1, status)) return;
    const float* x = smem + (size_t)st * LS_TOK * 2 * D;
    const float* xv = s_v + st * LS_TOK * CTA_COLS;
    const int here = min(LS_TOK, n - i * LS_TOK);
    int tt = 0;
#pragma unroll
    for (int b = 0; b < LS_TOK; b += 4) {
      if (b + 4 > here) break;
      Rows f[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) read(x, xv, b + u, f[u]);
      float a[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) a[u] = token(f[u]);
      float w0 = hi ? a[2] : a[0], w1 = hi ? a[3] : a[1];
      w0 += __shfl_xor_sync(0xffffffffu, hi ? a[0] : a[2], 2);
      w1 += __shfl_xor_sync(0xffffffffu, hi ? a[1] : a[3], 2);
      float out = hi2 ? w1 : w0;
      out += __shfl_xor_sync(0xffffffffu, hi2 ? w0 : w1, 4);
#pragma unroll
      for (int off = 8; off <= P; off <<= 1) out += __shfl_xor_sync(0xffffffffu, out, off);
      if (stores) ocol[(size_t)(i * LS_TOK + b) * H * V] = out;
      tt = b + 4;
    }
    for (; tt < here; ++tt) {
      Rows f;
      read(x, xv, tt, f);
      float a = token(f);
#pragma unroll
      for (int off = 2; off <= P; off <<= 1) a += __shfl_xor_sync(0xffffffffu, a, off);
      if (part == 0 && col_ok) o[(size_t)(t0 + i * LS_TOK + tt) * H * V + (size_t)h * V + v] = a;
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[st]);
  }
  if (col_ok) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int d = (i & 4) * 2 + (i & 3);
      S[(size_t)d * V] = ls_lo(s[i]);
      S[(size_t)(d + 4) * V] = ls_hi(s[i]);
    }
  }
}

}  // namespace hs

// Whether a step goes as a stream: sizes it is written for, and four tokens a request or more on
// average.  With fewer the blocks' set-up outweighs what a token saves (256 single
// tokens, 8 heads of 128: 145 us as a stream, 131 otherwise); the bits are the same
// either way.
static bool lightning_streams(int n_tokens, int n_requests, int D) {
  return (D == 64 || D == 128 || D == 256) && n_tokens >= 4ll * n_requests;
}

// Floats of scratch with which hs_lightning_recurrence takes many tokens a step.
HS_EXPORT int hs_lightning_scratch(int n_tokens, int n_requests, int H, int D, int V,
                                   long long* floats) {
  if (!floats || n_tokens < 0 || H <= 0 || D <= 0 || V <= 0) return HS_ERR_ARGUMENT;
  if (lightning_streams(n_tokens, n_requests, D)) {
    const int cols = hs::ls_cols(D);
    *floats = (long long)n_tokens * H * (2 * D + (V + cols - 1) / cols * cols);
  } else {
    *floats = D % 4 == 0 && V % 4 == 0 ? (long long)n_tokens * H * (2 * D + V) : 0;
  }
  return HS_OK;
}

// Floats of scratch with which requests of many tokens go in chunks (0: none can), and how many groups of heads
// take turns with it.
HS_EXPORT int hs_lightning_chunk_scratch(int n_tokens, int n_requests, int H, int D, int V, int rot_dims,
                                         long long* floats, int* groups) {
  if (!floats || !groups || n_tokens < 0 || n_requests < 0 || H <= 0 || D <= 0 || V <= 0) return HS_ERR_ARGUMENT;
  *floats = hs::lightning_takes_chunks(D, V, rot_dims)
                ? hs::lightning_chunk_floats(n_tokens, n_requests, H, D, V, rot_dims) : 0;
  const int heads = hs::lightning_chunk_heads(n_tokens, n_requests, H, D, V);
  *groups = (H + heads - 1) / heads;
  return HS_OK;
}

// proj: float32 rows of `stride` columns holding q (H*D at q_off), k (H*D at k_off) and v (H*V at
// v_off), head by head; o: float32 [tokens, H*V]; state: [slots, H*D*V] float32.  `scratch`
// (hs_lightning_scratch floats, or null): with it the activations are applied in a pass of their own
// and the recurrence streams the activated rows; the results are the same bits.  `chunks`
// (hs_lightning_chunk_scratch floats, or null): with it requests of hs::LC_MIN tokens and more go in chunks
// on the tensor cores (lightning_chunk.cu: sums in another order), each by its own length; `walks` 0 says that
// there are no others, so that nothing is launched for them.
HS_EXPORT int hs_lightning_recurrence(float* o, float* state, const float* proj,
                                      const float* decay, const int* req_start,
                                      const int* req_len, const int* req_slot, int n_requests,
                                      int n_tokens, int stride, int q_off, int k_off, int v_off,
                                      int H, int D, int V, int act, float* scratch,
                                      const int* tok_pos, const float* freq, int rot_dims,
                                      float k_scale, float* chunks, int walks, int* status, void* stream) {
  if (!o || !state || !proj || !decay || !req_start || !req_len || !req_slot)
    return HS_ERR_ARGUMENT;
  if (rot_dims < 0 || rot_dims % 2 || rot_dims > D || (rot_dims > 0 && (!freq || !tok_pos)))
    return HS_ERR_ARGUMENT;
  if (H <= 0 || D <= 0 || V <= 0 || D > 16 * hs::LA_ROWS || (act != HS_ACT_NONE && act != HS_ACT_SILU))
    return HS_ERR_UNSUPPORTED;
  if (n_requests <= 0 || n_tokens <= 0) return HS_OK;
  cudaStream_t st = (cudaStream_t)stream;
  int most = 0x7fffffff;                // tokens of the requests that are walked here
  if (chunks && hs::lightning_chunk_slots(n_tokens, n_requests) > 0 &&
      hs::lightning_takes_chunks(D, V, rot_dims) &&
      !(((uintptr_t)chunks | (uintptr_t)state) & 15) && !((uintptr_t)o & 7)) {
    if (int e = hs::lightning_chunks(o, state, proj, decay, req_start, req_len, req_slot, n_requests, n_tokens,
                                     stride, q_off, k_off, v_off, H, D, V, act, chunks, tok_pos, freq, rot_dims,
                                     k_scale, st))
      return e;
    if (!walks) return HS_OK;
    most = hs::LC_MIN - 1;
  }
  if (scratch && status && lightning_streams(n_tokens, n_requests, D) && !((uintptr_t)scratch & 15)) {
    // (measured, 2 x 1,024 tokens, 8 heads of 128 x 128: retention's mixer takes 176 us this way, 395
    // with the two kernels below)
    const int cols = hs::ls_cols(D), groups = (V + cols - 1) / cols;
    float* vals = scratch + (size_t)n_tokens * H * 2 * D;
    const int want = (8 * hs_sm_count() + n_tokens - 1) / n_tokens;     // blocks a token
    const int per = want >= H ? 1 : (H + want - 1) / want;
    cudaError_t e = hs_launch(hs::lightning_rows_kernel, dim3(n_tokens, (H + per - 1) / per),
                              dim3(256), 0, st,
                              hs_pdl_enabled(), scratch, vals, proj, n_tokens, stride, q_off, k_off,
                              v_off, H, D, V, act, tok_pos, freq, rot_dims, k_scale, per, req_start,
                              req_len, n_requests, most);
    if (e != cudaSuccess) return (int)e;
    const size_t smem = (size_t)hs::LS_STAGES * hs::LS_TOK * (2 * D + cols) * sizeof(float);
#define HS_LS(P)                                                                                 \
  do {                                                                                           \
    e = cudaFuncSetAttribute(hs::lightning_stream_kernel<P>,                                     \
                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);            \
    if (e == cudaSuccess)                                                                        \
      e = hs_launch(hs::lightning_stream_kernel<P>, dim3(groups, H, n_requests),                 \
                    dim3(hs::LS_WARPS * 32 + 32), smem, st, hs_pdl_enabled(), o, state,          \
                    (const float*)scratch, (const float*)vals, decay, req_start, req_len,        \
                    req_slot, n_tokens, H, V, most, status);                                           \
  } while (0)
    if (D == 64) HS_LS(4);
    else if (D == 128) HS_LS(8);
    else HS_LS(16);
#undef HS_LS
    return (int)e;
  }
  int P = 1;
  while (P * hs::LA_ROWS < D) P *= 2;
  const int cols = hs::LA_THREADS / P;
  const int ntok = P * hs::LA_ROWS > 128 ? hs::LA_TOK / 2 : hs::LA_TOK;   // at most 45 KB
  int bulk = 0;
  if (scratch && D % 4 == 0 && V % 4 == 0 && (((uintptr_t)scratch) & 15) == 0) {
    const int hd = H * D, hv = H * V;
    int blocks = n_tokens < 148 * 8 ? n_tokens : 148 * 8;
    cudaError_t e = hs_launch(hs::lightning_act_kernel, dim3(blocks), dim3(256), 0, st,
                              hs_pdl_enabled(), scratch, proj, n_tokens, stride, q_off, k_off,
                              v_off, hd, hv, act, D, tok_pos, freq, rot_dims, k_scale);
    if (e != cudaSuccess) return (int)e;
    proj = scratch;
    stride = 2 * hd + hv;
    q_off = 0; k_off = hd; v_off = 2 * hd;
    act = HS_ACT_NONE;
    rot_dims = 0;           // the rows are turned and scaled already
    k_scale = 1.0f;
    bulk = 1;
  }
  const size_t smem = (size_t)2 * ntok * (2 * P * hs::LA_PART + cols) * sizeof(float);
  dim3 grid((V + cols - 1) / cols, H, n_requests);
  cudaError_t e = hs_launch(hs::lightning_kernel, grid, dim3(hs::LA_THREADS), smem, st,
                            hs_pdl_enabled(), o, state, proj, decay, req_start, req_len, req_slot,
                            stride, q_off, k_off, v_off, H, D, V, P, act, ntok, bulk, tok_pos, freq,
                            rot_dims, k_scale, most);
  if (e != cudaSuccess) return (int)e;
  return HS_OK;
}
