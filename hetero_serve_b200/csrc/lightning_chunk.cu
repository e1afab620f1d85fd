// Lightning attention and retention (lightning.cu) over long prompt portions, in chunks of 64 tokens on
// the tensor cores (mma.sync m16n8k16, bfloat16 operands, float32 accumulators).
//
// With g the head's decay, S the state in front of a chunk of n tokens and S' the state behind it,
//
//     o_t = g^(t+1) S^T q_t + sum_{j <= t} g^(t-j) (q_t . k_j) v_j
//     S'  = g^n S + sum_j (g^(n-1-j) k_j) v_j^T
//
// so that everything but the chain of states is parallel over chunks, requests and heads:
//
//   chunk_state   the chunk's own contribution to S'
//   chunk_chain   S from chunk to chunk, element by element, in place of the contributions; the
//                 request's slot receives the last state
//   chunk_out     o
//
// Every operand is a float32 number and enters a product as the sum of three bfloat16 terms, its whole
// mantissa; of the nine products of terms the six above 2^-24 of the whole are formed, the small ones in
// an accumulator of their own.  Powers of the decay are formed in double.  The
// results are no further off float64 than the recurrence's.
//
// A chunk with a number that is not finite (or too large for its first term) is walked token by token
// instead, so that such a number stays behind its token as in the recurrence.
//
// A request's form depends on its own portion alone: chunks from LC_MIN tokens on, else lightning.cu's
// recurrence.  2 x 1,024 tokens, 8 heads: 148 us as a stream, 58 so (state 17, chain 8, outputs 28: a
// block's own chain of loads, terms and products; the tensor pipe is 30 % busy).
#include "lightning.cuh"
#include "mma_tiles.cuh"

namespace hs {

constexpr int LC_LEN = 64;           // tokens of a chunk
constexpr int LC_DS = LC_D + 8, LC_VS = LC_V + 8;    // bfloat16 numbers from row to row in shared memory
constexpr int LC_THREADS = 256;
constexpr float LC_BIG = 1e38f;      // a number beyond this may have no first term

struct LcShape {
  int H, stride, q_off, k_off, v_off, act, rot_dims, n_requests;
  int h0, heads;                     // the group of heads of this launch: from which on, how many
  float k_scale;
  const float2* turns;               // [tokens][rot_dims / 2] cosine and sine of the tokens' angles
};
// x / n and x % n, n fixed for a launch and mostly a power of two
struct LcDiv {
  int n, shift;
  __device__ __forceinline__ int over(int x) const { return shift >= 0 ? x >> shift : x / n; }
};
__device__ __forceinline__ LcDiv lc_div(int n) { return LcDiv{n, (n & (n - 1)) ? -1 : __ffs(n) - 1}; }

__device__ __forceinline__ void lc_ldsm_t(uint32_t* r, const __nv_bfloat16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"((uint32_t)__cvta_generic_to_shared(p)));
}
// the next bfloat16 term of a pair; what it leaves stays in v (exact)
__device__ __forceinline__ uint32_t lc_term(float2& v) {
  const __nv_bfloat162 b = __floats2bfloat162_rn(v.x, v.y);
  const uint32_t u = *(const uint32_t*)&b;
  v.x -= __uint_as_float(u << 16);
  v.y -= __uint_as_float(u & 0xffff0000u);
  return u;
}
__device__ __forceinline__ bool lc_odd(float2 v) {       // not a number that has three terms
  return !(fabsf(v.x) <= LC_BIG && fabsf(v.y) <= LC_BIG);
}
// three terms of a pair to their arrays, `size` numbers apart
__device__ __forceinline__ void lc_store(__nv_bfloat16* dst, int size, float2 v) {
#pragma unroll
  for (int k = 0; k < 3; ++k) *(uint32_t*)(dst + k * size) = lc_term(v);
}
// Six products of terms of N 16 x 8 x 16 steps, the steps' chains side by side: step i takes a[i / PER] and
// b[i % PER] (or b[i], with one a).  The tensor cores cut sums off below the last bit, so the large product
// starts from zero and is added with rounding.
template <int N, int PER>
__device__ __forceinline__ void lc_mma(float (*high)[4], float (*small)[4], const uint32_t (*a)[3][4],
                                       const uint32_t (*b)[3][2]) {
  float t[N][4];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const uint32_t *x = a[i / PER][0], *y = b[i % PER][0];
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%10,%10,%10,%10};"
        : "=f"(t[i][0]), "=f"(t[i][1]), "=f"(t[i][2]), "=f"(t[i][3])
        : "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(x[3]), "r"(y[0]), "r"(y[1]), "f"(0.f));
  }
  constexpr int TA[5] = {0, 2, 1, 0, 1}, TB[5] = {2, 0, 1, 1, 0};
#pragma unroll
  for (int k = 0; k < 5; ++k)
#pragma unroll
    for (int i = 0; i < N; ++i) mma_bf16(small[i], a[i / PER][TA[k]], b[i % PER][TB[k]]);
#pragma unroll
  for (int i = 0; i < N; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) high[i][e] += t[i][e];
}
// the operand of 16 columns as ldmatrix leaves it: two steps of eight
__device__ __forceinline__ void lc_two(uint32_t (*b)[3][2], int k, const uint32_t* r) {
  b[0][k][0] = r[0]; b[0][k][1] = r[1];
  b[1][k][0] = r[2]; b[1][k][1] = r[3];
}
__device__ __forceinline__ double lc_power(float g, int n) {
  double r = 1.0, b = g;
  for (; n; n >>= 1, b *= b)
    if (n & 1) r *= b;
  return r;
}
// chunk number `slot` of the step: which request's, and which of its chunks
__device__ __forceinline__ bool lc_find(const int* __restrict__ req_len, int n_requests, int slot, int& r,
                                        int& c) {
  for (r = 0; r < n_requests; ++r) {
    const int k = lc_chunks(req_len[r]);
    if (slot < k) {
      c = slot;
      return true;
    }
    slot -= k;
  }
  return false;
}

// Activated, turned and scaled rows of one head's q (if Q) and k for the chunk's tokens, as terms
// [3][LC_LEN][D + pad]; weights[j] multiplies row j of k.  Rows from n on are zeros.  Returns whether a
// number is odd.
template <bool Q>
__device__ __forceinline__ bool lc_rows(__nv_bfloat16* sq, __nv_bfloat16* sk, const float* __restrict__ proj,
                                        const LcShape& s, int h, int t0, int n, const float* weights) {
  constexpr int DS = LC_DS, size = LC_LEN * DS;
  const int half = s.rot_dims >> 1;
  const int turned = half >> 1, pairs = turned + (LC_D - s.rot_dims) / 2;
  const LcDiv per = lc_div(pairs);
  constexpr int B = Q ? 4 : 8;                             // items whose numbers are on their way together
  bool odd = false;
  for (int x0 = threadIdx.x; x0 < LC_LEN * pairs; x0 += B * LC_THREADS) {
    float2 lo[B][2], hi[B][2];                             // of q, k: numbers d, d + 1 and their partners
    float2 f0[B], f1[B];
#pragma unroll
    for (int u = 0; u < B; ++u) {
      const int x = x0 + u * LC_THREADS, i = per.over(x), p = x - i * pairs;
      const bool turn = p < turned;
      const int d = turn ? 2 * p : s.rot_dims + 2 * (p - turned);
      lo[u][0] = lo[u][1] = hi[u][0] = hi[u][1] = f0[u] = f1[u] = make_float2(0.f, 0.f);
      if (i < n) {
        const float* row = proj + (size_t)(t0 + i) * s.stride + h * LC_D + d;
#pragma unroll
        for (int m = Q ? 0 : 1; m < 2; ++m) {
          const float* v = row + (m == 0 ? s.q_off : s.k_off);
          lo[u][m] = make_float2(v[0], v[1]);
          if (turn) hi[u][m] = make_float2(v[half], v[half + 1]);
        }
        if (turn) {
          const float2* at = s.turns + (size_t)(t0 + i) * half + d;
          f0[u] = at[0];
          f1[u] = at[1];
        }
      }
    }
#pragma unroll
    for (int u = 0; u < B; ++u) {
      const int x = x0 + u * LC_THREADS, i = per.over(x), p = x - i * pairs;
      if (x >= LC_LEN * pairs) break;
      const bool turn = p < turned;
      const int d = turn ? 2 * p : s.rot_dims + 2 * (p - turned);
      const float c0 = f0[u].x, s0 = f0[u].y, c1 = f1[u].x, s1 = f1[u].y;
#pragma unroll
      for (int m = Q ? 0 : 1; m < 2; ++m) {
        const float mul = m == 0 ? 1.0f : s.k_scale;
        float2 a = lo[u][m], b = hi[u][m];
        if (i < n) {
          a = make_float2(la_act(a.x, s.act), la_act(a.y, s.act));
          if (turn) {                                      // as la_entry
            b = make_float2(la_act(b.x, s.act), la_act(b.y, s.act));
            const float2 a0 = a;
            a.x = fmaf(a.x, c0, -__fmul_rn(b.x, s0));
            a.y = fmaf(a.y, c1, -__fmul_rn(b.y, s1));
            b.x = fmaf(b.x, c0, __fmul_rn(a0.x, s0));
            b.y = fmaf(b.y, c1, __fmul_rn(a0.y, s1));
          }
        }
        a = make_float2(__fmul_rn(a.x, mul), __fmul_rn(a.y, mul));
        b = make_float2(__fmul_rn(b.x, mul), __fmul_rn(b.y, mul));
        odd = odd || lc_odd(a) || lc_odd(b);
        if (m == 1 && weights) {
          const float w = weights[i];
          a.x *= w; a.y *= w;
          b.x *= w; b.y *= w;
        }
        __nv_bfloat16* dst = (m == 0 ? sq : sk) + i * DS + d;
        lc_store(dst, size, a);
        if (turn) lc_store(dst + half, size, b);
      }
    }
  }
  return odd;
}

// Token after token on S [D][V]: the recurrence itself, for chunks with numbers that are not finite.  Two
// lanes share a column, each with half of its rows in registers; the token's k and q are formed once for the
// block, the next token's numbers are on their way meanwhile.  OUT: the outputs, else the state behind the
// chunk takes the place of S.  A state without a single number stays so: the rest of its outputs are none either.
// (2 x 1,024 tokens of 8 heads, all of them no numbers: 9,450 us with S in global memory and k and q formed by every
// thread, 41 so; 60 where all are finite, 150 token by token.)
template <bool OUT>
__device__ __noinline__ void lc_walk(float* S, float* o, const float* __restrict__ proj, const LcShape s, int h,
                                     int t0, int n, float g) {
  constexpr int ROWS = LC_D / 2, PART = ROWS + 4;          // (apart, so that the halves lie in other banks)
  __shared__ __align__(16) float s_kq[2][2 * PART];
  const int v = threadIdx.x >> 1, part = threadIdx.x & 1, half = s.rot_dims >> 1;
  float x[ROWS];
#pragma unroll
  for (int d = 0; d < ROWS; ++d) x[d] = S[(size_t)(part * ROWS + d) * LC_V + v];
  // the entry of k (the first half of the threads) or q this thread forms
  const int e = threadIdx.x & (LC_D - 1), which = threadIdx.x / LC_D;
  const int off = (which ? s.q_off : s.k_off) + h * LC_D;
  const bool mine = OUT || which == 0, turn = mine && e < s.rot_dims, low = e < half;
  const int partner = low ? off + e + half : off + e - half;
  float own = 0.f, other = 0.f, value;
  float2 f = make_float2(1.f, 0.f);
  auto fetch = [&](int t) {
    const float* row = proj + (size_t)t * s.stride;
    if (mine) own = row[off + e];
    value = row[s.v_off + h * LC_V + v];
    if (turn) {
      other = row[partner];
      f = s.turns[(size_t)t * half + (low ? e : e - half)];
    }
  };
  fetch(t0);
  for (int t = t0; t < t0 + n; ++t) {
    float entry = la_act(own, s.act);
    if (turn) {                                            // as la_entry
      const float cross = __fmul_rn(la_act(other, s.act), f.y);
      entry = fmaf(entry, f.x, low ? -cross : cross);
    }
    const float vt = la_act(value, s.act);
    if (t + 1 < t0 + n) fetch(t + 1);
    bool gone = (t - t0) % 8 == 1;                         // looked at now and then
    if (gone) {
#pragma unroll
      for (int d = 0; d < ROWS; ++d) gone = gone && x[d] != x[d];
    }
    if (__syncthreads_and(gone)) {                         // (and the token before is used up)
      if (OUT && part == 0)
        for (; t < t0 + n; ++t) o[((size_t)t * s.H + h) * LC_V + v] = x[0];
      break;
    }
    if (mine) s_kq[which][e + (e / ROWS) * 4] = __fmul_rn(entry, which ? 1.0f : s.k_scale);
    __syncthreads();
    float sum[4] = {};
#pragma unroll
    for (int d = 0; d < ROWS; d += 4) {
      const float4 k = *(const float4*)&s_kq[0][part * PART + d];
      x[d] = fmaf(k.x, vt, g * x[d]);
      x[d + 1] = fmaf(k.y, vt, g * x[d + 1]);
      x[d + 2] = fmaf(k.z, vt, g * x[d + 2]);
      x[d + 3] = fmaf(k.w, vt, g * x[d + 3]);
      if (OUT) {
        const float4 q = *(const float4*)&s_kq[1][part * PART + d];
        sum[0] = fmaf(x[d], q.x, sum[0]);
        sum[1] = fmaf(x[d + 1], q.y, sum[1]);
        sum[2] = fmaf(x[d + 2], q.z, sum[2]);
        sum[3] = fmaf(x[d + 3], q.w, sum[3]);
      }
    }
    if (OUT) {
      float all = (sum[0] + sum[1]) + (sum[2] + sum[3]);
      all += __shfl_xor_sync(0xffffffffu, all, 1);
      if (part == 0) o[((size_t)t * s.H + h) * LC_V + v] = all;
    }
  }
  if (!OUT)
#pragma unroll
    for (int d = 0; d < ROWS; ++d) S[(size_t)(part * ROWS + d) * LC_V + v] = x[d];
}

// ---- cosine and sine of every token's angles, once for all heads and both kernels ----------------
__global__ void lightning_turns_kernel(float2* __restrict__ turns, const int* __restrict__ tok_pos,
                                       const float* __restrict__ freq, int n_tokens, int half) {
  pdl_trigger();
  pdl_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_tokens * half) return;
  float2 f;
  pair_angle(tok_pos[i / half], freq[i % half], &f.x, &f.y);
  turns[i] = f;
}

// ---- the chunks' contributions ------------------------------------------------------------------
__global__ void __launch_bounds__(LC_THREADS)
lightning_chunk_state_kernel(float* __restrict__ dS, const float* __restrict__ proj,
                             const float* __restrict__ decay, const int* __restrict__ req_start,
                             const int* __restrict__ req_len, const LcShape s) {
  extern __shared__ __align__(16) uint8_t lc_smem[];
  __shared__ float s_w[LC_LEN];
  pdl_trigger();
  pdl_wait();
  const int slot = blockIdx.x, h = s.h0 + blockIdx.y;
  int r, c;
  if (!lc_find(req_len, s.n_requests, slot, r, c)) return;
  const int n = min(LC_LEN, req_len[r] - c * LC_LEN), t0 = req_start[r] + c * LC_LEN;
  const float g = decay[h];
  constexpr int DS = LC_DS, VS = LC_VS;
  __nv_bfloat16* sK = (__nv_bfloat16*)lc_smem;             // [3][LC_LEN][DS]
  __nv_bfloat16* sV = sK + 3 * LC_LEN * DS;                // [3][LC_LEN][VS]
  if (threadIdx.x < LC_LEN) s_w[threadIdx.x] = (float)lc_power(g, max(0, n - 1 - (int)threadIdx.x));
  __syncthreads();
  bool odd = threadIdx.x < n && !(fabsf(s_w[threadIdx.x]) <= LC_BIG);
  odd = lc_rows<false>(nullptr, sK, proj, s, h, t0, n, s_w) || odd;
  constexpr int vp = LC_V / 2;
  for (int x0 = threadIdx.x; x0 < LC_LEN * vp; x0 += 8 * LC_THREADS) {
    float2 a[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int x = x0 + u * LC_THREADS, i = x / vp, v = 2 * (x - i * vp);
      a[u] = make_float2(0.f, 0.f);
      if (i < n) {
        const float* src = proj + (size_t)(t0 + i) * s.stride + s.v_off + h * LC_V + v;
        a[u] = make_float2(src[0], src[1]);
      }
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int x = x0 + u * LC_THREADS, i = x / vp, v = 2 * (x - i * vp);
      if (x >= LC_LEN * vp) break;
      if (i < n) a[u] = make_float2(la_act(a[u].x, s.act), la_act(a[u].y, s.act));
      odd = odd || lc_odd(a[u]);
      lc_store(sV + i * VS + v, LC_LEN * VS, a[u]);
    }
  }
  float* out = dS + ((size_t)slot * s.heads + blockIdx.y) * LC_D * LC_V;
  if (__syncthreads_or(odd)) {
    for (int i = threadIdx.x; i < LC_D * LC_V; i += LC_THREADS) out[i] = 0.f;
    __syncthreads();
    lc_walk<false>(out, nullptr, proj, s, h, t0, n, g);
    return;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, mi = lane >> 3;
  const int m = warp, steps = (n + 15) / 16;               // a warp takes 16 rows of the state
  uint32_t a[LC_LEN / 16][1][3][4];
#pragma unroll
  for (int kk = 0; kk < LC_LEN / 16; ++kk)
#pragma unroll
    for (int k = 0; k < 3; ++k)
      lc_ldsm_t(a[kk][0][k], sK + (k * LC_LEN + kk * 16 + (mi >> 1) * 8 + (lane & 7)) * DS + m * 16 + (mi & 1) * 8);
#pragma unroll 1
  for (int v = 0; v < LC_V; v += 32) {
    float high[4][4] = {}, small[4][4] = {};
#pragma unroll
    for (int kk = 0; kk < LC_LEN / 16; ++kk) {
      if (kk >= steps) break;
      uint32_t b[4][3][2];
#pragma unroll
      for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          uint32_t r[4];
          lc_ldsm_t(r, sV + (k * LC_LEN + kk * 16 + (mi & 1) * 8 + (lane & 7)) * VS + v + 16 * g + (mi >> 1) * 8);
          lc_two(b + 2 * g, k, r);
        }
      lc_mma<4, 4>(high, small, a[kk], b);
    }
    const int row = m * 16 + (lane >> 2), col = v + 2 * (lane & 3);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      *(float2*)(out + (size_t)row * LC_V + col + 8 * i) =
          make_float2(high[i][0] + small[i][0], high[i][1] + small[i][1]);
      *(float2*)(out + (size_t)(row + 8) * LC_V + col + 8 * i) =
          make_float2(high[i][2] + small[i][2], high[i][3] + small[i][3]);
    }
  }
}

// ---- the chain of states ------------------------------------------------------------------------
// Blocks for as many requests as may go in chunks, not for all (600 tokens beside 60 single ones, 32 heads:
// lightning attention 288 us with all, 258 so).  The outputs' blocks are let in late: when they come while the
// contributions are being formed they share SMs and take longer (2 x 1,024 tokens of 4 heads 55 us, 50 so).
__global__ void __launch_bounds__(LC_THREADS)
lightning_chunk_chain_kernel(float* __restrict__ dS, float* __restrict__ state,
                             const float* __restrict__ decay, const int* __restrict__ req_len,
                             const int* __restrict__ req_slot, const LcShape s) {
  pdl_wait();
  pdl_trigger();
  const int h = s.h0 + blockIdx.y, size = LC_D * LC_V, i = (blockIdx.x * LC_THREADS + threadIdx.x) * 4;
  int r = 0, chunks = 0, first = 0;                        // the blockIdx.z-th request in chunks, the chunks before
  for (int nth = 0; r < s.n_requests; ++r) {
    chunks = lc_chunks(req_len[r]);
    if (chunks && nth++ == (int)blockIdx.z) break;
    first += chunks;
  }
  if (r == s.n_requests || i >= size) return;
  float4* slot = (float4*)(state + ((size_t)req_slot[r] * s.H + h) * size + i);
  float4* x = (float4*)(dS + ((size_t)first * s.heads + blockIdx.y) * size + i);
  const size_t next = (size_t)s.heads * size / 4;              // from a chunk to the next
  const float g = decay[h], whole = (float)lc_power(g, LC_LEN);
  const float end = (float)lc_power(g, req_len[r] - (chunks - 1) * LC_LEN);
  // a power that is below the range of numbers is zero, but no factor of the recurrence was: an infinity goes on
  auto beyond = [&](float w) { return w == 0.f && g != 0.f ? copysignf(1.f, w) : w; };
  const float whole_inf = beyond(whole), end_inf = beyond(end);
  float4 S = *slot;
  constexpr int B = 8;                                     // contributions on their way together
  for (int c0 = 0; c0 < chunks; c0 += B) {
    float4 d[B];
#pragma unroll
    for (int k = 0; k < B; ++k)
      if (c0 + k < chunks) d[k] = x[(c0 + k) * next];
#pragma unroll
    for (int k = 0; k < B; ++k)
      if (c0 + k < chunks) {
        x[(c0 + k) * next] = S;
        const bool more = c0 + k + 1 < chunks;
        const float w = more ? whole : end, w_inf = more ? whole_inf : end_inf;
        auto carry = [&](float x, float add) { return fmaf(fabsf(x) <= 3.402823466e38f ? w : w_inf, x, add); };
        S.x = carry(S.x, d[k].x); S.y = carry(S.y, d[k].y);
        S.z = carry(S.z, d[k].z); S.w = carry(S.w, d[k].w);
      }
  }
  *slot = S;
}

// ---- the outputs --------------------------------------------------------------------------------
__global__ void __launch_bounds__(LC_THREADS, 2)
lightning_chunk_out_kernel(float* __restrict__ o, float* __restrict__ states,
                           const float* __restrict__ proj, const float* __restrict__ decay,
                           const int* __restrict__ req_start, const int* __restrict__ req_len,
                           const LcShape s) {
  extern __shared__ __align__(16) uint8_t lc_smem[];
  __shared__ float s_p[LC_LEN + 1];                        // powers of the decay
  pdl_trigger();
  pdl_wait();
  const int slot = blockIdx.x, h = s.h0 + blockIdx.y;
  int r, c;
  if (!lc_find(req_len, s.n_requests, slot, r, c)) return;
  const int n = min(LC_LEN, req_len[r] - c * LC_LEN), t0 = req_start[r] + c * LC_LEN;
  const float g = decay[h];
  constexpr int DS = LC_DS, PS = LC_LEN + 8;
  __nv_bfloat16* sQ = (__nv_bfloat16*)lc_smem;             // [3][LC_LEN][DS]
  __nv_bfloat16* sK = sQ + 3 * LC_LEN * DS;                // the same; later the weights [3][LC_LEN][PS]
  if (threadIdx.x <= LC_LEN) s_p[threadIdx.x] = (float)lc_power(g, threadIdx.x);
  float* S = states + ((size_t)slot * s.heads + blockIdx.y) * LC_D * LC_V;
  bool odd = lc_rows<true>(sQ, sK, proj, s, h, t0, n, nullptr);
  if (__syncthreads_or(odd)) {                             // (nothing below would be of use)
    lc_walk<true>(S, o, proj, s, h, t0, n, g);
    return;
  }
  odd = threadIdx.x <= LC_LEN && !(fabsf(s_p[threadIdx.x]) <= LC_BIG);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int a_r = lane & 15, a_c = (lane >> 4) * 8;
  const int b_r = (lane & 7) + (lane >> 4) * 8, b_c = ((lane >> 3) & 1) * 8;
  const int g4 = lane >> 2, q2 = 2 * (lane & 3);
  // ---- weights g^(t-j) q_t . k_j: a warp takes 16 queries and half of the keys
  {
    const int m0 = (warp & 3) * 16, j0 = (warp >> 2) * 32;
    float high[4][4] = {}, small[4][4] = {};
    if (j0 <= m0 + 15) {
#pragma unroll 2
      for (int k0 = 0; k0 < LC_D; k0 += 16) {
        uint32_t a[1][3][4], b[4][3][2];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          ldmatrix_x4(a[0][k], sQ + (k * LC_LEN + m0 + a_r) * DS + k0 + a_c);
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            uint32_t r[4];
            ldmatrix_x4(r, sK + (k * LC_LEN + j0 + 16 * j + b_r) * DS + k0 + b_c);
            lc_two(b + 2 * j, k, r);
          }
        }
        lc_mma<4, 4>(high, small, a, b);
      }
    }
    __syncthreads();                                       // the keys are read: their place takes the weights
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int t = m0 + g4 + 8 * half, j = j0 + 8 * i + q2;
        float2 w = make_float2(0.f, 0.f);
        if (j <= t) w.x = s_p[t - j] * (high[i][2 * half] + small[i][2 * half]);
        if (j + 1 <= t) w.y = s_p[t - j - 1] * (high[i][2 * half + 1] + small[i][2 * half + 1]);
        odd = odd || lc_odd(w);
        lc_store(sK + t * PS + j, LC_LEN * PS, w);
      }
  }
  __syncthreads();
  // ---- outputs: a warp takes 16 value columns of all 64 queries; states and values come straight from
  // global memory (each is read by one warp) and are cut into terms in registers
  {
    const int v0 = warp * 16;
    float high[8][4] = {}, small[8][4] = {};               // [16 queries][eight columns]
    auto fetch = [&](float2 (&x)[2][2], int k0) {          // [columns 0-7, 8-15][numbers k0 + q2, + 8]
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const float* src = S + (size_t)(k0 + q2 + 8 * e) * LC_V + v0 + 8 * i + g4;
          x[i][e] = make_float2(src[0], src[LC_V]);
        }
    };
    float2 x[2][2], next[2][2], then[2][2];
    fetch(next, 0);
    fetch(then, 16);
    for (int k0 = 0; k0 < LC_D; k0 += 16) {
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          x[i][e] = next[i][e];
          next[i][e] = then[i][e];
          odd = odd || lc_odd(x[i][e]);
        }
      if (k0 + 32 < LC_D) fetch(then, k0 + 32);
      uint32_t b[2][3][2];
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
          for (int e = 0; e < 2; ++e) b[i][k][e] = lc_term(x[i][e]);
#pragma unroll
      for (int m = 0; m < 4; m += 2) {
        uint32_t a[2][3][4];
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
          for (int j = 0; j < 2; ++j) ldmatrix_x4(a[j][k], sQ + (k * LC_LEN + (m + j) * 16 + a_r) * DS + k0 + a_c);
        lc_mma<4, 2>(high + 2 * m, small + 2 * m, a, b);
      }
    }
    auto values = [&](float2 (&y)[2][2], int kk) {         // [columns 0-7, 8-15][keys 16 kk + q2, + 8]
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int j = kk * 16 + q2 + 8 * e;
          const float* src = proj + (size_t)(t0 + j) * s.stride + s.v_off + h * LC_V + v0 + 8 * i + g4;
          y[i][e].x = j < n ? src[0] : 0.f;
          y[i][e].y = j + 1 < n ? src[s.stride] : 0.f;
        }
    };
    values(next, 0);
    float acc[4][2][4];
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          acc[m][i][e] = s_p[m * 16 + g4 + 8 * (e >> 1) + 1] * (high[2 * m + i][e] + small[2 * m + i][e]);
          high[2 * m + i][e] = small[2 * m + i][e] = 0.f;
        }
#pragma unroll
    for (int kk = 0; kk < LC_LEN / 16; ++kk) {
      float2 y[2][2];
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          y[i][e] = make_float2(la_act(next[i][e].x, s.act), la_act(next[i][e].y, s.act));
          odd = odd || lc_odd(y[i][e]);
        }
      if (kk + 1 < LC_LEN / 16) values(next, kk + 1);
      uint32_t b[2][3][2];
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
          for (int e = 0; e < 2; ++e) b[i][k][e] = lc_term(y[i][e]);
#pragma unroll
      for (int m = kk & ~1; m < 4; m += 2) {               // (weights of queries before the keys are zeros)
        uint32_t a[2][3][4];
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
          for (int j = 0; j < 2; ++j) ldmatrix_x4(a[j][k], sK + (k * LC_LEN + (m + j) * 16 + a_r) * PS + kk * 16 + a_c);
        lc_mma<4, 2>(high + 2 * m, small + 2 * m, a, b);
      }
    }
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int t = m * 16 + g4 + 8 * half;
        if (t >= n) continue;
        float* dst = o + ((size_t)(t0 + t) * s.H + h) * LC_V + v0 + q2;
#pragma unroll
        for (int i = 0; i < 2; ++i)
          *(float2*)(dst + 8 * i) =
              make_float2(acc[m][i][2 * half] + (high[2 * m + i][2 * half] + small[2 * m + i][2 * half]),
                          acc[m][i][2 * half + 1] + (high[2 * m + i][2 * half + 1] + small[2 * m + i][2 * half + 1]));
      }
  }
  if (__syncthreads_or(odd)) lc_walk<true>(S, o, proj, s, h, t0, n, g);
}

bool lightning_takes_chunks(int D, int V, int rot_dims) { return D == LC_D && V == LC_V && rot_dims % 4 == 0; }

int lightning_chunks(float* o, float* state, const float* proj, const float* decay, const int* req_start,
                     const int* req_len, const int* req_slot, int n_requests, int n_tokens, int stride,
                     int q_off, int k_off, int v_off, int H, int D, int V, int act, float* scratch,
                     const int* tok_pos, const float* freq, int rot_dims, float k_scale, cudaStream_t st) {
  LcShape s;
  s.H = H; s.stride = stride; s.q_off = q_off; s.k_off = k_off; s.v_off = v_off;
  s.act = act; s.rot_dims = rot_dims; s.n_requests = n_requests; s.k_scale = k_scale;
  const int slots = lightning_chunk_slots(n_tokens, n_requests);
  const bool pdl = hs_pdl_enabled();
  const int smem_a = 3 * LC_LEN * (LC_DS + LC_VS) * 2, smem_c = 6 * LC_LEN * LC_DS * 2;
  const int group = lightning_chunk_heads(n_tokens, n_requests, H, D, V);
  s.turns = (const float2*)(scratch + (size_t)slots * group * D * V);
  cudaError_t e = cudaSuccess;
  if (rot_dims) {
    const int size = n_tokens * (rot_dims / 2);
    e = hs_launch(lightning_turns_kernel, dim3((size + 127) / 128), dim3(128), 0, st, pdl, (float2*)s.turns,
                  tok_pos, freq, n_tokens, rot_dims / 2);
    if (e != cudaSuccess) return (int)e;
  }
  e = cudaFuncSetAttribute(lightning_chunk_state_kernel,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, smem_a);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(lightning_chunk_out_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_c);
  if (e != cudaSuccess) return (int)e;
  const int most = n_requests < n_tokens / LC_MIN ? n_requests : n_tokens / LC_MIN;
  for (s.h0 = 0; s.h0 < H; s.h0 += group) {
    s.heads = H - s.h0 < group ? H - s.h0 : group;
    e = hs_launch(lightning_chunk_state_kernel, dim3(slots, s.heads), dim3(LC_THREADS), (size_t)smem_a, st, pdl,
                  scratch, proj, decay, req_start, req_len, s);
    if (e != cudaSuccess) return (int)e;
    e = hs_launch(lightning_chunk_chain_kernel, dim3((D * V / 4 + LC_THREADS - 1) / LC_THREADS, s.heads, most),
                  dim3(LC_THREADS), 0, st, pdl, scratch, state, decay, req_len, req_slot, s);
    if (e != cudaSuccess) return (int)e;
    e = hs_launch(lightning_chunk_out_kernel, dim3(slots, s.heads), dim3(LC_THREADS), (size_t)smem_c, st, pdl, o,
                  scratch, proj, decay, req_start, req_len, s);
    if (e != cudaSuccess) return (int)e;
  }
  return (int)e;
}

}  // namespace hs
