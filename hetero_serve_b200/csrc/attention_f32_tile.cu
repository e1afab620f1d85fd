// Causal attention over the paged cache in float32 on the CUDA cores, head size 64: the arithmetic
// of attention_simt.cu, operation for operation, laid out for tiles of queries (prompt portions) and,
// further down, for single tokens.
//
// A token's keys are taken 32 at a time; chunk c belongs to stream c mod 4.  A score is one chain of
// fused multiply-adds over d, times the scale; a stream keeps a running maximum, a running sum (the
// 32 weights of a chunk added by the butterfly's tree) and float32 accumulators that take the chunk's
// keys in order; the four streams are folded in stream order.  The order of every sum depends on the
// key positions alone, so a token's bits are those the one-token kernel gives it.
//
// attention_simt.cu serves at most four tokens a block: 4 KB of keys and values are read from shared
// memory for 4 x 32 scores, and each lane walks its own key's row.  Here a block serves 64 queries of
// one request and head; stream s is a group of 64 threads (s = threadIdx.x / 64) that works through
// its chunks on its own:
//     scores   8 queries x 4 keys a thread over d-major queries and keys, packed two queries an FMA;
//     softmax  a thread per query: its 32 scores from shared memory, the weights back to their place;
//     values   8 queries x 8 dimensions a thread, packed two dimensions an FMA.
// The keys of the next chunk are on their way from the end of the scores on, the values from the end
// of the values on.  113 KB of shared memory: two blocks can share an SM.  Keys arrive by 4-byte cp.async
// copies into d-major rows whose columns are XORed against bank conflicts.  Chunks that some query of
// the block does not see, or whose pages were refused, take a path that adds visible keys only, and so
// do chunks in which some query has no score above minus infinity: it leaves such a chunk out, as the
// one-token kernel does (its weights would be zeros, which make NaN of an infinite value).
// Bounded by each stream's chain of scores, softmax and values (FMA pipe 52 % busy, shared-memory pipe
// 40 %, with two blocks an SM).  Measured (2 x 512 tokens, 16 heads): 340 us in attention_simt.cu, 75 us
// here (14 TFLOP/s of causal work).
#include "common.cuh"

namespace hs {

constexpr int AF_Q = 64, AF_D = 64, AF_CHUNK = 32, AF_STREAMS = 4, AF_THREADS = 256;
// floats: queries [d][q] | per stream: keys [d][32], values [32][d], scores [32][q]
constexpr int AF_Q_FLOATS = AF_D * AF_Q, AF_K_FLOATS = AF_D * AF_CHUNK, AF_V_FLOATS = AF_CHUNK * AF_D,
              AF_S_FLOATS = AF_CHUNK * AF_Q;
constexpr int AF_STREAM_FLOATS = AF_K_FLOATS + AF_V_FLOATS + AF_S_FLOATS;
constexpr size_t AF_SMEM = (AF_Q_FLOATS + AF_STREAMS * AF_STREAM_FLOATS) * sizeof(float);

struct AfParams {
  float* out;
  const float *qkv, *pool;
  const int *table, *tile_info, *plan_head, *tok_req;
  int* status;
  int n_tokens;
  int n_heads, n_kv_heads, page_size, num_pages, max_pages, q_off, qkv_stride;
  float scale;
};

__device__ __forceinline__ void af_fma2(uint64_t& acc, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ uint64_t af_mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t af_twice(float a) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(a));
  return r;
}
__device__ __forceinline__ float af_lo(uint64_t a) { return __uint_as_float((uint32_t)a); }
__device__ __forceinline__ float af_hi(uint64_t a) { return __uint_as_float((uint32_t)(a >> 32)); }
__device__ __forceinline__ void af_copy4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void af_copy16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void af_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// the 64 threads of a stream
__device__ __forceinline__ void af_sync(int stream) {
  asm volatile("bar.sync %0, 64;" ::"r"(1 + stream) : "memory");
}

// ... and whether any of them says so
__device__ __forceinline__ bool af_sync_any(int stream, bool mine) {
  unsigned any;
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n barrier.cta.red.or.pred q, %2, 64, p;\n"
      " selp.u32 %0, 1, 0, q;\n}"
      : "=r"(any) : "r"((unsigned)mine), "r"(1 + stream) : "memory");
  return any != 0;
}

// BLOCKS an SM: two (128 registers a thread, some of them spilled) where there are more than two blocks
// an SM, else one (no such limit).  us, one block an SM against two, 12 heads: 64 portions of 16 tokens
// 59 and 45, 16 of 200 behind 300 positions 231 and 218; but one of 1,000 behind 3,000 507 and 567, 16
// of 8 tokens and 2 heads behind 3,000 218 and 287.
template <int BLOCKS>
__global__ void __launch_bounds__(AF_THREADS, BLOCKS)
attention_f32_tile_kernel(const AfParams p) {
  extern __shared__ __align__(16) float af_smem[];
  __shared__ float s_corr[AF_STREAMS][AF_Q];
  // rows of no request (a captured step's padding): zeros
  for (int i = blockIdx.x * AF_THREADS + threadIdx.x; i < p.n_tokens; i += gridDim.x * AF_THREADS)
    if (p.tok_req[i] < 0) {
      float* row = p.out + ((size_t)i * p.n_heads + blockIdx.y) * AF_D;
      for (int d = 0; d < AF_D; ++d) row[d] = 0.f;
    }
  if ((int)(blockIdx.x >> 1) >= p.plan_head[1]) return;
  const int4 ti = *(const int4*)(p.tile_info + 4 * (blockIdx.x >> 1));
  const int q0 = (blockIdx.x & 1) * AF_Q;
  const int nq = min(AF_Q, ti.y - q0), tok0 = ti.x + q0, r = ti.z, pos0 = ti.w + q0;
  if (nq <= 0 || r < 0 || pos0 < 0) return;
  const int h = blockIdx.y, hk = h / (p.n_heads / p.n_kv_heads);
  const int pos_last = pos0 + nq - 1;
  const int tid = threadIdx.x, lane = tid & 31, stream = tid >> 6, t = tid & 63, w = t >> 5;
  if (pos_last / p.page_size >= p.max_pages) {
    for (int i = tid; i < nq * AF_D; i += AF_THREADS)
      p.out[((size_t)(tok0 + i / AF_D) * p.n_heads + h) * AF_D + i % AF_D] = 0.f;
    return;
  }
  float* sQ = af_smem;
  float* sK = sQ + AF_Q_FLOATS + stream * AF_STREAM_FLOATS;
  float* sV = sK + AF_K_FLOATS;
  float* sS = sV + AF_V_FLOATS;
  const int* trow = p.table + (size_t)r * p.max_pages;
  const size_t tile = (size_t)p.page_size * AF_D, page_stride = 2 * (size_t)p.n_kv_heads * tile;
  const size_t v_off = (size_t)p.n_kv_heads * tile;

  // queries, d-major: a warp copies eight d of four queries at a time; rows past the last one
  // repeat it
  for (int i = tid >> 5; i < (AF_Q / 4) * (AF_D / 8); i += AF_THREADS / 32) {
    const int q = (i >> 3) * 4 + (lane >> 3), d = (i & 7) * 8 + (lane & 7);
    af_copy4(sQ + d * AF_Q + (q ^ ((d & 7) << 2)),
             p.qkv + (size_t)(tok0 + min(q, nq - 1)) * p.qkv_stride + p.q_off + h * AF_D + d);
  }
  // (they belong to the first group this thread commits)

  long long koff = -1;              // of the chunk being fetched: this lane's key row in the pool
  auto look_up = [&](int j0) {
    koff = -1;
    const int j = j0 + lane;
    if (j <= pos_last) {
      const int page = trow[j / p.page_size];
      if (page < 0 || page >= p.num_pages) atomicOr(p.status, HS_STATUS_BAD_PAGE);
      else koff = (long long)(page * page_stride + hk * tile + (size_t)(j % p.page_size) * AF_D);
    }
    return __ballot_sync(0xffffffffu, koff >= 0);
  };
  auto fetch_keys = [&] {
#pragma unroll
    for (int kg = 0; kg < 8; ++kg) {
      const int key = kg * 4 + (lane >> 3);
      const long long ko = __shfl_sync(0xffffffffu, koff, key);
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        const int d = (w * 4 + g) * 8 + (lane & 7);
        if (ko >= 0) af_copy4(sK + d * AF_CHUNK + (key ^ ((d & 7) << 2)), p.pool + ko + d);
      }
    }
    af_commit();
  };
  auto fetch_values = [&](long long rows) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int key = i * 4 + w * 2 + (lane >> 4);
      const long long ko = __shfl_sync(0xffffffffu, rows, key);
      if (ko >= 0)
        af_copy16(sV + key * AF_D + (lane & 15) * 4, p.pool + ko + v_off + (lane & 15) * 4);
    }
    af_commit();
  };

  // lanes: eight column groups on bits 1-3, four row groups on bits 0 and 4 (two wavefronts a read)
  const int cx = (lane >> 1) & 7, qg = ((lane & 1) | ((lane >> 3) & 2)) | (w << 2);
  uint64_t acc[8][4];               // queries qg*4..+3 and 32+qg*4..+3; dimensions likewise of cx
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0;
  float m = -INFINITY, l = 0.f;     // of query t
  const int pos_t = pos0 + t;

  int j0 = stream * AF_CHUNK;
  unsigned live = 0;
  if (j0 <= pos_last) {
    live = look_up(j0);
    fetch_keys();
    fetch_values(koff);
  } else {
    af_commit();
    af_commit();
  }
  asm volatile("cp.async.wait_group 1;" ::: "memory");
  __syncthreads();                                   // the queries are everyone's
  for (; j0 <= pos_last; j0 += AF_STREAMS * AF_CHUNK) {
    const int nxt = j0 + AF_STREAMS * AF_CHUNK;
    // ---- scores
    asm volatile("cp.async.wait_group 1;" ::: "memory");     // this chunk's keys
    af_sync(stream);
    {
      uint64_t s[4][4];                                      // [query pairs][keys]
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) s[i][j] = 0;
#pragma unroll 8
      for (int d = 0; d < AF_D; ++d) {
        const int sx = (d & 7) << 2;
        const ulonglong2 a = *(const ulonglong2*)(sQ + d * AF_Q + ((qg * 4) ^ sx));
        const ulonglong2 b = *(const ulonglong2*)(sQ + d * AF_Q + 32 + ((qg * 4) ^ sx));
        const float4 k = *(const float4*)(sK + d * AF_CHUNK + ((cx * 4) ^ sx));
        const uint64_t k2[4] = {af_twice(k.x), af_twice(k.y), af_twice(k.z), af_twice(k.w)};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          af_fma2(s[0][j], a.x, k2[j]);
          af_fma2(s[1][j], a.y, k2[j]);
          af_fma2(s[2][j], b.x, k2[j]);
          af_fma2(s[3][j], b.y, k2[j]);
        }
      }
      // [key][query], the query XORed with four times the key's group
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float* row = sS + (cx * 4 + j) * AF_Q + ((qg * 4) ^ (cx << 2));
        *(float4*)row = make_float4(af_lo(s[0][j]) * p.scale, af_hi(s[0][j]) * p.scale,
                                    af_lo(s[1][j]) * p.scale, af_hi(s[1][j]) * p.scale);
        *(float4*)(row + 32) = make_float4(af_lo(s[2][j]) * p.scale, af_hi(s[2][j]) * p.scale,
                                           af_lo(s[3][j]) * p.scale, af_hi(s[3][j]) * p.scale);
      }
    }
    af_sync(stream);
    const unsigned here = live;
    if (nxt <= pos_last) {
      live = look_up(nxt);
      fetch_keys();
    } else {
      af_commit();
    }
    // every query sees every key of the chunk
    bool whole = here == 0xffffffffu && j0 + AF_CHUNK - 1 <= pos0;
    // ---- softmax: query t
    bool left_out = false;
    {
      float x[AF_CHUNK];
      float* col = sS + (t & 32);
#pragma unroll
      for (int k = 0; k < AF_CHUNK; ++k) {
        x[k] = col[k * AF_Q + ((t & 31) ^ ((k >> 2) << 2))];
        if (!whole && (!((here >> k) & 1u) || j0 + k > pos_t)) x[k] = -INFINITY;
      }
      float cm = x[0];
#pragma unroll
      for (int k = 1; k < AF_CHUNK; ++k) cm = fmaxf(cm, x[k]);
      const float m_new = fmaxf(m, cm);
      float corr = 1.f;
      left_out = m_new == -INFINITY && j0 <= pos_t;          // (no corr below is negative)
      if (m_new == -INFINITY || j0 > pos_t) {                // nothing of the chunk is this query's
#pragma unroll
        for (int k = 0; k < AF_CHUNK; ++k) x[k] = 0.f;
      } else {
#pragma unroll
        for (int k = 0; k < AF_CHUNK; ++k) x[k] = (x[k] == -INFINITY) ? 0.f : expf(x[k] - m_new);
        corr = expf(m - m_new);
      }
#pragma unroll
      for (int k = 0; k < AF_CHUNK; ++k) col[k * AF_Q + ((t & 31) ^ ((k >> 2) << 2))] = x[k];
      if (!(m_new == -INFINITY || j0 > pos_t)) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)                     // the butterfly's tree
#pragma unroll
          for (int k = 0; k < o; ++k) x[k] += x[k + o];
        l = l * corr + x[0];
        m = m_new;
      }
      s_corr[stream][t] = left_out ? -1.f : corr;
    }
    asm volatile("cp.async.wait_group 1;" ::: "memory");     // this chunk's values
    if (af_sync_any(stream, left_out)) whole = false;
    // ---- values
    {
      const float4 c0 = *(const float4*)&s_corr[stream][qg * 4];
      const float4 c1 = *(const float4*)&s_corr[stream][32 + qg * 4];
      const float cr[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const uint64_t c2 = af_twice(cr[i] < 0.f ? 1.f : cr[i]);
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = af_mul2(acc[i][j], c2);
      }
#pragma unroll 4
      for (int k = 0; k < AF_CHUNK; ++k) {
        const float* prow = sS + k * AF_Q + ((qg * 4) ^ ((k >> 2) << 2));
        const float4 p0 = *(const float4*)prow, p1 = *(const float4*)(prow + 32);
        const ulonglong2 v0 = *(const ulonglong2*)(sV + k * AF_D + cx * 4);
        const ulonglong2 v1 = *(const ulonglong2*)(sV + k * AF_D + 32 + cx * 4);
        const float pv[8] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w};
        if (whole) {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const uint64_t p2 = af_twice(pv[i]);
            af_fma2(acc[i][0], p2, v0.x);
            af_fma2(acc[i][1], p2, v0.y);
            af_fma2(acc[i][2], p2, v1.x);
            af_fma2(acc[i][3], p2, v1.y);
          }
        } else if ((here >> k) & 1u) {
          const int first = j0 + k - pos0;                   // the first query that sees the key
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            if ((i < 4 ? qg * 4 + i : 28 + qg * 4 + i) < first || cr[i] < 0.f) continue;
            const uint64_t p2 = af_twice(pv[i]);
            af_fma2(acc[i][0], p2, v0.x);
            af_fma2(acc[i][1], p2, v0.y);
            af_fma2(acc[i][2], p2, v1.x);
            af_fma2(acc[i][3], p2, v1.y);
          }
        }
      }
    }
    af_sync(stream);                                         // weights and values may be overwritten
    if (nxt <= pos_last) fetch_values(koff);
    else af_commit();
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  // ---- fold the streams in stream order
  __syncthreads();
  float* fold = af_smem;                                     // [stream][query][d], 68 floats a row
  constexpr int LD = AF_D + 4;
  float(*s_m)[AF_Q] = (float(*)[AF_Q])(fold + AF_STREAMS * AF_Q * LD);      // behind the rows
  float(*s_l)[AF_Q] = s_m + AF_STREAMS;
  s_m[stream][t] = m;
  s_l[stream][t] = l;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    float* row = fold + (stream * AF_Q + (i < 4 ? qg * 4 + i : 28 + qg * 4 + i)) * LD;
    *(ulonglong2*)(row + cx * 4) = make_ulonglong2(acc[i][0], acc[i][1]);
    *(ulonglong2*)(row + 32 + cx * 4) = make_ulonglong2(acc[i][2], acc[i][3]);
  }
  __syncthreads();
  const int q = tid >> 2, dq = (tid & 3) * 4;                // dimensions dq, dq + 16, ...
  if (q >= nq) return;
  float M = -INFINITY, L = 0.f;
  float o[16];
#pragma unroll
  for (int c = 0; c < 16; ++c) o[c] = 0.f;
  for (int s = 0; s < AF_STREAMS; ++s) {
    const float ms = s_m[s][q];
    if (ms == -INFINITY) continue;                           // a stream without keys
    const float m_new = fmaxf(M, ms);
    const float c0 = expf(M - m_new), c1 = expf(ms - m_new);
    L = L * c0 + s_l[s][q] * c1;
    const float* row = fold + (s * AF_Q + q) * LD;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const float4 x = *(const float4*)(row + dq + 16 * c);
      o[4 * c] = fmaf(x.x, c1, o[4 * c] * c0);
      o[4 * c + 1] = fmaf(x.y, c1, o[4 * c + 1] * c0);
      o[4 * c + 2] = fmaf(x.z, c1, o[4 * c + 2] * c0);
      o[4 * c + 3] = fmaf(x.w, c1, o[4 * c + 3] * c0);
    }
    M = m_new;
  }
  const float inv = L > 0.f ? 1.0f / L : 0.f;
  float* orow = p.out + ((size_t)(tok0 + q) * p.n_heads + h) * AF_D + dq;
#pragma unroll
  for (int c = 0; c < 16; ++c) orow[16 * (c >> 2) + (c & 3)] = o[c] * inv;
}

// ---- single tokens --------------------------------------------------------------------------------
// One block per token and head, a warp per stream, as in attention_simt.cu and with its arithmetic.
// That kernel looks a chunk's pages up, copies it, waits and computes, chunk after chunk: every chunk
// costs two trips to the L2 or beyond.  Here NB chunks of a stream are on their way while one is
// worked on: a chunk's place in the ring is refilled as soon as its keys, and then its values, have
// been used, and the page of the chunk to fetch is read before the scores.  A whole chunk takes
// straight-line code: a score per lane (keys swizzled against bank conflicts), two dimensions of the
// values per lane.  Measured (8 tokens, 350-1,050 keys, 16 heads): 56 us in attention_simt.cu, 17 here.
template <int NB>
struct AfSingle {
  static constexpr int WARP_FLOATS = NB * 2 * AF_CHUNK * AF_D + AF_D + AF_CHUNK;
  static constexpr size_t SMEM = (size_t)AF_STREAMS * WARP_FLOATS * sizeof(float);
};

template <int NB>
__global__ void __launch_bounds__(AF_STREAMS * 32)
attention_f32_single_kernel(const AfParams p, const int* __restrict__ tok_pos,
                            const int* __restrict__ tok_req, const int* __restrict__ listed,
                            const int* __restrict__ n_listed) {
  extern __shared__ __align__(16) float af_smem[];
  if (listed != nullptr && (int)blockIdx.x >= *n_listed) return;
  const int tok = listed != nullptr ? listed[3 * blockIdx.x] : blockIdx.x;
  const int h = blockIdx.y, hk = h / (p.n_heads / p.n_kv_heads);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r = tok_req[tok], pos = tok_pos[tok];
  float* orow = p.out + ((size_t)tok * p.n_heads + h) * AF_D;
  if (r < 0 || pos < 0 || pos / p.page_size >= p.max_pages) {
    if (threadIdx.x < AF_D) orow[threadIdx.x] = 0.f;
    return;
  }
  float* sk = af_smem + warp * AfSingle<NB>::WARP_FLOATS;      // [NB][32 keys][64]
  float* sv = sk + NB * AF_CHUNK * AF_D;
  float* sq = sv + NB * AF_CHUNK * AF_D;
  float* sp = sq + AF_D;
  const int* trow = p.table + (size_t)r * p.max_pages;
  const size_t tile = (size_t)p.page_size * AF_D, page_stride = 2 * (size_t)p.n_kv_heads * tile;
  const size_t v_off = (size_t)p.n_kv_heads * tile;
  constexpr int STEP = AF_STREAMS * AF_CHUNK;

  auto page_of = [&](int j0) { return j0 + lane <= pos ? trow[(j0 + lane) / p.page_size] : -1; };
  auto row_of = [&](int j0, int page) -> long long {
    const int j = j0 + lane;
    if (j > pos) return -1;
    if (page < 0 || page >= p.num_pages) {
      atomicOr(p.status, HS_STATUS_BAD_PAGE);
      return -1;
    }
    return (long long)(page * page_stride + hk * tile + (size_t)(j % p.page_size) * AF_D);
  };
  // a warp copies two rows at a time, 16 pieces of 16 bytes each
  auto fetch = [&](float* dst, long long rows, size_t extra, bool swizzled) {
#pragma unroll
    for (int i = 0; i < AF_CHUNK / 2; ++i) {
      const int key = 2 * i + (lane >> 4), pc = lane & 15;
      const long long ko = __shfl_sync(0xffffffffu, rows, key);
      if (ko >= 0)
        af_copy16(dst + key * AF_D + (swizzled ? pc ^ (key & 7) : pc) * 4, p.pool + ko + extra + pc * 4);
    }
  };

  const int first = warp * AF_CHUNK;
  unsigned live[NB];
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    const int j0 = first + b * STEP;
    live[b] = 0;
    if (j0 <= pos) {
      const long long rows = row_of(j0, page_of(j0));
      live[b] = __ballot_sync(0xffffffffu, rows >= 0);
      fetch(sk + b * AF_CHUNK * AF_D, rows, 0, true);
      af_commit();
      fetch(sv + b * AF_CHUNK * AF_D, rows, v_off, false);
      af_commit();
    } else {
      af_commit();
      af_commit();
    }
  }
  const float* qrow = p.qkv + (size_t)tok * p.qkv_stride + p.q_off + h * AF_D;
  sq[lane] = qrow[lane];
  sq[lane + 32] = qrow[lane + 32];

  float m = -INFINITY, l = 0.f, o0 = 0.f, o1 = 0.f;            // dimensions 2 lane, 2 lane + 1
  for (int j00 = first; j00 <= pos; j00 += NB * STEP) {
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      const int j0 = j00 + b * STEP;
      if (j0 > pos) break;                                     // (the same for the whole warp)
      const int nxt = j0 + NB * STEP;
      const bool more = nxt <= pos;
      const int page = more ? page_of(nxt) : -1;
      float* kb = sk + b * AF_CHUNK * AF_D;
      float* vb = sv + b * AF_CHUNK * AF_D;
      asm volatile("cp.async.wait_group %0;" ::"n"(2 * NB - 1) : "memory");
      __syncwarp();
      const unsigned here = live[b];
      float s = -INFINITY;
      {
        float dot = 0.f;
        const float4* krow = (const float4*)(kb + lane * AF_D);
        const float4* q4 = (const float4*)sq;
#pragma unroll
        for (int c = 0; c < AF_D / 4; ++c) {
          const float4 k = krow[c ^ (lane & 7)], q = q4[c];
          dot = fmaf(q.x, k.x, dot);
          dot = fmaf(q.y, k.y, dot);
          dot = fmaf(q.z, k.z, dot);
          dot = fmaf(q.w, k.w, dot);
        }
        if ((here >> lane) & 1u) s = dot * p.scale;
      }
      __syncwarp();                                            // the keys' place is free
      long long rows = -1;
      if (more) {
        rows = row_of(nxt, page);
        live[b] = __ballot_sync(0xffffffffu, rows >= 0);
        fetch(kb, rows, 0, true);
      }
      af_commit();
      const float m_new = fmaxf(m, warp_max(s));
      asm volatile("cp.async.wait_group %0;" ::"n"(2 * NB - 1) : "memory");
      // a chunk whose pages were all refused leaves m_new at -inf: skip it
      if (m_new != -INFINITY) {
        const float w = (s == -INFINITY) ? 0.f : expf(s - m_new);
        const float corr = expf(m - m_new);
        sp[lane] = w;
        l = l * corr + warp_sum(w);
        o0 *= corr;
        o1 *= corr;
        m = m_new;
        __syncwarp();
        if (here == 0xffffffffu) {
#pragma unroll
          for (int k4 = 0; k4 < AF_CHUNK / 4; ++k4) {
            const float4 w4 = ((const float4*)sp)[k4];
            const float wk[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float2 v = *(const float2*)(vb + (4 * k4 + i) * AF_D + 2 * lane);
              o0 = fmaf(wk[i], v.x, o0);
              o1 = fmaf(wk[i], v.y, o1);
            }
          }
        } else {
          for (int k = 0; k < AF_CHUNK; ++k) {
            if (!((here >> k) & 1u)) continue;
            const float2 v = *(const float2*)(vb + k * AF_D + 2 * lane);
            o0 = fmaf(sp[k], v.x, o0);
            o1 = fmaf(sp[k], v.y, o1);
          }
        }
      }
      __syncwarp();                                            // the values' place is free
      if (more) fetch(vb, rows, v_off, false);
      af_commit();
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  // fold the streams in stream order
  __shared__ float s_fold[AF_STREAMS][AF_D + 2];
  s_fold[warp][2 * lane] = o0;
  s_fold[warp][2 * lane + 1] = o1;
  if (lane == 0) {
    s_fold[warp][AF_D] = m;
    s_fold[warp][AF_D + 1] = l;
  }
  __syncthreads();
  if (threadIdx.x >= AF_D) return;
  float M = -INFINITY, L = 0.f, o = 0.f;
  for (int i = 0; i < AF_STREAMS; ++i) {
    const float ms = s_fold[i][AF_D];
    if (ms == -INFINITY) continue;                             // a stream without keys
    const float m_new = fmaxf(M, ms);
    const float c0 = expf(M - m_new), c1 = expf(ms - m_new);
    L = L * c0 + s_fold[i][AF_D + 1] * c1;
    o = fmaf(s_fold[i][threadIdx.x], c1, o * c0);
    M = m_new;
  }
  const float inv = L > 0.f ? 1.0f / L : 0.f;
  orow[threadIdx.x] = o * inv;
}

}  // namespace hs

static_assert(hs::AF_STREAMS * hs::AF_Q * (hs::AF_D + 4 + 2) * sizeof(float) <= hs::AF_SMEM,
              "the folded accumulators, maxima and sums fit where queries, keys, values and scores were");
// (an SM has 228 KB; a block is charged its static array and 1 KB of the system's beside them)
static_assert(2 * (hs::AF_SMEM + hs::AF_STREAMS * hs::AF_Q * sizeof(float) + 1024) <= 228 * 1024,
              "two blocks share an SM");

// The plan's tiles (prompt portions): float32, head size 64, no window; `tile_info` entries of up to
// 128 queries (first token, queries, request row, first position).  Rows of tokens without a request
// (tok_req below zero) become zeros.
HS_EXPORT int hs_attention_f32_tiles(float* out, const float* qkv, const float* pool,
                                     const int* table, const int* tok_req, int n_tokens,
                                     const int* tile_info, const int* plan_head, int tile_cap,
                                     int n_heads, int n_kv_heads, int head_dim,
                                     int page_size, int num_pages, int max_pages, int q_off,
                                     int qkv_stride, float scale, int* status, void* stream) {
  using namespace hs;
  if (!out || !qkv || !pool || !table || !tok_req || !tile_info || !plan_head || !status)
    return HS_ERR_ARGUMENT;
  if (head_dim != AF_D || n_heads <= 0 || n_kv_heads <= 0 || n_heads % n_kv_heads ||
      n_heads > 65535 || page_size <= 0 || num_pages <= 0 || max_pages <= 0 ||
      ((uintptr_t)pool & 15) || ((uintptr_t)tile_info & 15) || tile_cap > (1 << 28))
    return HS_ERR_UNSUPPORTED;
  if (tile_cap <= 0) return HS_OK;
  AfParams p{out, qkv, pool, table, tile_info, plan_head, tok_req, status, n_tokens, n_heads,
             n_kv_heads, page_size, num_pages, max_pages, q_off, qkv_stride, scale};
  const bool two = 2ll * tile_cap * n_heads > 2ll * hs_sm_count();
  auto* kernel = two ? attention_f32_tile_kernel<2> : attention_f32_tile_kernel<1>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)AF_SMEM);
  if (e != cudaSuccess) return (int)e;
  kernel<<<dim3(2 * tile_cap, n_heads), AF_THREADS, AF_SMEM, (cudaStream_t)stream>>>(p);
  HS_LAUNCH_CHECK();
  return HS_OK;
}

// Single tokens: all n_tokens of the batch, or (listed: every third int names a token) the first
// *n_listed, n_tokens being the grid.
HS_EXPORT int hs_attention_f32_single(float* out, const float* qkv, const float* pool,
                                      const int* table, const int* tok_pos, const int* tok_req,
                                      const int* listed, const int* n_listed, int n_tokens,
                                      int n_heads, int n_kv_heads, int head_dim, int page_size,
                                      int num_pages, int max_pages, int q_off, int qkv_stride,
                                      float scale, int* status, void* stream) {
  using namespace hs;
  if (!out || !qkv || !pool || !table || !tok_pos || !tok_req || !status || (listed && !n_listed))
    return HS_ERR_ARGUMENT;
  if (head_dim != AF_D || n_heads <= 0 || n_kv_heads <= 0 || n_heads % n_kv_heads ||
      n_heads > 65535 || page_size <= 0 || num_pages <= 0 || max_pages <= 0 || ((uintptr_t)pool & 15))
    return HS_ERR_UNSUPPORTED;
  if (n_tokens <= 0) return HS_OK;
  AfParams p{out, qkv, pool, table, nullptr, nullptr, tok_req, status, n_tokens, n_heads,
             n_kv_heads, page_size, num_pages, max_pages, q_off, qkv_stride, scale};
  // up to a block an SM: the deepest ring; more blocks: three share an SM instead
  const bool deep = (long long)n_tokens * n_heads <= hs_sm_count();
  cudaError_t e;
#define HS_AF(NB)                                                                                 \
  do {                                                                                            \
    e = cudaFuncSetAttribute(attention_f32_single_kernel<NB>,                                     \
                             cudaFuncAttributeMaxDynamicSharedMemorySize,                         \
                             (int)AfSingle<NB>::SMEM);                                            \
    if (e == cudaSuccess)                                                                         \
      attention_f32_single_kernel<NB><<<dim3(n_tokens, n_heads), AF_STREAMS * 32,                 \
                                        AfSingle<NB>::SMEM, (cudaStream_t)stream>>>(              \
          p, tok_pos, tok_req, listed, n_listed);                                                 \
  } while (0)
  if (deep) HS_AF(3);
  else HS_AF(1);
#undef HS_AF
  if (e != cudaSuccess) return (int)e;
  HS_LAUNCH_CHECK();
  return HS_OK;
}
