// Token selection on the device: argmax, and temperature / top-k sampling by inverse CDF.
//
// The reference samples on the host (heteroserve/worker/worker.py:38-50): temperature <= 0
// takes the argmax; otherwise softmax(logits / temperature) over all tokens or, for
// 0 < top_k < V, over the top_k largest, and one draw from it.  Here the draw is one uniform
// number u in [0, 1) from Philox-4x32-10 keyed by the request's seed with the position of the
// new token as counter, so that (like the reference's reseeding with seed + n_kv,
// worker.py:647,694) a sampled token does not depend on how requests were batched.  The token
// is the first, in index order, whose cumulative unnormalised probability exceeds u * total.
// Ties in argmax and at the top-k threshold go to the lower index.  All arithmetic is float32.
#include "common.cuh"

namespace hs {

constexpr int SM_THREADS = 1024;

__device__ __forceinline__ void philox_round(uint32_t (&c)[4], uint32_t (&k)[2]) {
  const uint32_t M0 = 0xD2511F53u, M1 = 0xCD9E8D57u;
  const uint32_t hi0 = __umulhi(M0, c[0]), lo0 = M0 * c[0];
  const uint32_t hi1 = __umulhi(M1, c[2]), lo1 = M1 * c[2];
  const uint32_t n0 = hi1 ^ c[1] ^ k[0], n1 = lo1, n2 = hi0 ^ c[3] ^ k[1], n3 = lo0;
  c[0] = n0; c[1] = n1; c[2] = n2; c[3] = n3;
  k[0] += 0x9E3779B9u;
  k[1] += 0xBB67AE85u;
}

__device__ __forceinline__ float philox_uniform(uint32_t seed_lo, uint32_t seed_hi,
                                                uint32_t position) {
  uint32_t c[4] = {position, 0u, 0u, 0u};
  uint32_t k[2] = {seed_lo, seed_hi};
#pragma unroll
  for (int i = 0; i < 10; ++i) philox_round(c, k);
  return (float)(c[0] >> 8) * (1.0f / 16777216.0f);
}

__device__ __forceinline__ uint32_t order_key(float v) {
  uint32_t b = __float_as_uint(v);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

struct ArgMax {
  float v;
  int i;
};
__device__ __forceinline__ ArgMax better(ArgMax a, ArgMax b) {
  if (b.v > a.v || (b.v == a.v && b.i < a.i)) return b;
  return a;
}

// block-wide argmax of one row; every thread returns the result
__device__ ArgMax block_argmax(const float* row, int vocab) {
  __shared__ ArgMax sh[SM_THREADS / 32];
  __shared__ ArgMax result;
  ArgMax best{-INFINITY, 0x7fffffff};
  // 32 loads in flight per thread (a row of 50k logits is two rounds for 1,024 threads); within
  // a thread indices rise, so the first seen wins ties
  constexpr int INFLIGHT = 32;
  for (int base = threadIdx.x; base < vocab; base += INFLIGHT * blockDim.x) {
    float v[INFLIGHT];
#pragma unroll
    for (int j = 0; j < INFLIGHT; ++j) {
      const int i = base + j * blockDim.x;
      v[j] = i < vocab ? row[i] : -INFINITY;
    }
#pragma unroll
    for (int j = 0; j < INFLIGHT; ++j) {
      const int i = base + j * blockDim.x;
      if (i < vocab && (v[j] > best.v || best.i == 0x7fffffff)) best = ArgMax{v[j], i};
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ArgMax other{__shfl_xor_sync(0xffffffffu, best.v, o), __shfl_xor_sync(0xffffffffu, best.i, o)};
    best = better(best, other);
  }
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = best;
  __syncthreads();
  if (threadIdx.x == 0) {
    ArgMax b = sh[0];
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) b = better(b, sh[w]);
    if (b.i == 0x7fffffff) b.i = 0;
    result = b;
  }
  __syncthreads();
  ArgMax r = result;
  __syncthreads();
  return r;
}

__device__ int block_sum_int(int v) {
  __shared__ int sh[SM_THREADS / 32];
  __shared__ int total;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    int t = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += sh[w];
    total = t;
  }
  __syncthreads();
  int r = total;
  __syncthreads();
  return r;
}

// Inclusive scan over the block in thread order of a float and an int at once.
// Returns the block totals through `tot_f`, `tot_i`.
__device__ void block_scan(float& f, int& n, float& tot_f, int& tot_i) {
  __shared__ float wf[SM_THREADS / 32];
  __shared__ int wn[SM_THREADS / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float uf = __shfl_up_sync(0xffffffffu, f, o);
    const int un = __shfl_up_sync(0xffffffffu, n, o);
    if (lane >= o) {
      f += uf;
      n += un;
    }
  }
  if (lane == 31) {
    wf[warp] = f;
    wn[warp] = n;
  }
  __syncthreads();
  if (warp == 0) {
    const int nw = blockDim.x >> 5;
    float a = lane < nw ? wf[lane] : 0.f;
    int b = lane < nw ? wn[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float ua = __shfl_up_sync(0xffffffffu, a, o);
      const int ub = __shfl_up_sync(0xffffffffu, b, o);
      if (lane >= o) {
        a += ua;
        b += ub;
      }
    }
    if (lane < nw) {
      wf[lane] = a;
      wn[lane] = b;
    }
  }
  __syncthreads();
  if (warp > 0) {
    f += wf[warp - 1];
    n += wn[warp - 1];
  }
  tot_f = wf[(blockDim.x >> 5) - 1];
  tot_i = wn[(blockDim.x >> 5) - 1];
  __syncthreads();
}

__global__ void __launch_bounds__(SM_THREADS)
argmax_kernel(int* __restrict__ out, const float* __restrict__ logits, int vocab) {
  const float* row = logits + (size_t)blockIdx.x * vocab;
  ArgMax r = block_argmax(row, vocab);
  if (threadIdx.x == 0) out[blockIdx.x] = r.i;
}

__global__ void __launch_bounds__(SM_THREADS)
sample_kernel(int* __restrict__ out, const float* __restrict__ logits,
              const float* __restrict__ temperature, const int* __restrict__ top_k,
              const int* __restrict__ seed_lo, const int* __restrict__ seed_hi,
              const int* __restrict__ position, int vocab, int* __restrict__ feedback,
              const int* __restrict__ feedback_slot, const int* __restrict__ status_word) {
  const int rowi = blockIdx.x;
  const float* row = logits + (size_t)rowi * vocab;
  const float temp = temperature[rowi];
  pdl_wait();                       // the logits are what the previous kernel wrote
  // the engine's status word rides behind the tokens, so that one copy brings both to the host
  if (status_word != nullptr && rowi == 0 && threadIdx.x == 0) out[gridDim.x] = *status_word;
  const ArgMax top = block_argmax(row, vocab);
  // a row with a feedback slot also leaves its token there, for the next step's embedding
  const int fb = (feedback != nullptr && feedback_slot != nullptr) ? feedback_slot[rowi] : -1;
  if (!(temp > 0.f)) {
    if (threadIdx.x == 0) {
      out[rowi] = top.i;
      if (fb >= 0) feedback[fb] = top.i;
    }
    return;
  }
  const float mx = top.v / temp;
  int k = top_k[rowi];
  uint32_t thr = 0;   // order key of the k-th largest logit; 0 keeps everything
  int need_eq = 0;    // how many entries equal to the threshold are kept (lowest indices)
  const bool use_k = k > 0 && k < vocab;
  if (use_k) {
    for (int b = 31; b >= 0; --b) {
      const uint32_t cand = thr | (1u << b);
      int c = 0;
      for (int i = threadIdx.x; i < vocab; i += blockDim.x) c += order_key(row[i]) >= cand;
      if (block_sum_int(c) >= k) thr = cand;
    }
    int c = 0;
    for (int i = threadIdx.x; i < vocab; i += blockDim.x) c += order_key(row[i]) > thr;
    need_eq = k - block_sum_int(c);
  }
  const float u = philox_uniform((uint32_t)seed_lo[rowi], (uint32_t)seed_hi[rowi],
                                 (uint32_t)position[rowi]);
  __shared__ int found;
  if (threadIdx.x == 0) found = 0x7fffffff;
  float target = 0.f;
  int last_kept = 0;
  for (int pass = 0; pass < 2; ++pass) {
    float run = 0.f;
    int run_eq = 0;
    for (int base = 0; base < vocab; base += blockDim.x) {
      const int i = base + threadIdx.x;
      float e = 0.f;
      int eq = 0;
      uint32_t key = 0;
      if (i < vocab) {
        key = order_key(row[i]);
        eq = use_k && key == thr;
      }
      float sf = 0.f;
      int sn = eq;
      // the rank of an entry among those equal to the threshold needs the scan of `eq`
      // before its own probability is known, so scan the flags first
      float tf;
      int tn;
      block_scan(sf, sn, tf, tn);
      bool kept = false;
      if (i < vocab) {
        if (!use_k) kept = true;
        else if (key > thr) kept = true;
        else if (eq) kept = (run_eq + sn - 1) < need_eq;
        if (kept) e = expf(row[i] / temp - mx);
      }
      run_eq += tn;
      float cf = e;
      int dummy = kept ? 1 : 0;
      float chunk_total;
      int chunk_kept;
      block_scan(cf, dummy, chunk_total, chunk_kept);
      if (pass == 1) {
        if (kept && run + cf > target) atomicMin(&found, i);
        if (kept) last_kept = i;
        __syncthreads();
        if (found != 0x7fffffff) break;
      }
      run += chunk_total;
    }
    if (pass == 0) target = u * run;
  }
  __syncthreads();
  if (found == 0x7fffffff) {
    // u * total rounded up to the total itself: the last kept token
    __shared__ int lastk;
    if (threadIdx.x == 0) lastk = 0;
    __syncthreads();
    atomicMax(&lastk, last_kept);
    __syncthreads();
    if (threadIdx.x == 0) {
      out[rowi] = lastk;
      if (fb >= 0) feedback[fb] = lastk;
    }
  } else if (threadIdx.x == 0) {
    out[rowi] = found;
    if (fb >= 0) feedback[fb] = found;
  }
}

// ---- the same rule with the row held in shared memory ------------------------------------------
// A row of up to ~55k logits fits a CTA's shared memory.  It is read from global memory once;
// thread t owns the positions [t*C, (t+1)*C) (C odd: its walks are free of bank conflicts), so
// sums over threads in thread order are sums in index order.  The k-th largest logit is found
// by a radix select of four 8-bit digits over a 256-bin histogram, among the few entries that the
// threads' maxima leave in question, the kept entries' weights exp(x/T - max/T) replace the logits in place, one scan
// over the threads gives every thread the weight before its range, and the thread that holds
// the crossing of u * total finds the token.  Streaming the row from global memory for every
// pass (the kernel above, which stays for longer rows) took 90 us without top-k and 240-270 us
// with it at 50,257 logits.
constexpr int SS_THREADS = 1024;
constexpr int SS_CAND = 1024;       // entries that may be among the k largest
constexpr int SS_LIST_K = 512;      // the largest k for which they are listed ...
constexpr int SS_LIST_VOCAB = 12000;    // ... the shortest row ...
constexpr int SS_LIST_MAXIMA = 600;     // ... and the most maxima from the bound up (903 entries)

__device__ float block_max_f(float v) {
  __shared__ float sh[SS_THREADS / 32];
  __shared__ float res;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    float w = threadIdx.x < (blockDim.x >> 5) ? sh[threadIdx.x] : -INFINITY;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) w = fmaxf(w, __shfl_xor_sync(0xffffffffu, w, o));
    if (threadIdx.x == 0) res = w;
  }
  __syncthreads();
  const float r = res;
  __syncthreads();
  return r;
}

// Exclusive scan over the block in thread order of a float and an int; totals through tot_*.
__device__ void block_exclusive_scan(float& f, int& n, float& tot_f, int& tot_i) {
  __shared__ float wf[SS_THREADS / 32];
  __shared__ int wn[SS_THREADS / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float fi = f;
  int ni = n;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float uf = __shfl_up_sync(0xffffffffu, fi, o);
    const int un = __shfl_up_sync(0xffffffffu, ni, o);
    if (lane >= o) {
      fi += uf;
      ni += un;
    }
  }
  if (lane == 31) {
    wf[warp] = fi;
    wn[warp] = ni;
  }
  float fe = __shfl_up_sync(0xffffffffu, fi, 1);      // the warp's sum before this lane
  int ne = __shfl_up_sync(0xffffffffu, ni, 1);
  if (lane == 0) {
    fe = 0.f;
    ne = 0;
  }
  __syncthreads();
  if (warp == 0) {
    const int nw = blockDim.x >> 5;
    float a = lane < nw ? wf[lane] : 0.f;
    int b = lane < nw ? wn[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float ua = __shfl_up_sync(0xffffffffu, a, o);
      const int ub = __shfl_up_sync(0xffffffffu, b, o);
      if (lane >= o) {
        a += ua;
        b += ub;
      }
    }
    if (lane < nw) {
      wf[lane] = a;          // inclusive over the warps
      wn[lane] = b;
    }
  }
  __syncthreads();
  f = (warp > 0 ? wf[warp - 1] : 0.f) + fe;
  n = (warp > 0 ? wn[warp - 1] : 0) + ne;
  tot_f = wf[(blockDim.x >> 5) - 1];
  tot_i = wn[(blockDim.x >> 5) - 1];
  __syncthreads();
}

__global__ void __launch_bounds__(SS_THREADS)
sample_smem_kernel(int* __restrict__ out, const float* __restrict__ logits,
                   const float* __restrict__ temperature, const int* __restrict__ top_k,
                   const int* __restrict__ seed_lo, const int* __restrict__ seed_hi,
                   const int* __restrict__ position, int vocab, int* __restrict__ feedback,
                   const int* __restrict__ feedback_slot, const int* __restrict__ status_word) {
  extern __shared__ float s_row[];                  // [vocab]: logits, then weights (-1: dropped)
  __shared__ int hist[256];
  __shared__ int s_digit, s_above, s_same, s_found, s_last, s_n;
  __shared__ uint32_t s_cand[SS_CAND];
  const int rowi = blockIdx.x;
  const float* row = logits + (size_t)rowi * vocab;
  const float temp = temperature[rowi];
  pdl_wait();                       // the logits are what the previous kernel wrote
  if (status_word != nullptr && rowi == 0 && threadIdx.x == 0) out[gridDim.x] = *status_word;
  const int fb = (feedback != nullptr && feedback_slot != nullptr) ? feedback_slot[rowi] : -1;
  if (!(temp > 0.f)) {
    const ArgMax top = block_argmax(row, vocab);
    if (threadIdx.x == 0) {
      out[rowi] = top.i;
      if (fb >= 0) feedback[fb] = top.i;
    }
    return;
  }
  float m = -INFINITY;                              // the maximum needs no order: taken on the way in
#pragma unroll 16
  for (int i = threadIdx.x; i < vocab; i += blockDim.x) {
    const float v = row[i];
    s_row[i] = v;
    m = fmaxf(m, v);
  }
  if (threadIdx.x == 0) {
    s_found = 0x7fffffff;
    s_last = 0;
    s_n = 0;
  }
  const float top = block_max_f(m);                 // (its barriers also publish the row)
  const float mx = top / temp;
  int C = (vocab + blockDim.x - 1) / blockDim.x;
  C |= 1;                                           // odd
  const int lo = min(vocab, (int)threadIdx.x * C), hi = min(vocab, lo + C);

  const int k = top_k[rowi];
  const bool use_k = k > 0 && k < vocab;
  uint32_t thr = 0;     // order key of the k-th largest logit; 0 keeps everything
  int need_eq = 0;      // how many entries equal to the threshold are kept (lowest indices)
  bool all_eq = true;   // ... which is all of them
  if (use_k) {
    // the want-th largest of the keys that `walk` hands on, and among the keys equal to it: s_above
    // (of the last digit) lie above, s_same are equal
    int remaining = 0;
    auto select = [&](int want, auto walk) {
      uint32_t prefix = 0;
      remaining = want; // the want-th largest is the remaining-th largest among keys with the prefix
      for (int shift = 24; shift >= 0; shift -= 8) {
        if (threadIdx.x < 256) hist[threadIdx.x] = 0;
        __syncthreads();
        const uint32_t above_mask = shift == 24 ? 0u : (0xffffffffu << (shift + 8));
        // (one atomic per entry: adding once per warp and digit through __match_any_sync took
        // twice as long)
        walk([&](uint32_t key) {
          if ((key & above_mask) == prefix) atomicAdd(&hist[(key >> shift) & 255u], 1);
        });
        __syncthreads();
        if (threadIdx.x < 32) {
          // lane l owns digits 8l .. 8l+7; digits are taken from the largest down
          const int lane = threadIdx.x;
          int c[8], grp = 0;
#pragma unroll
          for (int b = 0; b < 8; ++b) {
            c[b] = hist[8 * lane + b];
            grp += c[b];
          }
          int incl = grp;             // inclusive sum over lanes lane .. 31
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_down_sync(0xffffffffu, incl, o);
            if (lane + o < 32) incl += u;
          }
          int run = incl - grp;       // keys with a digit above this lane's
          if (run < remaining && remaining <= incl) {
#pragma unroll
            for (int b = 7; b >= 0; --b) {
              if (run < remaining && remaining <= run + c[b]) {
                s_digit = 8 * lane + b;
                s_above = run;
                s_same = c[b];
              }
              run += c[b];
            }
          }
        }
        __syncthreads();
        prefix |= (uint32_t)s_digit << shift;
        remaining -= s_above;
      }
      return prefix;
    };
    auto whole_row = [&](auto take) {
      for (int i = lo; i < hi; ++i) take(order_key(s_row[i]));
    };
    // Few of the row's entries can be among the k largest: k of the threads' maxima, so k entries,
    // are no smaller than the k-th largest maximum.  In a row in no order about 1,024 ln(1024 / (1024
    // - k)) entries lie from there up (41 for k = 40, 710 for 512, the list's 1,024 at 647); they are
    // listed in one walk and the threshold is found among them.  A walk of the row per digit takes 4
    // us at 50,257 logits, the selection among the maxima 3 (32 rows, digits against list: k = 40 41.9
    // and 28.7 us, k = 512 44.2 and 33.3; 12,000 logits, k = 40 16.1 and 14.4, k = 512
    // 17.2 and 16.7; 5,000 logits, k = 40 10.7 and 11.4).  So the digits walk the row where k is larger or the row is short, where the maxima are mostly
    // equal (then the entries are too), and where the list overflows after all.
    bool listed = k <= SS_LIST_K && vocab >= SS_LIST_VOCAB;
    const uint32_t own = order_key(m);
    if (listed && !__syncthreads_and(own == order_key(top))) {
      const uint32_t bound = select(k, [&](auto take) { take(own); });
      // maxima from the bound up: k, and those equal to it that k leaves out
      listed = k - remaining + s_same <= SS_LIST_MAXIMA;
      for (int i = listed ? lo : hi; i < hi; ++i) {
        const uint32_t key = order_key(s_row[i]);
        if (key >= bound) {
          const int at = atomicAdd(&s_n, 1);
          if (at < SS_CAND) s_cand[at] = key;
        }
      }
      __syncthreads();
      listed = listed && s_n >= k && s_n <= SS_CAND;
    } else {
      listed = false;
    }
    if (listed) {
      const int n = s_n;
      thr = select(k, [&](auto take) {
        for (int i = threadIdx.x; i < n; i += blockDim.x) take(s_cand[i]);
      });
    } else {
      thr = select(k, whole_row);
    }
    need_eq = remaining;
    all_eq = s_same == remaining;
  }

  // entries equal to the threshold are kept in index order until k are reached
  int eq = 0;
  if (use_k && !all_eq) {                           // the same for the whole CTA
    for (int i = lo; i < hi; ++i) eq += order_key(s_row[i]) == thr;
    float unused = 0.f, tf;
    int tn;
    block_exclusive_scan(unused, eq, tf, tn);       // eq: equal entries before this range
  }
  float sum = 0.f;
  bool any = false;                                 // of this range's entries is kept
#pragma unroll 4
  for (int i = lo; i < hi; ++i) {
    const float v = s_row[i];
    bool kept = true;
    if (use_k) {
      const uint32_t key = order_key(v);
      kept = key > thr || (key == thr && (all_eq || eq++ < need_eq));
    }
    const float e = kept ? expf(v / temp - mx) : -1.f;
    s_row[i] = e;
    if (kept) {
      sum += e;
      any = true;
    }
  }
  float before = sum, total;
  int nz = 0, tnz;
  block_exclusive_scan(before, nz, total, tnz);     // before: weight of all kept entries below lo
  const float u = philox_uniform((uint32_t)seed_lo[rowi], (uint32_t)seed_hi[rowi],
                                 (uint32_t)position[rowi]);
  const float target = u * total;
  int cand = 0x7fffffff, last_kept = -1;
  float run = before;
  for (int i = any ? lo : hi; i < hi; ++i) {
    const float e = s_row[i];
    if (e >= 0.f) {
      run += e;
      if (cand == 0x7fffffff && run > target) cand = i;
      last_kept = i;
    }
  }
  if (cand != 0x7fffffff) atomicMin(&s_found, cand);
  if (last_kept >= 0) atomicMax(&s_last, last_kept);
  __syncthreads();
  if (threadIdx.x == 0) {
    // u * total rounded up to the total itself: the last kept token
    const int tok = s_found != 0x7fffffff ? s_found : s_last;
    out[rowi] = tok;
    if (fb >= 0) feedback[fb] = tok;
  }
}

// ---- a row over a cluster of eight blocks ------------------------------------------------------
// The same rule, decision for decision and sum for sum, for long rows: block c of the cluster does the work
// of threads 128 c .. 128 c + 127 of the kernel above and holds their positions.  Maxima, histograms and the
// warps' sums meet in shared memory of the cluster; the sums of a thread, of a warp and over the warps are
// formed in the order above, so the tokens are the same ones.  Of the maxima of each block's 64 groups of four
// threads the (k/8)-th largest is found by counting; the smallest of these eight bounds the k largest entries
// from below (there are k maxima, so k entries, from it up).  The entries from it up are listed, every block
// gathers all lists and counts again, where there are more than a block has threads each for the entries it listed
// itself (all of them in every block: 64 x 32,000, k = 200, 63 us against 27).  Where they are too many, and for k
// above 200, the threshold is found a digit of eight bits at a time with histograms that meet in the cluster (us, k =
// 200 and 256: 32 x 50,257 21.4 and 25.4, 64 x 32,000 27.0 and 26.6; as a list k = 256 took 47 and 101 in every block).
// One block a row leaves most SMs idle at the batches that sample, and its 50,257 exponentials and quotients take one SM
// 20 us.  us, a block a row against a cluster, without top-k, k = 40, k = 2,000 and greedy: 32 x 50,257 22.8 and 13.7,
// 29.1 and 16.5, 45.6 and 27.1, 7.9 and 5.1; 64 x 32,000 16.6 and 13.6, 22.1 and 17.9, 32.8 and 27.8, 5.4 and 4.9 (k of
// 80 to 400 is the range that loses there: 160 24.5 and 26.1; with 24,576 columns 21.7 and 25.8; 48 rows gain).  Shorter
// rows and larger batches gain nothing: 64 x 16,384 10.2 and 10.8, 128 x 32,000 16.6 and 20.3.
constexpr int SC_BLOCKS = 8, SC_THREADS = 256, SC_OWN = 128;   // of a cluster; a block; positions' owners
constexpr int SC_GROUPS = SC_THREADS / 4;                       // of four threads: a block's maxima
constexpr int SC_LIST_K = 200;                                  // the largest k that lists
constexpr int SC_LIST = 512, SC_CAND = 1024;                   // entries a block may list, a cluster
constexpr uint32_t SC_LOWEST = 0x007fffffu;                    // the key of minus infinity
constexpr int SC_VOCAB = 24576, SC_ROWS = 64;                  // the shortest row, the most rows

__device__ __forceinline__ uint32_t sc_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void sc_sync() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t sc_addr(const void* p, int rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
               : "=r"(r) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
  return r;
}
__device__ __forceinline__ int sc_read(const int* p, int rank) {
  int v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(sc_addr(p, rank)) : "memory");
  return v;
}
__device__ __forceinline__ float sc_read(const float* p, int rank) {
  return __int_as_float(sc_read((const int*)p, rank));
}
__device__ __forceinline__ void sc_write(int* p, int rank, int v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(sc_addr(p, rank)), "r"(v) : "memory");
}

// how many of n keys (a multiple of four) are larger than `key`, and how many equal to it
__device__ __forceinline__ int2 sc_rank_of(uint32_t key, const uint32_t* keys, int n) {
  int2 r = make_int2(0, 0);
#pragma unroll 4
  for (int i = 0; i < n; i += 4) {
    const uint4 x = *(const uint4*)(keys + i);
    r.x += (x.x > key) + (x.y > key) + (x.z > key) + (x.w > key);
    r.y += (x.x == key) + (x.y == key) + (x.z == key) + (x.w == key);
  }
  return r;
}

__global__ void __launch_bounds__(SC_THREADS)
sample_cluster_kernel(int* __restrict__ out, const float* __restrict__ logits,
                      const float* __restrict__ temperature, const int* __restrict__ top_k,
                      const int* __restrict__ seed_lo, const int* __restrict__ seed_hi,
                      const int* __restrict__ position, int rows, int vocab, int* __restrict__ feedback,
                      const int* __restrict__ feedback_slot, const int* __restrict__ status_word) {
  extern __shared__ float s_row[];                  // [SC_OWN * C]: logits, then weights (-1: dropped)
  __shared__ int hist[2][256], s_tot[256];
  __shared__ __align__(16) uint32_t s_key[SC_GROUPS], s_list[SC_LIST], s_cand[SC_CAND];
  __shared__ int s_digit, s_above, s_same, s_count, s_found, s_last, s_bound, s_n;
  __shared__ float s_max[SC_THREADS / 32], s_own, s_sum[SC_OWN / 32], s_warps[32];
  __shared__ int s_eq[SC_OWN / 32];
  __shared__ int s_v[32], s_i[32];                  // block 0: what the others hand over
  const int rank = (int)sc_rank(), rowi = blockIdx.x / SC_BLOCKS;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const float* row = logits + (size_t)rowi * vocab;
  pdl_trigger();
  const float temp = temperature[rowi];
  const int fb = (feedback != nullptr && feedback_slot != nullptr) ? feedback_slot[rowi] : -1;
  pdl_wait();                       // the logits are what the previous kernel wrote
  if (status_word != nullptr && blockIdx.x == 0 && tid == 0) out[rows] = *status_word;
  if (tid == 0) {
    s_found = 0x7fffffff;
    s_last = s_n = s_bound = 0;
  }
  if (!(temp > 0.f)) {              // (the same for the whole cluster) block_argmax over its 1,024 threads
    ArgMax best{-INFINITY, 0x7fffffff};
    if (tid < SC_OWN) {
      constexpr int INFLIGHT = 16;
      const int t = rank * SC_OWN + tid;
      for (int base = t; base < vocab; base += INFLIGHT * SS_THREADS) {
        float v[INFLIGHT];
#pragma unroll
        for (int j = 0; j < INFLIGHT; ++j) {
          const int i = base + j * SS_THREADS;
          v[j] = i < vocab ? row[i] : -INFINITY;
        }
#pragma unroll
        for (int j = 0; j < INFLIGHT; ++j) {
          const int i = base + j * SS_THREADS;
          if (i < vocab && (v[j] > best.v || best.i == 0x7fffffff)) best = ArgMax{v[j], i};
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        ArgMax other{__shfl_xor_sync(0xffffffffu, best.v, o), __shfl_xor_sync(0xffffffffu, best.i, o)};
        best = better(best, other);
      }
    }
    sc_sync();                      // block 0 has started: its memory may be written
    if (tid < SC_OWN && lane == 0) {
      sc_write(&s_v[rank * 4 + warp], 0, __float_as_int(best.v));
      sc_write(&s_i[rank * 4 + warp], 0, best.i);
    }
    sc_sync();
    if (rank == 0 && tid == 0) {
      ArgMax b{__int_as_float(s_v[0]), s_i[0]};
      for (int w = 1; w < 32; ++w) b = better(b, ArgMax{__int_as_float(s_v[w]), s_i[w]});
      if (b.i == 0x7fffffff) b.i = 0;
      out[rowi] = b.i;
      if (fb >= 0) feedback[fb] = b.i;
    }
    return;
  }

  const int C = ((vocab + SS_THREADS - 1) / SS_THREADS) | 1;
  const int from = min(vocab, rank * SC_OWN * C), size = min(vocab, (rank + 1) * SC_OWN * C) - from;
  float m = -INFINITY;
#pragma unroll 16
  for (int i = tid; i < size; i += SC_THREADS) {
    const float v = row[from + i];
    s_row[i] = v;
    m = fmaxf(m, v);
  }
  const int k = top_k[rowi];
  const bool use_k = k > 0 && k < vocab;
  {
    uint32_t key = tid < size ? order_key(m) : 0u;
    key = max(key, __shfl_xor_sync(0xffffffffu, key, 1));
    key = max(key, __shfl_xor_sync(0xffffffffu, key, 2));
    if ((tid & 3) == 0) s_key[tid >> 2] = key;
    const float w = warp_max(m);
    if (lane == 0) s_max[warp] = w;
    __syncthreads();
    if (tid == 0) {
      float b = s_max[0];
      for (int i = 1; i < SC_THREADS / 32; ++i) b = fmaxf(b, s_max[i]);
      s_own = b;
    }
  }
  const int share = (k + SC_BLOCKS - 1) / SC_BLOCKS;     // of the k maxima this block answers for
  if (use_k && k <= SC_LIST_K && tid < SC_GROUPS) {
    const int2 n = sc_rank_of(s_key[tid], s_key, SC_GROUPS);
    if (n.x < share && share <= n.x + n.y) s_bound = (int)s_key[tid];
  }
  sc_sync();
  float top = lane < SC_BLOCKS ? sc_read(&s_own, lane) : -INFINITY;
  top = warp_max(top);
  const float mx = top / temp;
  uint32_t thr = 0;     // order key of the k-th largest logit; 0 keeps everything
  int need_eq = 0;      // how many entries equal to the threshold are kept (lowest indices)
  bool all_eq = true;   // ... which is all of them
  uint32_t bound = 0;
  bool listed = false;
  if (use_k && k <= SC_LIST_K) {
    uint32_t b = lane < SC_BLOCKS ? (uint32_t)sc_read(&s_bound, lane) : 0xffffffffu;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) b = min(b, __shfl_xor_sync(0xffffffffu, b, o));
    bound = b;
    if (bound > SC_LOWEST) {                             // (from minus infinity up it would be the whole row)
#pragma unroll 4
      for (int i = tid; i < size; i += SC_THREADS) {
        const uint32_t key = order_key(s_row[i]);
        if (key >= bound) {
          const int at = atomicAdd(&s_n, 1);
          if (at < SC_LIST) s_list[at] = key;
        }
      }
      sc_sync();
      const int own = lane < SC_BLOCKS ? sc_read(&s_n, lane) : 0;      // of block `lane`
      listed = __all_sync(0xffffffffu, own <= SC_LIST);
      int incl = own;                                    // entries of the blocks up to it
#pragma unroll
      for (int o = 1; o < SC_BLOCKS; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
      }
      const int n = __shfl_sync(0xffffffffu, incl, SC_BLOCKS - 1);
      listed = listed && n >= k && n <= SC_CAND;
      if (listed) {
        for (int i0 = warp * 32; i0 < n; i0 += SC_THREADS) {
          const int i = i0 + lane;
          int c = 0, first = 0;
#pragma unroll
          for (int b = 0; b < SC_BLOCKS - 1; ++b) {
            const int end = __shfl_sync(0xffffffffu, incl, b);
            if (i >= end) { c = b + 1; first = end; }
          }
          if (i < n) s_cand[i] = (uint32_t)sc_read((const int*)&s_list[i - first], c);
        }
        for (int i = n + tid; i < ((n + 3) & ~3); i += SC_THREADS) s_cand[i] = 0;   // (no entry's key)
        __syncthreads();
        // few: every block counts for all of them; else each for its own and tells the others
        const bool shared = n > SC_THREADS;
        const int end = __shfl_sync(0xffffffffu, incl, rank);
        const int i = shared ? end - s_n + tid : tid;
        for (int j = i; j < (shared ? end : n); j += SC_THREADS) {
          const int2 r = sc_rank_of(s_cand[j], s_cand, (n + 3) & ~3);
          if (r.x < k && k <= r.x + r.y)                 // the same for all entries equal to it
#pragma unroll 1
            for (int b = shared ? 0 : rank; b <= (shared ? SC_BLOCKS - 1 : rank); ++b) {
              sc_write(&s_tot[0], b, (int)s_cand[j]);
              sc_write(&s_tot[1], b, r.x);
              sc_write(&s_tot[2], b, r.y);
            }
        }
        if (shared) sc_sync();
        else __syncthreads();
        thr = (uint32_t)s_tot[0];
        need_eq = k - s_tot[1];
        all_eq = s_tot[2] == need_eq;
      }
    }
  }
  if (use_k && !listed) {
    int turn = 0, remaining = 0;
    // the want-th largest of the keys that the blocks' walks hand on; false where there are fewer
    auto select = [&](int want, uint32_t& prefix, auto walk) {
      prefix = 0;
      remaining = want;
      for (int shift = 24; shift >= 0; shift -= 8, turn ^= 1) {
        int* h = hist[turn];
        h[tid] = 0;
        __syncthreads();
        const uint32_t above_mask = shift == 24 ? 0u : (0xffffffffu << (shift + 8));
        walk([&](uint32_t key) {
          if ((key & above_mask) == prefix) atomicAdd(&h[(key >> shift) & 255u], 1);
        });
        sc_sync();
        int sum = 0;
#pragma unroll
        for (int b = 0; b < SC_BLOCKS; ++b) sum += sc_read(&h[tid], b);
        s_tot[tid] = sum;
        __syncthreads();
        if (tid < 32) {
          // lane l owns digits 8l .. 8l+7; digits are taken from the largest down
          int c[8], grp = 0;
#pragma unroll
          for (int b = 0; b < 8; ++b) {
            c[b] = s_tot[8 * lane + b];
            grp += c[b];
          }
          int incl = grp;             // inclusive sum over lanes lane .. 31
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_down_sync(0xffffffffu, incl, o);
            if (lane + o < 32) incl += u;
          }
          if (lane == 0) s_count = incl;
          int run = incl - grp;       // keys with a digit above this lane's
          if (run < remaining && remaining <= incl) {
#pragma unroll
            for (int b = 7; b >= 0; --b) {
              if (run < remaining && remaining <= run + c[b]) {
                s_digit = 8 * lane + b;
                s_above = run;
                s_same = c[b];
              }
              run += c[b];
            }
          }
        }
        __syncthreads();
        const bool few = s_count < remaining;     // (only with the first digit, and in every block)
        const int digit = s_digit, above = s_above;
        __syncthreads();              // they are read before the next digit takes their place
        if (few) {
          turn ^= 1;
          return false;
        }
        prefix |= (uint32_t)digit << shift;
        remaining -= above;
      }
      return true;
    };
    auto entries = [&](auto take) {
      for (int i = tid; i < size; i += SC_THREADS) {
        const uint32_t key = order_key(s_row[i]);
        if (key >= bound) take(key);
      }
    };
    if (!select(k, thr, entries)) {   // maxima that are no entries (of threads with NaNs alone)
      bound = 0;
      select(k, thr, entries);
    }
    need_eq = remaining;
    all_eq = s_same == remaining;
  }
  const int lo = min(size, tid * C), hi = min(size, lo + C);   // (of the first SC_OWN threads)
  int eq = 0;
  if (use_k && !all_eq) {             // equal entries before each owner's positions
    if (tid < SC_OWN) {
      for (int i = lo; i < hi; ++i) eq += order_key(s_row[i]) == thr;
      int incl = eq;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
      }
      if (lane == 31) s_eq[warp] = incl;
      eq = incl - eq;
    }
    sc_sync();
    int before = 0;
    for (int w = 0; w < rank * 4 + min(warp, 4); ++w) before += sc_read(&s_eq[w & 3], w >> 2);
    eq += before;
  }
  __syncthreads();
  // the weights: position by position, and where only some of the equal entries are kept owner by owner
  const bool ordered = use_k && !all_eq;
  if (!ordered) {
#pragma unroll 4
    for (int i = tid; i < size; i += SC_THREADS) {
      const float v = s_row[i];
      s_row[i] = !use_k || order_key(v) >= thr ? expf(v / temp - mx) : -1.f;
    }
    __syncthreads();
  }
  float sum = 0.f;
  bool any = false;
  if (tid < SC_OWN) {
    for (int i = lo; i < hi; ++i) {
      float e = s_row[i];
      bool kept;
      if (ordered) {
        const uint32_t key = order_key(e);
        kept = key > thr || (key == thr && eq++ < need_eq);
        e = kept ? expf(e / temp - mx) : -1.f;
        s_row[i] = e;
      } else {
        kept = !use_k || !(e == -1.f);
      }
      if (kept) {
        sum += e;
        any = true;
      }
    }
  }
  // weight of all kept entries below lo: within a warp, then over the 32 warps of the cluster
  float before = 0.f, incl = sum;
  if (tid < SC_OWN) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float u = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += u;
    }
    if (lane == 31) s_sum[warp] = incl;
    before = __shfl_up_sync(0xffffffffu, incl, 1);
    if (lane == 0) before = 0.f;
  }
  sc_sync();
  if (warp == 0) {
    float a = sc_read(&s_sum[lane & 3], lane >> 2);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float u = __shfl_up_sync(0xffffffffu, a, o);
      if (lane >= o) a += u;
    }
    s_warps[lane] = a;
  }
  __syncthreads();
  if (tid < SC_OWN) {
    const int w = rank * 4 + warp;
    const float total = s_warps[31];
    float run = (w > 0 ? s_warps[w - 1] : 0.f) + before;
    const float u = philox_uniform((uint32_t)seed_lo[rowi], (uint32_t)seed_hi[rowi],
                                   (uint32_t)position[rowi]);
    const float target = u * total;
    int cand = 0x7fffffff, last_kept = -1;
    for (int i = any ? lo : hi; i < hi; ++i) {
      const float e = s_row[i];
      if (e >= 0.f) {
        run += e;
        if (cand == 0x7fffffff && run > target) cand = from + i;
        last_kept = from + i;
      }
    }
    if (cand != 0x7fffffff) atomicMin(&s_found, cand);
    if (last_kept >= 0) atomicMax(&s_last, last_kept);
  }
  __syncthreads();
  if (tid == 0) {
    sc_write(&s_v[rank], 0, s_found);
    sc_write(&s_i[rank], 0, s_last);
  }
  sc_sync();
  if (rank == 0 && tid == 0) {
    int found = 0x7fffffff, last = 0;
    for (int b = 0; b < SC_BLOCKS; ++b) {
      found = min(found, s_v[b]);
      last = max(last, s_i[b]);
    }
    // u * total rounded up to the total itself: the last kept token
    const int tok = found != 0x7fffffff ? found : last;
    out[rowi] = tok;
    if (fb >= 0) feedback[fb] = tok;
  }
}

}  // namespace hs

HS_EXPORT int hs_argmax(int* out, const float* logits, int rows, int vocab, void* stream) {
  if (!out || !logits) return HS_ERR_ARGUMENT;
  if (rows <= 0) return HS_OK;
  if (vocab <= 0) return HS_ERR_ARGUMENT;
  hs::argmax_kernel<<<rows, hs::SM_THREADS, 0, (cudaStream_t)stream>>>(out, logits, vocab);
  HS_LAUNCH_CHECK();
  return HS_OK;
}

// feedback / feedback_slot (both may be null): row i also stores its token to
// feedback[feedback_slot[i]] when that slot is not negative.  status_word (may be null): its
// value is stored to out[rows].
HS_EXPORT int hs_sample(int* out, const float* logits, const float* temperature, const int* top_k,
                        const int* seed_lo, const int* seed_hi, const int* position, int rows,
                        int vocab, int* feedback, const int* feedback_slot,
                        const int* status_word, void* stream) {
  if (!out || !logits || !temperature || !top_k || !seed_lo || !seed_hi || !position)
    return HS_ERR_ARGUMENT;
  if (rows <= 0) return HS_OK;
  if (vocab <= 0) return HS_ERR_ARGUMENT;
  // a row that fits shared memory (beside the kernel's own few KB) is read once
  const size_t row_bytes = (size_t)vocab * sizeof(float);
  cudaError_t le;
  if (row_bytes <= 220 * 1024 && vocab >= hs::SC_VOCAB && rows <= hs::SC_ROWS) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(rows * hs::SC_BLOCKS);
    cfg.blockDim = dim3(hs::SC_THREADS);
    cfg.dynamicSmemBytes = (size_t)hs::SC_OWN * (((vocab + hs::SS_THREADS - 1) / hs::SS_THREADS) | 1) * 4;
    cfg.stream = (cudaStream_t)stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = hs::SC_BLOCKS;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = hs_pdl_enabled() ? 2 : 1;
    le = cudaLaunchKernelEx(&cfg, hs::sample_cluster_kernel, out, logits, temperature, top_k, seed_lo, seed_hi,
                            position, rows, vocab, feedback, feedback_slot, status_word);
  } else if (row_bytes <= 220 * 1024) {
    static cudaError_t state = cudaErrorUnknown;
    if (state != cudaSuccess)
      state = cudaFuncSetAttribute(hs::sample_smem_kernel,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
    if (state != cudaSuccess) return (int)state;
    le = hs_launch(hs::sample_smem_kernel, dim3(rows), dim3(hs::SS_THREADS), row_bytes,
                   (cudaStream_t)stream, hs_pdl_enabled(), out, logits, temperature, top_k,
                   seed_lo, seed_hi, position, vocab, feedback, feedback_slot, status_word);
  } else {
    le = hs_launch(hs::sample_kernel, dim3(rows), dim3(hs::SM_THREADS), 0, (cudaStream_t)stream,
                   hs_pdl_enabled(), out, logits, temperature, top_k, seed_lo, seed_hi, position,
                   vocab, feedback, feedback_slot, status_word);
  }
  if (le != cudaSuccess) return (int)le;
  HS_LAUNCH_CHECK();
  return HS_OK;
}
