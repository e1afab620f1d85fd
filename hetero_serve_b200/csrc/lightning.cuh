// What lightning attention's recurrence (lightning.cu) and its chunks (lightning_chunk.cu) share.
#pragma once
#include "rotary.cuh"

namespace hs {

__device__ __forceinline__ float la_act(float z, int act) {
  return act == HS_ACT_SILU ? z / (1.0f + expf(-z)) : z;
}
// entry d of a head's q or k vector `vec`: activated, turned by position `pos` when d lies in the
// first rot_dims numbers (rot_dims 0: never), times `mul`
__device__ __forceinline__ float la_entry(const float* __restrict__ vec, int d, int act,
                                          int rot_dims, const float* __restrict__ freq, int pos,
                                          float mul) {
  float own = la_act(vec[d], act);
  if (d < rot_dims) {
    const int half = rot_dims >> 1;
    const bool low = d < half;
    const float partner = la_act(vec[low ? d + half : d - half], act);
    float c, sn;
    pair_angle(pos, freq[low ? d : d - half], &c, &sn);
    const float cross = __fmul_rn(partner, sn);
    own = fmaf(own, c, low ? -cross : cross);
  }
  return __fmul_rn(own, mul);
}

// Heads of 128 x 128; portions of LC_MIN tokens and more may go in chunks of 64 (each request for itself).
// (us, stream against chunks, 8 heads: 1 x 256 tokens 38 and 51, 1 x 384 52 and 52, 1 x 512 70 and 51, 8 x
// 512 179 and 115; with silu and no turning 1 x 512 71 and 60.  Heads of 64 gain nothing on a full device:
// 4 x 1,024 tokens of 32 heads 230 and 242.)
constexpr int LC_D = 128, LC_V = 128, LC_MIN = 512;
__host__ __device__ constexpr int lc_chunks(int tokens) { return tokens < LC_MIN ? 0 : (tokens + 63) / 64; }
// chunks a step can have at most
__host__ __device__ constexpr int lightning_chunk_slots(int n_tokens, int n_requests) {
  return n_tokens < LC_MIN ? 0 : n_tokens / 64 + (n_requests < n_tokens / LC_MIN ? n_requests : n_tokens / LC_MIN);
}

// Heads that go together: a state a chunk and head is scratch, 64 KB, and a step's heads share 128 MB of it (8,192
// tokens of 64 heads: 5 groups of 13, where all at once would keep 0.6 GB).
constexpr long long LC_SCRATCH = 1LL << 25;
constexpr int lightning_chunk_heads(int n_tokens, int n_requests, int H, int D, int V) {
  const long long a_head = (long long)lightning_chunk_slots(n_tokens, n_requests) * D * V;
  const long long most = a_head == 0 || LC_SCRATCH / a_head > H ? H : LC_SCRATCH / a_head < 1 ? 1 : LC_SCRATCH / a_head;
  const long long groups = (H + most - 1) / most;
  return (int)((H + groups - 1) / groups);
}
// floats of scratch: a state of these heads a chunk, the tokens' cosines and sines (0: no chunks)
constexpr long long lightning_chunk_floats(int n_tokens, int n_requests, int H, int D, int V, int rot_dims) {
  const long long slots = lightning_chunk_slots(n_tokens, n_requests);
  return slots ? slots * lightning_chunk_heads(n_tokens, n_requests, H, D, V) * D * V + (long long)n_tokens * rot_dims : 0;
}

bool lightning_takes_chunks(int D, int V, int rot_dims);
// Requests of LC_MIN tokens and more; the others are left alone.  scratch: lightning_chunk_floats,
// 16-byte aligned.
int lightning_chunks(float* o, float* state, const float* proj, const float* decay, const int* req_start,
                     const int* req_len, const int* req_slot, int n_requests, int n_tokens, int stride,
                     int q_off, int k_off, int v_off, int H, int D, int V, int act, float* scratch,
                     const int* tok_pos, const float* freq, int rot_dims, float k_scale, cudaStream_t st);

}  // namespace hs
