// What the routed feed-forward's kernels (moe.cu) and its tcgen05 tiles (moe_tiles_tc.cu) share.
#pragma once
#include "common.cuh"

namespace hs {

constexpr int MT_PAIRS = 256;         // pairs of one expert a tile takes at most

// act 0: g = min(g, limit), u = clamp(u, -limit, limit), g * sigmoid(1.702 g) * (u + 1); act 1:
// silu(g) * u; act 2: relu(u)^2 (an expert without a gate matrix)
template <int ACT>
__device__ __forceinline__ float expert_act(float g, float u, float limit) {
  if (ACT == 1) return g / (1.0f + expf(-g)) * u;
  if (ACT == 2) { const float r = fmaxf(u, 0.f); return r * r; }
  g = fminf(g, limit);
  u = fminf(fmaxf(u, -limit), limit);
  return g * (1.0f / (1.0f + expf(-1.702f * g))) * (u + 1.0f);
}
__device__ __forceinline__ float expert_act(float g, float u, float limit, int act) {
  return act == 1 ? expert_act<1>(g, u, limit) : act == 2 ? expert_act<2>(g, u, limit) : expert_act<0>(g, u, limit);
}

// The pairs sorted by expert: act_rows = activated gate / up rows (bfloat16 [pairs, ff]), down_rows =
// their down projections (float32 [pairs, width]).  tiles: [0] number, [1] rows of the widest (a multiple
// of 16), then (expert, first row, rows) a tile.  HS_ERR_UNSUPPORTED for operands that are not
// 16-byte aligned.
int moe_tiles_tc(__nv_bfloat16* act_rows, float* down_rows, const __nv_bfloat16* h,
                 const __nv_bfloat16* w_gate, const __nv_bfloat16* w_up, const __nv_bfloat16* w_down,
                 const int* tiles, int max_tiles, const int* row_token, int pairs, int width, int ff, int E, float limit, int act,
                 int* status, cudaStream_t st);

}  // namespace hs
