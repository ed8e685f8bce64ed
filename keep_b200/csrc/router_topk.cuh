// Pieces of the score function and top-k of one token that keepvq_routed_topk (router.cu) and the few-token
// layer kernel (few_tokens.cu) share: the same arithmetic in the same order, so the same picks and weights.
#pragma once

#include <math.h>

#include "router_logits.cuh"

namespace keepvq {

// Floats as unsigned keys of the same order (-inf lowest of the real values); 0 is below all of them.
__device__ __forceinline__ uint32_t ordered_key(float v) {
  const uint32_t u = __float_as_uint(v);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// The softmax's maximum (exact in any order), and the one-value score functions.
template <int NPL>
__device__ __forceinline__ float topk_max(const float (&lg)[NPL]) {
  float m = -INFINITY;
#pragma unroll
  for (int i = 0; i < NPL; ++i) m = fmaxf(m, lg[i]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xFFFFFFFFu, m, o));
  return m;
}
// ... and its sum: a lane's values in order, then a butterfly over the lanes.
template <int NPL>
__device__ __forceinline__ float topk_sum(const float (&ex)[NPL], int pool, int lane) {
  float s = 0.0f;
#pragma unroll
  for (int i = 0; i < NPL; ++i)
    if (lane + 32 * i < pool) s += ex[i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xFFFFFFFFu, s, o);
  return s;
}
__device__ __forceinline__ float topk_sigmoid(float v) { return 1.0f / (1.0f + expf(-v)); }
__device__ __forceinline__ float topk_sqrt_softplus(float v) { return sqrtf(v > 20.0f ? v : log1pf(expf(v))); }

// The top_k largest of a warp's keys, NQ per lane with their expert ids, in descending order, ties to the
// lowest id: lane j gets pick j (key 0 where there are none left).  A pick is a tree over the lane's
// registers, one warp max and one warp min (redux.sync): for warps that have the SM to themselves and wait for
// each step (routed_topk_reg_kernel scans, which is fewer instructions).
template <int NQ>
__device__ __forceinline__ void topk_select(uint32_t (&key)[NQ], const int (&id)[NQ], int top_k, int lane, uint32_t& my_key, int& my_e) {
  my_key = 0u;
  my_e = 0;
#pragma unroll 1
  for (int j = 0; j < top_k; ++j) {
    uint32_t best[NQ];
    int at[NQ];
#pragma unroll
    for (int i = 0; i < NQ; ++i) { best[i] = key[i]; at[i] = id[i]; }
#pragma unroll
    for (int step = 1; step < NQ; step *= 2)
#pragma unroll
      for (int i = 0; i + step < NQ; i += 2 * step)
        if (best[i + step] > best[i] || (best[i + step] == best[i] && at[i + step] < at[i])) { best[i] = best[i + step]; at[i] = at[i + step]; }
    const uint32_t top = __reduce_max_sync(0xFFFFFFFFu, best[0]);
    const int win = static_cast<int>(__reduce_min_sync(0xFFFFFFFFu, best[0] == top ? static_cast<uint32_t>(at[0]) : 0xFFFFFFFFu));
#pragma unroll
    for (int i = 0; i < NQ; ++i)
      if (id[i] == win) key[i] = 0u;
    if (lane == j) { my_key = top; my_e = win; }
  }
}
// A score with its selection bias as a key (at least 1).
__device__ __forceinline__ uint32_t topk_key(const float* bias, int e, float score) { return max(ordered_key(score + (bias ? bias[e] : 0.0f)), 1u); }

// Lane j < top_k has pick j of one of the two selections, the served picks (pass 0) or the demanded ones
// (pass 1), and its score: its slot and weight (pass 0); `write` stores the outputs.
__device__ __forceinline__ void topk_finish(const keepvq_routed_topk_args& a, int64_t t, int lane, int pass, int my_e, float my_raw, bool write, uint32_t& slot, float& weight) {
  const int K = a.top_k;
  float raw = 0.0f;
  bool live = false;
  if (lane < K) {
    raw = my_raw;
    live = pass == 1 || !a.served_bias || a.served_bias[my_e] > ABSENT_BIAS;
    if (!live) raw = 0.0f;  // a masked pick carries no weight (local_eval.py:87)
  }
  float sum = raw;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
  slot = KEEPVQ_NO_RESIDUAL;
  weight = 0.0f;
  if (lane < K) {
    const int e = my_e;
    const int64_t o = t * K + lane;
    if (pass == 0) {
      float w = raw;
      if (a.norm_topk_prob && K > 1) w = w / (sum + 1e-20f);
      w *= a.route_scale;
      weight = w;
      slot = live ? (a.slot_of ? a.slot_of[e] : static_cast<uint32_t>(e)) : KEEPVQ_NO_RESIDUAL;
      if (write) {
        a.served_weight[o] = w;
        a.served_expert[o] = live ? static_cast<uint32_t>(e) : KEEPVQ_NO_RESIDUAL;
        a.served_slot[o] = slot;
      }
    } else if (write) {
      a.want[o] = static_cast<uint32_t>(e);
      a.want_score[o] = raw;
      if (a.admit) {
        // the policy's own normalisation: always over the k demanded scores (omlx_routed.py:186)
        const float g = raw / (sum + 1e-20f) * a.route_scale;
        const bool absent = a.served_bias && a.served_bias[e] <= ABSENT_BIAS;
        a.admit[o] = (absent && g >= a.tau) ? e : -1;
      }
    }
  }
}
}  // namespace keepvq
