// Warp-level top-k selection of the router (one warp per token).
#pragma once
#include <cmath>

#include "common.cuh"

namespace blok {

// score: shared-memory array of `experts` floats owned by this warp, filled with s = sigmoid(logit) and __syncwarp()ed;
// sel[j]: this lane's s + bias of expert 32 j + lane (candidates past the last expert: -inf), N >= experts / 32.  Runs `topk`
// rounds of argmax with the reference's rule (strict '>' scanning ascending indices: the lowest index wins a tie, -inf and
// NaN are never taken, expert 0 where nothing is left; src/kimi_exec.cu:390-395).  Lane k < topk returns the k-th selected
// expert in my_id and its normalised, scaled weight in my_w.  The candidates stay in registers as integers of
// the same order, two warp reductions a round (shared memory and shuffles before).
template <int N>
__device__ __forceinline__ void warp_topk(const float *score, const float (&sel)[N], int topk, float routed_scale, int lane, int &my_id,
                                          float &my_w) {
  uint32_t key[N];
#pragma unroll
  for (int j = 0; j < N; ++j) {
    const uint32_t b = __float_as_uint(sel[j] + 0.0f);  // -0 becomes +0: equal to it, as a comparison has them
    key[j] = sel[j] > -INFINITY ? ((b >> 31) ? ~b : b | 0x80000000u) : 0u;
  }
  float sum = 0.f;
  my_w = 0.f;
  my_id = 0;
  for (int k = 0; k < topk; ++k) {
    uint32_t best = 0;
    int at = 0x7fffffff;
#pragma unroll
    for (int j = 0; j < N; ++j)
      if (key[j] > best) best = key[j], at = 32 * j + lane;
    const uint32_t top = __reduce_max_sync(0xffffffffu, best);
    int id = __reduce_min_sync(0xffffffffu, best == top ? at : 0x7fffffff);
    if (id == 0x7fffffff) id = 0;
    const float s = score[id];
    sum += s;
    if (lane == k) my_w = s, my_id = id;
#pragma unroll
    for (int j = 0; j < N; ++j)
      if (32 * j + lane == id) key[j] = 0;
  }
  my_w = my_w / (sum + 1.0e-20f) * routed_scale;
}

}  // namespace blok
