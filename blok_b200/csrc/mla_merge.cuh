// The merge behind the split-context attention cores (mla.cu, latent_attn.cu, grouped_attn.cu).
#pragma once
#include "common.cuh"

namespace blok {

// ---------------------------------------------------------------------------
// Merge of the split-KV partial results.  grid = (heads, B), 128 threads.
//   part_o fp32 [B, splits, heads, kv_rank] unnormalised, part_ml fp32 [B, splits, heads, 2] = (max, sum)
// parts, optional: entry b has parts[b].y <= splits partial results, one after another from parts[b].x on.
// Rows of o_lat are ldo values apart (0: heads * kv_rank).  gate, optional: bf16 [B, ld_gate]; head h's output times
// sigmoid(gate[b][h]).
// ---------------------------------------------------------------------------
template <int FLY>
static __global__ void mla_merge_kernel(const float *part_o, const float *part_ml, int splits, int heads, int kv_rank,
                                        uint16_t *__restrict__ o_lat, int ldo = 0, const uint16_t *gate = nullptr, int ld_gate = 0,
                                        const int2 *parts = nullptr) {
  extern __shared__ float s_wt[];  // [splits] weight of every split: exp(m_s - M), 0 for an empty split
  __shared__ float s_red[2][4];
  pdl_trigger();
  pdl_wait();
  const int h = blockIdx.x, b = blockIdx.y, tid = threadIdx.x;
  size_t first = (size_t)b * splits;
  if (parts) first = parts[b].x, splits = parts[b].y;
  // Four columns per thread, FLY partial results in flight per thread: they come from L2 or HBM (128 KB each for 64 heads of 512), and
  // the kernel is as fast as it keeps bytes in flight.  The first are asked for before the weights are known, and a remainder goes
  // like the rest.  Each column adds its splits in ascending order.
  const float4 *po4 = reinterpret_cast<const float4 *>(part_o + (first * heads + h) * kv_rank);
  const size_t stride4 = (size_t)heads * kv_rank / 4;
  float4 v[FLY];
  auto ask = [&](int s, int j4) {
#pragma unroll
    for (int i = 0; i < FLY; ++i)
      if (s + i < splits) v[i] = po4[(size_t)(s + i) * stride4 + j4];
  };
  if (tid < kv_rank / 4) ask(0, tid);
  const float2 *ml = reinterpret_cast<const float2 *>(part_ml) + first * heads + h;  // (max, sum) of split s at + s * heads
  const float2 own = tid < splits ? ml[(size_t)tid * heads] : make_float2(-INFINITY, 0.f);
  float M = own.x;
  for (int s = tid + blockDim.x; s < splits; s += blockDim.x) M = fmaxf(M, ml[(size_t)s * heads].x);
  M = warp_max(M);
  if ((tid & 31) == 0) s_red[0][tid >> 5] = M;
  __syncthreads();
  M = fmaxf(fmaxf(s_red[0][0], s_red[0][1]), fmaxf(s_red[0][2], s_red[0][3]));
  float L = 0.f;
  for (int s = tid; s < splits; s += blockDim.x) {
    const float2 m = s == tid ? own : ml[(size_t)s * heads];
    const float wt = m.x != -INFINITY ? expf(m.x - M) : 0.f;
    s_wt[s] = wt;
    L += wt * m.y;
  }
  L = warp_sum(L);
  if ((tid & 31) == 0) s_red[1][tid >> 5] = L;
  __syncthreads();
  L = (s_red[1][0] + s_red[1][1]) + (s_red[1][2] + s_red[1][3]);
  float inv = L > 0.f ? 1.0f / L : 0.f;
  if (gate) inv *= 1.0f / (1.0f + expf(-bf16_bits_to_f32(gate[(size_t)b * ld_gate + h])));
  if (!ldo) ldo = heads * kv_rank;
  for (int j4 = tid; j4 < kv_rank / 4; j4 += blockDim.x) {
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int s = 0; s < splits; s += FLY) {
      if (s > 0 || j4 != tid) ask(s, j4);
#pragma unroll
      for (int i = 0; i < FLY; ++i) {
        const float wt = s + i < splits ? s_wt[s + i] : 0.f;
        // an empty split holds no result: its weight of zero must not meet whatever lies there
        if (wt != 0.f) acc.x = fmaf(wt, v[i].x, acc.x), acc.y = fmaf(wt, v[i].y, acc.y), acc.z = fmaf(wt, v[i].z, acc.z), acc.w = fmaf(wt, v[i].w, acc.w);
      }
    }
    uint2 o;
    o.x = pack_bf16x2(acc.x * inv, acc.y * inv);
    o.y = pack_bf16x2(acc.z * inv, acc.w * inv);
    *reinterpret_cast<uint2 *>(o_lat + (size_t)b * ldo + (size_t)h * kv_rank + (size_t)j4 * 4) = o;
  }
}

// Few blocks have many parts of a sequence each, and sixteen in flight help; where blocks are many, the registers of eight let more of
// them run.  Core and merge alone, cold, us: one sequence of 3,000 tokens (47 parts) 33.8 with eight behind the weights and the remainder
// one by one, 25.6 with sixteen; 64 sequences of 64 tokens 27.6 with sixteen, 23.5 with eight.
inline auto mla_merge(int heads, int B) { return heads * B <= 2 * sm_count() ? mla_merge_kernel<16> : mla_merge_kernel<8>; }

}  // namespace blok
