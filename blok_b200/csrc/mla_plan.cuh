// How the attention core's CTAs share the tiles of a batch of sequences (mla_attend_tc.cu) and what the merge finds of it.
//
// The tiles of all sequences lie on one line, sequence after sequence, and CTA i takes the piece [i per, (i + 1) per) of it; its part
// of sequence b is partial result i + b: consecutive for a sequence, and fewer than CTAs + sequences in all.  Two ways:
//  - every sequence in pieces of its own, the longest as short as the CTAs allow (lead 0, each sequence's length on the line rounded
//    up to whole pieces).
//  - pieces over the sequences' borders, where that makes them shorter.  A further sequence costs a CTA about kMlaPlanLead tiles (its
//    queries, its result), so each has a lead of that length.
// Against a fixed number of parts per sequence (the longest one then sets the time), the block, us: 33 sequences of 1,500 to 6,000
// tokens 122 -> 110, 50 of 5,000 158 -> 147; where that number was as good the plan's way through memory costs 1 to 2.5 us
// (8 of 32,768 126 -> 128.5, one of 4,001 64.8 -> 65.4; the core alone, which makes the plan itself, over one of 3,000 23.5 -> 25.6).
#pragma once
#include "common.cuh"

namespace blok {

constexpr int kMlaPlanTile = 64, kMlaPlanLead = 2, kMlaPlanMax = 64;

struct MlaPlan {
  int per, lead;
  int start[kMlaPlanMax + 1];  // of a sequence's lead on the line
  int tokens[kMlaPlanMax];
};

// One whole warp; tokens(b): the length of sequence b < B <= kMlaPlanMax <= ctas.
template <typename F>
__device__ __forceinline__ void mla_plan(MlaPlan &p, int B, int ctas, F tokens) {
  const int lane = threadIdx.x & 31;
  const int ta = lane < B ? max(0, tokens(lane)) : 0, tc = lane + 32 < B ? max(0, tokens(lane + 32)) : 0;
  p.tokens[lane] = ta, p.tokens[lane + 32] = tc;
  int a = (ta + kMlaPlanTile - 1) / kMlaPlanTile, c = (tc + kMlaPlanTile - 1) / kMlaPlanTile;
  const int total = __reduce_add_sync(0xffffffffu, a + c);
  int per = max(1, (total + kMlaPlanLead * B + ctas - 1) / ctas), lead = kMlaPlanLead;
  // pieces of t tiles are enough for every sequence by itself where the number of pieces does not exceed the CTAs'
  auto pieces = [&](int t) { return __reduce_add_sync(0xffffffffu, (a + t - 1) / t + (c + t - 1) / t); };
  if (B == 1) {  // the search's result
    per = max(1, (total + ctas - 1) / ctas), lead = 0;
    a = (a + per - 1) / per * per;
  } else if (pieces(per + 1) <= ctas) {
    int lo = max(1, (total + ctas - 1) / ctas), hi = per + 1;
    while (lo < hi) {
      const int t = (lo + hi) / 2;
      if (pieces(t) <= ctas) hi = t;
      else lo = t + 1;
    }
    per = hi, lead = 0;
    a = (a + per - 1) / per * per, c = (c + per - 1) / per * per;
  } else {
    if (lane < B) a += lead;
    if (lane + 32 < B) c += lead;
  }
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int ua = __shfl_up_sync(0xffffffffu, a, o), uc = __shfl_up_sync(0xffffffffu, c, o);
    if (lane >= o) a += ua, c += uc;
  }
  const int half = __shfl_sync(0xffffffffu, a, 31);
  p.start[lane + 1] = a;
  p.start[lane + 33] = half + c;
  if (lane == 0) p.start[0] = 0, p.per = per, p.lead = lead;
  __syncwarp();
}

// The partial results of sequence b: the first, and how many (none: an empty sequence).
__device__ __forceinline__ int2 mla_plan_parts(const MlaPlan &p, int b) {
  const int tiles = (p.tokens[b] + kMlaPlanTile - 1) / kMlaPlanTile, tile0 = p.start[b] + p.lead, i0 = tile0 / p.per;
  return make_int2(i0 + b, tiles > 0 ? (tile0 + tiles - 1) / p.per - i0 + 1 : 0);
}

}  // namespace blok
