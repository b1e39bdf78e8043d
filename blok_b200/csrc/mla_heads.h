// The small kernels between the projections of the MLA block (mla_heads.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "mla_plan.cuh"

namespace blok {

// Entry b stands at position len[b], or (a chunk of one sequence) at len[0] + b; a sequence has cap rows.
struct MlaPositions {
  const int *len;
  int chunk;
  long cap;
};

// fp32 sums of the projections' K splits are [nz][B][ld].
struct MlaNorm {
  const float *part;  // q_a's q_rank columns, then kv_a's kv_rank + rope
  int nz, ld, q_rank, kv_rank, rope;
  float eps;
  const uint16_t *q_ln, *kv_ln;
  uint16_t *qa;  // [B, q_rank], normalised
  const float *inv_freq;
  MlaPositions pos;
  uint16_t *cache;  // dense: entry b's rows start at b * ctx_stride; paged: block_table
  long ctx_stride;
  const int *block_table, *slot_of;
  int table_stride, page_rows;
  int *seq;       // [B] position + 1
  MlaPlan *plan;  // how `ctas` CTAs of the attention core share the sequences,
  int2 *parts;    // [B] and what partial results they leave
  int ctas;
  unsigned *err;  // 1 + b of an entry outside its rows
};
int launch_mla_norm(const MlaNorm &a, int B, cudaStream_t stream);

struct MlaQuery {
  const float *part;  // sums of q_b's K split, ld = heads * (nope + rope); NULL: q
  const uint16_t *q;  // [B, heads, nope + rope]
  int nz, B, nope, rope, kv_rank;
  const float *inv_freq;
  MlaPositions pos;
  uint16_t *q_full;  // [B, heads, kv_rank + rope]
  unsigned *werr;    // set when a wait gives up
};
// wuk_t: [heads, kv_rank, nope].  The weights are fetched before the kernels in front of the launch have finished.
int launch_mla_query(const uint16_t *wuk_t, int heads, const MlaQuery &a, cudaStream_t stream);

struct MlaValue {
  const float *part_o, *part_ml;  // [partial result, heads, 512], [.., heads, 2]
  int B, nope, v_head;
  int splits;         // of every entry; 0: entry b has parts[b].y of them from parts[b].x on, fewer than ctas + B in all
  int ctas;
  const int2 *parts;  // there since before the attention core began
  uint16_t *out;  // [B, heads, v_head]
  unsigned *werr;
  int group;  // entries per CTA (set by the launch)
};
// kv_b: [heads, nope + v_head, 512].  The weights are fetched early, as above.
int launch_mla_value(const uint16_t *kv_b, int heads, MlaValue a, cudaStream_t stream);

}  // namespace blok
