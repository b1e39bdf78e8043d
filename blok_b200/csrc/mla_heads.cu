// The small kernels between the projections of the MLA block (mla.cu): the norms and the cache row behind the down projections,
// the absorbed query and its rotated part behind q_b, and the merge of the context splits with the per-head value product.
//
// Each stands where a few hundred kilobytes change hands between two weight streams, so what they cost is latency: every one takes
// its input as the kernel before leaves it (fp32 sums of a K split, partial results of the context splits), so that no launch
// exists only to add them, and the per-head products have their weights in shared memory before the wait for that input.  From one
// kernel's last store to the next one's first load pass about 1 us; of the rest (time stamps, one sequence / 8 / 64 tokens, us) the
// norms take 4 / 4 / 2, the query 2.5 / 3.5 / 5, merge and value product 7 / 13 / 9, where nine launches stood before.
#include <algorithm>

#include "gemm_tma.h"
#include "mla_heads.h"
#include "tc_pipe.cuh"

namespace blok {

// Four consecutive sums of a K split: nz parts, `stride` values apart, added in order; FLY loads in flight.
template <int FLY>
__device__ __forceinline__ float4 mh_sum4(const float *p, size_t stride, int nz) {
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
  for (int z = 0; z < nz; z += FLY) {
    float4 v[FLY];
#pragma unroll
    for (int i = 0; i < FLY; ++i, p += stride)
      if (z + i < nz) v[i] = *reinterpret_cast<const float4 *>(p);
#pragma unroll
    for (int i = 0; i < FLY; ++i)
      if (z + i < nz) acc.x += v[i].x, acc.y += v[i].y, acc.z += v[i].z, acc.w += v[i].w;
  }
  return acc;
}

constexpr int kMnThreads = 512;
// Values of a row that stay in shared memory between its two passes: 44 KB, which a launch gets without asking beside what the kernel
// keeps in static arrays.  Of longer rows the rest is added up from the parts a second time.
constexpr int kMnKept = 11264;

__device__ __forceinline__ float mh_block_sum(float v, float *red) {
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  return warp_sum((threadIdx.x & 31) < kMnThreads / 32 ? red[threadIdx.x & 31] : 0.f);
}

// The position of entry b.  One outside the sequence's rows (dense: ctx_cap rows; paged: the table's pages) must not become a
// store or a read: the row is not written, the attention is kept inside the rows, and the host learns of it from *err.
__device__ __forceinline__ int mh_position(const MlaPositions &p, int b, bool *in_range) {
  const int pos = p.chunk ? p.len[0] + b : p.len[b];
  *in_range = pos >= 0 && (long)pos < p.cap;
  return *in_range ? pos : (pos < 0 ? 0 : (int)(p.cap - 1));
}

// Interleaved pair (2 p, 2 p + 1) -> de-interleaved (p, half + p), every product rounded (src/kimi_exec.cu:346-357).
__device__ __forceinline__ void mh_rotate(float x0, float x1, float c, float s, uint16_t *lo, uint16_t *hi) {
  *lo = f32_to_bf16_bits(round_bf16(x0 * c) - round_bf16(x1 * s));
  *hi = f32_to_bf16_bits(round_bf16(x1 * c) + round_bf16(x0 * s));
}

// grid = (2, B); dynamic shared memory: the longer of the two rows, up to kMnKept floats.  Block 0 of an entry: q_a's sums -> bf16 -> RMSNorm
// (:813-815).  Block 1: kv_a's -> bf16, c_kv normalised, k_pe rotated, the row appended to the cache, the length of the sequence
// published (:816-824).  What the call was given (positions, tables, weights) is read before the wait, see decode_body.
__global__ void __launch_bounds__(kMnThreads) mla_norm_kernel(const MlaNorm a) {
  extern __shared__ float val[];
  __shared__ float red[kMnThreads / 32];
  const int b = blockIdx.y, tid = threadIdx.x, lat = a.kv_rank + a.rope, half = a.rope / 2;
  __shared__ MlaPlan s_plan;
  const bool kv = blockIdx.x != 0, plans = !kv && b == 0 && tid >= kMnThreads - 32;
  const int n = kv ? a.kv_rank : a.q_rank, all = kv ? lat : n;  // values under the norm, and in all
  pdl_trigger();
  const uint16_t *ln = kv ? a.kv_ln : a.q_ln;
  uint2 first_ln = make_uint2(0, 0);  // the thread's first four weights
  if (4 * tid < n) first_ln = make_uint2(ln[4 * tid] | (uint32_t)ln[4 * tid + 1] << 16, ln[4 * tid + 2] | (uint32_t)ln[4 * tid + 3] << 16);
  bool in_range = true;
  int pos = 0;
  float c = 0.f, s = 0.f;
  uint16_t *out = a.qa + (size_t)b * a.q_rank;
  if (kv) {
    pos = mh_position(a.pos, b, &in_range);
    if (tid < half) c = round_bf16(cosf(pos * a.inv_freq[tid])), s = round_bf16(sinf(pos * a.inv_freq[tid]));
    out = a.block_table ? a.cache + ((size_t)a.block_table[(size_t)(a.slot_of ? a.slot_of[b] : b) * a.table_stride + pos / a.page_rows] * a.page_rows +
                                     pos % a.page_rows) * lat
                        : a.cache + ((size_t)b * a.ctx_stride + pos) * lat;
  }
  if (plans)
    mla_plan(s_plan, gridDim.y, a.ctas, [&](int i) {
      bool in;
      return mh_position(a.pos, i, &in) + 1;
    });
  pdl_wait();
  if (plans) {
    for (int i = tid & 31; i < (int)gridDim.y; i += 32) a.parts[i] = mla_plan_parts(s_plan, i);
    for (int i = tid & 31; i < (int)(sizeof(MlaPlan) / sizeof(int)); i += 32) reinterpret_cast<int *>(a.plan)[i] = reinterpret_cast<const int *>(&s_plan)[i];
  }
  if (kv) {
    if (tid == 0) {
      a.seq[b] = pos + 1;
      if (!in_range) atomicExch(a.err, 1u + (unsigned)b);
    }
    if (!in_range) return;
  }
  const float *row = a.part + (size_t)b * a.ld + (kv ? a.q_rank : 0);
  auto sums = [&](int i) {
    float4 f = mh_sum4<16>(row + i, (size_t)gridDim.y * a.ld, a.nz);
    f.x = round_bf16(f.x), f.y = round_bf16(f.y), f.z = round_bf16(f.z), f.w = round_bf16(f.w);
    return f;
  };
  float v = 0.f;
  for (int i = 4 * tid; i < all; i += 4 * kMnThreads) {
    const float4 f = sums(i);
    if (i < kMnKept) *reinterpret_cast<float4 *>(val + i) = f;
    if (i < n) v = fmaf(f.x, f.x, fmaf(f.y, f.y, fmaf(f.z, f.z, fmaf(f.w, f.w, v))));
  }
  const float scale = rsqrtf(mh_block_sum(v, red) / n + a.eps);  // its barrier also orders val
  for (int i = 4 * tid; i < n; i += 4 * kMnThreads) {
    const float4 f = i < kMnKept ? *reinterpret_cast<const float4 *>(val + i) : sums(i);
    if (i != 4 * tid) first_ln = make_uint2(ln[i] | (uint32_t)ln[i + 1] << 16, ln[i + 2] | (uint32_t)ln[i + 3] << 16);
    *reinterpret_cast<uint2 *>(out + i) = make_uint2(pack_bf16x2(round_bf16(f.x * scale) * bf16lo(first_ln.x), round_bf16(f.y * scale) * bf16hi(first_ln.x)),
                                                     pack_bf16x2(round_bf16(f.z * scale) * bf16lo(first_ln.y), round_bf16(f.w * scale) * bf16hi(first_ln.y)));
  }
  if (kv && tid < half) mh_rotate(val[n + 2 * tid], val[n + 2 * tid + 1], c, s, out + n + tid, out + n + half + tid);
}

// Byte offset of 16 bytes (columns 8 c .. 8 c + 7) of a row in a K-major operand of 64 columns in the 128-byte swizzle.
__device__ __forceinline__ uint32_t mh_swizzled(int row, int c) { return (uint32_t)(row * 128 + ((c ^ (row & 7)) << 4)); }

// One block of 128 weight rows against N tokens: `boxes` pieces of 64 columns, weights at sw, tokens at sx.  A whole warp calls.
__device__ __forceinline__ void mh_mma(uint32_t tmem, uint32_t sw, uint32_t sx, int boxes, int N, bool more, uint32_t done) {
  tc_fence_after();
  if (tp_elect()) {
    for (int j = 0; j < boxes; ++j) {
      const uint64_t ad = tp_desc_k_sw128(sw + (uint32_t)j * 16384), bd = tp_desc_k_sw128(sx + (uint32_t)(j * N * 128));
#pragma unroll
      for (int k = 0; k < 4; ++k) tp_mma(tmem, ad + (uint64_t)(2 * k), bd + (uint64_t)(2 * k), tp_idesc_bf16(N), more || j || k);
    }
    tp_commit(done);
  }
}

// The accumulator's first n token columns to out, out + ld, ...: a lane owns a row.
__device__ __forceinline__ void mh_store(uint32_t tmem, int n, bool row, uint16_t *out, size_t ld, bool failed) {
#pragma unroll 1
  for (int t0 = 0; t0 < n; t0 += 16) {
    uint32_t v[16];
    tmem_ld16(tmem + t0, v);
    tmem_wait_ld();
#pragma unroll
    for (int j = 0; j < 16; ++j, out += ld)
      if (row && t0 + j < n) *out = f32_to_bf16_bits(__uint_as_float(failed ? 0x7fc00000u : v[j]));
  }
}

constexpr int kMqThreads = 256;
constexpr int kMqCols = 128;  // columns per piece (qk_nope: one piece for 128)

// grid = (heads, kv_rank / 128 + 1), 256 threads.  A CTA makes 128 rows of one head's absorbed query, W_UK^T q_nope (:366-369 folded
// into the query); the last one of a head rotates its rope part.  q: fp32 sums of q_b's K split, or bf16.
__global__ void __launch_bounds__(kMqThreads) mla_query_kernel(const __grid_constant__ CUtensorMap mw, const MlaQuery a) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) unsigned long long s_bar[2];
  __shared__ uint32_t s_tmem;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, h = blockIdx.x;
  const int N = (a.B + 15) / 16 * 16;
  const int qk = a.nope + a.rope;
  const size_t q_row = (size_t)gridDim.x * qk, stride = (size_t)a.B * q_row;
  // The trigger stands behind the wait: the attention core may then read before its own wait what the norm kernel left
  if (blockIdx.y == gridDim.y - 1) {
    const int half = a.rope / 2;
    uint32_t *cs = reinterpret_cast<uint32_t *>(smem_raw);  // [B][half] cosine and sine, before the wait
    for (int u = tid; u < a.B * half; u += kMqThreads) {
      bool in_range;
      const float ang = mh_position(a.pos, u / half, &in_range) * a.inv_freq[u % half];
      cs[u] = pack_bf16x2(cosf(ang), sinf(ang));
    }
    pdl_wait();
    pdl_trigger();
    for (int u = tid; u < a.B * half; u += kMqThreads) {  // the thread's own entries of cs
      const int tok = u / half, p = u % half;
      const size_t at = (size_t)tok * q_row + (size_t)h * qk + a.nope + 2 * p;
      float x0 = 0.f, x1 = 0.f;
      if (a.part) {
#pragma unroll 4
        for (int z = 0; z < a.nz; ++z) {
          const float2 f = *reinterpret_cast<const float2 *>(a.part + (size_t)z * stride + at);
          x0 += f.x, x1 += f.y;
        }
        x0 = round_bf16(x0), x1 = round_bf16(x1);
      } else {
        const uint32_t pair = *reinterpret_cast<const uint32_t *>(a.q + at);
        x0 = bf16lo(pair), x1 = bf16hi(pair);
      }
      uint16_t *o = a.q_full + ((size_t)tok * gridDim.x + h) * (a.kv_rank + a.rope) + a.kv_rank;
      mh_rotate(x0, x1, bf16lo(cs[u]), bf16hi(cs[u]), o + p, o + half + p);
    }
    return;
  }
  const uint32_t raw = (uint32_t)__cvta_generic_to_shared(smem_raw), sw = (raw + 1023u) & ~1023u;
  const uint32_t sx = sw + 2 * 16384;
  unsigned char *xp = smem_raw + (sx - raw);
  const uint32_t full = (uint32_t)__cvta_generic_to_shared(&s_bar[0]), done = full + 8;
  if (tid == 0) {
    tp_mbar_init(full, 1);
    tp_mbar_init(done, 1);
    tp_mbar_init_fence();
  }
  if (warp == 0) tp_tmem_alloc((uint32_t)__cvta_generic_to_shared(&s_tmem), 64);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s_tmem;
  auto boxes_of = [&](int c0) { return min(kMqCols / 64, (a.nope - c0 + 63) / 64); };
  auto fetch = [&](int c0) {  // columns past the matrix read as zeros
    const int n = boxes_of(c0);
    tp_expect_tx(full, (uint32_t)n * 16384);
    for (int j = 0; j < n; ++j) tp_load_2d(sw + (uint32_t)j * 16384, &mw, c0 + 64 * j, h * a.kv_rank + 128 * (int)blockIdx.y, full);
  };
  if (tid == 0) fetch(0);
  pdl_wait();
  pdl_trigger();
  // 16 bytes of one token's query: columns c .. c + 7 of the head
  auto query8 = [&](int tok, int c) -> uint4 {
    const size_t at = (size_t)tok * q_row + (size_t)h * qk + c;
    if (!a.part) return *reinterpret_cast<const uint4 *>(a.q + at);
    const float4 f = mh_sum4<4>(a.part + at, stride, a.nz), g = mh_sum4<4>(a.part + at + 4, stride, a.nz);
    return make_uint4(pack_bf16x2(f.x, f.y), pack_bf16x2(f.z, f.w), pack_bf16x2(g.x, g.y), pack_bf16x2(g.z, g.w));
  };
  bool failed = false;
  uint32_t turn = 0;
  for (int c0 = 0; c0 < a.nope; c0 += kMqCols, turn ^= 1) {
    const int n = boxes_of(c0);
    for (int u = tid; u < a.B * n * 8; u += kMqThreads) {
      const int tok = u / (n * 8), c = u % (n * 8), col = c0 + 8 * c;
      *reinterpret_cast<uint4 *>(xp + (c >> 3) * N * 128 + mh_swizzled(tok, c & 7)) = col < a.nope ? query8(tok, col) : make_uint4(0, 0, 0, 0);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
      if (!__all_sync(0xffffffffu, tp_wait(full, turn))) failed = true;
      else mh_mma(tmem, sw, sx, n, N, c0 > 0, done);
    }
    if (__syncthreads_or(failed || !tp_wait(done, turn))) {
      failed = true;
      break;
    }
    if (tid == 0 && c0 + kMqCols < a.nope) fetch(c0 + kMqCols);
  }
  tc_fence_after();
  if (warp < 4) {
    uint16_t *o = a.q_full + (size_t)h * (a.kv_rank + a.rope) + 128 * (int)blockIdx.y + 32 * warp + lane;
    mh_store(tmem + ((uint32_t)(32 * warp) << 16), a.B, true, o, (size_t)gridDim.x * (a.kv_rank + a.rope), failed);
  }
  if (failed && tid == 0) {
    tp_wait(full, turn);  // no copy may be in flight when the CTA leaves
    atomicExch(a.werr, 1u);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tp_tmem_free(tmem, 64);
}

constexpr int kMvThreads = 512;
constexpr int kMvRank = 512;                     // kv_rank
constexpr int kMvWBytes = (kMvRank / 64) * 16384;  // 128 rows of W_UV: 128 KB

struct MvMerge {
  int heads, G, N, quarter, j4;
  const int2 *parts;  // [G] first partial result and number of them
  const float4 *po;   // this thread's columns of partial result 0
  const float2 *ml;   // (max, sum) of partial result 0
  float *wt, *inv;    // weights of the partial results from parts[0].x on, [G] 1 / their sum
  float4 (*acc)[128];
  unsigned char *x;   // the merged rows, bf16, as the product reads them
};

__device__ __forceinline__ void mv_put(const MvMerge &m, int g, const float4 &acc) {
  const float inv = m.inv[g];
  const int c = m.j4 >> 1;  // 16-byte piece of the row; j4 & 1: its half
  *reinterpret_cast<uint2 *>(m.x + (c >> 3) * m.N * 128 + mh_swizzled(g, c & 7) + 8 * (m.j4 & 1)) =
      make_uint2(pack_bf16x2(acc.x * inv, acc.y * inv), pack_bf16x2(acc.z * inv, acc.w * inv));
}

// The merge of one head's splits over G entries.  Four groups of 128 threads, four columns a thread; a group takes every fourth
// entry, or (one or two entries) a part of an entry's splits.  Eight loads in flight per thread, of 8 / SP entries with up to SP
// splits (SP = 8: of one entry with any number); the first are asked for before the weights of the splits are known.
template <int SP>
__device__ __noinline__ void mv_merge(const MvMerge m) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int parts = SP == 8 ? (m.G == 1 ? 4 : (m.G == 2 ? 2 : 1)) : 1, part = m.quarter % parts, gstep = 4 / parts;
  const size_t split4 = (size_t)m.heads * (kMvRank / 4);
  float4 v[8];
  int2 e[8 / SP];  // the partial results of the entries in flight that this thread adds
  auto ask = [&](int g, int s) {
#pragma unroll
    for (int k = 0; k < 8 / SP; ++k) {
      e[k] = g + k * gstep < m.G ? m.parts[g + k * gstep] : make_int2(0, 0);
      if (parts > 1) {
        const int per = (e[k].y + parts - 1) / parts, n = max(0, min(e[k].y - part * per, per));
        e[k] = make_int2(e[k].x + part * per, n);
      }
#pragma unroll
      for (int i = 0; i < SP; ++i)
        if (s + i < e[k].y) v[k * SP + i] = m.po[(size_t)(e[k].x + s + i) * split4];
    }
  };
  int g = m.quarter / parts, s = 0;
  ask(g, s);
  const int base = m.parts[0].x;
#pragma unroll 1
  for (int i = warp; i < m.G; i += kMvThreads / 32) {
    const int2 p = m.parts[i];
    float M = -INFINITY, L = 0.f;
    float2 ms[5];  // up to 160 of them
#pragma unroll
    for (int k = 0; k < 5; ++k) ms[k] = lane + 32 * k < p.y ? m.ml[(size_t)(p.x + lane + 32 * k) * m.heads] : make_float2(-INFINITY, 0.f);
#pragma unroll
    for (int k = 0; k < 5; ++k) M = fmaxf(M, ms[k].x);
    M = warp_max(M);
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      const float w = ms[k].x != -INFINITY ? expf(ms[k].x - M) : 0.f;  // 0 for an empty split
      if (lane + 32 * k < p.y) m.wt[p.x - base + lane + 32 * k] = w;
      L += w * ms[k].y;
    }
    L = warp_sum(L);
    if (lane == 0) m.inv[i] = L > 0.f ? 1.0f / L : 0.f;
  }
  __syncthreads();
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
  while (g < m.G) {
    const int more = e[0].y;
#pragma unroll
    for (int k = 0; k < 8 / SP; ++k) {
#pragma unroll
      for (int i = 0; i < SP; ++i) {
        const float w = s + i < e[k].y ? m.wt[e[k].x + s + i - base] : 0.f;
        const float4 t = v[k * SP + i];
        // an empty split holds no result: its weight of zero must not meet whatever lies there
        if (w != 0.f) acc.x = fmaf(w, t.x, acc.x), acc.y = fmaf(w, t.y, acc.y), acc.z = fmaf(w, t.z, acc.z), acc.w = fmaf(w, t.w, acc.w);
      }
      if (SP < 8) {
        if (g + k * gstep < m.G) mv_put(m, g + k * gstep, acc);
        acc = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
    if (SP < 8) {
      g += (8 / SP) * gstep;
    } else if ((s += 8) >= more) {
      if (parts > 1) break;
      mv_put(m, g, acc);
      acc = make_float4(0.f, 0.f, 0.f, 0.f);
      s = 0, g += gstep;
    }
    ask(g, s);
  }
  if (parts > 1) {  // uniform
    const int i = m.quarter / parts;
    if (part) m.acc[m.quarter - i - 1][m.j4] = acc;
    __syncthreads();
    if (part == 0) {
      for (int p = 1; p < parts; ++p) {
        const float4 t = m.acc[m.quarter + p - i - 1][m.j4];
        acc.x += t.x, acc.y += t.y, acc.z += t.z, acc.w += t.w;
      }
      mv_put(m, i, acc);
    }
  }
}

// grid = (heads, ceil(v_head / 128), groups of a.group entries), 512 threads.  Merges the context splits of one head (weights
// exp(m_s - M), as mla_merge_kernel), rounds to bf16 and multiplies by the head's W_UV (:826 with V = W_UV c).
__global__ void __launch_bounds__(kMvThreads, 1) mla_value_kernel(const __grid_constant__ CUtensorMap mw, const MlaValue a) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) unsigned long long s_bar[2];
  __shared__ uint32_t s_tmem;
  __shared__ float s_inv[32];
  __shared__ float4 s_acc[3][128];
  __shared__ int2 s_parts[32];
  __shared__ int s_most;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, h = blockIdx.x, heads = gridDim.x;
  const int b0 = (int)blockIdx.z * a.group, G = min(a.group, a.B - b0), N = a.group <= 16 ? 16 : 32;
  pdl_trigger();
  const uint32_t raw = (uint32_t)__cvta_generic_to_shared(smem_raw), sw = (raw + 1023u) & ~1023u;
  const uint32_t sx = sw + kMvWBytes;
  unsigned char *xp = smem_raw + (sx - raw);
  float *wt = reinterpret_cast<float *>(xp + (kMvRank / 64) * N * 128);
  const uint32_t full = (uint32_t)__cvta_generic_to_shared(&s_bar[0]), done = full + 8;
  if (tid == 0) {
    tp_mbar_init(full, 1);
    tp_mbar_init(done, 1);
    tp_mbar_init_fence();
    tp_expect_tx(full, kMvWBytes);
    for (int j = 0; j < kMvRank / 64; ++j)
      tp_load_2d(sw + (uint32_t)j * 16384, &mw, 64 * j, h * (a.nope + a.v_head) + a.nope + 128 * (int)blockIdx.y, full);
  }
  if (warp == 0) tp_tmem_alloc((uint32_t)__cvta_generic_to_shared(&s_tmem), 32);
  if (warp == 1) {  // what the attention core leaves: known before the core began (it triggers behind its own wait)
    int2 p = make_int2((b0 + lane) * a.splits, a.splits);
    if (!a.splits && lane < G) p = a.parts[b0 + lane];
    if (lane < G) s_parts[lane] = p;
    const int most = __reduce_max_sync(0xffffffffu, lane < G ? p.y : 0);
    if (lane == 0) s_most = most;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_wait();
  MvMerge m;
  m.heads = heads, m.G = G, m.N = N, m.quarter = tid >> 7, m.j4 = tid & 127;
  m.parts = s_parts;
  m.po = reinterpret_cast<const float4 *>(a.part_o) + (size_t)h * (kMvRank / 4) + m.j4;
  m.ml = reinterpret_cast<const float2 *>(a.part_ml) + h;
  m.wt = wt, m.inv = s_inv, m.acc = s_acc, m.x = xp;
  // one instance per size of the lists, so that a launch fetches little code
  if (G <= 2 || s_most > 4) mv_merge<8>(m);
  else if (s_most > 2) mv_merge<4>(m);
  else mv_merge<2>(m);
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncthreads();
  bool failed = false;
  if (warp == 0) {
    if (!__all_sync(0xffffffffu, tp_wait(full, 0))) failed = true;
    else mh_mma(s_tmem, sw, sx, kMvRank / 64, N, false, done);
  }
  failed = __syncthreads_or(failed || !tp_wait(done, 0));
  tc_fence_after();
  const uint32_t tmem = s_tmem;
  if (warp < 4) {
    const int r = 128 * (int)blockIdx.y + 32 * warp + lane;
    mh_store(tmem + ((uint32_t)(32 * warp) << 16), G, r < a.v_head, a.out + ((size_t)b0 * heads + h) * a.v_head + r, (size_t)heads * a.v_head, failed);
  }
  if (failed && tid == 0) {
    tp_wait(full, 0);  // no copy may be in flight when the CTA leaves
    atomicExch(a.werr, 1u);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tp_tmem_free(tmem, 32);
}

int launch_mla_norm(const MlaNorm &a, int B, cudaStream_t stream) {
  const int lat = a.kv_rank + a.rope;
  BLOK_REQUIRE(lat <= kMnKept, BLOK_ERR_SHAPE, "mla norm: cache rows of %d values (at most %d)", lat, kMnKept);
  const size_t smem = (size_t)std::min(std::max(a.q_rank, lat), kMnKept) * sizeof(float);
  return launch_pdl("mla_norm_kernel", mla_norm_kernel, dim3(2, B), kMnThreads, smem, stream, a);
}

int launch_mla_query(const uint16_t *wuk_t, int heads, const MlaQuery &a, cudaStream_t stream) {
  CUtensorMap mw;
  if (int rc = gemm_operand_map(wuk_t, (long)heads * a.kv_rank, a.nope, a.nope, 128, &mw)) return rc;
  const int smem = 2 * 16384 + 2 * ((a.B + 15) / 16 * 16) * 128 + 1024;
  if (int rc = allow_smem(mla_query_kernel, smem)) return rc;
  return launch_pdl("mla_query_kernel", mla_query_kernel, dim3(heads, a.kv_rank / 128 + 1), kMqThreads, (size_t)smem, stream, mw, a);
}

int launch_mla_value(const uint16_t *kv_b, int heads, MlaValue a, cudaStream_t stream) {
  CUtensorMap mw;
  if (int rc = gemm_operand_map(kv_b, (long)heads * (a.nope + a.v_head), kMvRank, kMvRank, 128, &mw)) return rc;
  // two groups of entries from two on: 128 CTAs, each with its half of the partial results to add
  const int groups = a.B > 1 ? 2 : 1;
  a.group = (a.B + groups - 1) / groups;
  const int N = a.group <= 16 ? 16 : 32;
  // weights of the partial results: in the planned form those of consecutive entries are consecutive, fewer than CTAs + entries
  const int smem = kMvWBytes + (kMvRank / 64) * N * 128 + (a.splits ? a.group * a.splits : a.ctas + a.B) * (int)sizeof(float) + 1024;
  if (int rc = allow_smem(mla_value_kernel, smem)) return rc;
  return launch_pdl("mla_value_kernel", mla_value_kernel, dim3(heads, (a.v_head + 127) / 128, groups), kMvThreads, (size_t)smem, stream, mw, a);
}

}  // namespace blok
