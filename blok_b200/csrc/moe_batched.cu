// Batched routed-MoE layer: tokens are grouped by expert, every touched expert's
// INT4 weights are streamed once through the weight-streaming GEMM, and the
// per-assignment outputs are combined per token.  This is the per-token arithmetic
// of src/kimi_exec.cu:836-877 applied to T tokens; the reference itself only ever
// runs one token (:885-890).
#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "moe_layer.h"
#include "router_topk.cuh"
#include "wgemm.h"

namespace blok {

int launch_router_topk(const float *logits, const float *bias, int T, int experts, int topk, float routed_scale,
                       uint16_t *ids, float *wts, int *local_ids, int expert_base, cudaStream_t stream);

// The counting sort of the (token, slot) assignments by expert, stable, and the tile table (tiles of 64 sorted positions of one
// expert), in one launch.  A block places kMbChunk assignments: it counts all of them (and those before its own) by expert in shared
// memory, scans the counts, and a pair of threads counts the equals before an assignment inside the block's own.  Every block does the
// counting again, which costs less than a launch that it would have to wait for.  ids outside [0, n_local) belong to none.  Latency is all
// there is to it: one block that counted and, in a launch behind it, a warp per expert that walked all assignments took 15 us over
// 4,136 and 39 over 16,384 assignments (the gap between them with it), this one 8.4 and 9.9.  The counting is quadratic in all, but over
// 524,280 assignments of which nearly all belong to no expert a call takes 292 us where it took 1,321 with the two launches.
// Dynamic shared memory: [n_local] counts, [n_local] counts before the block's own, [n_local] offsets.
constexpr int kMbChunk = 512;
__global__ void __launch_bounds__(1024) mb_sort_kernel(const int *__restrict__ expert_local, const int *__restrict__ x_index, int row_div, int N,
                                                       int n_local, int *__restrict__ tile_expert, int *__restrict__ tile_start,
                                                       int *__restrict__ tile_count, int *__restrict__ num_tiles, int max_tiles,
                                                       int *__restrict__ sorted_assign, int *__restrict__ sorted_row) {
  extern __shared__ int s_dyn[];
  __shared__ __align__(16) int s_own[kMbChunk];
  __shared__ int s_rank[kMbChunk], s_warp[2][32];
  int *s_counts = s_dyn, *s_before = s_dyn + n_local, *s_offsets = s_before + n_local;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, start = blockIdx.x * kMbChunk;
  // the thread's own assignment, if any: both of its words are on their way before the first barrier
  const int at = start + tid;
  const bool has = tid < kMbChunk && at < N;
  const int own = has ? expert_local[at] : -1, row = has ? (x_index ? x_index[at] : at / row_div) : 0;
  const bool placed = own >= 0 && own < n_local;
  for (int e = tid; e < n_local; e += 1024) s_counts[e] = s_before[e] = 0;
  if (tid < kMbChunk) s_own[tid] = own, s_rank[tid] = 0;
  __syncthreads();
  constexpr int kFly = 8;
  if (gridDim.x == 1 && placed) atomicAdd(s_counts + own, 1);
  for (int a0 = tid; gridDim.x > 1 && a0 < N; a0 += kFly * 1024) {
    int e[kFly];
#pragma unroll
    for (int i = 0; i < kFly; ++i) e[i] = a0 + 1024 * i < N ? expert_local[a0 + 1024 * i] : -1;
#pragma unroll
    for (int i = 0; i < kFly; ++i) {
      if (e[i] < 0 || e[i] >= n_local) continue;
      atomicAdd(s_counts + e[i], 1);
      if (a0 + 1024 * i < start) atomicAdd(s_before + e[i], 1);
    }
  }
  {  // two threads an assignment: the equals among the first and the second half of those before it
    const int i = tid & (kMbChunk - 1), e = s_own[i], mid = (i / 2 + 3) / 4 * 4, j0 = tid < kMbChunk ? 0 : mid;
    const int j1 = e < 0 || e >= n_local ? 0 : (tid < kMbChunk ? min(mid, i) : i);
    int n = 0;
#pragma unroll 4
    for (int j = j0; j < j1; j += 4) {
      const int4 v = *reinterpret_cast<const int4 *>(s_own + j);
      n += (v.x == e) + (j + 1 < j1 && v.y == e) + (j + 2 < j1 && v.z == e) + (j + 3 < j1 && v.w == e);
    }
    if (n) atomicAdd(s_rank + i, n);
  }
  __syncthreads();
  // an expert per thread (n_local <= 1024): exclusive scans of the counts and of the tiles, in expert order
  const int c = tid < n_local ? s_counts[tid] : 0, nt = (c + kWgTileTokens - 1) / kWgTileTokens;
  int off = c, first = nt;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, off, d), v = __shfl_up_sync(0xffffffffu, first, d);
    if (lane >= d) off += u, first += v;
  }
  if (lane == 31) s_warp[0][warp] = off, s_warp[1][warp] = first;
  __syncthreads();
  off += __reduce_add_sync(0xffffffffu, lane < warp ? s_warp[0][lane] : 0) - c;
  first += __reduce_add_sync(0xffffffffu, lane < warp ? s_warp[1][lane] : 0) - nt;
  if (tid < n_local) {
    s_offsets[tid] = off + s_before[tid];
    if (blockIdx.x == 0) {
      for (int k = 0; k < nt && first + k < max_tiles; ++k) {
        tile_expert[first + k] = tid;
        tile_start[first + k] = off + k * kWgTileTokens;
        tile_count[first + k] = min(kWgTileTokens, c - k * kWgTileTokens);
      }
    }
  }
  if (blockIdx.x == 0 && tid == 1023) *num_tiles = min(first + nt, max_tiles);
  __syncthreads();
  if (placed) {
    const int p = s_offsets[own] + s_rank[tid];
    sorted_assign[p] = at;
    sorted_row[p] = row;
  }
}

// What stands between the first products of a layer of up to kWgStreamTokens tokens and the rest of it, in one launch: block 0
// routes (the sums of the router's K split added in order, top-k, a warp per token), sorts the assignments by expert and writes
// the tile table; the other blocks make the shared expert's gated vector from its sums.  Each of these kernels by itself is
// a few microseconds of latency, most of it the fetch of its instructions (the weights that stream between two calls leave
// nothing of them in L2): reduce, top-k, plan and reduce took 22 us over 6 tokens, this one 8.7.  With the front launch and the
// combination that adds the second half's sums, layers of 6 and 2 tokens (7168 x 2048, 384 experts) 285 -> 257, 151 -> 121 us, of 3, 40
// and 64 (2048 x 1024, 128 experts) 76 -> 61, 152 -> 127, 157 -> 139; of 1, 5 and 16 (2048 x 512, 512 experts) 73 -> 45, 94 -> 67, 124 -> 97.  A pass over stale sums before the wait, to have the
// instructions there, is slower (64 tokens 139 -> 148).
struct MbRoute {
  const float *part;  // [nz][T][ld]: the shared expert's gate columns, its up columns, the router's
  int nz, ld, T, experts, topk, shared;
  const float *bias;
  float scale;
  uint16_t *ids;
  float *wts;
  int *local_ids, *tile_expert, *tile_start, *tile_count, *num_tiles, *sorted_assign, *sorted_row;
  int max_tiles;
  uint16_t *mid;  // [T][shared]
};
// Most experts: the scores of 64 tokens stay in shared memory (512 experts 137 KB, 1,024 would be 268), one instance per width of a lane's
// share of them.
constexpr int kMbRouteExperts = 512;

template <int N>
__global__ void __launch_bounds__(1024) mb_route_kernel(const MbRoute a) {
  extern __shared__ int s_dyn[];
  __shared__ int s_warp[2][32];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const size_t stride = (size_t)a.T * a.ld;
  pdl_trigger();
  if (blockIdx.x > 0) {
    const int i = ((int)(blockIdx.x - 1) * 1024 + tid) * 4;  // four columns of one token
    pdl_wait();
    if (i >= a.T * a.shared) return;
    const int t = i / a.shared, c = i - t * a.shared;
    const float *p = a.part + (size_t)t * a.ld + c;
    float g[4] = {0.f, 0.f, 0.f, 0.f}, u[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (int z = 0; z < a.nz; ++z, p += stride) {
      const float4 v = *reinterpret_cast<const float4 *>(p), w = *reinterpret_cast<const float4 *>(p + a.shared);
      g[0] += v.x, g[1] += v.y, g[2] += v.z, g[3] += v.w;
      u[0] += w.x, u[1] += w.y, u[2] += w.z, u[3] += w.w;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float gv = round_bf16(g[k]);
      g[k] = round_bf16(gv / (1.0f + expf(-gv))) * round_bf16(u[k]);
    }
    *reinterpret_cast<uint2 *>(a.mid + i) = make_uint2(pack_bf16x2(g[0], g[1]), pack_bf16x2(g[2], g[3]));
    return;
  }
  const int n = a.T * a.topk, n4 = (n + 3) / 4 * 4;
  int *s_local = s_dyn, *s_counts = s_dyn + n4, *s_offsets = s_counts + a.experts;
  float *s_bias = reinterpret_cast<float *>(s_offsets + a.experts), *score = s_bias + a.experts;  // [T][experts]
  for (int e = tid; e < a.experts; e += 1024) s_counts[e] = 0, s_bias[e] = a.bias[e];
  if (tid < n4 - n) s_local[n + tid] = -1;
  __syncthreads();
  pdl_wait();
  const float *router = a.part + a.ld - a.experts;
  for (int i = 4 * tid; i < a.T * a.experts; i += 4096) {  // four experts of one token
    const int tok = i / a.experts, e = i - tok * a.experts;
    const float *p = router + (size_t)tok * a.ld + e;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
    for (int z = 0; z < a.nz; z += 4) {
      float4 f[4];
#pragma unroll
      for (int k = 0; k < 4; ++k, p += stride)
        if (z + k < a.nz) f[k] = *reinterpret_cast<const float4 *>(p);
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (z + k < a.nz) v.x += f[k].x, v.y += f[k].y, v.z += f[k].z, v.w += f[k].w;
    }
    *reinterpret_cast<float4 *>(score + i) = make_float4(1.0f / (1.0f + expf(-v.x)), 1.0f / (1.0f + expf(-v.y)), 1.0f / (1.0f + expf(-v.z)), 1.0f / (1.0f + expf(-v.w)));
  }
  __syncthreads();
#pragma unroll 1
  for (int tok = warp; tok < a.T; tok += 32) {
    float sel[N];
#pragma unroll
    for (int j = 0; j < N; ++j) {
      const int e = 32 * j + lane;
      sel[j] = e < a.experts ? score[tok * a.experts + e] + s_bias[e] : -INFINITY;
    }
    int my_id;
    float my_w;
    warp_topk(score + tok * a.experts, sel, a.topk, a.scale, lane, my_id, my_w);
    if (lane < a.topk) {
      const int at = tok * a.topk + lane;
      a.ids[at] = (uint16_t)my_id;
      a.local_ids[at] = my_id;
      a.wts[at] = my_w;
      s_local[at] = my_id;
      atomicAdd(s_counts + my_id, 1);
    }
  }
  __syncthreads();
  // an expert per thread: exclusive scans of the counts and of the tiles, in expert order
  const int c = tid < a.experts ? s_counts[tid] : 0, nt = (c + kWgTileTokens - 1) / kWgTileTokens;
  int off = c, first = nt;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, off, d), v = __shfl_up_sync(0xffffffffu, first, d);
    if (lane >= d) off += u, first += v;
  }
  if (lane == 31) s_warp[0][warp] = off, s_warp[1][warp] = first;
  __syncthreads();
  const int before = __reduce_add_sync(0xffffffffu, lane < warp ? s_warp[0][lane] : 0), tiles = __reduce_add_sync(0xffffffffu, lane < warp ? s_warp[1][lane] : 0);
  off += before - c, first += tiles - nt;
  if (tid < a.experts) {
    s_offsets[tid] = off;
    for (int k = 0; k < nt && first + k < a.max_tiles; ++k) {
      a.tile_expert[first + k] = tid;
      a.tile_start[first + k] = off + k * kWgTileTokens;
      a.tile_count[first + k] = min(kWgTileTokens, c - k * kWgTileTokens);
    }
    if (tid == a.experts - 1) *a.num_tiles = min(first + nt, a.max_tiles);
  }
  __syncthreads();
  // an assignment per thread: its place among its expert's is the number of them before it
  for (int i = tid; i < n; i += 1024) {
    const int e = s_local[i];
    int rank = 0;
#pragma unroll 4
    for (int j = 0; j < i; j += 4) {
      const int4 v = *reinterpret_cast<const int4 *>(s_local + j);
      rank += (v.x == e) + (j + 1 < i && v.y == e) + (j + 2 < i && v.z == e) + (j + 3 < i && v.w == e);
    }
    a.sorted_assign[s_offsets[e] + rank] = i;
    a.sorted_row[s_offsets[e] + rank] = i / a.topk;
  }
}

static int launch_mb_route(const MbRoute &a, cudaStream_t stream) {
  const size_t smem = (size_t)((a.T * a.topk + 3) / 4 * 4 + (3 + a.T) * a.experts) * sizeof(int);
  const int blocks = 1 + (a.T * a.shared / 4 + 1023) / 1024;
  auto kernel = a.experts <= 128 ? mb_route_kernel<4> : (a.experts <= 384 ? mb_route_kernel<12> : mb_route_kernel<16>);
  if (int rc = allow_smem(kernel, smem)) return rc;
  return launch_pdl("mb_route_kernel", kernel, blocks, 1024, smem, stream, a);
}

// out[t, c] = bf16( bf16(sum_k w[t,k] * y[t*topk + k, c]) + shared[t, c] ), slot order as :868-871, :684.
// The shared expert's output is bf16, or (sums) the nz fp32 parts of its K split, added in order and rounded here.
// V columns per thread: 8 (16-byte loads, eight slots in flight: bound by HBM, 264 MB at 2,048 tokens), or 2 where the rows'
// length or alignment does not allow that.
template <int V>
__global__ void mb_combine_kernel(const uint16_t *y, const float *wts, const uint16_t *shared, const float *sums, int nz, int hidden, int topk,
                                  uint16_t *out) {
  pdl_wait();
  pdl_trigger();
  using Words = typename std::conditional<V == 8, uint4, uint32_t>::type;
  const int t = blockIdx.y;
  const int c = (blockIdx.x * blockDim.x + threadIdx.x) * V;
  if (c >= hidden) return;
  float o[V];
#pragma unroll
  for (int i = 0; i < V; ++i) o[i] = 0.f;
  for (int k0 = 0; k0 < topk; k0 += 8) {
    union {
      Words v;
      uint32_t w[V / 2];
    } q[8];
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (k0 + k < topk) q[k].v = *reinterpret_cast<const Words *>(y + ((size_t)t * topk + k0 + k) * hidden + c);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (k0 + k < topk) {
        const float w = wts[(size_t)t * topk + k0 + k];
#pragma unroll
        for (int i = 0; i < V / 2; ++i) {
          o[2 * i] = fmaf(bf16lo(q[k].w[i]), w, o[2 * i]);
          o[2 * i + 1] = fmaf(bf16hi(q[k].w[i]), w, o[2 * i + 1]);
        }
      }
    }
  }
  union {
    Words v;
    uint32_t w[V / 2];
  } s, r;
  if (sums) {
    float f[V];
#pragma unroll
    for (int i = 0; i < V; ++i) f[i] = 0.f;
    const size_t part = (size_t)gridDim.y * hidden;
    const float *p = sums + (size_t)t * hidden + c;
#pragma unroll 4
    for (int z = 0; z < nz; ++z, p += part) {
#pragma unroll
      for (int i = 0; i < V; i += 2) {
        const float2 v = *reinterpret_cast<const float2 *>(p + i);
        f[i] += v.x, f[i + 1] += v.y;
      }
    }
#pragma unroll
    for (int i = 0; i < V / 2; ++i) s.w[i] = pack_bf16x2(f[2 * i], f[2 * i + 1]);
  } else if (shared) {
    s.v = *reinterpret_cast<const Words *>(shared + (size_t)t * hidden + c);
  }
#pragma unroll
  for (int i = 0; i < V / 2; ++i) {
    float lo = round_bf16(o[2 * i]), hi = round_bf16(o[2 * i + 1]);
    if (shared || sums) {
      lo = round_bf16(lo + bf16lo(s.w[i]));
      hi = round_bf16(hi + bf16hi(s.w[i]));
    }
    r.w[i] = pack_bf16x2(lo, hi);
  }
  *reinterpret_cast<Words *>(out + (size_t)t * hidden + c) = r.v;
}

static int launch_combine(bool overlap, const uint16_t *y, const float *wts, const uint16_t *shared, const float *sums, int nz, int T, int topk, int hidden,
                          uint16_t *out, cudaStream_t stream) {
  const uintptr_t at = reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(shared) | reinterpret_cast<uintptr_t>(out);
  if (hidden % 8 == 0 && at % 16 == 0)
    return launch_pdl_if(overlap, "mb_combine_kernel", mb_combine_kernel<8>, dim3((hidden / 8 + 127) / 128, T), 128, 0, stream, y, wts, shared, sums, nz, hidden, topk, out);
  return launch_pdl_if(overlap, "mb_combine_kernel", mb_combine_kernel<2>, dim3((hidden / 2 + 255) / 256, T), 256, 0, stream, y, wts, shared, sums, nz, hidden, topk, out);
}

// The front launch and the routing kernel read the operands 16 bytes at a time.
static bool wgemm_front_aligned(const blok_moe_weights &w, const uint16_t *x) {
  uintptr_t at = reinterpret_cast<uintptr_t>(w.router_w) | reinterpret_cast<uintptr_t>(x);
  if (w.shared_inter > 0)
    at |= reinterpret_cast<uintptr_t>(w.shared_gate) | reinterpret_cast<uintptr_t>(w.shared_up) | reinterpret_cast<uintptr_t>(w.shared_down);
  return at % 16 == 0;
}

static size_t al(size_t v) { return (v + 255) / 256 * 256; }

int batched_alloc(blok_moe_layer *L) {
  const blok_moe_weights &w = L->w;
  const size_t T = L->max_tokens, N = T * w.topk;
  const int nl = std::max(w.experts_local, 1);
  L->b_max_assign = (int)N;
  L->b_max_tiles = (int)((N + kWgTileTokens - 1) / kWgTileTokens) + nl;
  size_t off = 0;
  auto take = [&](size_t b) { size_t at = off; off = al(off + b); return at; };
  size_t o_counts = take((nl + 1) * 4), o_offsets = take((nl + 1) * 4), o_sa = take(N * 4), o_sr = take(N * 4);
  size_t o_te = take(L->b_max_tiles * 4), o_ts = take(L->b_max_tiles * 4), o_tc = take(L->b_max_tiles * 4), o_nt = take(4);
  size_t o_mid = take(N * (size_t)w.inter * 2), o_y = take(N * (size_t)w.hidden * 2);
  size_t o_smid = take(T * (size_t)std::max(w.shared_inter, 8) * 2), o_sout = take(T * (size_t)w.hidden * 2);
  // K-split partial sums of the bf16 products over few tiles of tokens (router, shared gate/up, shared down)
  L->b_splitk_bytes = std::max(wgemm_splitk_bytes(WG_BF16_PLAIN, w.hidden, w.experts, (int)T),
                               std::max(wgemm_splitk_bytes(WG_BF16_SWIGLU, w.hidden, std::max(w.shared_inter, 8), (int)T),
                                        wgemm_splitk_bytes(WG_BF16_PLAIN, std::max(w.shared_inter, 8), w.hidden, (int)T)));
  L->b_front_split = wgemm_stream_pair_split(WG_BF16_SWIGLU, w.hidden, std::max(w.shared_inter, 8), w.experts);
  // The launches over up to kWgStreamTokens tokens that leave their sums to another kernel want room for one part also where K is not split.
  const size_t few = std::min<size_t>(T, kWgStreamTokens) * sizeof(float);
  L->b_splitk_bytes = std::max({L->b_splitk_bytes, L->b_front_split * few * (2 * w.shared_inter + w.experts), w.shared_inter > 0 ? few * w.hidden : 0});
  size_t o_sk = take(std::max(L->b_splitk_bytes, (size_t)16)), o_err = take(4);
  BLOK_CUDA(cudaMalloc(&L->bws, off));
  unsigned char *b = static_cast<unsigned char *>(L->bws);
  L->b_counts = (int *)(b + o_counts); L->b_offsets = (int *)(b + o_offsets);
  L->b_sorted_assign = (int *)(b + o_sa); L->b_sorted_row = (int *)(b + o_sr);
  L->b_tile_expert = (int *)(b + o_te); L->b_tile_start = (int *)(b + o_ts); L->b_tile_count = (int *)(b + o_tc);
  L->b_num_tiles = (int *)(b + o_nt);
  L->b_mid = (uint16_t *)(b + o_mid); L->b_y = (uint16_t *)(b + o_y);
  L->b_smid = (uint16_t *)(b + o_smid); L->b_sout = (uint16_t *)(b + o_sout);
  L->b_splitk = (float *)(b + o_sk);
  L->b_err = (unsigned *)(b + o_err);
  BLOK_CUDA(cudaMemset(L->b_err, 0, sizeof(unsigned)));
  return BLOK_OK;
}

// The products behind the plan (sorted order and tile table in the handle).
static int planned_experts(blok_moe_layer *L, const uint16_t *x, int N, uint16_t *y, bool overlap, cudaStream_t stream) {
  const blok_moe_weights &w = L->w;
  const int nl = w.experts_local;
  WgArgs g;
  g.w_a = w.gate_w; g.w_b = w.up_w; g.s_a = w.gate_s; g.s_b = w.up_s; g.expert_stride_rows = w.inter;
  g.x = x; g.x_index = L->b_sorted_row; g.K = w.hidden; g.R = w.inter; g.out_bf16 = L->b_mid; g.out_f32 = nullptr;
  g.tile_expert = L->b_tile_expert; g.tile_start = L->b_tile_start; g.tile_count = L->b_tile_count;
  g.num_tiles = L->b_num_tiles; g.out_index = nullptr; g.n_rows = N; g.err = L->b_err; g.overlap = overlap;
  const int max_tiles = std::min(L->b_max_tiles, (N + kWgTileTokens - 1) / kWgTileTokens + nl);
  WgArgs d = g;
  d.w_a = w.down_w; d.w_b = nullptr; d.s_a = w.down_s; d.s_b = nullptr; d.expert_stride_rows = w.hidden;
  d.x = L->b_mid; d.x_index = nullptr; d.K = w.inter; d.R = w.hidden; d.out_bf16 = y; d.out_index = L->b_sorted_assign;
  return launch_wgemm_experts(g, d, L->b_y, N, max_tiles, stream);  // b_y is not written before the down projection
}

// y[a, :] = bf16(expert_{e_a}(x[row_a, :])) for N assignments; row_a = x_index[a], or a / row_div.
int grouped_experts(blok_moe_layer *L, const uint16_t *x, const int *x_index, int row_div, const int *expert_local, int N,
                    uint16_t *y, cudaStream_t stream) {
  const int nl = L->w.experts_local;
  mb_sort_kernel<<<(N + kMbChunk - 1) / kMbChunk, 1024, (size_t)3 * nl * sizeof(int), stream>>>(
      expert_local, x_index, row_div, N, nl, L->b_tile_expert, L->b_tile_start, L->b_tile_count, L->b_num_tiles, L->b_max_tiles, L->b_sorted_assign,
      L->b_sorted_row);
  if (int rc = launch_status("mb_sort_kernel")) return rc;
  return planned_experts(L, x, N, y, false, stream);
}

}  // namespace blok

using namespace blok;

extern "C" int blok_moe_experts_grouped(blok_moe_layer_t *L, const blok_bf16_t *x, const int *x_index,
                                        const int *expert_local, int N, blok_bf16_t *y, blok_stream_t stream) {
  BLOK_REQUIRE(L, BLOK_ERR_ARG, "blok_moe_experts_grouped: null layer");
  if (N == 0) return BLOK_OK;  // empty inputs may carry null pointers
  BLOK_REQUIRE(x && expert_local && y, BLOK_ERR_ARG, "blok_moe_experts_grouped: null pointer");
  BLOK_REQUIRE(L->bws, BLOK_ERR_STATE, "blok_moe_experts_grouped: the layer was created with max_tokens = 1");
  BLOK_REQUIRE(N >= 0 && N <= L->b_max_assign, BLOK_ERR_SHAPE, "blok_moe_experts_grouped: N=%d exceeds capacity %d", N,
               L->b_max_assign);
  BLOK_REQUIRE(L->w.hidden % 512 == 0 && L->w.inter % 512 == 0, BLOK_ERR_SHAPE,
               "blok_moe_experts_grouped: hidden and inter must be multiples of 512");
  if (N == 0) return BLOK_OK;
  return grouped_experts(L, x, x_index, 1, expert_local, N, y, (cudaStream_t)stream);
}

extern "C" int blok_moe_batched(blok_moe_layer_t *L, const blok_bf16_t *x, int T, blok_bf16_t *y, uint16_t *ids_out,
                                float *wts_out, blok_stream_t stream_) {
  BLOK_REQUIRE(L && x && y, BLOK_ERR_ARG, "blok_moe_batched: null pointer");
  const blok_moe_weights &w = L->w;
  BLOK_REQUIRE(L->bws, BLOK_ERR_STATE, "blok_moe_batched: the layer was created with max_tokens = 1");
  BLOK_REQUIRE(T >= 0 && T <= L->max_tokens, BLOK_ERR_SHAPE, "blok_moe_batched: T=%d exceeds max_tokens %d", T, L->max_tokens);
  BLOK_REQUIRE(w.experts_local == w.experts && w.expert_base == 0, BLOK_ERR_ROUTE,
               "blok_moe_batched: needs every expert local; use blok_router + blok_moe_experts_grouped under expert parallelism");
  BLOK_REQUIRE(w.hidden % 512 == 0 && w.inter % 512 == 0 && w.experts % 128 == 0 && w.shared_inter % 512 == 0,
               BLOK_ERR_SHAPE, "blok_moe_batched: hidden/inter/shared_inter must be multiples of 512 and experts of 128");
  if (T == 0) return BLOK_OK;
  cudaStream_t stream = (cudaStream_t)stream_;
  const int N = T * w.topk;
  int rc;
  if (T <= kWgStreamTokens && !wgemm_forced_impl() && w.experts <= kMbRouteExperts && wgemm_front_aligned(w, x)) {
    // the router and the shared expert's first half in one launch, whose sums the routing kernel takes; the shared expert's second
    // half; the grouped experts; the combination, which adds the sums of the second half
    WgArgs f = {};
    f.identity_tiles = 1; f.n_rows = T; f.x = x; f.K = w.hidden; f.keep_sums = true;
    f.splitk_ws = L->b_splitk; f.splitk_bytes = L->b_splitk_bytes; f.err = L->b_err; f.max_splits = L->b_front_split;
    MbRoute m = {};
    if (w.shared_inter > 0) {
      f.w_a = w.shared_gate; f.w_b = w.shared_up; f.R = w.shared_inter; f.w_2 = w.router_w; f.R2 = w.experts;
    } else {
      f.w_a = w.router_w; f.R = w.experts;
    }
    if ((rc = launch_wgemm_stream(w.shared_inter > 0 ? WG_BF16_SWIGLU : WG_BF16_PLAIN, f, &m.nz, stream))) return rc;
    m.part = L->b_splitk; m.ld = 2 * w.shared_inter + w.experts; m.T = T; m.experts = w.experts; m.topk = w.topk; m.shared = w.shared_inter;
    m.bias = w.router_bias; m.scale = w.routed_scale; m.ids = L->ids; m.wts = L->wts; m.local_ids = L->local_ids;
    m.tile_expert = L->b_tile_expert; m.tile_start = L->b_tile_start; m.tile_count = L->b_tile_count; m.num_tiles = L->b_num_tiles;
    m.sorted_assign = L->b_sorted_assign; m.sorted_row = L->b_sorted_row; m.max_tiles = L->b_max_tiles; m.mid = L->b_smid;
    if ((rc = launch_mb_route(m, stream))) return rc;
    int nz = 0;
    if (w.shared_inter > 0) {
      WgArgs d = f;
      d.w_a = w.shared_down; d.w_b = nullptr; d.w_2 = nullptr; d.R2 = 0; d.x = L->b_smid; d.K = w.shared_inter; d.R = w.hidden;
      d.max_splits = 0; d.weights_early = true;
      if ((rc = launch_wgemm_stream(WG_BF16_PLAIN, d, &nz, stream))) return rc;
    }
    if ((rc = planned_experts(L, x, N, L->b_y, true, stream))) return rc;
    if ((rc = launch_combine(true, L->b_y, L->wts, nullptr, nz ? L->b_splitk : nullptr, nz, T, w.topk, w.hidden, y, stream))) return rc;
    if (ids_out) BLOK_CUDA(cudaMemcpyAsync(ids_out, L->ids, (size_t)N * sizeof(uint16_t), cudaMemcpyDeviceToDevice, stream));
    if (wts_out) BLOK_CUDA(cudaMemcpyAsync(wts_out, L->wts, (size_t)N * sizeof(float), cudaMemcpyDeviceToDevice, stream));
    return BLOK_OK;
  }
  // router: logits through the weight-streaming GEMM (fp32, unrounded, :297), then the top-k kernel
  const int tt = (T + kWgTileTokens - 1) / kWgTileTokens;
  WgArgs r;
  r.w_a = w.router_w; r.w_b = nullptr; r.s_a = r.s_b = nullptr; r.expert_stride_rows = 0; r.x = x; r.x_index = nullptr;
  r.K = w.hidden; r.R = w.experts; r.out_bf16 = nullptr; r.out_f32 = L->logits;
  r.tile_expert = r.tile_start = r.tile_count = r.num_tiles = nullptr;
  r.out_index = nullptr; r.n_rows = T; r.identity_tiles = 1;
  r.splitk_ws = L->b_splitk; r.splitk_bytes = L->b_splitk_bytes; r.err = L->b_err;
  r.max_splits = L->b_front_split;  // the expert-parallel layer's: the two agree bit for bit
  if ((rc = launch_wgemm(WG_BF16_PLAIN, r, tt, stream))) return rc;
  if ((rc = launch_router_topk(L->logits, w.router_bias, T, w.experts, w.topk, w.routed_scale, L->ids, L->wts, L->local_ids,
                               w.expert_base, stream)))
    return rc;
  if ((rc = grouped_experts(L, x, nullptr, w.topk, L->local_ids, N, L->b_y, stream))) return rc;
  const uint16_t *shared = nullptr;
  if (w.shared_inter > 0) {
    WgArgs s = r;
    s.w_a = w.shared_gate; s.w_b = w.shared_up; s.R = w.shared_inter; s.out_bf16 = L->b_smid; s.out_f32 = nullptr;
    s.weights_early = true;  // the router's launch and others are in between
    if ((rc = launch_wgemm(WG_BF16_SWIGLU, s, tt, stream))) return rc;
    WgArgs d = r;
    d.w_a = w.shared_down; d.x = L->b_smid; d.K = w.shared_inter; d.R = w.hidden; d.out_bf16 = L->b_sout; d.out_f32 = nullptr;
    d.max_splits = 0;
    d.weights_early = true;
    if ((rc = launch_wgemm(WG_BF16_PLAIN, d, tt, stream))) return rc;
    shared = L->b_sout;
  }
  if ((rc = launch_combine(false, L->b_y, L->wts, shared, nullptr, 0, T, w.topk, w.hidden, y, stream))) return rc;
  if (ids_out) BLOK_CUDA(cudaMemcpyAsync(ids_out, L->ids, (size_t)N * sizeof(uint16_t), cudaMemcpyDeviceToDevice, stream));
  if (wts_out) BLOK_CUDA(cudaMemcpyAsync(wts_out, L->wts, (size_t)N * sizeof(float), cudaMemcpyDeviceToDevice, stream));
  return BLOK_OK;
}

extern "C" int blok_moe_shared(blok_moe_layer_t *L, const blok_bf16_t *x, int T, blok_bf16_t *out, blok_stream_t stream_) {
  BLOK_REQUIRE(L && x && out, BLOK_ERR_ARG, "blok_moe_shared: null pointer");
  const blok_moe_weights &w = L->w;
  BLOK_REQUIRE(L->bws, BLOK_ERR_STATE, "blok_moe_shared: the layer was created with max_tokens = 1");
  BLOK_REQUIRE(w.shared_inter > 0 && w.shared_inter % 512 == 0 && w.hidden % 512 == 0, BLOK_ERR_SHAPE,
               "blok_moe_shared: needs a shared expert with sizes that are multiples of 512");
  BLOK_REQUIRE(T >= 0 && T <= L->max_tokens, BLOK_ERR_SHAPE, "blok_moe_shared: T=%d exceeds max_tokens %d", T, L->max_tokens);
  if (T == 0) return BLOK_OK;
  cudaStream_t stream = (cudaStream_t)stream_;
  const int tt = (T + kWgTileTokens - 1) / kWgTileTokens;
  int rc;
  WgArgs s;
  s.w_a = w.shared_gate; s.w_b = w.shared_up; s.s_a = s.s_b = nullptr; s.expert_stride_rows = 0; s.x = x; s.x_index = nullptr;
  s.K = w.hidden; s.R = w.shared_inter; s.out_bf16 = L->b_smid; s.out_f32 = nullptr;
  s.tile_expert = s.tile_start = s.tile_count = s.num_tiles = nullptr;
  s.out_index = nullptr; s.n_rows = T; s.identity_tiles = 1;
  s.splitk_ws = L->b_splitk; s.splitk_bytes = L->b_splitk_bytes; s.err = L->b_err;
  s.max_splits = L->b_front_split;  // blok_moe_batched's: the two agree bit for bit
  if ((rc = launch_wgemm(WG_BF16_SWIGLU, s, tt, stream))) return rc;
  WgArgs d = s;
  d.max_splits = 0;
  d.weights_early = true;
  d.w_a = w.shared_down; d.w_b = nullptr; d.x = L->b_smid; d.K = w.shared_inter; d.R = w.hidden; d.out_bf16 = out;
  return launch_wgemm(WG_BF16_PLAIN, d, tt, stream);
}

extern "C" int blok_moe_combine(const blok_bf16_t *y_assign, const float *wts, const blok_bf16_t *shared, int T, int topk,
                                int hidden, blok_bf16_t *out, blok_stream_t stream) {
  BLOK_REQUIRE(y_assign && wts && out, BLOK_ERR_ARG, "blok_moe_combine: null pointer");
  BLOK_REQUIRE(T >= 0 && topk >= 1 && hidden > 0 && hidden % 2 == 0, BLOK_ERR_SHAPE, "blok_moe_combine: bad shape");
  if (T == 0) return BLOK_OK;
  return launch_combine(false, y_assign, wts, shared, nullptr, 0, T, topk, hidden, out, (cudaStream_t)stream);
}
