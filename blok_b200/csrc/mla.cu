// MLA decode attention in the absorbed form over a bf16 latent cache.
// Reference: src/kimi_exec.cu:813-826 (projections, RMSNorm, RoPE, KV store, o_proj)
// and :692-716 / :414-475 (three-pass softmax attention over materialised K/V).
//
// The reference stores, per token and layer, the full K [64 x 192] and V [64 x 128]
// in fp32 (81,920 B) and re-reads K three times.  Both are functions of the bf16
// latent row (normed c_kv [512], roped k_pe [64]) that the reference computes at
// :817-823, so the cache here is that row, 1,152 B per token, and the attention is
// evaluated in the latent space:
//   q_abs_h = W_UK_h^T q_nope_h        W_UK_h = kv_b rows [h*256, h*256+128)   (:366-369)
//   s_t     = (q_abs_h . c_t + q_rope_h . kpe_t) * scale
//   o_lat_h = sum_t softmax(s)_t c_t
//   out_h   = W_UV_h o_lat_h           W_UV_h = kv_b rows [h*256+128, h*256+256)
// One pass over the cache with an online softmax; the sequence is split over CTAs
// (flash-decoding) and the partial results are merged by a second kernel.
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <new>

#include "mla_heads.h"
#include "mla_merge.cuh"
#include "wgemm.h"

namespace blok {

// W_UK^T: out[h][j][d] = kv_b[h*(nope+v) + d][j]  (a pure re-arrangement, no arithmetic)
__global__ void transpose_wuk_kernel(const uint16_t *__restrict__ kv_b, uint16_t *__restrict__ out, int heads, int nope,
                                     int v_head, int kv_rank) {
  long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  long total = (long)heads * kv_rank * nope;
  if (i >= total) return;
  int d = (int)(i % nope);
  long r = i / nope;
  int j = (int)(r % kv_rank);
  int h = (int)(r / kv_rank);
  out[i] = kv_b[((size_t)h * (nope + v_head) + d) * kv_rank + j];
}

size_t mla_attend_smem_bytes();
int launch_mla_attend(const uint16_t *q, const uint16_t *cache, long ctx_stride, const int *seq_len, int B, int splits,
                      float scale, float *part_o, float *part_ml, cudaStream_t stream);
int launch_mla_attend_tc(const uint16_t *q, const uint16_t *cache, long ctx_stride, long total_rows, const int *seq_len, int B, int ctas,
                         float scale, float *part_o, float *part_ml, const MlaPlan *plan, int2 *parts, cudaStream_t stream);
int launch_mla_attend_tc_paged(const uint16_t *q, const uint16_t *pool, long pool_rows, const int *block_table, const int *slot_of,
                               int table_stride, int page_rows, const int *seq_len, int B, int ctas, float scale, float *part_o,
                               float *part_ml, const MlaPlan *plan, int2 *parts, cudaStream_t stream);
int mla_attend_tc_take_error(unsigned *out);
int mla_attend_tc_trace(long long *host_out, int max_entries);
int launch_mla_attend_paged(const uint16_t *q, const uint16_t *pool, const int *block_table, const int *slot_of,
                            int table_stride, int page_rows, const int *seq_len, int B, int splits, float scale,
                            float *part_o, float *part_ml, cudaStream_t stream);

static size_t align256(size_t v) { return (v + 255) / 256 * 256; }

constexpr int kMlaMaxBatch = 64;  // sequences (or tokens of a prefill chunk) per call: what one pass of the weight-streaming kernel covers

}  // namespace blok

struct blok_mla_layer {
  blok_mla_weights w;
  int max_batch = 0;
  int max_splits = 0;
  float scale = 0.f;
  void *ws = nullptr;
  uint16_t *wuk_t = nullptr;   // [heads, kv_rank, qk_nope]
  float *inv_freq = nullptr;   // [qk_rope / 2]
  uint16_t *qa = nullptr;      // [B, q_rank]
  uint16_t *q = nullptr;       // [B, heads, nope + rope]
  uint16_t *q_full = nullptr;  // [B, heads, kv_rank + rope]
  uint16_t *av = nullptr;      // [B, heads * v_head]
  int *seq = nullptr;          // [B]
  unsigned *err = nullptr;     // [2] 1 + b when entry b of a call had a position outside its sequence's rows; a product gave up
  float *wg_ws = nullptr;      // fp32 sums of the projections (wgemm_stream.cu), one projection's at a time
  size_t wg_bytes = 0;
  bool weights_stay = false;   // see mla_layer_weights_stay
  float *part_o = nullptr;     // [max_splits + max_batch partial results, heads, kv_rank]
  float *part_ml = nullptr;
  blok::MlaPlan *plan = nullptr;  // of the call's sequences
  int2 *parts = nullptr;       // [B] and the sequences' partial results
};

using namespace blok;

// For a layer whose calls follow an ordinary launch of the same program that stands behind the last write of its weights, positions
// and tables (a model's embedding): the first launch of a call, too, may fetch its weights early.
namespace blok {
void mla_layer_weights_stay(blok_mla_layer_t *L);
}
void blok::mla_layer_weights_stay(blok_mla_layer_t *L) { L->weights_stay = true; }

// YaRN inverse frequencies, src/kimi_exec.cu:325-344 with the factor as a parameter.
static void yarn_inv_freq_host(const blok_mla_weights &w, float *out) {
  const float dim = (float)w.qk_rope;
  auto corr = [&](float rotations) {
    return dim * logf(w.yarn_original_ctx / (rotations * 2.0f * 3.141592654f)) / (2.0f * logf(w.rope_theta));
  };
  float low = fmaxf(floorf(corr(w.yarn_beta_fast)), 0.0f);
  float high = fminf(ceilf(corr(w.yarn_beta_slow)), dim - 1.0f);
  if (low == high) high += 0.001f;
  for (int p = 0; p < w.qk_rope / 2; ++p) {
    float extra = powf(w.rope_theta, -2.0f * (float)p / dim);
    float inter = extra / w.yarn_factor;
    float ramp = fminf(1.0f, fmaxf(0.0f, ((float)p - low) / (high - low)));
    float mask = 1.0f - ramp;
    out[p] = inter * (1.0f - mask) + extra * mask;
  }
}

extern "C" float blok_mla_softmax_scale(const blok_mla_weights *w) {
  if (!w) return 0.f;
  float mscale = 0.1f * w->yarn_mscale_all_dim * logf(w->yarn_factor) + 1.0f;
  return (1.0f / sqrtf((float)(w->qk_nope + w->qk_rope))) * mscale * mscale;
}

extern "C" int blok_mla_layer_create(const blok_mla_weights *w, int max_batch, int max_ctx, blok_mla_layer_t **out) {
  BLOK_REQUIRE(w && out, BLOK_ERR_ARG, "blok_mla_layer_create: null pointer");
  BLOK_REQUIRE(max_batch >= 1 && max_batch <= kMlaMaxBatch && max_ctx >= 1, BLOK_ERR_ARG,
               "blok_mla_layer_create: need 1 <= max_batch <= %d and max_ctx >= 1", kMlaMaxBatch);
  BLOK_REQUIRE(w->heads == 64 && w->kv_rank == 512 && w->qk_rope == 64 && w->qk_nope % 32 == 0 && w->v_head % 16 == 0 &&
                   w->hidden % 32 == 0 && w->q_rank % 32 == 0,
               BLOK_ERR_SHAPE,
               "blok_mla_layer_create: the attention kernel is built for 64 heads, kv_rank 512, qk_rope 64 (got %d, %d, %d)",
               w->heads, w->kv_rank, w->qk_rope);
  BLOK_REQUIRE(w->q_a && w->q_a_ln && w->q_b && w->kv_a && w->kv_a_ln && w->kv_b && w->o, BLOK_ERR_ARG,
               "blok_mla_layer_create: weight pointer missing");
  BLOK_REQUIRE(w->yarn_factor > 0.f && w->rope_theta > 1.f, BLOK_ERR_ARG, "blok_mla_layer_create: bad rope parameters");
  blok_mla_layer *L = new (std::nothrow) blok_mla_layer();
  BLOK_REQUIRE(L, BLOK_ERR_ARG, "blok_mla_layer_create: out of host memory");
  L->w = *w;
  L->max_batch = max_batch;
  L->max_splits = std::min(sm_count(), 160);  // what mla_value_kernel holds
  L->scale = blok_mla_softmax_scale(w);
  const int lat_w = w->kv_rank + w->qk_rope, qk_head = w->qk_nope + w->qk_rope;
  size_t off = 0;
  auto take = [&](size_t bytes) {
    size_t at = off;
    off = align256(off + bytes);
    return at;
  };
  size_t o_wuk = take((size_t)w->heads * w->kv_rank * w->qk_nope * 2);
  size_t o_freq = take((size_t)(w->qk_rope / 2) * 4);
  size_t o_qa = take((size_t)max_batch * w->q_rank * 2);
  size_t o_q = take((size_t)max_batch * w->heads * qk_head * 2);
  size_t o_qf = take((size_t)max_batch * w->heads * lat_w * 2);
  size_t o_av = take((size_t)max_batch * w->heads * w->v_head * 2);
  size_t o_seq = take((size_t)max_batch * 4);
  size_t o_err = take(8);
  size_t o_plan = take(sizeof(MlaPlan));
  size_t o_parts = take((size_t)max_batch * sizeof(int2));
  size_t o_po = take((size_t)(L->max_splits + max_batch) * w->heads * w->kv_rank * 4);
  size_t o_pml = take((size_t)(L->max_splits + max_batch) * w->heads * 2 * 4);
  const size_t q_rows = (size_t)w->heads * qk_head;
  L->wg_bytes = (size_t)max_batch * sizeof(float) *
                std::max(std::max((size_t)wgemm_stream_pair_split(WG_BF16_PLAIN, w->hidden, w->q_rank, lat_w) * (w->q_rank + lat_w),
                                  wgemm_stream_split(WG_BF16_PLAIN, w->q_rank, (int)q_rows) * q_rows),
                         (size_t)wgemm_stream_split(WG_BF16_PLAIN, w->heads * w->v_head, w->hidden) * w->hidden);
  size_t o_wg = take(L->wg_bytes);
  cudaError_t e = cudaMalloc(&L->ws, off);
  if (e != cudaSuccess) {
    delete L;
    return cuda_fail(e, "cudaMalloc(mla layer workspace)");
  }
  e = cudaMemset(L->ws, 0, off);  // the error words start at zero
  if (e != cudaSuccess) {
    cudaFree(L->ws);
    delete L;
    return cuda_fail(e, "cudaMemset(mla layer workspace)");
  }
  unsigned char *b = static_cast<unsigned char *>(L->ws);
  L->wuk_t = reinterpret_cast<uint16_t *>(b + o_wuk);
  L->inv_freq = reinterpret_cast<float *>(b + o_freq);
  L->qa = reinterpret_cast<uint16_t *>(b + o_qa);
  L->q = reinterpret_cast<uint16_t *>(b + o_q);
  L->q_full = reinterpret_cast<uint16_t *>(b + o_qf);
  L->av = reinterpret_cast<uint16_t *>(b + o_av);
  L->seq = reinterpret_cast<int *>(b + o_seq);
  L->err = reinterpret_cast<unsigned *>(b + o_err);
  L->plan = reinterpret_cast<MlaPlan *>(b + o_plan);
  L->parts = reinterpret_cast<int2 *>(b + o_parts);
  L->part_o = reinterpret_cast<float *>(b + o_po);
  L->part_ml = reinterpret_cast<float *>(b + o_pml);
  L->wg_ws = reinterpret_cast<float *>(b + o_wg);
  float freq[128];
  yarn_inv_freq_host(*w, freq);
  e = cudaMemcpy(L->inv_freq, freq, (size_t)(w->qk_rope / 2) * 4, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    long total = (long)w->heads * w->kv_rank * w->qk_nope;
    transpose_wuk_kernel<<<(unsigned)((total + 255) / 256), 256>>>(w->kv_b, L->wuk_t, w->heads, w->qk_nope, w->v_head,
                                                                   w->kv_rank);
    count_launch();
    e = cudaDeviceSynchronize();
  }
  if (e != cudaSuccess) {
    cudaFree(L->ws);
    delete L;
    return cuda_fail(e, "blok_mla_layer_create: set-up");
  }
  (void)max_ctx;
  *out = L;
  return BLOK_OK;
}

extern "C" int blok_mla_layer_refresh(blok_mla_layer_t *L) {
  BLOK_REQUIRE(L, BLOK_ERR_ARG, "blok_mla_layer_refresh: null pointer");
  const blok_mla_weights &w = L->w;
  const long total = (long)w.heads * w.kv_rank * w.qk_nope;
  transpose_wuk_kernel<<<(unsigned)((total + 255) / 256), 256>>>(w.kv_b, L->wuk_t, w.heads, w.qk_nope, w.v_head, w.kv_rank);
  count_launch();
  BLOK_CUDA(cudaDeviceSynchronize());
  return launch_status("transpose_wuk_kernel");
}

extern "C" int blok_mla_layer_destroy(blok_mla_layer_t *L) {
  if (!L) return BLOK_OK;
  cudaError_t e = L->ws ? cudaFree(L->ws) : cudaSuccess;
  delete L;
  return e == cudaSuccess ? BLOK_OK : cuda_fail(e, "cudaFree(mla layer workspace)");
}

extern "C" int blok_mla_attend_trace(long long *host_out, int max_entries) {
  if (!host_out || max_entries <= 0) return 0;
  return mla_attend_tc_trace(host_out, max_entries);
}

extern "C" int blok_mla_layer_check(blok_mla_layer_t *L, blok_stream_t stream) {
  BLOK_REQUIRE(L, BLOK_ERR_ARG, "blok_mla_layer_check: null pointer");
  BLOK_CUDA(cudaStreamSynchronize((cudaStream_t)stream));
  unsigned tc_err = 0;
  if (int rc = mla_attend_tc_take_error(&tc_err)) return rc;
  if (tc_err) {
    set_error("blok_mla_decode: the attention core gave up on wait %u (1 tile buffer, 2-5 MMA thread, 6-9 softmax warps)", tc_err);
    return BLOK_ERR_TIMEOUT;
  }
  unsigned err[2] = {0, 0};
  BLOK_CUDA(cudaMemcpy(err, L->err, sizeof(err), cudaMemcpyDeviceToHost));
  if (err[0] == 0 && err[1] == 0) return BLOK_OK;
  BLOK_CUDA(cudaMemset(L->err, 0, sizeof(err)));
  if (err[1]) {
    set_error("blok_mla_decode: a product gave up on a barrier");
    return BLOK_ERR_TIMEOUT;
  }
  set_error("blok_mla_decode: entry %u had a position outside its sequence's cache rows; its row was not stored", err[0] - 1);
  return BLOK_ERR_SHAPE;
}

// Where the latent rows of the sequences of a call live.
struct CacheRef {
  uint16_t *base = nullptr;         // dense cache, or the page pool
  long seq_stride = 0;              // dense: rows between consecutive sequences; 0 = every entry is the same sequence
  long ctx_cap = 0;                 // rows one sequence can hold (bounds the context splits)
  const int *block_table = nullptr; // paged when non-null: int32 [slots, table_stride] page numbers
  const int *slot_of = nullptr;     // paged: table row of batch entry b (null: b)
  int table_stride = 0, page_rows = 0;
};

// The mma.sync core's context splits per sequence: enough CTAs to fill the GPU, but never more than one per 64 rows of the cache
// allocation (the sequence lengths live on the device; the capacity bounds them), so that a short cache is not cut
// into slivers whose merge costs more than the attention.
static int splits_for(const blok_mla_layer *L, int B, long ctx_cap) {
  long s = L->max_splits / B;
  const long cap = (ctx_cap + 63) / 64;
  if (s > cap) s = cap;
  return s < 1 ? 1 : (int)s;
}

// The attention core: partial results in L->part_o and L->part_ml.  *splits: of every sequence, or 0: as the plan for L->max_splits
// CTAs says; planned: that is in L->plan and L->parts already, else the core makes it.
static int attend(blok_mla_layer *L, const uint16_t *q, const CacheRef &c, const int *seq_len, int B, float scale, bool planned, int *splits,
                  cudaStream_t stream) {
  const MlaPlan *plan = planned ? L->plan : nullptr;
  // the tcgen05 core by default; BLOK_MLA_ATTEND_IMPL=mma (read at every call) selects the mma.sync kernel, which also
  // serves page sizes that are not a multiple of the tcgen05 core's 64-token tile
  const char *impl = getenv("BLOK_MLA_ATTEND_IMPL");
  const bool tc = !(impl && strcmp(impl, "mma") == 0) && (!c.block_table || c.page_rows % 64 == 0);
  *splits = tc ? 0 : splits_for(L, B, c.ctx_cap);
  if (tc) {
    // the rows the tensor map may address: the whole dense cache (reads past it give zeros); a paged tile never leaves
    // its page, so the pool needs no tighter bound than the coordinate range
    const long dense_rows = c.seq_stride > 0 ? (long)B * c.seq_stride : c.ctx_cap;
    return c.block_table ? launch_mla_attend_tc_paged(q, c.base, (1l << 31) - 64, c.block_table, c.slot_of, c.table_stride, c.page_rows, seq_len,
                                                      B, L->max_splits, scale, L->part_o, L->part_ml, plan, L->parts, stream)
                         : launch_mla_attend_tc(q, c.base, c.seq_stride, dense_rows, seq_len, B, L->max_splits, scale, L->part_o, L->part_ml, plan, L->parts,
                                                stream);
  }
  return c.block_table ? launch_mla_attend_paged(q, c.base, c.block_table, c.slot_of, c.table_stride, c.page_rows, seq_len, B,
                                                 *splits, scale, L->part_o, L->part_ml, stream)
                       : launch_mla_attend(q, c.base, c.seq_stride, seq_len, B, *splits, scale, L->part_o, L->part_ml, stream);
}

static int attend_and_merge(blok_mla_layer *L, const uint16_t *q, const CacheRef &c, const int *seq_len, int B, float scale,
                            uint16_t *o_lat, cudaStream_t stream) {
  int splits;
  if (int rc = attend(L, q, c, seq_len, B, scale, false, &splits, stream)) return rc;
  const int most = splits ? splits : L->max_splits;
  return launch_pdl("mla_merge_kernel", mla_merge(L->w.heads, B), dim3(L->w.heads, B), 128, (size_t)most * sizeof(float), stream, L->part_o, L->part_ml, most,
                    L->w.heads, L->w.kv_rank, o_lat, 0, nullptr, 0, splits ? nullptr : L->parts);
}

static int check_paged(const char *who, const void *pool, const int *block_table, int table_stride, int page_rows) {
  BLOK_REQUIRE(pool && block_table, BLOK_ERR_ARG, "%s: null pointer", who);
  BLOK_REQUIRE((reinterpret_cast<uintptr_t>(pool) & 15) == 0, BLOK_ERR_ARG, "%s: the pool must be 16-byte aligned", who);
  BLOK_REQUIRE(table_stride >= 1 && page_rows >= 32 && page_rows % 32 == 0, BLOK_ERR_SHAPE,
               "%s: page_rows (%d) must be a positive multiple of 32 and table_stride (%d) >= 1", who, page_rows, table_stride);
  return BLOK_OK;
}

extern "C" int blok_mla_attend(blok_mla_layer_t *L, const blok_bf16_t *q, const blok_bf16_t *cache, long ctx_stride,
                               const int *seq_len, int B, float softmax_scale, blok_bf16_t *o_lat,
                               blok_stream_t stream) {
  BLOK_REQUIRE(L && q && cache && seq_len && o_lat, BLOK_ERR_ARG, "blok_mla_attend: null pointer");
  BLOK_REQUIRE(B >= 1 && B <= L->max_batch && ctx_stride >= 1, BLOK_ERR_SHAPE, "blok_mla_attend: B=%d outside [1, %d]", B,
               L->max_batch);
  BLOK_REQUIRE((reinterpret_cast<uintptr_t>(q) & 15) == 0 && (reinterpret_cast<uintptr_t>(cache) & 15) == 0, BLOK_ERR_ARG,
               "blok_mla_attend: q and cache must be 16-byte aligned");
  CacheRef c;
  c.base = const_cast<uint16_t *>(cache);
  c.seq_stride = c.ctx_cap = ctx_stride;
  return attend_and_merge(L, q, c, seq_len, B, softmax_scale, o_lat, (cudaStream_t)stream);
}

extern "C" int blok_mla_attend_paged(blok_mla_layer_t *L, const blok_bf16_t *q, const blok_bf16_t *pool, const int *block_table,
                                     const int *slot_of, int table_stride, int page_rows, const int *seq_len, int B,
                                     float softmax_scale, blok_bf16_t *o_lat, blok_stream_t stream) {
  BLOK_REQUIRE(L && q && seq_len && o_lat, BLOK_ERR_ARG, "blok_mla_attend_paged: null pointer");
  BLOK_REQUIRE(B >= 1 && B <= L->max_batch, BLOK_ERR_SHAPE, "blok_mla_attend_paged: B=%d outside [1, %d]", B, L->max_batch);
  BLOK_REQUIRE((reinterpret_cast<uintptr_t>(q) & 15) == 0, BLOK_ERR_ARG, "blok_mla_attend_paged: q must be 16-byte aligned");
  if (int rc = check_paged("blok_mla_attend_paged", pool, block_table, table_stride, page_rows)) return rc;
  CacheRef c;
  c.base = const_cast<uint16_t *>(pool);
  c.ctx_cap = (long)table_stride * page_rows;
  c.block_table = block_table;
  c.slot_of = slot_of;
  c.table_stride = table_stride;
  c.page_rows = page_rows;
  return attend_and_merge(L, q, c, seq_len, B, softmax_scale, o_lat, (cudaStream_t)stream);
}

static_assert(kMlaMaxBatch <= kWgStreamTokens, "a call's entries are one pass of the weight-streaming kernel");

// The attention block for B entries (sequences, or the tokens of a prefill chunk: chunk, ctx_len then holds the first position):
// three passes of the weight-streaming kernel and, between them, kernels that take each pass's fp32 sums as they lie (mla_heads.cu).
// From the second launch on every kernel with weights fetches them before the kernels in front of it have finished: the first one
// (weights_early unset) starts the others only when everything before the call is done.
static int decode_body(blok_mla_layer *L, const uint16_t *n, const CacheRef &c, const int *ctx_len, bool chunk, int B, uint16_t *out,
                       cudaStream_t stream) {
  const blok_mla_weights &w = L->w;
  const int lat_w = w.kv_rank + w.qk_rope, qk_head = w.qk_nope + w.qk_rope;
  const MlaPositions pos = {ctx_len, chunk, c.ctx_cap};
  int rc, nz = 1;
  WgArgs g = {};
  g.identity_tiles = 1;
  g.n_rows = B;
  g.splitk_ws = L->wg_ws;
  g.splitk_bytes = L->wg_bytes;
  g.err = L->err + 1;
  // q_a and kv_a, then the norms and the cache row   (:813-824)
  g.w_a = w.q_a; g.R = w.q_rank; g.w_2 = w.kv_a; g.R2 = lat_w; g.x = n; g.K = w.hidden;
  g.keep_sums = true;
  g.weights_early = L->weights_stay;
  if ((rc = launch_wgemm_stream(WG_BF16_PLAIN, g, &nz, stream))) return rc;
  MlaNorm m = {};
  m.part = L->wg_ws; m.nz = nz; m.ld = w.q_rank + lat_w; m.q_rank = w.q_rank; m.kv_rank = w.kv_rank; m.rope = w.qk_rope;
  m.eps = w.rms_eps; m.q_ln = w.q_a_ln; m.kv_ln = w.kv_a_ln; m.qa = L->qa; m.inv_freq = L->inv_freq; m.pos = pos;
  m.cache = c.base; m.ctx_stride = c.seq_stride; m.block_table = c.block_table; m.slot_of = c.slot_of;
  m.table_stride = c.table_stride; m.page_rows = c.page_rows; m.seq = L->seq; m.plan = L->plan; m.parts = L->parts; m.ctas = L->max_splits; m.err = L->err;
  if ((rc = launch_mla_norm(m, B, stream))) return rc;
  // q_b, then q_abs = W_UK^T q_nope and the rotated rope part.  The head kernels read a head's sums four times over: with many
  // entries one part and bf16
  g.w_a = w.q_b; g.R = w.heads * qk_head; g.w_2 = nullptr; g.R2 = 0; g.x = L->qa; g.K = w.q_rank; g.out_bf16 = L->q;
  g.keep_sums = false; g.max_splits = B > 16 ? 1 : 0; g.weights_early = true;
  if ((rc = launch_wgemm_stream(WG_BF16_PLAIN, g, &nz, stream))) return rc;
  MlaQuery q = {};
  q.part = nz > 1 ? L->wg_ws : nullptr; q.q = L->q; q.nz = nz; q.B = B; q.nope = w.qk_nope; q.rope = w.qk_rope; q.kv_rank = w.kv_rank;
  q.inv_freq = L->inv_freq; q.pos = pos; q.q_full = L->q_full; q.werr = L->err + 1;
  if ((rc = launch_mla_query(L->wuk_t, w.heads, q, stream))) return rc;
  int splits;
  if ((rc = attend(L, L->q_full, c, L->seq, B, L->scale, true, &splits, stream))) return rc;
  // the splits merged, out_h = W_UV o_lat_h, then o_proj   (:826)
  MlaValue v = {};
  v.part_o = L->part_o; v.part_ml = L->part_ml; v.B = B; v.splits = splits; v.ctas = L->max_splits; v.parts = L->parts; v.nope = w.qk_nope; v.v_head = w.v_head; v.out = L->av;
  v.werr = L->err + 1;
  if ((rc = launch_mla_value(w.kv_b, w.heads, v, stream))) return rc;
  g.w_a = w.o; g.R = w.hidden; g.x = L->av; g.K = w.heads * w.v_head; g.out_bf16 = out; g.max_splits = 0;
  if ((rc = launch_wgemm_stream(WG_BF16_PLAIN, g, &nz, stream))) return rc;
  return nz > 1 ? launch_wgemm_splitk_reduce(WG_BF16_PLAIN, g, nz, stream) : BLOK_OK;
}

extern "C" int blok_mla_decode(blok_mla_layer_t *L, const blok_bf16_t *n, blok_bf16_t *cache, long ctx_stride,
                               const int *ctx_len, int B, blok_bf16_t *out, blok_stream_t stream_) {
  BLOK_REQUIRE(L && n && cache && ctx_len && out, BLOK_ERR_ARG, "blok_mla_decode: null pointer");
  BLOK_REQUIRE(B >= 1 && B <= L->max_batch && ctx_stride >= 1, BLOK_ERR_SHAPE, "blok_mla_decode: B=%d outside [1, %d]", B,
               L->max_batch);
  BLOK_REQUIRE((reinterpret_cast<uintptr_t>(n) & 15) == 0 && (reinterpret_cast<uintptr_t>(cache) & 15) == 0, BLOK_ERR_ARG,
               "blok_mla_decode: n and cache must be 16-byte aligned");
  CacheRef c;
  c.base = cache;
  c.seq_stride = c.ctx_cap = ctx_stride;
  return decode_body(L, n, c, ctx_len, false, B, out, (cudaStream_t)stream_);
}

extern "C" int blok_mla_prefill(blok_mla_layer_t *L, const blok_bf16_t *n, blok_bf16_t *cache, long ctx_cap, const int *first_pos,
                                int T, blok_bf16_t *out, blok_stream_t stream_) {
  BLOK_REQUIRE(L && n && cache && first_pos && out, BLOK_ERR_ARG, "blok_mla_prefill: null pointer");
  BLOK_REQUIRE(T >= 1 && T <= L->max_batch && ctx_cap >= T, BLOK_ERR_SHAPE,
               "blok_mla_prefill: T=%d outside [1, %d] or larger than the cache (%ld rows)", T, L->max_batch, ctx_cap);
  BLOK_REQUIRE((reinterpret_cast<uintptr_t>(n) & 15) == 0 && (reinterpret_cast<uintptr_t>(cache) & 15) == 0, BLOK_ERR_ARG,
               "blok_mla_prefill: n and cache must be 16-byte aligned");
  CacheRef c;
  c.base = cache;
  c.seq_stride = 0;  // every token of the chunk appends to, and reads, the same sequence
  c.ctx_cap = ctx_cap;
  return decode_body(L, n, c, first_pos, true, T, out, (cudaStream_t)stream_);
}

extern "C" int blok_mla_decode_paged(blok_mla_layer_t *L, const blok_bf16_t *n, blok_bf16_t *pool, const int *block_table,
                                     const int *slot_of, int table_stride, int page_rows, const int *ctx_len, int B,
                                     blok_bf16_t *out, blok_stream_t stream_) {
  BLOK_REQUIRE(L && n && ctx_len && out, BLOK_ERR_ARG, "blok_mla_decode_paged: null pointer");
  BLOK_REQUIRE(B >= 1 && B <= L->max_batch, BLOK_ERR_SHAPE, "blok_mla_decode_paged: B=%d outside [1, %d]", B, L->max_batch);
  BLOK_REQUIRE((reinterpret_cast<uintptr_t>(n) & 15) == 0, BLOK_ERR_ARG, "blok_mla_decode_paged: n must be 16-byte aligned");
  if (int rc = check_paged("blok_mla_decode_paged", pool, block_table, table_stride, page_rows)) return rc;
  CacheRef c;
  c.base = pool;
  c.ctx_cap = (long)table_stride * page_rows;
  c.block_table = block_table;
  c.slot_of = slot_of;
  c.table_stride = table_stride;
  c.page_rows = page_rows;
  return decode_body(L, n, c, ctx_len, false, B, out, (cudaStream_t)stream_);
}
