// bf16 weights against up to 64 rows of activations (a decode step, a rank's share of a small batch):
//   out[token, row] = sum_c W[row, c] * x[token, c]          (matvec_bf16_k, src/kimi_exec.cu:272-284, per token)
// with the SwiGLU front half as an option (gate and up rows of the same index, :255, :674-686).
//
// At these counts the product is the weight stream.  The weights are the M = 128 side of tcgen05.mma and the tokens its N side
// (16 to 64), so a weight byte passes shared memory once whatever the token count and no warp spends an instruction on it: one
// thread brings 128 rows x 64 columns of weights and the same columns of the tokens per step by TMA, four to six steps in flight
// (about 100 KB per CTA, two CTAs per SM), one lane issues the MMAs, four warps store the accumulator (a lane owns a weight row).
//
// Matrices with few rows are split over K (blockIdx.y) so that about two CTAs per SM run; the partial sums go to the caller's
// scratch in the layout of wgemm_splitk_reduce_kernel, which adds them in split order.
//
// The mma.sync form before it (a warp's cp.async ring of its own 16 rows, tokens staged in shared memory) read eight times the
// weights' bytes from shared memory at 64 tokens.  The three projections of the attention block, 202 MB, with what stands between
// them (mla_heads.cu), us: one sequence 92 -> 67 (mat-vec kernels), 33 sequences 209 -> 140, a 64-token chunk 200 -> 126.
//
// The kernel becomes resident while the kernel before it runs (launch_pdl), and where the caller knows that the weights have long
// been there (WgArgs::weights_early) the first steps' weights are on their way before the wait: the ramp of the stream is hidden
// behind the kernel before.  Shared memory keeps it at two CTAs per SM, so early CTAs spread evenly.
//
// A launch reads every weight once, and they are the first that L2 gives up: what other kernels find there (caches, activations, the rest
// of a small model) stays.  Without that the vocabulary's 134 MB, which had gone through the mat-vec kernel, pushed the layers' weights out
// at every step: small Nomozen and Pamopel models of four layers, one sequence of 1,024 tokens, us a step: mat-vec 301 / 282, weight
// stream 336 / 306, with the hint 301 / 277.
//
// Every wait is bounded; a CTA that gives up sets the error word, stores NaN, waits for its copies and frees its tensor memory.
#include <algorithm>

#include "gemm_tma.h"
#include "tc_pipe.cuh"
#include "wgemm.h"

namespace blok {

constexpr int kStRows = 128;     // weight rows per CTA (SwiGLU: 64 gate + 64 up rows)
constexpr int kStCols = 64;      // columns per step
constexpr int kStMinSteps = 8;   // a split of K has at least so many
constexpr int kStThreads = 192;  // warps 0..3: stores, 4: copies, 5: MMA
constexpr int kStMaxStages = 6;
constexpr int kStTmemCols = 64;
constexpr uint32_t kStWBytes = kStRows * kStCols * 2;

__device__ unsigned g_wgemm_stream_error = 0;

struct StArgs {
  float *part;         // fp32 [split][token][ld] where K is split, else NULL
  uint16_t *out_bf16;  // [token][R]
  float *out_f32;
  int T, N, K, R, R2, tiles1, ld, stages, early;  // tiles from tiles1 on: the second matrix's; its sums follow the first's columns
  unsigned *err;
};

template <bool SWIGLU>
__global__ void __launch_bounds__(kStThreads) wgemm_stream_kernel(const __grid_constant__ CUtensorMap mx, const __grid_constant__ CUtensorMap mwa,
                                                                  const __grid_constant__ CUtensorMap mwb, const __grid_constant__ CUtensorMap mw2,
                                                                  const StArgs a) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) unsigned long long s_bar[2 * kStMaxStages + 1];
  __shared__ uint32_t s_tmem;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // Without early weights the kernels behind this one must not start before everything before it has finished: they may fetch
  // theirs before their own wait, on the word of a caller who knows this launch to be in between.
  if (!a.early) pdl_wait();
  pdl_trigger();
  const uint32_t sbase = ((uint32_t)__cvta_generic_to_shared(smem_raw) + 1023u) & ~1023u;
  const uint32_t full = (uint32_t)__cvta_generic_to_shared(&s_bar[0]), empty = full + 8 * kStMaxStages, done = full + 16 * kStMaxStages;
  const int S = a.stages;
  if (tid == 0) {
    for (int s = 0; s < S; ++s) {
      tp_mbar_init(full + 8 * s, 1);
      tp_mbar_init(empty + 8 * s, 1);
    }
    tp_mbar_init(done, 1);
    tp_mbar_init_fence();
  }
  if (warp == 0) tp_tmem_alloc((uint32_t)__cvta_generic_to_shared(&s_tmem), kStTmemCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s_tmem;
  const bool second = (int)blockIdx.x >= a.tiles1, gated = SWIGLU && !second;
  const int tile = second ? (int)blockIdx.x - a.tiles1 : (int)blockIdx.x;
  const int all_steps = (a.K + kStCols - 1) / kStCols, nz = (int)gridDim.y, z = (int)blockIdx.y;
  const int first = all_steps * z / nz, nsteps = all_steps * (z + 1) / nz - first;
  const uint32_t xbytes = (uint32_t)a.N * (kStCols * 2), stage = kStWBytes + xbytes;
  bool failed = false;

  if (warp == 4) {
    if (lane == 0) {
      const uint64_t once = tp_read_once();
      auto weights = [&](int c, uint32_t dst, uint32_t bar) {
        const int k = (first + c) * kStCols;
        tp_expect_tx(bar, stage);
        if (gated) {
          tp_load_2d_hint(dst, &mwa, k, tile * (kStRows / 2), bar, once);
          tp_load_2d_hint(dst + kStWBytes / 2, &mwb, k, tile * (kStRows / 2), bar, once);
        } else {
          tp_load_2d_hint(dst, second ? &mw2 : &mwa, k, tile * kStRows, bar, once);
        }
      };
      const int pre = min(S, nsteps);
      for (int c = 0; c < pre; ++c) weights(c, sbase + (uint32_t)c * stage, full + 8 * c);
      pdl_wait();
      asm volatile("fence.proxy.async;" ::: "memory");  // the tokens' rows were written by ordinary stores
      for (int c = 0; c < pre; ++c) tp_load_2d(sbase + (uint32_t)c * stage + kStWBytes, &mx, (first + c) * kStCols, 0, full + 8 * c);
      int issued = pre, s = 0;
      uint32_t turn = 0;
      for (int c = pre; c < nsteps; ++c) {
        if (!tp_wait(empty + 8 * s, turn)) {
          failed = true;
          break;
        }
        weights(c, sbase + (uint32_t)s * stage, full + 8 * s);
        tp_load_2d(sbase + (uint32_t)s * stage + kStWBytes, &mx, (first + c) * kStCols, 0, full + 8 * s);
        issued = c + 1;
        if (++s == S) s = 0, turn ^= 1;
      }
      // no copy may be in flight when the CTA leaves; the MMA lane has seen all of them unless a wait gave up
      for (int c = max(0, issued - S); c < issued; ++c) tp_wait(full + 8 * (c % S), (uint32_t)((c / S) & 1));
    }
  } else if (warp == 5) {
    // the whole warp walks the steps, so that addresses and descriptors stay warp-uniform; one lane issues
    const bool issues = tp_elect();
    const uint32_t idesc = tp_idesc_bf16(a.N);
    pdl_wait();  // the bound below is for this kernel's own copies, not for what the kernels in front still have to do
    int s = 0;
    uint32_t turn = 0;
    for (int c = 0; c < nsteps; ++c) {
      if (!__all_sync(0xffffffffu, tp_wait(full + 8 * s, turn))) {
        failed = true;
        break;
      }
      tc_fence_after();
      const uint64_t ad = tp_desc_k_sw128(sbase + (uint32_t)s * stage), bd = tp_desc_k_sw128(sbase + (uint32_t)s * stage + kStWBytes);
      if (issues) {
#pragma unroll
        for (int k = 0; k < kStCols / 16; ++k) tp_mma(tmem, ad + (uint64_t)(2 * k), bd + (uint64_t)(2 * k), idesc, (c | k) ? 1u : 0u);
        tp_commit(empty + 8 * s);
        if (c == nsteps - 1) tp_commit(done);
      }
      if (++s == S) s = 0, turn ^= 1;
    }
  } else {
    pdl_wait();  // the kernel before may still read what this one writes
    failed = __any_sync(0xffffffffu, !tp_wait(done, 0));
    tc_fence_after();
    const int r = 32 * warp + lane;
    const uint32_t at = tmem + ((uint32_t)(32 * warp) << 16);
    const int R = second ? a.R2 : a.R;
    if (gated && !a.part) {
      // the sums to the ring's memory (every copy into it has been consumed): [token][64 gate, 64 up]
      float *sums = reinterpret_cast<float *>(smem_raw) + r;
#pragma unroll 1
      for (int c0 = 0; c0 < a.T; c0 += 16) {
        uint32_t v[16];
        tmem_ld16(at + c0, v);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 16; ++j)
          if (c0 + j < a.T) sums[(c0 + j) * kStRows] = __uint_as_float(failed ? 0x7fc00000u : v[j]);
      }
    } else {
      const int row = gated ? tile * (kStRows / 2) + (r & 63) : tile * kStRows + r;
      const int col = second ? a.ld - a.R2 + row : (gated && r >= 64 ? R + row : row);  // of the partial sums
      const size_t ld = a.part ? a.ld : R;
      float *f32 = a.part ? a.part + (size_t)z * a.T * ld + col : (a.out_f32 ? a.out_f32 + row : nullptr);
      uint16_t *b16 = a.out_bf16 + row;
#pragma unroll 1
      for (int c0 = 0; c0 < a.T; c0 += 16) {
        uint32_t v[16];
        tmem_ld16(at + c0, v);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          if (row < R && c0 + j < a.T) {
            const float f = __uint_as_float(failed ? 0x7fc00000u : v[j]);
            if (f32) f32[j * ld] = f;
            else b16[j * ld] = f32_to_bf16_bits(f);
          }
        }
        if (f32) f32 += 16 * ld;
        else b16 += 16 * ld;
      }
    }
  }
  if (failed) atomicExch(a.err ? a.err : &g_wgemm_stream_error, 1u);
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tp_tmem_free(tmem, kStTmemCols);
  if (gated && !a.part) {
    // All warps gate, a thread every third token of one row: exponential and quotient are a long chain for every value.  With the gate's
    // two warps alone a launch over 64 rows took 17 us where its plain twin takes 10; a dense layer of 256 x 512 over 64 rows 27.5 -> 19.5.
    const int row = tile * (kStRows / 2) + (tid & 63);
    const float *sums = reinterpret_cast<const float *>(smem_raw) + (tid & 63);
    if (row < a.R) {
#pragma unroll 4
      for (int tok = tid >> 6; tok < a.T; tok += kStThreads / 64) {
        const float f = round_bf16(sums[tok * kStRows]);
        const float m = round_bf16(f / (1.0f + expf(-f))) * round_bf16(sums[tok * kStRows + 64]);
        a.out_bf16[(size_t)tok * a.R + row] = f32_to_bf16_bits(round_bf16(m));
      }
    }
  }
}

static bool st_aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

bool wgemm_stream_supports(int mode, const WgArgs &a) {
  if (mode != WG_BF16_PLAIN && mode != WG_BF16_SWIGLU) return false;
  if (!a.identity_tiles || a.n_rows < 1 || a.n_rows > kWgStreamTokens || a.x_index || a.out_index) return false;
  if (a.K % 256 || a.R % (mode == WG_BF16_SWIGLU ? 8 : 16)) return false;
  return st_aligned16(a.w_a) && st_aligned16(a.x) && (mode != WG_BF16_SWIGLU || st_aligned16(a.w_b));
}

static int st_tiles(int mode, int R) {
  const int per = mode == WG_BF16_SWIGLU ? kStRows / 2 : kStRows;
  return (R + per - 1) / per;
}
// About two CTAs per SM, at least kStMinSteps steps each.
static int st_split(int K, int tiles) { return std::max(1, std::min((K + kStCols - 1) / kStCols / kStMinSteps, 2 * sm_count() / tiles)); }
int wgemm_stream_split(int mode, int K, int R) {
  if (mode != WG_BF16_PLAIN && mode != WG_BF16_SWIGLU) return 1;
  return st_split(K, st_tiles(mode, R));
}
int wgemm_stream_pair_split(int mode, int K, int R, int R2) { return st_split(K, st_tiles(mode, R) + st_tiles(WG_BF16_PLAIN, R2)); }

bool wgemm_stream_takes_few(int mode, const WgArgs &args) { return wgemm_stream_supports(mode, args) && st_tiles(mode, args.R) >= sm_count(); }
// Products of up to 8 rows with fewer tiles than SMs: K in parts and a launch that adds them, against the mat-vec kernel, the dense
// layer's two products measured together (hidden x ffn, rows: mat-vec / here, us).
//  - gate and up: 7168 x 8192, 1 row 72 / 62, 8 rows 101 / 63; 16384 x 4096, 1 row 81 / 69; 2048 x 8192, 1 row 27.3 / 25.8, 8 rows 30.7 /
//    27.0; but 7168 x 2048, 59 MB, 1 row 24.6 / 26.7 (4 rows 24.7 / 23.6), 1024 x 4096, 17 MB, 4 rows 14.3 / 15.7.
//  - down: 7168 x 18432, 1 row 145 / 124, 4 rows 188 / 124; 4096 x 14336, 1 row 72 / 62; 1024 x 4096, 1 row 14.4 / 13.4; but K = 2,048 of
//    7,168 rows, 1 row 23.7 / 24.6 (4 rows 26.2 / 24.7).
bool wgemm_stream_takes_parts(int mode, const WgArgs &args, size_t room) {
  const bool gated = mode == WG_BF16_SWIGLU, one = args.n_rows == 1;
  const size_t weights = (size_t)args.R * args.K * (gated ? 4 : 2), sums = (size_t)args.n_rows * args.R * (gated ? 8 : 4);
  if (gated ? weights < (one ? size_t(64) : size_t(32)) * 1000000 : one && args.K < 4096) return false;
  return wgemm_stream_supports(mode, args) && room >= wgemm_stream_split(mode, args.K, args.R) * sums;
}

// Launches the kernel; *splits = the K-split it used (> 1: the partial sums wait in args.splitk_ws for the reduce kernel).
int launch_wgemm_stream(int mode, const WgArgs &args, int *splits, cudaStream_t stream) {
  const bool swiglu = mode == WG_BF16_SWIGLU;
  BLOK_REQUIRE(args.K % 8 == 0 && args.R >= 1 && args.n_rows >= 1 && args.n_rows <= kWgStreamTokens && (!args.R2 || args.keep_sums), BLOK_ERR_SHAPE,
               "streaming product: %d rows x %d columns over %d tokens", args.R, args.K, args.n_rows);
  StArgs a;
  a.tiles1 = st_tiles(mode, args.R);
  const int tiles = a.tiles1 + (args.R2 ? st_tiles(WG_BF16_PLAIN, args.R2) : 0);
  a.ld = (swiglu ? 2 * args.R : args.R) + args.R2;
  const size_t per_split = (size_t)args.n_rows * a.ld * sizeof(float);
  const size_t room = args.splitk_ws ? args.splitk_bytes / per_split : 0;
  BLOK_REQUIRE(!args.keep_sums || room >= 1, BLOK_ERR_WORKSPACE, "streaming product: no room for the sums");
  const int nz = (int)std::max<size_t>(1, std::min<size_t>(args.max_splits > 0 ? std::min(args.max_splits, st_split(args.K, tiles)) : st_split(args.K, tiles), room));
  a.part = nz > 1 || args.keep_sums ? args.splitk_ws : nullptr;
  a.out_bf16 = args.out_bf16;
  a.out_f32 = args.out_f32;
  a.T = args.n_rows;
  a.N = (args.n_rows + 15) / 16 * 16;
  a.K = args.K;
  a.R = args.R;
  a.R2 = args.R2;
  a.early = args.weights_early;
  a.err = args.err;
  // as many steps as two CTAs per SM leave room for: 108, 100, 88 and 96 KB
  a.stages = a.N == 16 ? 6 : (a.N == 32 ? 5 : 4);
  const int smem = a.stages * (int)(kStWBytes + a.N * kStCols * 2) + 1024;
  CUtensorMap mx, mwa, mwb, mw2;
  int rc;
  if ((rc = gemm_operand_map(args.x, args.n_rows, args.K, args.K, a.N, &mx))) return rc;
  if ((rc = gemm_operand_map(args.w_a, args.R, args.K, args.K, swiglu ? kStRows / 2 : kStRows, &mwa))) return rc;
  mwb = mw2 = mwa;
  if (swiglu && (rc = gemm_operand_map(args.w_b, args.R, args.K, args.K, kStRows / 2, &mwb))) return rc;
  if (args.R2 && (rc = gemm_operand_map(args.w_2, args.R2, args.K, args.K, kStRows, &mw2))) return rc;
  auto kernel = swiglu ? wgemm_stream_kernel<true> : wgemm_stream_kernel<false>;
  if (int rc = allow_smem(kernel, smem)) return rc;
  *splits = nz;
  return launch_pdl("wgemm_stream_kernel", kernel, dim3(tiles, nz), kStThreads, (size_t)smem, stream, mx, mwa, mwb, mw2, a);
}

int wgemm_stream_take_error(unsigned *out) {
  unsigned zero = 0;
  BLOK_CUDA(cudaMemcpyFromSymbol(out, g_wgemm_stream_error, sizeof(unsigned)));
  if (*out) BLOK_CUDA(cudaMemcpyToSymbol(g_wgemm_stream_error, &zero, sizeof(unsigned)));
  return BLOK_OK;
}

int wgemm_stream_set_error(unsigned code) {
  BLOK_CUDA(cudaMemcpyToSymbol(g_wgemm_stream_error, &code, sizeof(unsigned)));
  return BLOK_OK;
}

// Adds the K-split partial sums in split order and applies the epilogue of the GEMM kernels.  grid = (ceil(R / 256), n_rows).
template <bool SWIGLU>
__global__ void wgemm_splitk_reduce_kernel(const WgArgs a, int nz) {
  const int p = blockIdx.y, row = blockIdx.x * blockDim.x + threadIdx.x;
  pdl_trigger();
  pdl_wait();
  if (row >= a.R) return;
  const int cols = SWIGLU ? 2 * a.R : a.R;
  const float *ps = a.splitk_ws + (size_t)p * cols + row;
  const size_t stride = (size_t)a.n_rows * cols;
  float v = 0.f, u = 0.f;
  for (int z = 0; z < nz; ++z) {
    v += ps[z * stride];
    if (SWIGLU) u += ps[z * stride + a.R];
  }
  const size_t o = (a.out_index ? (size_t)a.out_index[p] : (size_t)p) * a.R + row;
  if (SWIGLU) {
    const float gv = round_bf16(v), uv = round_bf16(u);
    a.out_bf16[o] = f32_to_bf16_bits(round_bf16(round_bf16(gv / (1.0f + expf(-gv))) * uv));
  } else if (a.out_f32) {
    a.out_f32[o] = v;
  } else {
    a.out_bf16[o] = f32_to_bf16_bits(v);
  }
}

int launch_wgemm_splitk_reduce(int mode, const WgArgs &args, int nz, cudaStream_t stream) {
  const dim3 rg((args.R + 255) / 256, args.n_rows);
  if (mode == WG_BF16_SWIGLU || mode == WG_I4_SWIGLU) return launch_pdl("wgemm_splitk_reduce_kernel", wgemm_splitk_reduce_kernel<true>, rg, 256, 0, stream, args, nz);
  return launch_pdl("wgemm_splitk_reduce_kernel", wgemm_splitk_reduce_kernel<false>, rg, 256, 0, stream, args, nz);
}

// The mma.sync kernel (wgemm.cu) has 128 weight rows per CTA (64 + 64 for SwiGLU) and splits whole 512-column chunks.
int wgemm_splitk_factor(int mode, int K, int R, int tiles) {
  if (mode != WG_BF16_PLAIN && mode != WG_BF16_SWIGLU) return 1;
  const int rows_per_cta = mode == WG_BF16_SWIGLU ? 64 : 128;
  if (R % rows_per_cta || K % 512 || tiles < 1) return 1;
  const int ctas = R / rows_per_cta * tiles, chunks = K / 512;
  return std::max(1, std::min(chunks, 2 * sm_count() / ctas));
}
// The TMA-fed GEMM: parts of at least 16 of its 64-column steps, so that its pipeline fills.  Up to 128 rows of x tiles of 128
// outputs and two CTAs per SM; more, pairs of CTAs with tiles of 256 rows by 256 weight rows (the 384-expert router over 517
// tokens: 6 tiles, 7 parts).
int wgemm_tma_split(int mode, int K, int R, int rows) {
  if (mode != WG_BF16_PLAIN && mode != WG_BF16_SWIGLU) return 1;
  if (rows > 128) {
    const int tiles = ((mode == WG_BF16_SWIGLU ? 2 * R : R) + 255) / 256 * ((rows + 255) / 256);
    return std::max(1, std::min((K + 63) / 64 / 16, sm_count() / 2 / tiles));
  }
  const int ctas = (R + 127) / 128 * ((rows + 127) / 128);
  return std::max(1, std::min((K + 63) / 64 / 16, 2 * sm_count() / ctas));
}
size_t wgemm_splitk_bytes(int mode, int K, int R, int max_rows) {
  size_t worst = 0;
  for (int rows = 128; max_rows > kWgStreamTokens; rows += 128) {
    const int nz = wgemm_tma_split(mode, K, R, rows);
    if (nz > 1) worst = std::max(worst, (size_t)nz * std::min(rows, max_rows) * (mode == WG_BF16_SWIGLU ? 2 * R : R) * sizeof(float));
    if (nz <= 1 || rows >= max_rows) break;  // the factor falls as the rows grow
  }
  {  // the weight-streaming kernel over up to kWgStreamTokens rows
    const int nz = wgemm_stream_split(mode, K, R);
    if (nz > 1) worst = std::max(worst, (size_t)nz * std::min(max_rows, kWgStreamTokens) * (mode == WG_BF16_SWIGLU ? 2 * R : R) * sizeof(float));
  }
  for (int tiles = 1; tiles <= (max_rows + kWgTileTokens - 1) / kWgTileTokens; ++tiles) {
    const int nz = wgemm_splitk_factor(mode, K, R, tiles);
    if (nz <= 1) break;  // the factor falls as the tiles grow in number
    const size_t rows = (size_t)std::min(max_rows, tiles * kWgTileTokens);
    worst = std::max(worst, (size_t)nz * rows * (mode == WG_BF16_SWIGLU ? 2 * R : R) * sizeof(float));
  }
  return worst;
}

WgArgs wgemm_rows(const void *w_a, const void *w_b, const uint16_t *x, uint16_t *out_bf16, float *out_f32, int R, int K, int T) {
  WgArgs r;
  r.w_a = w_a; r.w_b = w_b; r.s_a = r.s_b = nullptr; r.expert_stride_rows = 0; r.x = x; r.x_index = nullptr;
  r.K = K; r.R = R; r.out_bf16 = out_bf16; r.out_f32 = out_f32;
  r.tile_expert = r.tile_start = r.tile_count = r.num_tiles = nullptr; r.out_index = nullptr;
  r.identity_tiles = 1; r.n_rows = T;
  return r;
}

int launch_wgemm_rows(int mode, const void *w_a, const void *w_b, const uint16_t *x, uint16_t *out_bf16, float *out_f32, int R, int K,
                      int T, float *splitk_ws, size_t splitk_bytes, cudaStream_t stream, bool weights_early, unsigned *err) {
  WgArgs r = wgemm_rows(w_a, w_b, x, out_bf16, out_f32, R, K, T);
  r.splitk_ws = splitk_ws; r.splitk_bytes = splitk_bytes; r.weights_early = weights_early; r.err = err;
  BLOK_REQUIRE(wgemm_stream_supports(mode, r), BLOK_ERR_SHAPE, "wgemm rows: %d rows x %d columns over %d tokens is outside the streaming kernel",
               R, K, T);
  int nz = 1;
  if (int rc = launch_wgemm_stream(mode, r, &nz, stream)) return rc;
  return nz > 1 ? launch_wgemm_splitk_reduce(mode, r, nz, stream) : BLOK_OK;
}

}  // namespace blok
