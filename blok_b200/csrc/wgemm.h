// Products of several tokens with bf16 or INT4 weights: which kernel takes a launch (wgemm.cu) and the kernels (wgemm.cu, wgemm_stream.cu,
// wgemm_tc.cu, wgemv_small.cu).
#pragma once
#include <cuda_runtime.h>
#include <cstddef>
#include <cstdint>

namespace blok {

enum { WG_BF16_PLAIN = 0, WG_BF16_SWIGLU = 1, WG_I4_SWIGLU = 2, WG_I4_PLAIN = 3 };
constexpr int kWgTileTokens = 64;
constexpr int kWgStreamTokens = 64;  // bf16 weights over up to this many rows take the weight-streaming kernel (wgemm_stream.cu)
// Grouped INT4 products of up to this many assignments take the mat-vec-style kernel (wgemv_small.cu: four tokens per pass),
// more take the tcgen05 kernel
constexpr int kWgSmallRows = 40;

struct WgArgs {
  const void *w_a;
  const void *w_b;
  const uint16_t *s_a;
  const uint16_t *s_b;
  long expert_stride_rows;
  const uint16_t *x;
  const int *x_index;
  int K;
  int R;
  uint16_t *out_bf16;
  float *out_f32;
  const int *tile_expert;
  const int *tile_start;
  const int *tile_count;
  const int *num_tiles;
  const int *out_index;
  int identity_tiles = 0;  // the tiles are consecutive 64-row blocks of x (one group: a dense layer over n_rows tokens)
  int n_rows = 0;  // rows of x the launch covers (tokens, or token-expert assignments): picks the kernel
  // bf16 modes over identity tiles: scratch for the K-split partial sums, see wgemm_splitk_bytes; NULL: no split
  float *splitk_ws = nullptr;
  size_t splitk_bytes = 0;
  // INT4 modes, where the host knows only a bound of them: the assignments that pick the kernel, a device word (launch_wgemm_experts)
  const int *total = nullptr;
  // The weight-streaming kernel only.  keep_sums: fp32 sums in splitk_ws also where K is not split, for a kernel of the caller's that
  // takes them.  A second matrix over the same rows (w_2, R2 rows; with keep_sums): its tiles follow the first's, its sums the first's
  // columns.  max_splits: a bound of the K split (0: none).  weights_early: the weights may be fetched before the kernels in front of
  // this launch have finished (the caller has launched one since they were written, in this call).
  const void *w_2 = nullptr;
  int R2 = 0, max_splits = 0;
  bool keep_sums = false, weights_early = false;
  // INT4 modes: the launches become resident while the ones before them run.  For few tokens, where they are short: layers of 3, 64 (2048 x
  // 1024, 128 experts) and 6 (7168 x 2048) tokens 59 -> 56, 139 -> 130, 259 -> 254 us; over 2,048 tokens 1 to 2 % slower (blocks that come
  // early hold registers that the many blocks of the layout and the combination want).
  bool overlap = false;
  unsigned *err = nullptr;  // set to 1 when a tcgen05 kernel's wait gives up: a word of the handle the launch is for
};

// Picks the kernel of a launch.  INT4 modes: the mma.sync kernel (see launch_wgemm_experts for the others).  bf16 modes: up to
// kWgStreamTokens rows of a dense product the weight-streaming kernel (wgemm_stream.cu); more, the TMA-fed tcgen05 GEMM
// (gemm_tma.cu; over more than 128 rows gemm_pair.cu), K split where its tiles are few; for shapes the others do not cover the mma.sync kernel with its K-split.
// BLOK_WGEMM_IMPL=mma / =tc in the environment forces one GEMM kernel for every row (no small-group or streaming kernel).
int launch_wgemm(int mode, const WgArgs &args, int max_tiles, cudaStream_t stream);
int wgemm_forced_impl();  // 0: none forced

// A bf16 product over few tiles of tokens has (R / 128 or R / 64) x tiles CTAs, far fewer than the GPU has SMs (3 per
// tile for a 384-expert router): the mma.sync kernel then splits K over blockIdx.z so that about two CTAs per SM run,
// writes fp32 partial sums to args.splitk_ws and a second kernel adds them in split order and applies the epilogue.
// The factor depends on the launch's shape (mode, K, R, number of token tiles), so two launches of the same shape give
// the same bits.  wgemm_splitk_bytes: the scratch that serves every launch of up to max_rows rows.
int wgemm_splitk_factor(int mode, int K, int R, int tiles);
size_t wgemm_splitk_bytes(int mode, int K, int R, int max_rows);
int wgemm_tma_split(int mode, int K, int R, int rows);  // the same for the TMA-fed GEMM

// The INT4 modes over few assignments: streams the weights like the batch-1 decode kernel (BLOK_WGEMM_SMALL=0 in the
// environment: through the GEMM kernels as well).
bool wgemv_small_supports(int mode, const WgArgs &args, int max_rows);
int launch_wgemv_small(int mode, const WgArgs &args, cudaStream_t stream);

// The bf16 modes over 1..kWgStreamTokens rows of x (identity tiles): the weights streamed by TMA as the M side of tcgen05.mma
// (wgemm_stream.cu).  *splits > 1: K was split and the partial sums wait in args.splitk_ws for wgemm_splitk_reduce_kernel
// (launch_wgemm runs it) or a kernel that adds them itself.  wgemm_stream_split, _pair_split: the split of a shape at most.
// wgemm_stream_supports: what launch_wgemm hands to it; the launch itself takes any K % 8 == 0 and R.
bool wgemm_stream_supports(int mode, const WgArgs &args);
int wgemm_stream_split(int mode, int K, int R);
int wgemm_stream_pair_split(int mode, int K, int R, int R2);
// Matrices with a tile for every SM: up to 8 rows of x too go through it rather than the mat-vec kernels (bf16_kernels.cu), which
// spend an instruction on every 16 bytes.  One row, 2 x 18,432 gated rows of 7,168 (528 MB) 93 us and 77, 32,768 (470 MB) 92 and 75.
bool wgemm_stream_takes_few(int mode, const WgArgs &args);
// Fewer tiles, K in parts; room: bytes for their sums.
bool wgemm_stream_takes_parts(int mode, const WgArgs &args, size_t room);
// *out becomes non-zero if a CTA without an error word of its own has given up since the last call (the flag is cleared).
int wgemm_stream_take_error(unsigned *out);
int wgemm_stream_set_error(unsigned code);  // for tests
// The reduction behind a K-split launch: adds the nz partial sums in split order and applies the epilogue.
int launch_wgemm_splitk_reduce(int mode, const WgArgs &args, int nz, cudaStream_t stream);
int launch_wgemm_stream(int mode, const WgArgs &args, int *splits, cudaStream_t stream);
// One dense product through launch_wgemm without tile tables: out[T, R] = W[R, K] x[T, K] (mode WG_BF16_PLAIN; bf16 or
// fp32 output) or the SwiGLU front half of (w_a = gate, w_b = up) (mode WG_BF16_SWIGLU), for 1 <= T <= kWgStreamTokens.
int launch_wgemm_rows(int mode, const void *w_a, const void *w_b, const uint16_t *x, uint16_t *out_bf16, float *out_f32, int R, int K,
                      int T, float *splitk_ws, size_t splitk_bytes, cudaStream_t stream, bool weights_early = false, unsigned *err = nullptr);
WgArgs wgemm_rows(const void *w_a, const void *w_b, const uint16_t *x, uint16_t *out_bf16, float *out_f32, int R, int K, int T);  // its launch

// Both products of the grouped experts, INT4: mid = SwiGLU front half of x (up: WG_I4_SWIGLU), then the down projection
// (down: WG_I4_PLAIN, its x is up's output).  Up to kWgSmallRows rows through the mat-vec-style kernel (wgemv_small.cu), else
// through the tcgen05 kernel (wgemm_tc.cu) where it covers the shapes; else, or with BLOK_WGEMM_IMPL=mma, launch_wgemm twice.
// With up.total both kernels are launched and the word decides on the device (the other one leaves at once).  xs: scratch of
// `rows` x up.K values, where `rows` is the number of sorted positions that up.out_bf16 and xs hold (it may be the buffer of
// down's output).
int launch_wgemm_experts(const WgArgs &up, const WgArgs &down, uint16_t *xs, long rows, int max_tiles, cudaStream_t stream);
bool wgemm_i4_supports(const WgArgs &up, const WgArgs &down);
int launch_wgemm_i4(const WgArgs &up, const WgArgs &down, uint16_t *xs, long rows, int max_tiles, cudaStream_t stream);

}  // namespace blok
