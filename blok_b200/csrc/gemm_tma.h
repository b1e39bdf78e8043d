// bf16 GEMM on tcgen05 with TMA-fed operands (gemm_tma.cu): out[t, r] = act(sum_k x[t, k] W[r, k]), fp32 accumulation.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace blok {

// GEMM_ACT_SWIGLU_REF: the gated product with the reference's rounding points (both products, SiLU and the result to bf16).
enum { GEMM_ACT_NONE = 0, GEMM_ACT_RELU2 = 1, GEMM_ACT_SILU = 2, GEMM_ACT_SWIGLU = 3, GEMM_ACT_SWIGLU_REF = 4 };
constexpr int kGtTileRows = 128;  // rows of x per tile

// A 2-D tensor map: rows of `cols` elements, `pitch` bytes apart (a multiple of 16; base 16-byte aligned), copied in boxes
// of box_rows x box_cols; elements past the ends read as zeros.
int tensor_map_2d(const void *base, CUtensorMapDataType type, long rows, long cols, long pitch, int box_rows, int box_cols,
                  CUtensorMapSwizzle swizzle, CUtensorMap *out);

// A matrix operand: bf16 [rows, cols], rows `pitch` elements apart (pitch a multiple of 8, base 16-byte aligned).
// `box`: rows per copied box (128 for x, 128 or 256 for weights).
int gemm_operand_map(const void *base, long rows, int cols, long pitch, int box, CUtensorMap *out);

struct GemmTma {
  const CUtensorMap *x = nullptr;              // boxes of kGtTileRows rows
  const CUtensorMap *w128 = nullptr, *w256 = nullptr;  // the weights in boxes of 128 and of 256 rows
  const CUtensorMap *w64 = nullptr;            // and of 64 (more than 128 rows of x over few weight rows), or NULL
  int T = 0;                                   // rows of x
  int R = 0, K = 0;                            // weight rows (a multiple of 4) and columns (a multiple of 8)
  void *out = nullptr;                         // bf16 or fp32 [T, ldo]
  bool out_f32 = false;
  int ldo = 0;
  int act = GEMM_ACT_NONE;
  int act_cols = 0;                            // GEMM_ACT_SILU: the first so many columns (a multiple of 4) only; bf16 output
  // GEMM_ACT_SWIGLU: out[t, r] = silu(row r) * (row up_row + r), bf16 (R counts the outputs; the weights hold both halves)
  int up_row = 0;
  // GEMM_ACT_SWIGLU_REF: the up weights, a matrix of their own (w128: the gate weights)
  const CUtensorMap *up128 = nullptr;
  // > 1: K is cut into so many parts (grid.z), `out` is fp32 [splits][T][ldo] and holds the parts' sums (of both products, gate
  // columns then up columns, ldo = 2 R, for a gated product); no activation
  int splits = 1;
  // Set to 1 by a CTA whose wait gave up (its outputs are NaN); NULL: a word of the process, gemm_tma_take_error.
  unsigned *err = nullptr;
  // Grouped form: tile i covers rows [tile_start[i], + tile_count[i]) of x (at most kGtTileRows) and weight rows
  // [tile_expert[i] * R, + R); at most max_tiles tiles, *num_tiles of them valid.  NULL: consecutive tiles of one matrix.
  const int *tile_expert = nullptr, *tile_start = nullptr, *tile_count = nullptr, *num_tiles = nullptr;
  int max_tiles = 0;
};
int launch_gemm_tma(const GemmTma &g, cudaStream_t stream);
// *out becomes non-zero if a CTA has given up on a barrier since the last call (the flag is cleared).
int gemm_tma_take_error(unsigned *out);
int gemm_pair_take_error(unsigned *out);  // the same for the kernel that takes more than 128 rows

}  // namespace blok
