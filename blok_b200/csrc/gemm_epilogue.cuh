// What the TMA-fed GEMM kernels (gemm_tma.cu, gemm_pair.cu) do with their sums.
#pragma once
#include "gemm_tma.h"
#include "tc_pipe.cuh"

namespace blok {

struct GtArgs {
  void *out;
  const int *tile_expert, *tile_start, *tile_count, *num_tiles;
  int T, R, K, ldo, act_cols, up_row;
  unsigned *err;
  int wide;  // bf16 rows start on 16 bytes and R is a multiple of 8: sixteen bytes a store
};

template <int ACT>
__device__ __forceinline__ float gt_act(float v) {
  if (ACT == GEMM_ACT_RELU2) {
    v = fmaxf(v, 0.f);
    return v * v;
  }
  if (ACT == GEMM_ACT_SILU) return __fdividef(v, 1.0f + __expf(-v));  // the result is rounded to bf16
  return v;
}

// Groups of four bf16 columns of one row from column `col` on, up to column R.
template <int N>
__device__ __forceinline__ void gt_store(const GtArgs &a, uint16_t *row, int col, const uint2 (&w)[N]) {
#pragma unroll
  for (int j = 0; j < N; j += 2) {
    if (a.wide) {
      if (col + 4 * j < a.R) *reinterpret_cast<uint4 *>(row + col + 4 * j) = make_uint4(w[j].x, w[j].y, w[j + 1].x, w[j + 1].y);
    } else {
      if (col + 4 * j < a.R) *reinterpret_cast<uint2 *>(row + col + 4 * j) = w[j];
      if (col + 4 * j + 4 < a.R) *reinterpret_cast<uint2 *>(row + col + 4 * j + 4) = w[j + 1];
    }
  }
}

// The epilogue of one warp (0..3) over its 32 lanes of an accumulator at tensor-memory column `tmem`: row (in the output with its part
// of a K split; stored if valid), BN columns from output column n0 on, half of them gate and half up for a gated product.
template <int BN, int ACT, bool F32>
__device__ __forceinline__ void gt_epilogue(const GtArgs &a, uint32_t tmem, int warp, size_t row, bool valid, int n0, bool failed) {
  constexpr bool kGated = ACT == GEMM_ACT_SWIGLU || ACT == GEMM_ACT_SWIGLU_REF;
  constexpr int kCols = kGated ? BN / 2 : BN;
  const size_t o = row * a.ldo;
  if constexpr (kGated) {
#pragma unroll 1
    for (int c0 = 0; c0 < kCols; c0 += 16) {
      if (n0 + c0 >= a.R) break;
      uint32_t gate[16], up[16];
      const uint32_t at = tmem + ((uint32_t)(32 * warp) << 16) + c0;
      tmem_ld16(at, gate);
      tmem_ld16(at + kCols, up);
      tmem_wait_ld();
      if (failed) {  // nothing that looks like a result
#pragma unroll
        for (int j = 0; j < 16; ++j) gate[j] = up[j] = 0x7fc00000u;
      }
      if (valid) {
        uint2 words[4];
#pragma unroll
        for (int j = 0; j < 16; j += 4) {
          const int col = n0 + c0 + j;
          if (col < a.R) {
            if (F32) {  // the parts of a K split
              *reinterpret_cast<uint4 *>(static_cast<float *>(a.out) + o + col) = make_uint4(gate[j], gate[j + 1], gate[j + 2], gate[j + 3]);
              *reinterpret_cast<uint4 *>(static_cast<float *>(a.out) + o + a.R + col) = make_uint4(up[j], up[j + 1], up[j + 2], up[j + 3]);
              continue;
            }
            float f[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              if (ACT == GEMM_ACT_SWIGLU_REF) {
                const float g = round_bf16(__uint_as_float(gate[j + i]));
                f[i] = round_bf16(g / (1.0f + expf(-g))) * round_bf16(__uint_as_float(up[j + i]));
              } else {
                f[i] = gt_act<GEMM_ACT_SILU>(__uint_as_float(gate[j + i])) * __uint_as_float(up[j + i]);
              }
            }
            words[j / 4] = make_uint2(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]));
          }
        }
        if (!F32) gt_store<4>(a, static_cast<uint16_t *>(a.out) + o, n0 + c0, words);
      }
    }
  } else {
#pragma unroll 1
    for (int c0 = 0; c0 < BN; c0 += 32) {
      if (n0 + c0 >= a.R) break;
      uint32_t v[32];
      tmem_ld32(tmem + ((uint32_t)(32 * warp) << 16) + c0, v);
      tmem_wait_ld();
      if (failed) {
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = 0x7fc00000u;
      }
      if (valid) {
        uint2 words[8];
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
          const int col = n0 + c0 + j;
          if (col < a.R) {  // R is a multiple of 4
            float f0 = __uint_as_float(v[j]), f1 = __uint_as_float(v[j + 1]), f2 = __uint_as_float(v[j + 2]), f3 = __uint_as_float(v[j + 3]);
            if (ACT != GEMM_ACT_SILU || col < a.act_cols) f0 = gt_act<ACT>(f0), f1 = gt_act<ACT>(f1), f2 = gt_act<ACT>(f2), f3 = gt_act<ACT>(f3);
            if (F32) *reinterpret_cast<float4 *>(static_cast<float *>(a.out) + o + col) = make_float4(f0, f1, f2, f3);
            else words[j / 4] = make_uint2(pack_bf16x2(f0, f1), pack_bf16x2(f2, f3));
          }
        }
        if (!F32) gt_store<8>(a, static_cast<uint16_t *>(a.out) + o, n0 + c0, words);
      }
    }
  }
}

}  // namespace blok
