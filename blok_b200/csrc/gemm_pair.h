// The TMA-fed GEMM over pairs of CTAs (gemm_pair.cu): what launch_gemm_tma hands to it.
#pragma once
#include "gemm_tma.h"

namespace blok {

bool gemm_pair_takes(const GemmTma &g);
int launch_gemm_pair(const GemmTma &g, cudaStream_t stream);
int gt_wide(const GemmTma &g);  // sixteen-byte stores of the output

}  // namespace blok
