// bf16 GEMM over more than 128 rows of x with pairs of CTAs: out[t, r] = act(sum_k x[t, k] W[r, k]), as gemm_tma.cu.
//
// What bounds the one-CTA kernel is the way from L2 to the SM: a tile of 128 x 256 wants 48 KB per 64-column step, 512 cycles of the
// tensor pipe, at about 64 bytes a cycle (128 x 128: 32 KB for 256 cycles).  Here two SMs share a tile of 256 rows of x by BN weight
// rows (tcgen05.mma.cta_group::2): each CTA brings its 128 rows of x and half of the weight rows, 32 KB per 512 cycles, and the
// tensor cores read the halves from both.  One CTA per SM, persistent; two accumulators in tensor memory, so that a tile is
// stored while the next one is summed.
//
// Measured, one CTA per tile / pairs, us: 1,000 rows, gated product of 2 x 8,192 by 2,048 70 / 52 (1.3 PFLOP/s), 8,512 by 2,048 43 / 31,
// 2,048 by 8,192 49.5 / 41; a prompt of 130 / 1,000 / 2,040 tokens through four layers 966 / 1,340 / 2,090 -> 832 / 1,196 / 1,770 (with the
// K parts of sublayer_product and overlapped launches 517 / 956 / 1,600 since).  A step
// takes 0.41 us of the wide tile, 0.32 of the narrow one; over a whole launch the tensor pipe is 78 % busy (gated), 66 and 46 % (the other
// two), and 8.3 to 9.5 TB/s come from L2 to the SMs.
//
// Both CTAs' copies count on the leader's mbarrier (the copy's cta_group::2 form; no multicast); the leader's MMA warp issues for
// the pair, its commits free the slots of both.  A gated product's tile is 128 gate rows (the leader's half) and the up rows of the
// same outputs.  Tiles walk the rows of x first, so that CTAs at work share weight rows in L2.
//
// Every wait is bounded; a CTA that gives up records it and stores NaN; the pair meets before either leaves.
#include <algorithm>
#include <atomic>

#include "gemm_epilogue.cuh"
#include "gemm_pair.h"

namespace blok {

constexpr int kGpThreads = 192;  // warps 0..3: epilogue, 4: copies, 5: MMA (leader)
constexpr int kGpRows = 256;     // rows of x per tile
constexpr int kGpStep = 64;
constexpr uint32_t kGpABytes = 128 * kGpStep * 2;

template <int BN>
struct GpCfg {
  static constexpr uint32_t kBBytes = BN / 2 * kGpStep * 2, kStage = kGpABytes + kBBytes;
  static constexpr int kStages = BN == 256 ? 6 : 8;  // 192 KB
  static constexpr int kSmem = kStages * (int)kStage + 1024;
};

__device__ unsigned g_gemm_pair_error = 0;

__device__ __forceinline__ uint32_t gp_rank() {
  uint32_t r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// The address of this CTA's shared-memory word in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t gp_map(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void gp_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void gp_arrive_remote(uint32_t cluster_mbar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_mbar) : "memory");
}
// Like tp_load_2d, the mbarrier in either CTA of the pair.
__device__ __forceinline__ void gp_load_2d(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t cluster_mbar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
               "l"(map), "r"(x), "r"(y), "r"(cluster_mbar)
               : "memory");
}
// bf16 x bf16 -> fp32, M = 256 over the pair, both operands K-major.
__host__ __device__ constexpr uint32_t gp_idesc(int n) { return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((256u >> 4) << 24); }
__device__ __forceinline__ void gp_mma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t"
      "}\n" ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrives at the same mbarrier of both CTAs when the MMAs so far are done.
__device__ __forceinline__ void gp_commit(uint32_t mbar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(mbar), "h"((uint16_t)3)
               : "memory");
}
// tp_wait for a phase that the other CTA completes.
__device__ __forceinline__ bool gp_wait(uint32_t mbar, uint32_t parity) {
  for (unsigned it = 0; it < kTpSpinLimit; ++it) {
    uint32_t ok;
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t"
        "}\n"
        : "=r"(ok)
        : "r"(mbar), "r"(parity)
        : "memory");
    if (ok) return true;
    if (it > 64) __nanosleep(64);
  }
  return false;
}

struct GpTiles {
  int rows, cols, parts;  // tiles along x, along the weights, parts of K
};

template <int BN, int ACT, bool F32>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kGpThreads, 1)
    gemm_pair_kernel(const __grid_constant__ CUtensorMap mx, const __grid_constant__ CUtensorMap mw, const __grid_constant__ CUtensorMap mup,
                     const GtArgs a, const GpTiles tl) {
  using Cfg = GpCfg<BN>;
  constexpr int S = Cfg::kStages;
  constexpr bool kGated = ACT == GEMM_ACT_SWIGLU || ACT == GEMM_ACT_SWIGLU_REF;
  constexpr int kCols = kGated ? BN / 2 : BN;
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) unsigned long long s_bar[2 * S + 4];
  __shared__ uint32_t s_tmem;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t rank = gp_rank();
  const uint32_t sbase = ((uint32_t)__cvta_generic_to_shared(smem_raw) + 1023u) & ~1023u;
  const uint32_t full = (uint32_t)__cvta_generic_to_shared(&s_bar[0]), empty = full + 8 * S, dfull = full + 16 * S, dempty = dfull + 16;
  if (tid == 0) {
    for (int s = 0; s < S; ++s) {
      tp_mbar_init(full + 8 * s, 1);
      tp_mbar_init(empty + 8 * s, 1);
    }
    for (int i = 0; i < 2; ++i) {
      tp_mbar_init(dfull + 8 * i, 1);
      tp_mbar_init(dempty + 8 * i, 8);  // an arrival per epilogue warp of the pair
    }
    tp_mbar_init_fence();
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"((uint32_t)__cvta_generic_to_shared(&s_tmem)), "r"(2u * BN)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  gp_cluster_sync();
  tc_fence_after();
  const uint32_t tmem = s_tmem;
  pdl_wait();
  pdl_trigger();
  const int all_steps = (a.K + kGpStep - 1) / kGpStep;
  const int tiles = tl.rows * tl.cols * tl.parts, pairs = (int)gridDim.x / 2, pair = (int)blockIdx.x / 2;
  bool failed = false;

  if (warp == 4) {
    if (lane == 0) {
      int s = 0, issued = 0;
      uint32_t turn = 0;
      for (int t = pair; t < tiles && !failed; t += pairs) {
        const int m = t % tl.rows, n = t / tl.rows % tl.cols, z = t / (tl.rows * tl.cols);
        const int first = all_steps * z / tl.parts, nsteps = all_steps * (z + 1) / tl.parts - first;
        const int xrow = m * kGpRows + 128 * (int)rank;
        // this CTA's half of the tile's weight rows
        const int wrow = kGated ? (rank ? a.up_row : 0) + n * kCols : n * BN + (BN / 2) * (int)rank;
        const CUtensorMap *map = kGated && rank ? &mup : &mw;
        for (int c = 0; c < nsteps; ++c) {
          if (issued >= S && !gp_wait(empty + 8 * s, turn ^ 1)) {
            failed = true;
            break;
          }
          const uint32_t dst = sbase + (uint32_t)s * Cfg::kStage, bar = gp_map(full + 8 * s, 0);
          if (rank == 0) tp_expect_tx(full + 8 * s, 2 * Cfg::kStage);
          gp_load_2d(dst, &mx, (first + c) * kGpStep, xrow, bar);
          gp_load_2d(dst + kGpABytes, map, (first + c) * kGpStep, wrow, bar);
          ++issued;
          if (++s == S) s = 0, turn ^= 1;
        }
      }
      // no copy may be in flight and no commit on its way when the CTA leaves: the last use of every slot has been consumed
      for (int c = max(0, issued - S); c < issued; ++c) gp_wait(empty + 8 * (c % S), (uint32_t)((c / S) & 1));
    }
  } else if (warp == 5) {
    if (rank == 0) {
      // the whole warp walks the steps, so that addresses and descriptors stay warp-uniform; one lane issues
      const bool issues = tp_elect();
      int s = 0, buf = 0, used = 0;
      uint32_t turn = 0, dturn = 0;
      for (int t = pair; t < tiles && !failed; t += pairs) {
        const int z = t / (tl.rows * tl.cols);
        const int nsteps = all_steps * (z + 1) / tl.parts - all_steps * z / tl.parts;
        if (used >= 2 && !__all_sync(0xffffffffu, gp_wait(dempty + 8 * buf, dturn ^ 1))) {
          failed = true;
          break;
        }
        tc_fence_after();
        const uint32_t d = tmem + (uint32_t)(buf * BN);
        for (int c = 0; c < nsteps; ++c) {
          if (!__all_sync(0xffffffffu, gp_wait(full + 8 * s, turn))) {
            failed = true;
            break;
          }
          tc_fence_after();
          const uint64_t ad = tp_desc_k_sw128(sbase + (uint32_t)s * Cfg::kStage), bd = tp_desc_k_sw128(sbase + (uint32_t)s * Cfg::kStage + kGpABytes);
          if (issues) {
#pragma unroll
            for (int k = 0; k < kGpStep / 16; ++k) gp_mma(d, ad + (uint64_t)(2 * k), bd + (uint64_t)(2 * k), gp_idesc(BN), (c | k) ? 1u : 0u);
            gp_commit(empty + 8 * s);
            if (c == nsteps - 1) gp_commit(dfull + 8 * buf);
          }
          __syncwarp();
          if (++s == S) s = 0, turn ^= 1;
        }
        ++used;
        if (++buf == 2) buf = 0, dturn ^= 1;
      }
    }
  } else {
    int buf = 0;
    uint32_t turn = 0;
    for (int t = pair; t < tiles; t += pairs) {
      const int m = t % tl.rows, n = t / tl.rows % tl.cols, z = t / (tl.rows * tl.cols);
      if (!failed) failed = !__all_sync(0xffffffffu, gp_wait(dfull + 8 * buf, turn));
      tc_fence_after();
      const int r = m * kGpRows + 128 * (int)rank + 32 * warp + lane;
      gt_epilogue<BN, ACT, F32>(a, tmem + (uint32_t)(buf * BN), warp, (size_t)z * a.T + r, r < a.T, n * kCols, failed);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) gp_arrive_remote(gp_map(dempty + 8 * buf, 0));
      if (++buf == 2) buf = 0, turn ^= 1;
    }
  }
  if (failed) atomicExch(a.err ? a.err : &g_gemm_pair_error, 1u);
  tc_fence_before();
  __syncthreads();
  gp_cluster_sync();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2u * BN) : "memory");
}

// Rows past the first 128: below that half of every pair would have nothing to do.  Against the one-CTA kernel, us, weights in L2 / from HBM:
//  - few columns are mostly the stores of a tile's sums, which 256 x 256 outputs make once per pair and 128 x 128 in smaller pieces:
//    gated, 2 x 8,192 by 256 over 1,000 rows 25 / 31 here, 21 / 27 there; 1,024 by 256 (fp32) over 513 rows 7.4 / 12.2, 8.7 / 10.2.  At 512
//    columns the launch's own ramp, hidden behind the kernel before, decides: geometric mean over 200 products 0.93 / 1.03 of the other.
//  - rows that leave half of the last tile empty, among three tiles or fewer, cost a fifth or more of the products: 4,096 and 8,192 by 512
//    over 513 rows 12.5 / 17.2 and 19 / 24.6 here, 10.7 / 14.3 and 14.9 / 20.5 there; by 2,048 they are even.
//  - with a few tiles only the one-CTA kernel is 4 to 11 % faster from L2 (64 by 8,192: 33.3 / 37.0), and 20 % slower from HBM.
bool gemm_pair_takes(const GemmTma &g) {
  if (g.tile_start || g.T <= 128 || g.K < 512) return false;
  const bool gated = g.act == GEMM_ACT_SWIGLU || g.act == GEMM_ACT_SWIGLU_REF;
  const long row_tiles = (g.T + kGpRows - 1) / kGpRows, tiles = row_tiles * (((gated ? 2 * g.R : g.R) + 255) / 256);
  const bool half_empty = (g.T - 1) % kGpRows < 128 && (row_tiles == 2 || row_tiles == 3);
  return !(half_empty && g.K < 2048 && tiles > sm_count() / 4);
}

// Pairs of SMs that hold a pair of CTAs at once (an odd SM of a GPC has no partner): a persistent grid must not be larger.
template <int BN, int ACT, bool F32>
static int gp_pairs(int *out) {
  static std::atomic<int> known{0};
  if (!known.load()) {
    auto kernel = gemm_pair_kernel<BN, ACT, F32>;
    if (int rc = allow_smem(kernel, GpCfg<BN>::kSmem)) return rc;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = sm_count() / 2 * 2;
    cfg.blockDim = kGpThreads;
    cfg.dynamicSmemBytes = GpCfg<BN>::kSmem;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    BLOK_CUDA(cudaOccupancyMaxActiveClusters(&n, kernel, &cfg));
    known = std::max(1, std::min(n, sm_count() / 2));
  }
  *out = known.load();
  return BLOK_OK;
}

template <int BN, int ACT, bool F32>
static int gp_launch(const GemmTma &g, cudaStream_t stream) {
  constexpr bool kGated = ACT == GEMM_ACT_SWIGLU || ACT == GEMM_ACT_SWIGLU_REF;
  const GtArgs a = {g.out, nullptr, nullptr, nullptr, nullptr, g.T, g.R, g.K, g.ldo, g.act_cols, g.up_row, g.err, gt_wide(g)};
  GpTiles tl;
  tl.rows = (g.T + kGpRows - 1) / kGpRows;
  tl.cols = (g.R + (kGated ? BN / 2 : BN) - 1) / (kGated ? BN / 2 : BN);
  tl.parts = g.splits;
  int pairs = 1;
  if (int rc = gp_pairs<BN, ACT, F32>(&pairs)) return rc;
  pairs = std::min(tl.rows * tl.cols * tl.parts, pairs);
  auto kernel = gemm_pair_kernel<BN, ACT, F32>;
  if (int rc = allow_smem(kernel, GpCfg<BN>::kSmem)) return rc;
  const CUtensorMap &w = BN == 128 && !kGated ? *g.w64 : *g.w128;
  return launch_pdl("gemm_pair_kernel", kernel, 2 * pairs, kGpThreads, (size_t)GpCfg<BN>::kSmem, stream, *g.x, w, g.up128 ? *g.up128 : *g.w128, a, tl);
}

int launch_gemm_pair(const GemmTma &g, cudaStream_t stream) {
  if (g.act == GEMM_ACT_SWIGLU_REF) {
    BLOK_REQUIRE(g.up128 && (g.splits > 1) == g.out_f32, BLOK_ERR_SHAPE, "gemm: a gated product is bf16 and not grouped");
    return g.out_f32 ? gp_launch<256, GEMM_ACT_SWIGLU_REF, true>(g, stream) : gp_launch<256, GEMM_ACT_SWIGLU_REF, false>(g, stream);
  }
  if (g.act == GEMM_ACT_SWIGLU) {
    BLOK_REQUIRE(!g.out_f32, BLOK_ERR_SHAPE, "gemm: a gated product is bf16 and not grouped");
    return gp_launch<256, GEMM_ACT_SWIGLU, false>(g, stream);
  }
  // The wide tile costs 512 cycles a step, the narrow one about 390 (its 24 KB set the time): whichever leaves fewer of them to
  // the pair with most
  const long rows = (g.T + kGpRows - 1) / kGpRows, pairs = sm_count() / 2;
  const long wide = (rows * ((g.R + 255) / 256) * g.splits + pairs - 1) / pairs * 512, narrow = (rows * ((g.R + 127) / 128) * g.splits + pairs - 1) / pairs * 390;
  const bool use256 = !g.w64 || wide <= narrow;
  if (g.act == GEMM_ACT_SILU) {
    BLOK_REQUIRE(!g.out_f32 && g.act_cols % 4 == 0, BLOK_ERR_SHAPE, "gemm: SiLU on %d columns of an fp32 output", g.act_cols);
    return use256 ? gp_launch<256, GEMM_ACT_SILU, false>(g, stream) : gp_launch<128, GEMM_ACT_SILU, false>(g, stream);
  }
#define BLOK_GP(BN)                                                                             \
  return g.act == GEMM_ACT_RELU2 ? (g.out_f32 ? gp_launch<BN, GEMM_ACT_RELU2, true>(g, stream)   \
                                              : gp_launch<BN, GEMM_ACT_RELU2, false>(g, stream)) \
                                 : (g.out_f32 ? gp_launch<BN, GEMM_ACT_NONE, true>(g, stream)    \
                                              : gp_launch<BN, GEMM_ACT_NONE, false>(g, stream));
  if (use256) {
    BLOK_GP(256)
  }
  BLOK_GP(128)
#undef BLOK_GP
}

int gemm_pair_take_error(unsigned *out) {
  unsigned zero = 0;
  BLOK_CUDA(cudaMemcpyFromSymbol(out, g_gemm_pair_error, sizeof(unsigned)));
  if (*out) BLOK_CUDA(cudaMemcpyToSymbol(g_gemm_pair_error, &zero, sizeof(unsigned)));
  return BLOK_OK;
}

}  // namespace blok
