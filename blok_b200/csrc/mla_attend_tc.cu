// The attention core of absorbed MLA decode on the 5th-generation tensor cores (tcgen05, accumulators in tensor
// memory), its cache tiles brought in by TMA: one pass over the bf16 latent cache with an online softmax, split over
// the sequence (flash-decoding).  Replaces attn_tile_score_k / max / sum / accum (src/kimi_exec.cu:414-475) and the
// three-pass tiled_attention (:692-716).  Same interface and partial results as mla_attend_kernel (mla_attend.cu),
// which stays as the fallback.
//
// All 64 heads of a sequence share one latent row per token: per token 1,152 bytes are read once from HBM and feed
// 64 x (576 + 512) multiply-adds.  A CTA walks its share of the batch, a range of tokens of one sequence after another's
// (mla_plan.cuh; FINE: of one sequence), in tiles of 64 tokens:
//
//   S [heads x tokens]     = Q [heads x 576] . C^T          36 MMAs M64 N64 K16: A = Q (shared memory, as a tile lies),
//                                                            B = the tile read K-major; two partial sums
//   P = exp2(S * scale * log2 e - m)                         a quad of lanes per pair of head rows, bf16, to shared memory
//   O^T [latent x heads]  += C^T [latent x tokens] . P^T     16 MMAs M128 N64 K16: A = the SAME tile bytes read MN-major
//                                                            (four blocks of 128 latent columns), B = P (K-major)
//
// A tile lies in shared memory as nine chunks of [64 tokens x 128 bytes] in the 128-byte swizzle, each written by one
// cp.async.bulk.tensor (no multicast; the tensor map covers this GPU's cache only).  Read K-major a chunk is 64 columns
// of a [64 tokens x 576] operand; read MN-major the same bytes are 64 rows of a [512 x 64 tokens] operand: one copy from
// HBM serves both products, and no thread touches the bytes on their way.
//
// What bounds it: the chain load -> scores -> softmax -> P.C of a tile with two tile buffers beside Q, and in it the fixed cost of
// an MMA of this size, about 40 cycles for the warp that issues it (43 with N = 32, 61 with N = 64; so tiles of 32 tokens in four
// buffers are slower, 131 against 126 us below).  So two warps issue; a tile is loaded and released in two halves, its scores
// begin with the first; whichever product can go next goes; and all 32 lanes of a softmax warp work.  A tile took 2.83 us, takes
// 1.92 (8 x 32,768 tokens: the block 147 -> 126 us; 33 paged sequences 140 -> 122; HBM's share of an SM would be 1.67 us).
//
// The running maximum is kept lazily: a head's reference m changes only when a tile's maximum exceeds it by more than
// 40 (natural units); then all four consumer warps rescale O^T in tensor memory.  exp(s - m) stays far inside fp32 and
// bf16 range meanwhile, and the merge over the splits needs a consistent (m, sum, O) only.
//
// FINE: the weights enter the second product as two bf16 parts, high and low (17 bits of each weight; the sum of the weights
// is fp32), for models whose attention weights are fp32.  The low part needs no shared memory of its own: a tile's chunk of
// rope columns is read by the score product only, so once the tile's scores have been taken the low parts go there, and
// the tile's release frees both.  seq_len then holds positions (the token itself included).  Any number of heads in groups of 64 (blockIdx.z).
//
// Warps: 0..3 consumers (the M = 64 accumulator S keeps head rows 16 w .. 16 w + 15 in lanes 0..15 of warp w's quarter of
// tensor memory; all four own the 128 lanes of O^T), 4: the TMA producer, 5 and 6: one lane of each issues the MMAs.  Every mbarrier
// wait is bounded; on a timeout the CTA records an error, still releases its tensor memory and returns.
#include <cuda.h>

#include <mutex>

#include "common.cuh"
#include "gemm_tma.h"
#include "mla_plan.cuh"
#include "tmem_io.cuh"

namespace blok {

constexpr int kTaHeads = 64, kTaD = 576, kTaDV = 512;
constexpr int kTaTile = 64;                              // tokens per tile
constexpr int kTaChunks = kTaD / 64;                     // 128-byte column chunks of a cache row
constexpr int kTaChunkBytes = kTaTile * 128;             // 8,192
constexpr int kTaHalfChunks = 4;                         // chunks of a tile's first half (latent columns 0..255)
constexpr int kTaTileBytes = kTaChunks * kTaChunkBytes;  // 73,728
constexpr int kTaLbo = kTaHeads * 16;                    // P (64 rows, no swizzle): bytes between 16-byte column groups
constexpr int kTaSbo = 128;                              // ... and between 8-row groups
constexpr int kTaQBytes = kTaChunks * kTaHeads * 128;    // 73,728
constexpr int kTaPBytes = (kTaTile / 8) * kTaLbo;        // P: [64 heads x 64 tokens] bf16, K (token) major
constexpr int kTaSmemBytes = 2 * kTaTileBytes + kTaQBytes + kTaPBytes + 1024;  // + 1024: the tiles start on a 1,024-byte boundary
constexpr int kTaConsumers = 128;
constexpr int kTaThreads = kTaConsumers + 96;
constexpr int kTaTmemCols = 512;                         // S: 2 buffers x 2 partial sums x 64 columns, O^T: 4 x 64 columns
constexpr int kTaColO = 256;
constexpr unsigned kTaSpinLimit = 1u << 21;
constexpr float kTaLazy = 57.7f;                         // 40 natural units in the log2 domain
constexpr int kTaTraceTiles = 64;

__device__ unsigned g_mla_tc_error = 0;

__device__ __forceinline__ float ta_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// bf16 pair (hi in the upper half), both rounded to nearest even
__device__ __forceinline__ uint32_t ta_pack_bf16x2(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
// True in one lane of a converged warp.
__device__ __forceinline__ bool ta_elect() {
  uint32_t is;
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t"
      "}\n"
      : "=r"(is));
  return is != 0;
}
// Shared-memory matrix descriptors (start address, leading and stride byte offsets in 16-byte units, version 1).
// No swizzle, K-major (P): leading = between 16-byte column groups along K, stride = between 8-row groups.
__device__ __forceinline__ uint64_t ta_desc_plain(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) | (1ull << 46);
}
// 128-byte swizzle (layout type 2).  K-major: rows of 128 bytes, stride = 1,024 between 8-row groups, leading unused
// (1); a K = 16 step inside the 128-byte row advances the start address by 32 bytes.  MN-major: 64 contiguous
// elements along M, leading = between 64-element chunks along M, stride = 1,024 between 8-row groups along K.
__device__ __forceinline__ uint64_t ta_desc_sw128(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void ta_mma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t"
      "}\n" ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void ta_commit(uint32_t mbar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
}
__device__ __forceinline__ void ta_arrive(uint32_t mbar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(mbar) : "memory");
}
__device__ __forceinline__ void ta_expect_tx(uint32_t mbar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar), "r"(bytes) : "memory");
}
// One box of the 2-D tensor map (x: column in elements, a multiple of 64; y: cache row) into shared memory; the bytes
// are counted on the mbarrier.
__device__ __forceinline__ void ta_tma_2d(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t mbar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
               "l"(map), "r"(x), "r"(y), "r"(mbar)
               : "memory");
}
__device__ __forceinline__ bool ta_test(uint32_t mbar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t"
      "}\n"
      : "=r"(ok)
      : "r"(mbar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait for the given phase parity; false (and the error word set) on a timeout.
__device__ __forceinline__ bool ta_wait(uint32_t mbar, uint32_t parity, unsigned code) {
  for (unsigned it = 0; it < kTaSpinLimit; ++it) {
    uint32_t ok;
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t"
        "}\n"
        : "=r"(ok)
        : "r"(mbar), "r"(parity)
        : "memory");
    if (ok) return true;
    __nanosleep(64);
  }
  atomicExch(&g_mla_tc_error, code);
  return false;
}
// Barrier of the 128 consumer threads that also ORs their failure flags: after a timeout all of them leave together.
__device__ __forceinline__ bool ta_consumers_sync(bool failed) {
  uint32_t any;
  asm volatile(
      "{\n\t"
      ".reg .pred p, q;\n\t"
      "setp.ne.u32 q, %1, 0;\n\t"
      "bar.red.or.pred p, 1, %2, q;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t"
      "}\n"
      : "=r"(any)
      : "r"((uint32_t)failed), "n"(kTaConsumers)
      : "memory");
  return any != 0;
}

size_t mla_attend_tc_smem_bytes() { return kTaSmemBytes; }

// Arguments as mla_attend_kernel, plus the tensor maps of the cache ([rows, 576] bf16) and of the queries ([B x heads, 576]), both in
// boxes of 64 rows x 64 columns, 128-byte swizzle.  PAGED: page_rows is a multiple of the 64-token tile.  planned > 0: so many
// sequences, shared out over a one-dimensional grid as mla_plan.cuh says (plan: made by a kernel before this one; NULL: made here, and
// CTA 0 leaves each sequence's partial results in parts); planned = 0: grid = (splits, B, groups of heads), every sequence in `splits` equal parts.
template <bool PAGED, bool FINE>
__global__ void __launch_bounds__(kTaThreads, 1)
    mla_attend_tc_kernel(const __grid_constant__ CUtensorMap tmap, const __grid_constant__ CUtensorMap qmap, const uint16_t *cache,
                         long ctx_stride, const int *seq_len, float scale, float *__restrict__ part_o,
                         float *__restrict__ part_ml, const int *block_table, const int *slot_of,
                         int table_stride, int page_rows, long long *__restrict__ trace, int heads, int planned,
                         const MlaPlan *plan, int2 *__restrict__ parts) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) unsigned long long s_bar[16];
  __shared__ uint32_t s_tmem;
  __shared__ float s_alpha[kTaHeads];
  __shared__ int s_need[2][4];
  __shared__ MlaPlan s_plan;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // the swizzle is a function of the address: the tiles start on a 1,024-byte boundary
  const uint32_t raw = (uint32_t)__cvta_generic_to_shared(smem_raw);
  const uint32_t sT = (raw + 1023u) & ~1023u;
  unsigned char *smem = smem_raw + (sT - raw);
  const uint32_t sQ = sT + 2 * kTaTileBytes;
  const uint32_t sP = sQ + kTaQBytes;
  unsigned char *Pp = smem + 2 * kTaTileBytes + kTaQBytes;
  const uint32_t bar0 = (uint32_t)__cvta_generic_to_shared(&s_bar[0]);
  // A tile comes and goes in two halves: chunks 0..3 (latent columns 0..255) and 4..8.  tma[buf][half]: the half's bytes have
  // landed; fix[buf]: the rows past the sequence's end are zeroed (its last tile only); sfull[buf]: the S MMAs' commits, one of each
  // MMA warp; sfree[buf]: the softmax warps have read S; pfull: they have written P; empty[buf][half]: the commit behind the P.C
  // MMAs of the half's columns (the half of the buffer is free, with both halves P too); q: the queries have landed
  const uint32_t bar_tma = bar0, bar_fix = bar0 + 32, bar_sfull = bar0 + 48, bar_sfree = bar0 + 64, bar_empty = bar0 + 80, bar_pfull = bar0 + 112,
                 bar_q = bar0 + 120;
  if (tid == 0) {
    for (int i = 0; i < 16; ++i)  // sfree and pfull: an arrival per softmax warp
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar0 + 8 * i), "r"(i == 8 || i == 9 || i == 14 ? 4 : (i == 6 || i == 7 ? 2 : 1)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"((uint32_t)__cvta_generic_to_shared(&s_tmem)),
                 "r"((uint32_t)kTaTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (plan) {  // made by a kernel that had finished before the one in front of this launch let it begin; a word a thread
    static_assert(sizeof(MlaPlan) / sizeof(int) <= kTaThreads, "a word of the plan to a thread");
    if (tid < (int)(sizeof(MlaPlan) / sizeof(int))) reinterpret_cast<int *>(&s_plan)[tid] = reinterpret_cast<const int *>(plan)[tid];
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s_tmem;
  pdl_wait();
  pdl_trigger();  // after the wait: the kernel behind this one may read what was there before this one, the plan's parts
  const int h0 = blockIdx.z * kTaHeads, nh = min(kTaHeads, heads - h0);  // this CTA's heads
  auto length = [&](int b) { return FINE ? min(seq_len[b] + 1, table_stride * page_rows) : seq_len[b]; };
  if (planned && !plan) {
    if (warp == 0) {
      mla_plan(s_plan, planned, gridDim.x, length);
      if (blockIdx.x == 0)
        for (int b = lane; b < planned; b += 32) parts[b] = mla_plan_parts(s_plan, b);
    }
    __syncthreads();
  }
  // The CTA's segments in order: nt tiles of sequence b from tile ts on, partial result `slot`; `partial`: the last of them holds
  // rows past the sequence's end.
  struct Segment {
    int b, ts, nt, slot, seq;
    bool partial;
  };
  const int lo = planned ? (int)blockIdx.x * s_plan.per : 0, hi = planned ? lo + s_plan.per : 0;
  int b_first = 0;  // the first sequence that ends behind the piece's begin
  if (planned) {
    b_first = __popc(__ballot_sync(0xffffffffu, lane < planned && s_plan.start[lane + 1] <= lo)) +
              __popc(__ballot_sync(0xffffffffu, lane + 32 < planned && s_plan.start[lane + 33] <= lo));
  }
  auto segment = [&](int &next, Segment &g) -> bool {
    if (planned) {
      for (; next < planned && s_plan.start[next] < hi; ++next) {
        const int tile0 = s_plan.start[next] + s_plan.lead, ntiles = (s_plan.tokens[next] + kTaTile - 1) / kTaTile;
        const int t0 = max(lo - tile0, 0), t1 = min(hi - tile0, ntiles);
        if (t1 <= t0) continue;
        g.b = next, g.ts = t0, g.nt = t1 - t0, g.slot = (int)blockIdx.x + next, g.seq = s_plan.tokens[next];
        g.partial = g.seq % kTaTile != 0 && ntiles == t1;
        ++next;
        return true;
      }
      return false;
    }
    if (next > 0) return false;
    next = 1;
    const int split = blockIdx.x, splits = gridDim.x;
    g.b = blockIdx.y, g.slot = g.b * splits + split, g.seq = length(g.b);
    const int ntiles = (g.seq + kTaTile - 1) / kTaTile, per = (ntiles + splits - 1) / splits;
    g.ts = split * per, g.nt = max(0, min(ntiles, g.ts + per) - g.ts);
    g.partial = g.seq % kTaTile != 0 && g.ts + g.nt == ntiles;
    if (g.nt == 0 && tid < nh) {  // nothing to do for this split: mark it empty for the merge
      float *ml = part_ml + ((size_t)g.slot * heads + h0) * 2;
      ml[tid * 2] = -INFINITY;
      ml[tid * 2 + 1] = 0.f;
    }
    return g.nt > 0;
  };
  bool failed = false;
  // diagnostics (trace != NULL): CTA (0, 0) stamps, per tile, [0] buffer free, [1] TMA issued, [2] S issued, [3] S seen
  // by the softmax warps, [4] P handed over, [5] P.C issued, [8] S read, [9] softmax done (nanoseconds)
  auto stamp = [&](int n, int slot) {
    if (trace && blockIdx.x == 0 && blockIdx.y == 0 && n < kTaTraceTiles) {
      long long t;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
      trace[n * 16 + slot] = t;
    }
  };
  Segment g;
  int next_b = b_first;

  if (warp == 4) {
    // ---- the producer: nine boxes for the queries, nine per tile, counted on the mbarrier of their half ----
    int issued = 0, at = 0;  // halves asked for, tile of the CTA
    for (int sg = 0; !failed && segment(next_b, g); ++sg) {
      const uint16_t *cache_b = PAGED ? cache : cache + (size_t)g.b * ctx_stride * kTaD;
      const int *table_b = PAGED ? block_table + (size_t)(slot_of ? slot_of[g.b] : g.b) * table_stride : nullptr;
      auto first_row = [&](int tok0) -> long {  // the tensor map's row of the tile's first token
        if (PAGED) return (long)table_b[tok0 / page_rows] * page_rows + tok0 % page_rows;
        return (long)g.b * ctx_stride + tok0;
      };
      // the queries of the segment before are free behind its last scores
      if (at > 0 && !__all_sync(0xffffffffu, ta_wait(bar_sfull + 8 * ((at - 1) & 1), (uint32_t)(((at - 1) >> 1) & 1), 12u))) {
        failed = true;
        break;
      }
      if (lane == 0) {
        ta_expect_tx(bar_q, kTaQBytes);
#pragma unroll 1
        for (int c = 0; c < kTaChunks; ++c) ta_tma_2d(sQ + c * kTaChunkBytes, &qmap, 64 * c, g.b * heads + h0, bar_q);
      }
      for (int n = 0; n < g.nt; ++n, ++at) {
        const int buf = at & 1;
        const int tok0 = (g.ts + n) * kTaTile, row = (int)first_row(tok0);
        const uint32_t dst = sT + buf * kTaTileBytes;
#pragma unroll 1
        for (int half = 0; half < 2; ++half) {
          // (the second half also holds FINE's low parts, which both warps read; it comes after the first)
          if (at >= 2 && !__all_sync(0xffffffffu, ta_wait(bar_empty + 16 * buf + 8 * half, (uint32_t)(((at >> 1) - 1) & 1), 1u))) {
            failed = true;
            break;
          }
          if (lane == 0) {
            if (half == 0) stamp(at, 0);
            const int c0 = half ? kTaHalfChunks : 0, c1 = half ? kTaChunks : kTaHalfChunks;
            const uint32_t bar = bar_tma + 16 * buf + 8 * half;
            ta_expect_tx(bar, (uint32_t)(c1 - c0) * kTaChunkBytes);
#pragma unroll 1
            for (int c = c0; c < c1; ++c) ta_tma_2d(dst + c * kTaChunkBytes, &tmap, 64 * c, row, bar);
          }
          issued = 2 * at + half + 1;
        }
        if (failed) break;
        if (lane == 0) {
          if (n + 2 < g.nt) {
            // The buffer's next tile starts its way from HBM to L2 now: by the time the buffer is free again (this
            // tile's two products later) the copy finds it there, and HBM has been busy meanwhile.  A tile is contiguous
            // (dense cache, or inside a page); only rows of the sequence are touched.
            const int ptok = tok0 + 2 * kTaTile;
            const int prow = min(kTaTile, g.seq - ptok);
            const uint16_t *pp = PAGED ? cache + (size_t)first_row(ptok) * kTaD : cache_b + (size_t)ptok * kTaD;
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(pp), "r"((uint32_t)(prow * kTaD * 2)) : "memory");
          }
          stamp(at, 1);
        }
        if (g.partial && n == g.nt - 1) {
          // rows past the sequence's end hold whatever the allocation holds: zero them (their P is zero, and zero times
          // a stray NaN would not be), whole 128-byte rows, which the swizzle only permutes within
          const uint32_t turn = (uint32_t)((at >> 1) & 1);
          if (!__all_sync(0xffffffffu, ta_wait(bar_tma + 16 * buf, turn, 10u) && ta_wait(bar_tma + 16 * buf + 8, turn, 10u))) {
            failed = true;
            break;
          }
          const int valid = g.seq - tok0;
          unsigned char *tile = smem + (size_t)buf * kTaTileBytes;
          for (int idx = lane; idx < (kTaTile - valid) * kTaChunks * 8; idx += 32) {
            const int r = valid + idx / (kTaChunks * 8), rem = idx % (kTaChunks * 8);
            *reinterpret_cast<uint4 *>(tile + (rem >> 3) * kTaChunkBytes + r * 128 + (rem & 7) * 16) = make_uint4(0, 0, 0, 0);
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if (lane == 0) ta_arrive(bar_fix + 8 * buf);
        }
      }
    }
    // no copy may be in flight when the CTA leaves; the MMA warps have seen all of them unless a wait gave up
    for (int i = max(0, issued - 4); i < issued; ++i) ta_wait(bar_tma + 16 * ((i >> 1) & 1) + 8 * (i & 1), (uint32_t)((i >> 2) & 1), 11u);
  } else if (warp >= 5) {
    // ---- two MMA warps: the fixed cost of an MMA of this size is larger than its work, and two warps share it.  All lanes walk,
    // so that addresses and descriptors stay warp-uniform; one issues ----
    const int wi = warp - 5;
    const bool issues = ta_elect();
    const uint32_t idesc_128 = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kTaTile >> 3) << 17) | ((128u >> 4) << 24);
    const uint32_t idesc_s = (idesc_128 & ~(31u << 24)) | ((64u >> 4) << 24);  // M = 64
    const uint32_t idesc_pv = idesc_128 | (1u << 15);                          // A (the tile) MN-major
    const uint64_t q_desc = ta_desc_sw128(sQ, 16, 1024);
    const uint64_t p_desc = ta_desc_plain(sP, kTaLbo, kTaSbo);
    // every descriptor below is a per-tile base plus a constant: the start address sits in the low bits (16-byte units,
    // 14 bits for 256 KB) and no offset used here carries out of them
    auto issue_s = [&](int n, int half) {
      const int buf = n & 1;
      const uint64_t c_desc = ta_desc_sw128(sT + buf * kTaTileBytes, 16, 1024);
      if (issues) {
        const int c0 = half ? kTaHalfChunks : 0, c1 = half ? kTaChunks : kTaHalfChunks;
#pragma unroll 1
        for (int c = c0; c < c1; ++c) {
#pragma unroll
          for (int k4 = 0; k4 < 4; k4 += 2) {
            // K step of 16 columns: 32 bytes of the chunk's rows, of the queries and of the tile alike.  The first warp takes the
            // even steps, the second one the odd ones, each into a partial sum of its own
            const uint64_t at = (uint64_t)((c * kTaChunkBytes + (k4 + wi) * 32) >> 4);
            ta_mma(tmem + 128 * buf + 64 * wi, q_desc + at, c_desc + at, idesc_s, c > 0 || k4 > 0 ? 1u : 0u);
          }
        }
        if (half) {
          ta_commit(bar_sfull + 8 * buf);
          if (wi == 0) stamp(n, 2);
        }
      }
      __syncwarp();
    };
    // Latent blocks of 128 columns = chunks 2 j and 2 j + 1, two of them to a warp; a K step is 16 tokens = two 8-row groups.  The
    // blocks take turns, so that consecutive MMAs accumulate into different columns of tensor memory.
    auto issue_pv = [&](int n, bool first) {
      const int buf = n & 1;
      const uint64_t a_desc = ta_desc_sw128(sT + buf * kTaTileBytes + 4 * wi * kTaChunkBytes, kTaChunkBytes, 1024);
      const uint64_t lo_desc = ta_desc_plain(sT + buf * kTaTileBytes + (kTaChunks - 1) * kTaChunkBytes, kTaLbo, kTaSbo);  // FINE: the low parts
      if (issues) {
#pragma unroll
        for (int part = 0; part < (FINE ? 2 : 1); ++part) {
#pragma unroll
          for (int kk = 0; kk < kTaTile / 16; ++kk) {
#pragma unroll
            for (int j = 0; j < 2; ++j)
              ta_mma(tmem + kTaColO + 128 * wi + 64 * j, a_desc + (uint64_t)((2 * j * kTaChunkBytes + kk * 2048) >> 4),
                     (part ? lo_desc : p_desc) + (uint64_t)(kk * ((2 * kTaLbo) >> 4)), idesc_pv, (!first || kk > 0 || part > 0) ? 1u : 0u);
          }
        }
        ta_commit(bar_empty + 16 * buf + 8 * wi);
        if (wi == 0) stamp(n, 5);
      }
      __syncwarp();
    };
    // true where the whole warp sees the phase complete
    auto seen = [&](uint32_t bar, uint32_t parity) -> bool { return __all_sync(0xffffffffu, ta_test(bar, parity)); };
    // Whatever can go next goes: a tile's P.C product frees its buffer and comes first; the scores of the tile behind it are
    // issued half by half as they land, so that neither product waits long behind the other in the tensor pipe.
    int sn = 0, pn = 0;   // next scores, next P.C product: tiles of the CTA
    uint32_t fix_turn = 0;  // a bit per buffer
    for (int sg = 0; !failed && segment(next_b, g); ++sg) {
      const int first = pn, end = pn + g.nt, last_partial = g.partial ? end - 1 : -1;
      int sh = 0;  // half of the scores
      if (!__all_sync(0xffffffffu, ta_wait(bar_q, (uint32_t)(sg & 1), 4u))) failed = true;
      unsigned idle = 0;
      while (pn < end && !failed) {
        bool went = false;
        if (pn < sn && seen(bar_pfull, (uint32_t)(pn & 1))) {
          tc_fence_after();
          issue_pv(pn, pn == first);
          ++pn;
          went = true;
        } else if (sn < end && sn <= pn + 1) {
          const int sb = sn & 1;
          const uint32_t turn = (uint32_t)((sn >> 1) & 1);
          bool ready = seen(bar_tma + 16 * sb + 8 * sh, turn);
          if (ready && sn == last_partial) ready = seen(bar_fix + 8 * sb, (fix_turn >> sb) & 1u);
          if (ready && sh == 0 && sn >= 2) ready = seen(bar_sfree + 8 * sb, turn ^ 1);
          if (ready) {
            tc_fence_after();
            issue_s(sn, sh);
            if (sh && sn == last_partial) fix_turn ^= 1u << sb;
            sn += sh;
            sh ^= 1;
            went = true;
          }
        }
        if (went) {
          idle = 0;
        } else if (++idle > 64) {
          __nanosleep(32);
          if (idle > kTaSpinLimit) {
            if (lane == 0) atomicExch(&g_mla_tc_error, 3u);
            failed = true;
          }
        }
      }
    }
  } else {
    // ---- consumers: warp w holds head rows 16 w .. 16 w + 15 of S; a lane has rows r0 and r0 + 8, 16 tokens of each ----
    const float sl2 = scale * 1.4426950408889634f;
    const int r0 = 16 * warp + (lane >> 2), tq = 2 * (lane & 3);
    auto done_with = [&](int n, unsigned code) -> bool {  // both warps' P.C products of tile n
      const uint32_t turn = (uint32_t)((n >> 1) & 1);
      return ta_wait(bar_empty + 16 * (n & 1), turn, code) && ta_wait(bar_empty + 16 * (n & 1) + 8, turn, code);
    };
    int n = 0;  // tile of the CTA
    while (!failed && segment(next_b, g)) {
      float m_ref[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
      for (int i = 0; i < g.nt; ++i, ++n) {
        const int buf = n & 1;
        uint32_t pk[2][8], pl[2][FINE ? 8 : 1];  // [row][column group of 8 tokens]: this lane's pair of tokens
        bool need = false;
        if (!failed && !__all_sync(0xffffffffu, ta_wait(bar_sfull + 8 * buf, (uint32_t)((n >> 1) & 1), 6u))) failed = true;
        if (!failed) {
          if (tid == 0) stamp(n, 3);
          tc_fence_after();
          uint32_t r[32];
          {
            uint32_t r2[32];  // the two partial sums of the score product
            tmem_ld_rows16(tmem + ((uint32_t)(32 * warp) << 16) + 128 * buf, r);
            tmem_ld_rows16(tmem + ((uint32_t)(32 * warp) << 16) + 128 * buf + 64, r2);
            tmem_wait_ld();
#pragma unroll
            for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) + __uint_as_float(r2[j]));
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) ta_arrive(bar_sfree + 8 * buf);
          if (tid == 0) stamp(n, 8);
          const int tok0 = (g.ts + i) * kTaTile;
          if (tok0 + kTaTile > g.seq) {  // the sequence's last tile: tokens past the end take no weight
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (tok0 + 8 * (j >> 2) + tq + (j & 1) >= g.seq) r[j] = 0xff800000u;
          }
#pragma unroll
          for (int y = 0; y < 2; ++y) {
            float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              mx0 = fmaxf(mx0, __uint_as_float(r[4 * e + 2 * y]));
              mx1 = fmaxf(mx1, __uint_as_float(r[4 * e + 2 * y + 1]));
            }
            float mx = fmaxf(mx0, mx1);
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2)) * sl2;  // the scale is positive
            float alpha = 1.f;
            if (i == 0) {
              m_ref[y] = mx;  // the segment's first tile holds at least one token
            } else if (mx > m_ref[y] + kTaLazy) {
              alpha = exp2f(m_ref[y] - mx);
              m_ref[y] = mx;
              need = true;
            }
            if ((lane & 3) == 0) s_alpha[r0 + 8 * y] = alpha;
            const float nm = -m_ref[y];
            float sum0 = 0.f, sum1 = 0.f;
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              // the probabilities enter the second product rounded to bf16 (as the reference rounds them, :466); the
              // normaliser sums the same rounded values (FINE: two parts, and the normaliser sums the weights themselves)
              const float p0 = ta_ex2(fmaf(__uint_as_float(r[4 * e + 2 * y]), sl2, nm)), p1 = ta_ex2(fmaf(__uint_as_float(r[4 * e + 2 * y + 1]), sl2, nm));
              const uint32_t pa = ta_pack_bf16x2(p0, p1);
              if (FINE) {
                sum0 += p0;
                sum1 += p1;
                pl[y][FINE ? e : 0] = ta_pack_bf16x2(p0 - __uint_as_float(pa << 16), p1 - __uint_as_float(pa & 0xffff0000u));
              } else {
                sum0 += __uint_as_float(pa << 16);
                sum1 += __uint_as_float(pa & 0xffff0000u);
              }
              pk[y][e] = pa;
            }
            l[y] = l[y] * alpha + (sum0 + sum1);
          }
          if (tid == 0) stamp(n, 9);
        }
        need = __any_sync(0xffffffffu, need);
        if (lane == 0) s_need[buf][warp] = need ? 1 : 0;
        if (ta_consumers_sync(failed)) {
          failed = true;
          break;
        }
        if (s_need[buf][0] | s_need[buf][1] | s_need[buf][2] | s_need[buf][3]) {
          // a head's reference maximum moved (never in a segment's first tile): every lane of O^T scales its 4 x 64 head columns, once the
          // previous tile's MMAs have finished with them
          if (!__all_sync(0xffffffffu, done_with(n - 1, 7u))) failed = true;
          if (!failed) {
            tc_fence_after();
#pragma unroll 1
            for (int j = 0; j < kTaDV / 128; ++j) {
              uint32_t o[64];
              const uint32_t ta = tmem + ((uint32_t)(32 * warp) << 16) + kTaColO + 64 * j;
              tmem_ld64(ta, o);
              tmem_wait_ld();
#pragma unroll
              for (int c = 0; c < 64; ++c) o[c] = __float_as_uint(__uint_as_float(o[c]) * s_alpha[c]);
              tmem_st64(ta, o);
            }
            tmem_wait_st();
            tc_fence_before();
          }
          if (ta_consumers_sync(failed)) {
            failed = true;
            break;
          }
        }
        if (!failed) {
          if (n > 0 && !__all_sync(0xffffffffu, done_with(n - 1, 8u))) {
            failed = true;  // reaches the others at the next tile's barrier
          } else {
            unsigned char *lo = smem + (size_t)buf * kTaTileBytes + (kTaChunks - 1) * kTaChunkBytes;
#pragma unroll
            for (int y = 0; y < 2; ++y) {
#pragma unroll
              for (int kg = 0; kg < kTaTile / 8; ++kg) {
                const int at = kg * kTaLbo + (r0 + 8 * y) * 16 + 2 * tq;
                *reinterpret_cast<uint32_t *>(Pp + at) = pk[y][kg];
                if (FINE) *reinterpret_cast<uint32_t *>(lo + at) = pl[y][FINE ? kg : 0];
              }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) ta_arrive(bar_pfull);
            if (tid == 0) stamp(n, 4);
          }
        }
      }
      // ---- the segment's partial result: O^T [latent lane x head column] -> part_o [head][512], (m, sum) per head ----
      if (!failed && !__all_sync(0xffffffffu, done_with(n - 1, 9u))) failed = true;
      failed = ta_consumers_sync(failed);
      if (!failed) {
        tc_fence_after();
        float *po = part_o + ((size_t)g.slot * heads + h0) * kTaDV, *my_ml = part_ml + ((size_t)g.slot * heads + h0) * 2;
#pragma unroll 1
        for (int j = 0; j < kTaDV / 128; ++j) {
#pragma unroll 1
          for (int half = 0; half < 2; ++half) {
            uint32_t o[32];
            tmem_ld32(tmem + ((uint32_t)(32 * warp) << 16) + kTaColO + 64 * j + 32 * half, o);
            tmem_wait_ld();
#pragma unroll
            for (int c = 0; c < 32; ++c)
              if (32 * half + c < nh) po[(size_t)(32 * half + c) * kTaDV + 128 * j + 32 * warp + lane] = __uint_as_float(o[c]);
          }
        }
#pragma unroll
        for (int y = 0; y < 2; ++y) {
          float sum = l[y] + __shfl_xor_sync(0xffffffffu, l[y], 1);
          sum += __shfl_xor_sync(0xffffffffu, sum, 2);
          const int head = r0 + 8 * y;
          if ((lane & 3) == 0 && head < nh) {
            my_ml[head * 2] = m_ref[y] * 0.6931471805599453f;  // back to natural units
            my_ml[head * 2 + 1] = sum;
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)kTaTmemCols) : "memory");
}

// Reads and clears the error word of the kernels above (0: no wait ever gave up).
int mla_attend_tc_take_error(unsigned *out) {
  unsigned zero = 0;
  BLOK_CUDA(cudaMemcpyFromSymbol(out, g_mla_tc_error, sizeof(unsigned)));
  if (*out) BLOK_CUDA(cudaMemcpyToSymbol(g_mla_tc_error, &zero, sizeof(unsigned)));
  return BLOK_OK;
}

// BLOK_MLA_TRACE=1 in the environment at the first launch: CTA (0, 0) of every launch records the time stamps described
// in the kernel; blok_mla_attend_trace copies them out.
static long long *g_trace_buf = nullptr;
static long long *trace_buffer() {
  static bool asked = false;
  if (!asked) {
    asked = true;
    const char *e = getenv("BLOK_MLA_TRACE");
    if (e && e[0] == '1' && cudaMalloc(&g_trace_buf, kTaTraceTiles * 16 * sizeof(long long)) == cudaSuccess)
      cudaMemset(g_trace_buf, 0, kTaTraceTiles * 16 * sizeof(long long));
  }
  return g_trace_buf;
}
int mla_attend_tc_trace(long long *host_out, int max_entries) {
  if (!g_trace_buf) return 0;
  const int n = max_entries < kTaTraceTiles * 16 ? max_entries : kTaTraceTiles * 16;
  if (cudaDeviceSynchronize() != cudaSuccess ||
      cudaMemcpy(host_out, g_trace_buf, (size_t)n * sizeof(long long), cudaMemcpyDeviceToHost) != cudaSuccess)
    return 0;
  return n;
}

// The tensor map of a cache of `rows` rows of 576 bf16 at `base`: boxes of 64 rows x 64 columns in the 128-byte swizzle;
// rows at or past `rows` read as zeros.  The last few maps are kept (a model's layers pass the same caches step after step).
// keep: false for operands that move from call to call (the queries).
static int cache_tensor_map(const uint16_t *base, long rows, bool keep, CUtensorMap *out) {
  struct Entry {
    const void *base;
    long rows;
    CUtensorMap map;
  };
  static std::mutex mu;
  static Entry kept[128];
  static int n_kept = 0, next = 0;
  std::lock_guard<std::mutex> lock(mu);
  for (int i = 0; i < n_kept && keep; ++i)
    if (kept[i].base == base && kept[i].rows == rows) {
      *out = kept[i].map;
      return BLOK_OK;
    }
  CUtensorMap map;
  if (int rc = tensor_map_2d(base, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rows, kTaD, kTaD * 2, kTaTile, 64, CU_TENSOR_MAP_SWIZZLE_128B, &map)) return rc;
  *out = map;
  if (!keep) return BLOK_OK;
  kept[next] = Entry{base, rows, map};
  next = (next + 1) % 128;
  if (n_kept < 128) ++n_kept;
  return BLOK_OK;
}

// total_rows: the rows of the cache allocation from `cache` on (reads past them give zeros).  Up to kMlaPlanMax sequences over `ctas`
// CTAs; plan, parts: see the kernel.
int launch_mla_attend_tc(const uint16_t *q, const uint16_t *cache, long ctx_stride, long total_rows, const int *seq_len, int B, int ctas,
                         float scale, float *part_o, float *part_ml, const MlaPlan *plan, int2 *parts, cudaStream_t stream) {
  if (int rc = allow_smem(mla_attend_tc_kernel<false, false>, kTaSmemBytes)) return rc;
  CUtensorMap map, qmap;
  if (int rc = cache_tensor_map(cache, total_rows, true, &map)) return rc;
  if (int rc = cache_tensor_map(q, (long)B * kTaHeads, false, &qmap)) return rc;
  return launch_pdl("mla_attend_tc_kernel", mla_attend_tc_kernel<false, false>, dim3(ctas), kTaThreads, kTaSmemBytes, stream, map, qmap, cache, ctx_stride, seq_len, scale, part_o, part_ml, nullptr, nullptr, 0, 0, trace_buffer(), kTaHeads, B, plan, parts);
}

// The same over a paged pool of pool_rows rows: page_rows must be a positive multiple of the 64-token tile.
template <bool FINE>
static int launch_paged(const uint16_t *q, const uint16_t *pool, long pool_rows, const int *block_table, const int *slot_of, int table_stride,
                        int page_rows, const int *seq_len, int B, int heads, dim3 grid, float scale, float *part_o, float *part_ml,
                        int planned, const MlaPlan *plan, int2 *parts, cudaStream_t stream) {
  if (int rc = allow_smem(mla_attend_tc_kernel<true, FINE>, kTaSmemBytes)) return rc;
  CUtensorMap map, qmap;
  if (int rc = cache_tensor_map(pool, pool_rows, true, &map)) return rc;
  if (int rc = cache_tensor_map(q, (long)B * heads, false, &qmap)) return rc;
  return launch_pdl("mla_attend_tc_kernel(paged)", mla_attend_tc_kernel<true, FINE>, grid, kTaThreads, kTaSmemBytes, stream, map, qmap, pool, 0, seq_len, scale, part_o, part_ml, block_table, slot_of, table_stride, page_rows, trace_buffer(), heads, planned, plan, parts);
}
int launch_mla_attend_tc_paged(const uint16_t *q, const uint16_t *pool, long pool_rows, const int *block_table, const int *slot_of,
                               int table_stride, int page_rows, const int *seq_len, int B, int ctas, float scale, float *part_o,
                               float *part_ml, const MlaPlan *plan, int2 *parts, cudaStream_t stream) {
  return launch_paged<false>(q, pool, pool_rows, block_table, slot_of, table_stride, page_rows, seq_len, B, kTaHeads, dim3(ctas), scale, part_o,
                             part_ml, B, plan, parts, stream);
}
// Any number of heads; the weights in two bf16 parts; entry b attends to rows 0..pos[b].
int launch_mla_attend_tc_fine(const uint16_t *q, const uint16_t *pool, long pool_rows, const int *block_table, const int *slot_of, int table_stride,
                              int page_rows, const int *pos, int B, int heads, int splits, float scale, float *part_o, float *part_ml,
                              cudaStream_t stream) {
  return launch_paged<true>(q, pool, pool_rows, block_table, slot_of, table_stride, page_rows, pos, B, heads, dim3(splits, B, (heads + kTaHeads - 1) / kTaHeads), scale,
                            part_o, part_ml, 0, nullptr, nullptr, stream);
}

}  // namespace blok
