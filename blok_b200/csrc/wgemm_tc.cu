// Grouped GEMM on the 5th-generation tensor cores (tcgen05, accumulators in tensor memory) for the INT4 experts of the
// batched routed-MoE layer:
//   out[token, row] = sum_c bf16(q[row, c] * scale[row, c / 32]) * x[token, c]
// Reference arithmetic: matvec_i4_bf16_scale_k (src/kimi_exec.cu:300-323) applied per token; the dequantised weight is the
// reference's bf16(q * s) bit for bit (:312).  The weight rows are the M = 128 dimension of tcgen05.mma, the tokens the N
// dimension, so a weight byte is read from HBM and dequantised once per tile whatever the token count.  Every mbarrier wait
// is bounded; on a timeout the CTA records an error, waits for its copies, releases its tensor memory and returns.
#include <algorithm>

#include "common.cuh"
#include "gemm_tma.h"
#include "tc_pipe.cuh"
#include "wgemm.h"

namespace blok {

constexpr int kTcN = kWgTileTokens;  // token columns of a tile

__device__ __forceinline__ uint32_t tc_bf16x2_mul(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ uint32_t tc_bf16x2_fma(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t r;
  asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
  return r;
}

// Dequantisation with one instruction per pair of weights besides the masks.  The bits of a nibble n = q + 8 in the low four
// bits of a bf16 are the number n 2^-133, in the next four n 2^-129 (below and just above the smallest normal number the
// encoding is linear), so w & 0x000f000f and w & 0x00f000f0 are pairs of nibbles as they lie, and
//   fma(n 2^-129, s 2^117, -s 2^-9) = bf16(q s 2^-12) = 2^-12 bf16(q s)
// with one rounding, the reference's (:312): a power of two does not change it while s 2^121 is finite and q s 2^-12 normal
// (s = 0 or 2^-114 <= |s| < 2^7).  The epilogue takes the 2^12 back, exactly.  A larger power would cover larger scales and lose
// smaller sums: with 2^29 results below 1e-31 lost bits, with 2^12 below 1e-36.  (Adding an exponent to the nibble, subtracting
// 136 and multiplying took 15 instructions a word instead of 9.)  No checkpoint has other scales, but any bf16 is accepted:
// i4_outside finds them, and i4_plain_rows takes the place of the unit's epilogue.
constexpr uint32_t kI4Hi = 0x7a007a00u, kI4Lo = 0x7c007c00u, kI4Off = 0xbb00bb00u;  // 2^117, 2^121, -2^-9
constexpr float kI4Unscale = 4096.f;                                                // 2^12
struct I4Scale {
  uint32_t hi, lo, off;
  __device__ __forceinline__ explicit I4Scale(uint32_t s2) : hi(tc_bf16x2_mul(s2, kI4Hi)), lo(tc_bf16x2_mul(s2, kI4Lo)), off(tc_bf16x2_mul(s2, kI4Off)) {}
};
// The pairs (q_j s, q_{j+4} s), j = 0..3, of one packed word: its eight columns in the order 0 4 1 5 2 6 3 7.
__device__ __forceinline__ void i4_dequant(uint32_t w, const I4Scale &s, uint32_t *o) {
  const uint32_t t = w >> 8;
  o[0] = tc_bf16x2_fma(w & 0x000f000fu, s.lo, s.off);
  o[1] = tc_bf16x2_fma(w & 0x00f000f0u, s.hi, s.off);
  o[2] = tc_bf16x2_fma(t & 0x000f000fu, s.lo, s.off);
  o[3] = tc_bf16x2_fma(t & 0x00f000f0u, s.hi, s.off);
}

// A unit is (tile of up to 64 tokens of one expert) x 256 weight rows (128 gate + 128 up rows of the same indices, or 256
// rows of the down projection); a persistent CTA per SM walks the units, and every role runs ahead across their boundaries:
//   warps 0, 1    MMAs of row block 0 and 1: 8 K = 16 steps per piece of 128 columns
//   warp 2        activations by TMA: four slots of 128 columns
//   warp 3        weights and scales by TMA: four stages of 256 rows x 128 bytes, scales 32 bytes (512 columns) per row
//   warps 4..7    epilogue of the unit before (two accumulator buffers)
//   warps 8..     unpack: two sets of eight warps, one for each piece of a stage; a thread owns one row of one block and writes
//                 the piece's exact bf16(q * s) to TENSOR MEMORY as the MMA's A operand
// The activations arrive in sorted order with the columns of every packed word in the order 0 4 1 5 2 6 3 7 (the order the
// unpacking leaves the weights in): i4_rows_kernel lays them out once per launch, the SwiGLU epilogue writes them so.
//
// Bound: the weight stream where a group has few tokens, then the tensor cores and the power of both.  What it took, gate/up
// product of 384 experts of 7168 x 2048 over 4,136 assignments (6.3 GB): cp.async producers that also fetched the activations,
// two CTAs per SM 1,447 us and 835 us more for the groups of up to 8 (mat-vec-style kernel); TMA, roles, one CTA 1,687 us;
// dequantisation in 9 instead of 15 instructions a word 1,437; MMAs of the two blocks by two warps 1,389; scales on the
// weights' barrier 1,301; operands of the MMAs in uniform registers 1,255; pieces of 128 columns instead of 64 and 16
// unpacking warps instead of 24 1,138 us (5.6 TB/s).  With a hand-over every 64 columns the MMA warps' waits were the limit,
// whatever the others did.  At 16,384 assignments 2,190 us before, 1,537 now; at 512 1,017 before, 800 now.
// Unpacking is bound by its instructions: the test of the scales' range (four of about 190 a piece) cost the layer 0.7 % at 6
// tokens and 1 to 2.5 % from 64 on; the walk by pairs of stages, whose slots and parities are constants, took that back: 6 / 64 /
// 517 / 2,048 tokens 291 / 1,575 / 2,220 / 3,180 us before, 287 / 1,495 / 2,127 / 3,110 now.
constexpr int kI4Unpack = 16, kI4Epi = 4;                       // warps
constexpr int kI4FirstUnpack = 4 + kI4Epi;
constexpr int kI4Threads = (kI4FirstUnpack + kI4Unpack) * 32;
constexpr int kI4Cols = 256;                                    // columns per weight stage
constexpr int kI4WStages = 4, kI4WBytes = 256 * (kI4Cols / 2);  // 32 KB
constexpr int kI4SStages = 3, kI4SBytes = 256 * 32;             // scales of 512 columns: whole 32-byte sectors
constexpr int kI4XStages = 4, kI4XHalf = kTcN * 128, kI4XBytes = 2 * kI4XHalf;  // 64 tokens x 2 x 64 columns
constexpr int kI4Smem = kI4WStages * kI4WBytes + kI4SStages * kI4SBytes + kI4XStages * kI4XBytes + 1024;
constexpr int kI4Piece = 2;                                     // 64-column parts per piece: a slot of the activations
constexpr int kI4Pieces = 4 / kI4Piece;                         // per weight stage; each has its own tensor-memory buffer
constexpr int kI4TmemCols = 512;                                // 2 x 2 accumulators of 64 columns, 4 pieces x 2 blocks x 32 columns of weights
constexpr int kI4ACol = 4 * kTcN;

struct I4Args {
  uint16_t *out;
  const int *out_index, *tile_expert, *tile_start, *tile_count, *num_tiles;
  int K, R, stride_rows;
  const int *total;       // up to kWgSmallRows here: the launch is the mat-vec-style kernel's; NULL: no
  const void *w_a, *w_b;  // the operands again, for i4_plain_rows
  const uint16_t *s_a, *s_b, *x;
  unsigned *err;
  // the launch before is the gate/up product of the same experts: weights, scales and the tile table are there, what that product
  // writes and reads (activations, results' buffer) only behind the wait
  int early;
};

// The epilogue of a thread's two sums for one token: gate and up, or two rows of the down projection 128 apart.
template <bool SWIGLU>
__device__ __forceinline__ void i4_store(uint16_t *out, float va, float vb) {
  if (SWIGLU) {
    const float gv = round_bf16(va), uv = round_bf16(vb);
    *out = f32_to_bf16_bits(round_bf16(gv / (1.0f + expf(-gv))) * uv);
  } else {
    out[0] = f32_to_bf16_bits(va);
    out[128] = f32_to_bf16_bits(vb);
  }
}

// Two scales: |s| 2^7 or more (infinities and NaN too), or below 2^-114 and not zero.  |s| - 1 with the top bit on: zero wraps to
// the smallest unsigned and the largest signed value.
__device__ __forceinline__ bool i4_outside(uint32_t s2) {
  const uint32_t v = (s2 | 0x80008000u) - 0x00010001u;
  return __vmaxu2(v, 0xc2fec2feu) != 0xc2fec2feu || __vmins2(v, 0x867f867fu) != 0x867f867fu;
}

// A thread's two rows of a unit that holds scales i4_dequant does not cover, in place of what the MMAs summed: the product q s
// rounded to bf16 as the reference has it, whatever the scale, in plain loops (7168 columns: 0.23 ms a token of the tile; four tokens
// per look at a weight took as long for 64 and longer for one).  row: weight row inside the expert; col: output column.
template <bool SWIGLU>
__device__ __noinline__ void i4_plain_rows(const I4Args &a, int tile, int row, int col) {
  const int p0 = a.tile_start[tile], cnt = a.tile_count[tile], blocks = a.K / 32;
  const size_t at = ((size_t)a.tile_expert[tile] * a.stride_rows + row) * blocks;
  const uint4 *w[2] = {reinterpret_cast<const uint4 *>(a.w_a) + at, reinterpret_cast<const uint4 *>(SWIGLU ? a.w_b : a.w_a) + at + (SWIGLU ? 0 : 128 * (size_t)blocks)};
  const uint16_t *s[2] = {a.s_a + at, (SWIGLU ? a.s_b : a.s_a) + at + (SWIGLU ? 0 : 128 * (size_t)blocks)};
  for (int tok = 0; tok < cnt; ++tok) {
    const uint2 *x = reinterpret_cast<const uint2 *>(a.x + (size_t)(p0 + tok) * a.K);
    float acc[2] = {0.f, 0.f};
    for (int b = 0; b < blocks; ++b) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint32_t *words = reinterpret_cast<const uint32_t *>(w[h] + b);
        const float scale = bf16_bits_to_f32(s[h][b]);
        for (int i = 0; i < 8; ++i) {  // half a word: columns j and j + 4 are neighbours in x
          const uint2 v = x[8 * b + i];
          const int q = (int)(words[i >> 1] >> (8 * (i & 1)));
          acc[h] = fmaf(round_bf16((float)((q & 15) - 8) * scale), bf16lo(v.x), acc[h]);
          acc[h] = fmaf(round_bf16((float)((q >> 16 & 15) - 8) * scale), bf16hi(v.x), acc[h]);
          acc[h] = fmaf(round_bf16((float)((q >> 4 & 15) - 8) * scale), bf16lo(v.y), acc[h]);
          acc[h] = fmaf(round_bf16((float)((q >> 20 & 15) - 8) * scale), bf16hi(v.y), acc[h]);
        }
      }
    }
    const size_t p = a.out_index ? (size_t)a.out_index[p0 + tok] : (size_t)(p0 + tok);
    i4_store<SWIGLU>(a.out + p * a.R + col, acc[0], acc[1]);
  }
}

__device__ __forceinline__ uint4 i4_lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t i4_lds32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}

// Bounded wait, longer than a unit of i4_plain_rows (64 tokens of 32,768 columns: 70 ms); a warp that has time (SLEEP ns between tries) leaves the issue slots to the unpacking warps.
template <int SLEEP>
__device__ __forceinline__ bool i4_wait(uint32_t mbar, uint32_t parity) {
  for (unsigned it = 0; it < (1u << 23); ++it) {
    uint32_t ok;
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, 1000;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t"
        "}\n"
        : "=r"(ok)
        : "r"(mbar), "r"(parity)
        : "memory");
    if (ok) return true;
    if (SLEEP) __nanosleep(SLEEP);
  }
  return false;
}

// A ring's position: slot and the parity of the slot's current use.
template <int N>
struct I4Ring {
  int slot = 0;
  uint32_t turn = 0;
  __device__ __forceinline__ void next() {
    if (++slot == N) slot = 0, turn ^= 1;
  }
};

struct I4Mma {
  uint32_t x_full, x_empty, a_full, a_empty, d_full, d_empty, xbase;
};
// The MMAs of one row block; false: a wait gave up.  The whole warp walks the pieces and one lane issues: every address is
// a constant or a loop variable and stays in uniform registers.
template <int BLK>
__device__ __forceinline__ bool i4_mma(const I4Mma &m, const I4Args &a, int units, int blocks, int stages) {
  const bool issues = tp_elect();
  I4Ring<kI4XStages> xr;
  I4Ring<2> dr;
  uint32_t aturn = 0;
  for (int u = blockIdx.x; u < units; u += gridDim.x) {
    const uint32_t idesc = tp_idesc_bf16(((a.tile_count[u / blocks] + 15) >> 4) << 4);
    if (!__all_sync(0xffffffffu, i4_wait<0>(m.d_empty + 8 * dr.slot, dr.turn ^ 1))) return false;
    const uint32_t d = (uint32_t)(dr.slot * 2 + BLK) * kTcN;
    for (int st = 0; st < stages; ++st) {
#pragma unroll
      for (int c = 0; c < kI4Pieces; ++c) {
        const bool ok = i4_wait<0>(m.x_full + 8 * xr.slot, xr.turn) && i4_wait<0>(m.a_full + 16 * c + 8 * BLK, aturn);
        if (!__all_sync(0xffffffffu, ok)) return false;
        tc_fence_after();
        const uint64_t bd = tp_desc_k_sw128(m.xbase + xr.slot * kI4XBytes);
        constexpr uint32_t ta = kI4ACol + BLK * 32;
        if (issues) {
#pragma unroll
          for (int z = 0; z < kI4Piece; ++z)
#pragma unroll
            for (int k = 0; k < 4; ++k)
              tp_mma_ts(d, ta + (c * kI4Piece + z) * 64 + 8 * k, bd + (uint64_t)(z * (kI4XHalf / 16) + 2 * k), idesc,
                        (st | c | z | k) ? 1u : 0u);
          tp_commit(m.a_empty + 16 * c + 8 * BLK);
          tp_commit(m.x_empty + 8 * xr.slot);
          if (c == kI4Pieces - 1 && st == stages - 1) tp_commit(m.d_full + 8 * dr.slot);
        }
        xr.next();
      }
      aturn ^= 1;
    }
    dr.next();
  }
  return true;
}

template <bool SWIGLU>
__global__ void __launch_bounds__(kI4Threads, 1)
    wgemm_tc_kernel(const __grid_constant__ CUtensorMap mwa, const __grid_constant__ CUtensorMap mwb, const __grid_constant__ CUtensorMap msa,
                    const __grid_constant__ CUtensorMap msb, const __grid_constant__ CUtensorMap mx, const __grid_constant__ I4Args a) {
  if (!a.early) pdl_wait();
  pdl_trigger();  // behind the wait of the gate/up product: the down projection reads weights and tile table before its own
  if (a.total && *a.total <= kWgSmallRows) return;
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) unsigned long long s_bar[2 * (kI4WStages + kI4XStages + 8 + 2)];
  __shared__ uint32_t s_tmem;
  __shared__ volatile int s_odd[2];  // per accumulator buffer: 1 + the last unit in it that has a scale i4_dequant does not cover
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr int kRows = SWIGLU ? 128 : 256;
  const int blocks = a.R / kRows, units = *a.num_tiles * blocks;
  const int stages = a.K / kI4Cols;
  const uint32_t wbase = ((uint32_t)__cvta_generic_to_shared(smem_raw) + 1023u) & ~1023u;
  const uint32_t sbase = wbase + kI4WStages * kI4WBytes, xbase = sbase + kI4SStages * kI4SBytes;
  const uint32_t w_full = (uint32_t)__cvta_generic_to_shared(&s_bar[0]), w_empty = w_full + 8 * kI4WStages;
  const uint32_t x_full = w_empty + 8 * kI4WStages, x_empty = x_full + 8 * kI4XStages;
  const uint32_t a_full = x_empty + 8 * kI4XStages, a_empty = a_full + 64, d_full = a_empty + 64, d_empty = d_full + 16;
  if (tid == 0) {
    for (int s = 0; s < kI4WStages; ++s) tp_mbar_init(w_full + 8 * s, 1), tp_mbar_init(w_empty + 8 * s, kI4Pieces * 8);
    for (int s = 0; s < kI4XStages; ++s) tp_mbar_init(x_full + 8 * s, 1), tp_mbar_init(x_empty + 8 * s, 2);
    for (int s = 0; s < 8; ++s) tp_mbar_init(a_full + 8 * s, 4), tp_mbar_init(a_empty + 8 * s, 1);  // [piece of a stage][row block]
    for (int s = 0; s < 2; ++s) tp_mbar_init(d_full + 8 * s, 2), tp_mbar_init(d_empty + 8 * s, kI4Epi);
    tp_mbar_init_fence();
    s_odd[0] = s_odd[1] = 0;
  }
  if (warp == 0) tp_tmem_alloc((uint32_t)__cvta_generic_to_shared(&s_tmem), kI4TmemCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  constexpr uint32_t tmem = 0;  // all columns are this CTA's, so they start at 0: a constant keeps the MMAs' operands in uniform registers
  bool failed = false;

  if (warp >= kI4FirstUnpack) {
    // c: the piece of every stage that this set takes, and the tensor-memory buffer it goes to.  Two stages at a time: they share
    // a slot of scales, and the slots and parities inside the pair are constants.
    const int c = (warp - kI4FirstUnpack) >> 3, blk = (warp >> 2) & 1, row = 32 * (warp & 3) + lane;
    const uint32_t wrow = wbase + (uint32_t)(blk * (128 * 128) + row * 128);
    const uint32_t srow = sbase + (uint32_t)(blk * (128 * 32) + row * 32 + c * 4 * kI4Piece);
    const uint32_t ta = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)(kI4ACol + blk * 32 + c * kI4Piece * 64);
    const uint32_t ready = a_full + 16 * c + 8 * blk, free = a_empty + 16 * c + 8 * blk;
    I4Ring<kI4WStages / 2> wr;
    I4Ring<kI4SStages> sr;
    int dslot = 0;
    for (int u = blockIdx.x; u < units && !failed; u += gridDim.x) {
      bool odd = false;
      for (int st = 0; st < stages && !failed; st += 2) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const uint32_t ws = 2 * wr.slot + e;
          if (!__all_sync(0xffffffffu, i4_wait<0>(w_full + 8 * ws, wr.turn))) {
            failed = true;
            break;
          }
          uint4 q[2 * kI4Piece];
          uint32_t sc[kI4Piece];
#pragma unroll
          for (int h = 0; h < 2 * kI4Piece; ++h) q[h] = i4_lds128(wrow + ws * kI4WBytes + (((2 * kI4Piece * c + h) ^ (row & 7)) << 4));
#pragma unroll
          for (int h = 0; h < kI4Piece; ++h) sc[h] = i4_lds32(srow + sr.slot * kI4SBytes + ((e ^ ((row >> 2) & 1)) << 4) + h * 4);
          __syncwarp();
          if (lane == 0) tp_arrive(w_empty + 8 * ws);
#pragma unroll
          for (int z = 0; z < kI4Piece; ++z) {
            uint32_t av[32];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const I4Scale s2(__byte_perm(sc[z], 0, h ? 0x3232 : 0x1010));
              const uint32_t w[4] = {q[2 * z + h].x, q[2 * z + h].y, q[2 * z + h].z, q[2 * z + h].w};
#pragma unroll
              for (int k = 0; k < 4; ++k) i4_dequant(w[k], s2, av + (h * 4 + k) * 4);
            }
            if (z == 0) {
              if (!__all_sync(0xffffffffu, i4_wait<0>(free, e ^ 1))) {  // the first use finds it free
                failed = true;
                break;
              }
              tc_fence_after();
            }
            tmem_st32(ta + z * 64, av);
          }
          if (failed) break;
          // while the stores are on their way; exponents that begin 01 are 2^-63 <= |s| < 2, for the few others the exact test
          if (((sc[0] ^ 0x20002000u) | (sc[1] ^ 0x20002000u)) & 0x60006000u) odd = odd || i4_outside(sc[0]) || i4_outside(sc[1]);
          if (e && st + 2 == stages && odd) s_odd[dslot] = u + 1;
          tmem_wait_st();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) tp_arrive(ready);
        }
        wr.next();
        sr.next();
      }
      dslot ^= 1;
    }
  } else if (warp >= 4) {
    const int quarter = warp & 3, row = 32 * quarter + lane;
    I4Ring<2> dr;
    pdl_wait();
    for (int u = blockIdx.x; u < units; u += gridDim.x) {
      const int tile = u / blocks, row0 = (u - tile * blocks) * kRows;
      const int p0 = a.tile_start[tile], cnt = a.tile_count[tile];
      if (!__all_sync(0xffffffffu, i4_wait<400>(d_full + 8 * dr.slot, dr.turn))) {
        failed = true;
        break;
      }
      tc_fence_after();
      const uint32_t td = tmem + ((uint32_t)(32 * quarter) << 16) + (uint32_t)(dr.slot * 2 * kTcN);
      // a row of the intermediate vector is a column of the down projection's activations
      const int col = row0 + (SWIGLU ? (row & ~7) | ((row & 3) << 1) | ((row >> 2) & 1) : row);
      for (int n0 = 0; n0 < cnt; n0 += 16) {
        uint32_t ra[16], rb[16];
        tmem_ld16(td + n0, ra);
        tmem_ld16(td + kTcN + n0, rb);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const int tok = n0 + j;
          if (tok < cnt) {
            const size_t p = a.out_index ? (size_t)a.out_index[p0 + tok] : (size_t)(p0 + tok);
            const float va = __uint_as_float(ra[j]) * kI4Unscale, vb = __uint_as_float(rb[j]) * kI4Unscale;
            i4_store<SWIGLU>(a.out + p * a.R + col, va, vb);
          }
        }
      }
      if (s_odd[dr.slot] == u + 1) i4_plain_rows<SWIGLU>(a, tile, row0 + row, col);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) tp_arrive(d_empty + 8 * dr.slot);
      dr.next();
    }
  } else if (warp == 3) {
    if (lane == 0) {
      I4Ring<kI4WStages> wr;
      I4Ring<kI4SStages> sr;
      long issued = 0;
      for (int u = blockIdx.x; u < units && !failed; u += gridDim.x) {
        const int tile = u / blocks, row0 = (u - tile * blocks) * kRows;
        const int r = a.tile_expert[tile] * a.stride_rows + row0, rb = SWIGLU ? r : r + 128;
        for (int st = 0; st < stages; ++st) {
          if (!i4_wait<100>(w_empty + 8 * wr.slot, wr.turn ^ 1)) {
            failed = true;
            break;
          }
          const uint32_t dst = wbase + wr.slot * kI4WBytes, bar = w_full + 8 * wr.slot;
          tp_expect_tx(bar, kI4WBytes + (st & 1 ? 0 : kI4SBytes));
          if (!(st & 1)) {
            // scales ride with the even stage; the slot's last readers, stages st - 6 and st - 5, left before stage st - 1 was asked for
            const uint32_t sdst = sbase + sr.slot * kI4SBytes;
            tp_load_2d(sdst, &msa, st * (kI4Cols / 16), r, bar);
            tp_load_2d(sdst + kI4SBytes / 2, SWIGLU ? &msb : &msa, st * (kI4Cols / 16), rb, bar);
            sr.next();
          }
          tp_load_2d(dst, &mwa, st * (kI4Cols / 2), r, bar);
          tp_load_2d(dst + kI4WBytes / 2, SWIGLU ? &mwb : &mwa, st * (kI4Cols / 2), rb, bar);
          wr.next();
          ++issued;
        }
      }
      // no copy may be in flight when the CTA leaves: the last use of every slot
      for (long c = issued > kI4WStages ? issued - kI4WStages : 0; c < issued; ++c)
        i4_wait<0>(w_full + 8 * (int)(c % kI4WStages), (uint32_t)((c / kI4WStages) & 1));
    }
  } else if (warp == 2) {
    if (lane == 0) {
      I4Ring<kI4XStages> xr;
      long issued = 0;
      pdl_wait();
      for (int u = blockIdx.x; u < units && !failed; u += gridDim.x) {
        const int tile = u / blocks, p0 = a.tile_start[tile], rows16 = (a.tile_count[tile] + 15) >> 4;
        for (int c = 0; c < 2 * stages; ++c) {
          if (!i4_wait<20>(x_empty + 8 * xr.slot, xr.turn ^ 1)) {
            failed = true;
            break;
          }
          const uint32_t dst = xbase + xr.slot * kI4XBytes, bar = x_full + 8 * xr.slot;
          tp_expect_tx(bar, rows16 * 4096);
          for (int n = 0; n < rows16; ++n) {
            tp_load_2d(dst + n * 2048, &mx, c * 128, p0 + 16 * n, bar);
            tp_load_2d(dst + kI4XHalf + n * 2048, &mx, c * 128 + 64, p0 + 16 * n, bar);
          }
          xr.next();
          ++issued;
        }
      }
      for (long c = issued > kI4XStages ? issued - kI4XStages : 0; c < issued; ++c)
        i4_wait<0>(x_full + 8 * (int)(c % kI4XStages), (uint32_t)((c / kI4XStages) & 1));
    }
  } else {
    const I4Mma m = {x_full, x_empty, a_full, a_empty, d_full, d_empty, xbase};
    failed = warp ? !i4_mma<1>(m, a, units, blocks, stages) : !i4_mma<0>(m, a, units, blocks, stages);
  }
  if (failed && a.err) atomicExch(a.err, 1u);
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tp_tmem_free(tmem, kI4TmemCols);
}

// xs[p] = x[x_index ? x_index[p] : p] for the sorted positions p of every tile, the columns of each packed word in the
// order 0 4 1 5 2 6 3 7.  grid = (tile slots, parts of a tile).
__global__ void __launch_bounds__(256) i4_rows_kernel(const uint16_t *x, const int *x_index, int K, const int *tile_start, const int *tile_count,
                                                      const int *num_tiles, const int *total, uint16_t *xs) {
  pdl_wait();
  pdl_trigger();
  if (total && *total <= kWgSmallRows) return;
  const int ntiles = *num_tiles, per_row = K / 8;
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int p0 = tile_start[tile], n = tile_count[tile] * per_row;
    for (int u = blockIdx.y * 256 + threadIdx.x; u < n; u += gridDim.y * 256) {
      const int r = u / per_row, c = u - r * per_row;
      const size_t src = x_index ? (size_t)x_index[p0 + r] : (size_t)(p0 + r);
      const uint4 v = reinterpret_cast<const uint4 *>(x + src * K)[c];
      uint4 o;
      o.x = __byte_perm(v.x, v.z, 0x5410);
      o.y = __byte_perm(v.x, v.z, 0x7632);
      o.z = __byte_perm(v.y, v.w, 0x5410);
      o.w = __byte_perm(v.y, v.w, 0x7632);
      reinterpret_cast<uint4 *>(xs + (size_t)(p0 + r) * K)[c] = o;
    }
  }
}

static bool tc_aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

bool wgemm_i4_supports(const WgArgs &up, const WgArgs &down) {
  if (up.K % 512 || up.R % 512 || down.K != up.R || down.R != up.K) return false;
  for (const void *p : {up.w_a, up.w_b, down.w_a, (const void *)up.s_a, (const void *)up.s_b, (const void *)down.s_a, (const void *)up.x,
                        (const void *)up.out_bf16})
    if (!tc_aligned16(p)) return false;
  return true;
}

static int i4_launch(bool swiglu, const WgArgs &g, const uint16_t *x, long x_rows, cudaStream_t stream) {
  // rows past the last expert are never addressed: the coordinates come from the tile table
  constexpr long kRows = 1l << 31;
  CUtensorMap wa, wb, sa, sb, mx;
  int rc;
  if ((rc = tensor_map_2d(g.w_a, CU_TENSOR_MAP_DATA_TYPE_UINT8, kRows, g.K / 2, g.K / 2, 128, kI4Cols / 2, CU_TENSOR_MAP_SWIZZLE_128B, &wa))) return rc;
  if ((rc = tensor_map_2d(g.s_a, CU_TENSOR_MAP_DATA_TYPE_UINT8, kRows, g.K / 16, g.K / 16, 128, 32, CU_TENSOR_MAP_SWIZZLE_32B, &sa))) return rc;
  wb = wa;
  sb = sa;
  if (swiglu) {
    if ((rc = tensor_map_2d(g.w_b, CU_TENSOR_MAP_DATA_TYPE_UINT8, kRows, g.K / 2, g.K / 2, 128, kI4Cols / 2, CU_TENSOR_MAP_SWIZZLE_128B, &wb))) return rc;
    if ((rc = tensor_map_2d(g.s_b, CU_TENSOR_MAP_DATA_TYPE_UINT8, kRows, g.K / 16, g.K / 16, 128, 32, CU_TENSOR_MAP_SWIZZLE_32B, &sb))) return rc;
  }
  if ((rc = tensor_map_2d(x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, x_rows, g.K, (long)g.K * 2, 16, 64, CU_TENSOR_MAP_SWIZZLE_128B, &mx))) return rc;
  const I4Args a = {g.out_bf16, g.out_index, g.tile_expert, g.tile_start, g.tile_count, g.num_tiles, g.K, g.R, (int)g.expert_stride_rows, g.total,
                    g.w_a, g.w_b, g.s_a, g.s_b, x, g.err, g.overlap && !swiglu};
  auto kernel = swiglu ? wgemm_tc_kernel<true> : wgemm_tc_kernel<false>;
  if (int rc = allow_smem(kernel, kI4Smem)) return rc;
  return launch_pdl_if(g.overlap, "wgemm_tc_kernel", kernel, sm_count(), kI4Threads, (size_t)kI4Smem, stream, wa, wb, sa, sb, mx, a);
}

int launch_wgemm_i4(const WgArgs &up, const WgArgs &down, uint16_t *xs, long rows, int max_tiles, cudaStream_t stream) {
  // a tile's rows are shared by a few CTAs: 64 rows of 7,168 columns are 57,344 16-byte pieces
  int rc = launch_pdl_if(up.overlap, "i4_rows_kernel", i4_rows_kernel, dim3(std::min(max_tiles, 1024), 4), 256, 0, stream, up.x, up.x_index, up.K, up.tile_start,
                      up.tile_count, up.num_tiles, up.total, xs);
  if (rc) return rc;
  if ((rc = i4_launch(true, up, xs, rows, stream))) return rc;
  return i4_launch(false, down, up.out_bf16, rows, stream);
}

}  // namespace blok
