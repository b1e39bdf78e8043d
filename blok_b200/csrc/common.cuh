// Shared device/host helpers for the sm_100a kernels.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cstdint>
#include <cstdio>

#include "../../include/blok_b200.h"

namespace blok {

// ---- error plumbing (host) -------------------------------------------------
void set_error(const char *fmt, ...);
int cuda_fail(cudaError_t e, const char *what);

#define BLOK_CUDA(call)                                        \
  do {                                                         \
    cudaError_t e_ = (call);                                   \
    if (e_ != cudaSuccess) return ::blok::cuda_fail(e_, #call); \
  } while (0)

#define BLOK_REQUIRE(cond, code, ...) \
  do {                                \
    if (!(cond)) {                    \
      ::blok::set_error(__VA_ARGS__); \
      return (code);                  \
    }                                 \
  } while (0)

void count_launch();
void count_launches(long long n);  // kernels replayed from a CUDA graph
long long launches_so_far();

inline int launch_status(const char *what) {
  count_launch();
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? BLOK_OK : cuda_fail(e, what);
}

int sm_count();

// Lets a kernel be launched with `dynamic` bytes of dynamic shared memory: a launch gets 48 KB, its static arrays among them, without asking.
// The limit is the function's, for all threads of the program, so it is always set to the same value: a smaller one could come between
// another thread's call and its launch.
int allow_smem_of(const void *kernel, size_t dynamic);
template <typename... P>
inline int allow_smem(void (*kernel)(P...), size_t dynamic) {
  return allow_smem_of(reinterpret_cast<const void *>(kernel), dynamic);
}

// Launches a kernel that begins with pdl_wait(): its blocks may become resident while the kernel before it runs (programmatic
// dependent launch), which takes the launch and the start of its blocks off the critical path; captured into graphs like any
// other launch.  Some forty launches of 5 to 50 us in a prompt of 60 / 130 / 1,000 tokens: 547 / 612 / 1,050 -> 500 / 517 / 956 us; over
// 2,048 tokens of routed experts, where a launch takes 800 us, it costs 1 to 2 %.  For kernels whose blocks fill an SM (shared memory) or are few and small.  Not for the mat-vec kernels: blocks
// that come early crowd on the SMs that have room, and the stream of weights is then uneven (o_proj over 8 rows 29 -> 80 us).
// overlap false: an ordinary launch of the same kernel.
template <typename... P, typename... A>
inline int launch_pdl_if(bool overlap, const char *what, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A... args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = overlap ? 1 : 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  count_launch();
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
  return e == cudaSuccess ? BLOK_OK : cuda_fail(e, what);
}
template <typename... P, typename... A>
inline int launch_pdl(const char *what, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A... args) {
  return launch_pdl_if(true, what, kernel, grid, block, smem, stream, args...);
}

// ---- device helpers ----------------------------------------------------------
// The kernel behind this one may become resident as soon as every block of this one has started.
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// Everything before this launch has finished and is visible; nothing that it reads or writes may be touched earlier.  Without the launch attribute both do nothing.
// The kernel is resident while others write what it will read, so its inputs are plain pointers: const __restrict__ or __ldg would
// promise that nobody writes them while it lives, and let the compiler and the read-only path fetch them before the wait.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ float bf16_bits_to_f32(uint32_t h) { return __uint_as_float(h << 16); }
__device__ __forceinline__ float bf16lo(uint32_t pair) { return __uint_as_float(pair << 16); }
__device__ __forceinline__ float bf16hi(uint32_t pair) { return __uint_as_float(pair & 0xffff0000u); }

__device__ __forceinline__ uint16_t f32_to_bf16_bits(float f) {
  return __bfloat16_as_ushort(__float2bfloat16_rn(f));
}
__device__ __forceinline__ float round_bf16(float f) { return __bfloat162float(__float2bfloat16_rn(f)); }

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  return (uint32_t)f32_to_bf16_bits(lo) | ((uint32_t)f32_to_bf16_bits(hi) << 16);
}

// 128-bit streaming load of weights that are read exactly once per pass.
__device__ __forceinline__ uint4 ldg_stream(const uint4 *p) {
  uint4 v;
  asm("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}

// D(16x8, fp32) += A(16x16, bf16, row) * B(16x8, bf16, col).
__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                               uint32_t b0, uint32_t b1) {
  asm(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

__device__ __forceinline__ float silu_mul_f32(float g, float u) { return g / (1.0f + __expf(-g)) * u; }

}  // namespace blok
