// Error plumbing and small ABI-level helpers.
#include <atomic>
#include <cstdarg>
#include <cstring>
#include <mutex>

#include "common.cuh"

namespace blok {

static thread_local char g_error[512] = "";

void set_error(const char *fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_error, sizeof(g_error), fmt, ap);
  va_end(ap);
}

int cuda_fail(cudaError_t e, const char *what) {
  cudaGetLastError();  // reported here: the program's next CUDA call must not find it
  set_error("%s: %s", what, cudaGetErrorString(e));
  return BLOK_ERR_CUDA;
}

static std::atomic<long long> g_launches{0};
void count_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }
void count_launches(long long n) { g_launches.fetch_add(n, std::memory_order_relaxed); }
long long launches_so_far() { return g_launches.load(std::memory_order_relaxed); }
long long launches() { return g_launches.load(std::memory_order_relaxed); }

int sm_count() {
  static thread_local int cached_dev = -1, cached = 0;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 148;
  if (dev != cached_dev) {
    cudaDeviceProp p;
    if (cudaGetDeviceProperties(&p, dev) != cudaSuccess) return 148;
    cached = p.multiProcessorCount;
    cached_dev = dev;
  }
  return cached;
}

// The bytes of a kernel's static arrays, which do not change; a table without allocations.
static int static_smem_of(const void *kernel, size_t *bytes) {
  struct Known {
    std::atomic<const void *> kernel{nullptr};
    size_t bytes = 0;  // written before the kernel is
  };
  constexpr size_t kSlots = 512;
  static Known known[kSlots];
  static std::mutex mu;
  const size_t home = reinterpret_cast<uintptr_t>(kernel) / 16 % kSlots;
  auto find = [&]() -> Known * {  // its slot, or the free one; NULL: the table is full
    for (size_t i = 0; i < kSlots; ++i) {
      Known *k = known + (home + i) % kSlots;
      const void *is = k->kernel.load(std::memory_order_acquire);
      if (is == kernel || !is) return k;
    }
    return nullptr;
  };
  Known *k = find();
  if (k && k->kernel.load(std::memory_order_acquire) == kernel) {
    *bytes = k->bytes;
    return BLOK_OK;
  }
  cudaFuncAttributes a;
  BLOK_CUDA(cudaFuncGetAttributes(&a, kernel));
  *bytes = a.sharedSizeBytes;
  std::lock_guard<std::mutex> lock(mu);
  if ((k = find()) && !k->kernel.load(std::memory_order_relaxed)) {
    k->bytes = a.sharedSizeBytes;
    k->kernel.store(kernel, std::memory_order_release);
  }
  return BLOK_OK;
}

constexpr size_t kFreeSmem = 48 * 1024, kMostSmem = 227 * 1024;  // of a block, static arrays included: unasked, and at most

int allow_smem_of(const void *kernel, size_t dynamic) {
  size_t fixed = 0;
  if (int rc = static_smem_of(kernel, &fixed)) return rc;
  if (fixed + dynamic <= kFreeSmem) return BLOK_OK;
  BLOK_REQUIRE(fixed + dynamic <= kMostSmem, BLOK_ERR_SHAPE, "a kernel wants %zu bytes of shared memory (at most %zu)", fixed + dynamic, kMostSmem);
  BLOK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kMostSmem - fixed)));
  return BLOK_OK;
}

}  // namespace blok

extern "C" const char *blok_last_error(void) { return blok::g_error; }
extern "C" int blok_abi_version(void) { return BLOK_ABI_VERSION; }
extern "C" long long blok_kernel_launch_count(void) { return blok::launches(); }
