// A launch in front of the weight stream that lets it begin at once and takes its time (test_gpu_slow_front.py).
#include "wgemm.h"

#include "common.cuh"

namespace blok {

// Copies n values after about `us` microseconds; the kernel behind may become resident meanwhile.
__global__ void slow_copy_kernel(const uint16_t *from, uint16_t *to, int n, int us) {
  pdl_trigger();
  pdl_wait();
  for (int i = 0; i < us; ++i) __nanosleep(1000);
  for (int i = threadIdx.x; i < n; i += blockDim.x) to[i] = from[i];
}

}  // namespace blok

using namespace blok;

// out[t, r] = sum_k w[r, k] x[t, k], x a copy of x_from that the launch in front makes; *err as the kernel leaves it.
extern "C" int slow_front_product(const uint16_t *w, const uint16_t *x_from, uint16_t *x, float *out, int R, int K, int T, int us, unsigned *err,
                                  void *stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (int rc = launch_pdl("slow_copy_kernel", slow_copy_kernel, 1, 256, 0, stream, x_from, x, T * K, us)) return rc;
  WgArgs a = wgemm_rows(w, nullptr, x, nullptr, out, R, K, T);
  a.weights_early = true;
  a.err = err;
  int splits = 1;
  return launch_wgemm_stream(WG_BF16_PLAIN, a, &splits, stream);
}
