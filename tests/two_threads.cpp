// Two host threads that call the same function with different arguments as fast as they can (test_gpu_two_threads.py).
#include <atomic>
#include <cstddef>
#include <thread>

struct MlpCall {
  const void *gate, *up, *down, *x;
  void *y;
  int hidden, ffn, T;
  void *ws;
  size_t ws_bytes;
  void *stream;
};
typedef int (*mlp_fn)(const void *, const void *, const void *, const void *, void *, int, int, int, void *, size_t, void *);

// The number of calls that failed.
extern "C" int two_threads(mlp_fn fn, const MlpCall *a, const MlpCall *b, int calls) {
  std::atomic<int> failed{0}, ready{0};
  auto work = [&](const MlpCall *c) {
    for (++ready; ready < 2;) {
    }
    for (int i = 0; i < calls; ++i)
      if (fn(c->gate, c->up, c->down, c->x, c->y, c->hidden, c->ffn, c->T, c->ws, c->ws_bytes, c->stream)) ++failed;
  };
  std::thread other(work, b);
  work(a);
  other.join();
  return failed;
}
