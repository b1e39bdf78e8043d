// Two host threads that call the same function with different arguments as fast as they can (test_gpu_two_threads.py).
#include <atomic>
#include <cstddef>
#include <cstdio>
#include <thread>

struct MlpCall {
  const void *gate, *up, *down, *x;
  void *y;
  int hidden, ffn, T;
  void *ws;
  size_t ws_bytes;
  void *stream;
};
typedef const char *(*message_fn)();
typedef int (*mlp_fn)(const void *, const void *, const void *, const void *, void *, int, int, int, void *, size_t, void *);

// The number of calls that failed; their threads' last messages to stderr.
extern "C" int two_threads(mlp_fn fn, message_fn message, const MlpCall *a, const MlpCall *b, int calls) {
  std::atomic<int> failed{0}, ready{0};
  auto work = [&](const MlpCall *c) {
    for (++ready; ready < 2;) {
    }
    int own = 0;
    for (int i = 0; i < calls; ++i)
      if (fn(c->gate, c->up, c->down, c->x, c->y, c->hidden, c->ffn, c->T, c->ws, c->ws_bytes, c->stream)) ++own;
    if (own) fprintf(stderr, "%d of %d calls over %d rows failed: %s\n", own, calls, c->T, message());
    failed += own;
  };
  std::thread other(work, b);
  work(a);
  other.join();
  return failed;
}
