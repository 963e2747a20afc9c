// Host worker threads shared by the library's host phases.
#pragma once
#include <cstdint>
#include <functional>

namespace fem2d {

// host threads that a phase may use (the hardware's, at most 64)
int num_host_threads();

// f(t) for t = 0 .. nt - 1, spread over the calling thread and the kept workers; returns when all are done.
// Any number of threads may call it at once: callers share the workers, and a caller runs whatever of its
// own calls no worker has taken, so none waits for another's. The first exception of f is rethrown here.
void run_threads(int nt, const std::function<void(int)>& f);

// f(begin, end) over [0, n) in contiguous chunks, inline below `grain` elements
template <class F>
void parallel_for(int64_t n, F f, int64_t grain = 4096) {
  const int nt = n < grain ? 1 : num_host_threads();
  if (nt <= 1) {
    f((int64_t)0, n);
    return;
  }
  const int64_t chunk = (n + nt - 1) / nt;
  run_threads((int)((n + chunk - 1) / chunk), [&](int t) {
    const int64_t a = t * chunk, b = a + chunk < n ? a + chunk : n;
    f(a, b);
  });
}

}  // namespace fem2d
