// Thread-parallel loop for host work over O(1e5) entries (the long-double ACAT
// terms of a scan).
#pragma once
#include <stdint.h>

#include <algorithm>
#include <thread>
#include <vector>

namespace eqtl {

// f(i) for i in [0, n), split into contiguous ranges over the host threads;
// small n runs inline.
template <class F>
void parallel_for(size_t n, F&& f, size_t min_per_thread = 4096) {
  const size_t hw = std::max(1u, std::thread::hardware_concurrency());
  const size_t nt = std::min(hw, (n + min_per_thread - 1) / std::max<size_t>(min_per_thread, 1));
  if (nt <= 1) {
    for (size_t i = 0; i < n; ++i) f(i);
    return;
  }
  std::vector<std::thread> th;
  th.reserve(nt);
  const size_t step = (n + nt - 1) / nt;
  for (size_t t = 0; t < nt; ++t) {
    const size_t lo = t * step, hi = std::min(n, lo + step);
    if (lo >= hi) break;
    th.emplace_back([&f, lo, hi] {
      for (size_t i = lo; i < hi; ++i) f(i);
    });
  }
  for (auto& x : th) x.join();
}

}  // namespace eqtl
