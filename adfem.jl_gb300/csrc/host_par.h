// Host threading of the set-up code.
#pragma once
#include <stdint.h>

#include <algorithm>
#include <thread>
#include <vector>

namespace adfem {

// run f(lo, hi) over [0, n) on up to 32 host threads
template <class F>
static void parallel_for(int64_t n, F f) {
  unsigned nt = std::thread::hardware_concurrency();
  nt = std::max(1u, std::min(nt, 32u));
  if (n < 50000) nt = 1;
  if (nt == 1) {
    f((int64_t)0, n);
    return;
  }
  std::vector<std::thread> th;
  for (unsigned t = 0; t < nt; t++) {
    int64_t lo = n * t / nt, hi = n * (t + 1) / nt;
    th.emplace_back([=] { f(lo, hi); });
  }
  for (auto& x : th) x.join();
}

}  // namespace adfem
