// Host threading of the set-up code.
#pragma once
#include <stdint.h>

#include <algorithm>
#include <exception>
#include <thread>
#include <vector>

namespace adfem {

// run f(lo, hi) over [0, n) on up to 32 host threads (fewer where no more can be had); the first
// exception of a part is thrown again here when all have ended
template <class F>
static void parallel_for(int64_t n, F f) {
  unsigned nt = std::thread::hardware_concurrency();
  nt = std::max(1u, std::min(nt, 32u));
  if (n < 50000) nt = 1;
  if (nt == 1) {
    f((int64_t)0, n);
    return;
  }
  std::vector<std::exception_ptr> err(nt);
  auto part = [&](unsigned t) {
    try {
      f(n * t / nt, n * (t + 1) / nt);
    } catch (...) {
      err[t] = std::current_exception();
    }
  };
  std::vector<std::thread> th;
  th.reserve(nt);
  unsigned t = 1;
  try {
    for (; t < nt; t++) th.emplace_back(part, t);
  } catch (...) {  // (no further thread: their parts are run here)
  }
  part(0);
  for (; t < nt; t++) part(t);
  for (auto& x : th) x.join();
  for (auto& e : err)
    if (e) std::rethrow_exception(e);
}

}  // namespace adfem
