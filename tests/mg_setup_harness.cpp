// CPU harness for the multigrid set-up code (adfem.jl_gb300/csrc/mg_setup.cpp, host_par.h), built and
// run by tests/test_mg_setup_cpu.py.  Test infrastructure only: nothing in the library uses it.
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <new>
#include <stdexcept>

#include "host_par.h"
#include "mg.cuh"

namespace adfem {
Mg::~Mg() {}
void DevBuf::release() {}
}  // namespace adfem
using namespace adfem;

// the k-th following allocation fails, whichever thread makes it (k < 0: none)
static std::atomic<long long> g_fail{-1};
void* operator new(std::size_t n) {
  if (g_fail.load() >= 0 && g_fail.fetch_sub(1) == 0) throw std::bad_alloc();
  if (void* p = std::malloc(n ? n : 1)) return p;
  throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }

#define REQUIRE(c)                                          \
  do {                                                      \
    if (!(c)) {                                             \
      std::printf("failed at line %d: %s\n", __LINE__, #c); \
      std::exit(1);                                         \
    }                                                       \
  } while (0)

// graph of a square of m x n cells with one diagonal each
static void graph(int64_t m, int64_t n, std::vector<int32_t>& rp, std::vector<int32_t>& ci) {
  rp.assign(1, 0);
  ci.clear();
  for (int64_t i = 0; i < (m + 1) * (n + 1); i++) {
    const int64_t x = i % (m + 1), y = i / (m + 1);
    for (int dy = -1; dy <= 1; dy++)
      for (int dx = -1; dx <= 1; dx++) {
        if (dx * dy == 1 || x + dx < 0 || x + dx > m || y + dy < 0 || y + dy > n) continue;
        ci.push_back((int32_t)((y + dy) * (m + 1) + x + dx));
      }
    rp.push_back((int32_t)ci.size());
  }
}

static bool build(int64_t m, int64_t n, std::vector<MgHostLevel>& lv, int64_t limit = INT32_MAX) {
  std::vector<int32_t> rp, ci;
  graph(m, n, rp, ci);
  return mg_build_host((m + 1) * (n + 1), std::move(rp), std::move(ci), 1, 1, {}, {}, lv, limit);
}

static int64_t sliced_entries(int64_t n, const MgPattern& P) {
  int64_t s = 0;
  for (int64_t r0 = 0; r0 < n; r0 += 32) {
    int w = 0;
    for (int64_t r = r0; r < n && r < r0 + 32; r++) w = std::max(w, P.rp[r + 1] - P.rp[r]);
    s += 32 * w;
  }
  return s;
}

// every index of the hierarchy is in range, and the largest pattern (sliced) has `most` entries
static void check(const std::vector<MgHostLevel>& lv, int64_t* most) {
  *most = 0;
  for (size_t l = 0; l < lv.size(); l++) {
    const MgHostLevel& L = lv[l];
    for (int32_t c : L.A.ci) REQUIRE(c >= 0 && c < L.n);
    *most = std::max(*most, sliced_entries(L.n, L.A));
    if (l + 1 == lv.size()) continue;
    const int64_t nc = lv[l + 1].n;
    for (int32_t a : L.agg) REQUIRE(a >= 0 && a < nc);
    for (int32_t c : L.P.ci) REQUIRE(c >= 0 && c < nc);
    for (int32_t c : L.AP.ci) REQUIRE(c >= 0 && c < nc);
    for (int64_t J = 0; J < nc; J++)
      for (int32_t k = L.PT.rp[J]; k < L.PT.rp[J + 1]; k++)
        REQUIRE(L.P.ci[L.P.rp[L.PT.ci[k]] + L.PTslot[k]] == J);
    *most = std::max(*most, std::max(sliced_entries(L.n, L.P), sliced_entries(L.n, L.AP)));
    *most = std::max(*most, sliced_entries(nc, L.PT));
  }
}

int main(int argc, char** argv) {
  REQUIRE(argc == 2);
  if (!std::strcmp(argv[1], "limit")) {
    // patterns with more entries than can be numbered are refused, whichever of them it is
    std::vector<MgHostLevel> lv;
    int64_t most = 0;
    REQUIRE(build(90, 70, lv));
    check(lv, &most);
    REQUIRE(build(90, 70, lv, most));
    for (int64_t limit = most - 1; limit > 0; limit /= 2) REQUIRE(!build(90, 70, lv, limit));
  }
  if (!std::strcmp(argv[1], "exceptions")) {
    // an exception of one thread's part reaches the caller, after all parts have ended
    std::atomic<int64_t> done{0};
    bool caught = false;
    try {
      parallel_for(100000, [&](int64_t lo, int64_t hi) {
        done += hi - lo;
        if (lo <= 70000 && 70000 < hi) throw std::runtime_error("part");
      });
    } catch (const std::runtime_error&) {
      caught = true;
    }
    REQUIRE(caught && done.load() == 100000);
    // every allocation of a set-up (90k nodes: threaded, the threads' own included) fails in turn: the
    // caller gets std::bad_alloc (or the whole hierarchy, where only a thread was not to be had) and
    // still has the graph
    std::vector<int32_t> rp0, ci0;
    graph(299, 299, rp0, ci0);
    int64_t most = 0;
    int thrown = 0;
    bool whole = false;
    for (long long k = 0; !whole; k += 1 + k / 16) {
      std::vector<MgHostLevel> lv;
      std::vector<int32_t> rp = rp0, ci = ci0;
      g_fail = k;
      try {
        REQUIRE(mg_build_host(90000, std::move(rp), std::move(ci), 1, 1, {}, {}, lv));
        whole = g_fail.exchange(-1) >= 0;
        check(lv, &most);
      } catch (const std::bad_alloc&) {
        g_fail = -1;
        thrown++;
        REQUIRE(lv.empty() ? rp == rp0 && ci == ci0 : lv[0].A.rp == rp0 && lv[0].A.ci == ci0);
      }
    }
    REQUIRE(thrown > 20);
  }
  std::printf("mg setup ok\n");
  return 0;
}
