// CPU harness for the multigrid set-up code (adfem.jl_gb300/csrc/mg_setup.cpp, host_par.h), built and
// run by tests/test_mg_setup_cpu.py.  Test infrastructure only: nothing in the library uses it.
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "mg.cuh"

namespace adfem {
Mg::~Mg() {}
void DevBuf::release() {}
}  // namespace adfem
using namespace adfem;

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
  std::printf("mg setup ok\n");
  return 0;
}
