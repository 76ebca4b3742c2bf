// Host part of the multigrid hierarchy: aggregation of the matrix graph and the patterns of
// interpolation, A P and the coarse operators.  Runs once per system; no values.
#include "host_par.h"
#include "mg.cuh"

namespace adfem {
namespace {

// Aggregates of the graph.  First pass, in node order: a node none of whose neighbours is
// taken becomes the root of an aggregate of itself and its neighbours; with short_first, nodes with
// fewer neighbours than the average before the others (P2: edges, 9 entries a row, before
// vertices, 19, which makes aggregates of 9 instead of 16: 33 instead of 42 iterations at 5k DOF,
// 35 instead of 43 at 44k, 40 instead of 42 at 243k).  Second pass: the
// nodes left over join the neighbouring first-pass aggregate with which they share the most
// edges (the lowest-numbered of equals); nodes without one become aggregates of their own.
// Nodes without neighbours (eliminated rows of a user's matrix, whose interpolation is zero) are
// dealt over the aggregates in node order: on their own they would be unknowns of every level.
int64_t aggregate(int64_t n, const MgPattern& A, std::vector<int32_t>& agg, bool short_first) {
  agg.assign(n, -1);
  int32_t na = 0;
  auto alone = [&](int64_t i) {
    return A.rp[i + 1] == A.rp[i] || (A.rp[i + 1] == A.rp[i] + 1 && A.ci[A.rp[i]] == i);
  };
  for (int pass = short_first ? 0 : 1; pass < 2; pass++)
    for (int64_t i = 0; i < n; i++) {
      if (agg[i] >= 0 || alone(i)) continue;
      if (pass == 0 && n * (A.rp[i + 1] - A.rp[i]) >= (int64_t)A.rp[n]) continue;
      bool free = true;
      for (int32_t k = A.rp[i]; k < A.rp[i + 1] && free; k++) free = agg[A.ci[k]] < 0;
      if (!free) continue;
      agg[i] = na;
      for (int32_t k = A.rp[i]; k < A.rp[i + 1]; k++) agg[A.ci[k]] = na;
      na++;
    }
  std::vector<std::pair<int64_t, int32_t>> late;
  std::vector<int32_t> c;
  for (int64_t i = 0; i < n; i++) {
    if (agg[i] >= 0 || alone(i)) continue;
    c.clear();
    for (int32_t k = A.rp[i]; k < A.rp[i + 1]; k++)
      if (agg[A.ci[k]] >= 0) c.push_back(agg[A.ci[k]]);
    if (c.empty()) {
      late.emplace_back(i, na++);
      continue;
    }
    std::sort(c.begin(), c.end());
    int32_t best = c[0];
    size_t most = 0;
    for (size_t a = 0; a < c.size();) {
      size_t b = a;
      while (b < c.size() && c[b] == c[a]) b++;
      if (b - a > most) {
        most = b - a;
        best = c[a];
      }
      a = b;
    }
    late.emplace_back(i, best);
  }
  for (auto& p : late) agg[p.first] = p.second;
  if (na == 0) return n;  // no edges at all
  for (int64_t i = 0; i < n; i++)
    if (agg[i] < 0) agg[i] = (int32_t)(i * na / n);
  return na;
}

// Pattern whose row i is the sorted set of the columns (below nc) that emit(i, add) adds.  (Repeated
// ones are dropped as they come, by the row that last had the column: a coarse row meets each of its
// some 7 columns 15 to 20 times.)  Returns the longest row's entries, or kTooMany for more than limit
// entries in all (which are counted with 64 bits, but kept as 32).
constexpr int64_t kTooMany = INT64_MAX;
template <class F>
int64_t pattern(int64_t n, int64_t nc, int64_t limit, MgPattern& P, F emit) {
  constexpr int64_t kChunk = 16384;
  const int64_t nch = (n + kChunk - 1) / kChunk;
  std::vector<std::vector<int32_t>> part(nch);
  P.rp.assign(n + 1, 0);
  // (parallel_for splits by index; scale the chunk count up so that it threads)
  const int64_t m = n < 50000 ? nch : std::max<int64_t>(nch, 50000);
  parallel_for(m, [&](int64_t lo, int64_t hi) {
    std::vector<int32_t> v, seen(nc, -1);
    for (int64_t c = lo * nch / m; c < hi * nch / m; c++)
      for (int64_t i = c * kChunk; i < std::min(n, (c + 1) * kChunk); i++) {
        v.clear();
        emit(i, [&](int32_t j) {
          if (seen[j] == (int32_t)i) return;
          seen[j] = (int32_t)i;
          v.push_back(j);
        });
        std::sort(v.begin(), v.end());
        part[c].insert(part[c].end(), v.begin(), v.end());
        P.rp[i + 1] = (int32_t)v.size();
      }
  });
  int64_t w = 0, total = 0;
  for (int64_t i = 0; i < n; i++) {
    w = std::max<int64_t>(w, P.rp[i + 1]);
    total += P.rp[i + 1];
    if (total > limit) return kTooMany;
    P.rp[i + 1] = (int32_t)total;
  }
  P.ci.resize(P.rp[n]);
  parallel_for(m, [&](int64_t lo, int64_t hi) {
    for (int64_t c = lo * nch / m; c < hi * nch / m; c++)
      std::copy(part[c].begin(), part[c].end(), P.ci.begin() + P.rp[c * kChunk]);
  });
  return w;
}

// whether a pattern in slices of 32 rows has at most limit / nb entries (a slice has at most 32 times
// its rows' entries: no need to look at most patterns)
bool fits(int64_t n, const MgPattern& P, int nb, int64_t limit) {
  if (32 * (int64_t)P.rp[n] * nb <= limit) return true;
  int64_t s = 0;
  for (int64_t r0 = 0; r0 < n; r0 += 32) {
    int64_t w = 0;
    for (int64_t r = r0; r < std::min(n, r0 + 32); r++) w = std::max<int64_t>(w, P.rp[r + 1] - P.rp[r]);
    s += 32 * w;
  }
  return s * nb <= limit;
}

}  // namespace

bool mg_build_host(int64_t n, std::vector<int32_t>&& rp, std::vector<int32_t>&& ci, int nb0, int nbc,
                   std::vector<double>&& x, std::vector<double>&& y, std::vector<MgHostLevel>& lv, int64_t limit) {
  lv.clear();
  lv.emplace_back();
  lv[0].n = n;
  lv[0].A.rp = std::move(rp);
  lv[0].A.ci = std::move(ci);
  lv[0].x = std::move(x);
  lv[0].y = std::move(y);
  for (;;) {
    MgHostLevel& L = lv.back();
    const int nb = lv.size() == 1 ? nb0 : nbc;
    if (!fits(L.n, L.A, nb, limit)) return false;
    if (L.n * nb <= kMgDense) break;
    if ((int)lv.size() == kMgMaxLevels) return false;
    // (rows of two kinds: on the system's own level, where the longest is 1.5 times the average)
    int64_t longest = 0;
    if (lv.size() == 1)
      for (int64_t i = 0; i < L.n; i++) longest = std::max<int64_t>(longest, L.A.rp[i + 1] - L.A.rp[i]);
    const int64_t nc = aggregate(L.n, L.A, L.agg, 2 * longest * L.n >= 3 * (int64_t)L.A.rp[L.n]);
    if (2 * nc > L.n) return false;  // hardly any edges: no hierarchy
    auto rows = [](const MgPattern& Q, int64_t i, auto&& add) {
      for (int32_t k = Q.rp[i]; k < Q.rp[i + 1]; k++) add(Q.ci[k]);
    };
    if (pattern(L.n, nc, limit, L.P, [&](int64_t i, auto&& add) {
          for (int32_t k = L.A.rp[i]; k < L.A.rp[i + 1]; k++) add(L.agg[L.A.ci[k]]);
        }) > kMgMaxP)
      return false;
    if (pattern(L.n, nc, limit, L.AP, [&](int64_t i, auto&& add) {
          for (int32_t k = L.A.rp[i]; k < L.A.rp[i + 1]; k++) rows(L.P, L.A.ci[k], add);
        }) > kMgMaxAP)
      return false;
    // transpose of P, nodes ascending within each aggregate's row
    L.PT.rp.assign(nc + 1, 0);
    for (int32_t J : L.P.ci) L.PT.rp[J + 1]++;
    for (int64_t J = 0; J < nc; J++) L.PT.rp[J + 1] += L.PT.rp[J];
    L.PT.ci.resize(L.P.ci.size());
    L.PTslot.resize(L.P.ci.size());
    {
      std::vector<int32_t> fill(L.PT.rp.begin(), L.PT.rp.end() - 1);
      for (int64_t i = 0; i < L.n; i++)
        for (int32_t k = L.P.rp[i]; k < L.P.rp[i + 1]; k++) {
          const int32_t q = fill[L.P.ci[k]]++;
          L.PT.ci[q] = (int32_t)i;
          L.PTslot[q] = k - L.P.rp[i];
        }
    }
    if (!fits(L.n, L.P, 1, limit) || !fits(L.n, L.AP, 1, limit) || !fits(nc, L.PT, 1, limit)) return false;
    MgHostLevel C;
    C.n = nc;
    if (pattern(nc, nc, limit, C.A, [&](int64_t J, auto&& add) {
          for (int32_t q = L.PT.rp[J]; q < L.PT.rp[J + 1]; q++) rows(L.AP, L.PT.ci[q], add);
        }) > kMgMaxA)
      return false;
    if (!L.x.empty()) {
      C.x.assign(nc, 0.0);
      C.y.assign(nc, 0.0);
      std::vector<int32_t> cnt(nc, 0);
      for (int64_t i = 0; i < L.n; i++) {
        C.x[L.agg[i]] += L.x[i];
        C.y[L.agg[i]] += L.y[i];
        cnt[L.agg[i]]++;
      }
      for (int64_t J = 0; J < nc; J++) {
        C.x[J] /= cnt[J];
        C.y[J] /= cnt[J];
      }
    }
    lv.push_back(std::move(C));
  }
  return true;
}

}  // namespace adfem
