// Multigrid-preconditioned CG of the resident systems (sm_103a).
//
// Jacobi-CG needs 5,000 to 16,000 iterations at 1M to 4M unknowns, each near the memory
// bound already, so the time of a solve is their number.  Here the preconditioner is one
// V-cycle of smoothed aggregation in FP32, and the CG around it is FP64: iterate, residual,
// direction, products with K and every sum (r.z is the FP64 sum over the cycle's FP32 input and
// output).  Iterations at 625 to 4M unknowns: P1 Poisson 14 to 36, P2 33 to 53, elasticity 36 to 70.
//  * Patterns (aggregates, interpolation, A P, coarse operators) are made once per system on
//    the host (mg_setup.cpp); after an assembly the kernels below fill in the values.
//  * Level 0 is S K S, S = diag(K_ii^-1/2) as in the Jacobi iterations, so the stopping
//    quantity is unchanged; the coarse operators are scaled to unit diagonal as well.
//  * Interpolation: P = P0 - (c / q_i) A P0, q_i the weighted absolute row sum (2 for a row
//    of an M-matrix with zero sum), c = 1.6 on level 0 and 1.8 below it, 1.8 and 2.2 for elasticity
//    (q_i, a bound, is further from the spectrum on blocks; 1.6 throughout: 38 instead of 36
//    iterations at 4M DOF, 68 instead of 58 for elasticity at 320k); P0 is piecewise constant on the aggregates, plus the
//    rotation about the aggregate's centre for 2-D elasticity.
//  * Smoother: Chebyshev of degree 2 on level 0 and 4 below (the coarse levels are cheap and
//    the V-cycle gains most there), on [fr lam, lam] with lam = max q_i, an upper bound of the
//    spectrum, so the cycle is symmetric positive definite for every input.
//  * Every sum is formed by one thread or a fixed shuffle tree: results repeat bit for bit.
//  * A solve is one launch up to kMgTailDofs unknowns (k_mg_tail), above that one CUDA graph: a
//    while node around one iteration, left when a residual
//    evaluated in FP64 from the iterate meets the tolerance (or the iteration ends otherwise);
//    the host waits once.
#include <cmath>
#include <cstring>
#include <mutex>
#include <thread>
#include <type_traits>

#include "cg_common.cuh"
#include "checks.cuh"
#include "host_par.h"

namespace adfem {

Mg::~Mg() {
  if (solve) cudaGraphExecDestroy(solve);
}

namespace {

constexpr float kFrac0 = 0.125f, kFrac = 0.06f;  // lower end of the Chebyshev interval over lam
constexpr int kCoef = 2 * kMgDeg;
constexpr size_t kTailSmem = 224 * 1024;  // shared memory of a tail block, at most

template <int NB>
struct Vec {
  float v[NB];
};
template <int NB>
__device__ __forceinline__ Vec<NB> load_vec(const float* p, int64_t i) {
  Vec<NB> r;
  if constexpr (NB == 2) {
    const float2 t = reinterpret_cast<const float2*>(p)[i];
    r.v[0] = t.x;
    r.v[1] = t.y;
  } else {
#pragma unroll
    for (int c = 0; c < NB; c++) r.v[c] = p[NB * i + c];
  }
  return r;
}
template <int NB>
__device__ __forceinline__ void store_vec(float* __restrict__ p, int64_t i, const Vec<NB>& r) {
  if constexpr (NB == 2) reinterpret_cast<float2*>(p)[i] = make_float2(r.v[0], r.v[1]);
  else
#pragma unroll
    for (int c = 0; c < NB; c++) p[NB * i + c] = r.v[c];
}
// R x C blocks of an array of n entries: 2 x 2 blocks as one 16-byte word each, other blocks as
// R C planes of n floats (a warp's loads of one component are then consecutive; 36-byte blocks
// side by side cost nine times the L1 wavefronts).
template <int R, int C>
__device__ __forceinline__ void load_block(const float* __restrict__ m, int idx, int n, float (&v)[R * C]) {
  if constexpr (R == 2 && C == 2) {
    const float4 t = reinterpret_cast<const float4*>(m)[idx];
    v[0] = t.x;
    v[1] = t.y;
    v[2] = t.z;
    v[3] = t.w;
  } else {
#pragma unroll
    for (int e = 0; e < R * C; e++) v[e] = m[(int64_t)e * n + idx];
  }
}
template <int R, int C>
__device__ __forceinline__ int64_t block_at(int e, int64_t idx, int n) {
  return R == 2 && C == 2 ? 4 * idx + e : (int64_t)e * n + idx;
}
// acc += M x
template <int R, int C>
__device__ __forceinline__ void block_fma(const float* __restrict__ m, int idx, int n, const Vec<C>& x,
                                          Vec<R>& acc) {
  float v[R * C];
  load_block<R, C>(m, idx, n, v);
#pragma unroll
  for (int r = 0; r < R; r++)
#pragma unroll
    for (int c = 0; c < C; c++) acc.v[r] = fmaf(v[r * C + c], x.v[c], acc.v[r]);
}
template <int NB, int LPR>
__device__ __forceinline__ void lane_sum(Vec<NB>& a) {
#pragma unroll
  for (int o = LPR / 2; o > 0; o >>= 1)
#pragma unroll
    for (int c = 0; c < NB; c++) a.v[c] += __shfl_xor_sync(0xffffffffu, a.v[c], o);
}

// rows of sliced patterns: first entry and width
__device__ __forceinline__ void slice_row(const int32_t* __restrict__ sptr, int r, int64_t& base, int& w) {
  const int32_t s0 = __ldg(sptr + (r >> 5)), s1 = __ldg(sptr + (r >> 5) + 1);
  base = (int64_t)s0 + (r & 31);
  w = (s1 - s0) >> 5;
}

// column of entry k (at idx) of row r of the level's operator
template <bool D16>
struct Cols {
  const MgLev& L;
  int r, so;
  __device__ __forceinline__ Cols(const MgLev& lv, int row) : L(lv), r(row), so(-1) {
    if (D16) so = __ldg(L.spat + (row >> 5));
  }
  __device__ __forceinline__ int at(int k, int idx) const {
    if (D16) return r + (int)(so >= 0 ? __ldg(L.pat + so + k) : __ldg(reinterpret_cast<const int16_t*>(L.col) + idx));
    return __ldg(reinterpret_cast<const int32_t*>(L.col) + idx);
  }
};

// Row r of the level's operator for one of its LPR lanes.  The first group of entries is loaded
// ahead: the operators do not change while a solve runs, so a kernel has its first rows in
// registers when the launch before it ends.
template <int NB, bool D16, int LPR>
struct RowHead {
  // entries in groups whose loads are all in flight at once
  static constexpr int U = LPR == 1 ? (NB == 1 ? 8 : 4) : 2;
  float v[U][NB * NB];
  int j[U];
  int base = 0, w = 0;
  __device__ __forceinline__ void load(const MgLev& L, int r, int lane) {
    const int s0 = __ldg(L.sptr + (r >> 5));
    w = (__ldg(L.sptr + (r >> 5) + 1) - s0) >> 5;
    base = s0 + (r & 31);
    const Cols<D16> cols(L, r);
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int k = lane + u * LPR;
      j[u] = k < w ? cols.at(k, base + 32 * k) : r;
      if (!ADFEM_DCHECK(j[u] >= 0 && j[u] < L.n)) j[u] = r;
      if (k < w) load_block<NB, NB>(L.val, base + 32 * k, L.nv, v[u]);
    }
  }
  // (A x)_r (every lane gets the sum)
  __device__ __forceinline__ Vec<NB> product(const MgLev& L, int r, int lane, const float* x) const {
    Vec<NB> acc;
#pragma unroll
    for (int c = 0; c < NB; c++) acc.v[c] = 0.0f;
#pragma unroll
    for (int u = 0; u < U; u++)
      if (lane + u * LPR < w) {
        const Vec<NB> t = load_vec<NB>(x, j[u]);
#pragma unroll
        for (int a = 0; a < NB; a++)
#pragma unroll
          for (int c = 0; c < NB; c++) acc.v[a] = fmaf(v[u][a * NB + c], t.v[c], acc.v[a]);
      }
    const Cols<D16> cols(L, r);
    for (int k0 = lane + U * LPR; k0 < w; k0 += U * LPR) {
      int i[U];
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int k = k0 + u * LPR;
        i[u] = k < w ? cols.at(k, base + 32 * k) : r;
        if (!ADFEM_DCHECK(i[u] >= 0 && i[u] < L.n)) i[u] = r;
      }
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int k = k0 + u * LPR;
        if (k < w) block_fma<NB, NB>(L.val, base + 32 * k, L.nv, load_vec<NB>(x, i[u]), acc);
      }
    }
    if (LPR > 1) lane_sum<NB, LPR>(acc);
    return acc;
  }
};

// Sums over a grid: every block leaves its partial sum (block_partial), and the kernel that needs
// the total forms it in each of its blocks, in one order, from the same words (grid_total).  The
// kernel boundary in between is there anyway; a last block that adds up instead costs every block
// a fence and a count (some 2 us in which its place on the SM is idle) and the registers of the
// addition (last sweep of level 0 with its dot product: 45 against 34 us at 4M rows, 22 against 14 us
// at 240k rows of P2).
// A block's values go through shared memory to its first warp, eight to a lane (13 warp additions a
// block instead of 40 of shuffle trees in every warp).  The products are FP64 too, as in the Jacobi
// iterations: in FP32 and FP32 pairs an iteration takes 235 instead of 243 us at 1M unknowns, 42.4
// instead of 44.5 at 4225, 194 instead of 198 for elasticity at 320k, and the iterations are the same.
__device__ __forceinline__ void block_partial(double x, double* partials) {
  __shared__ double sh[kT];
  const int lane = threadIdx.x;
  sh[threadIdx.x] = x;
  __syncthreads();
  if (threadIdx.x >= 32) return;
  double s = sh[lane];
#pragma unroll
  for (int k = 1; k < kT / 32; k++) s += sh[lane + 32 * k];
  s = warp_sum(s);
  if (lane == 0) partials[blockIdx.x] = s;
}
// The total as f makes two words of it.  (One warp adds and one thread runs f: an FP64 warp
// instruction holds the SM's FP64 pipe for 16 cycles, and a division is some twenty of them, one
// after the other: run by every thread, f cost 7 us a kernel.  So the state keeps reciprocals.
// f also looks at st->done, which the first block may be setting: a block goes by one reading.)
template <class F>
__device__ __forceinline__ double2 grid_total(const double* partials, int count, F f) {
  __shared__ double2 out;
  if (threadIdx.x < 32) {
    constexpr int K = 20;
    double s[4] = {0.0, 0.0, 0.0, 0.0};
    for (int b0 = 0; b0 < count; b0 += 32 * K) {
      double v[K];
#pragma unroll
      for (int k = 0; k < K; k++) {
        const int b = b0 + 32 * k + (int)threadIdx.x;
        v[k] = b < count ? partials[b] : 0.0;
      }
#pragma unroll
      for (int k = 0; k < K; k++)
        if (b0 + 32 * k < count) s[k & 3] += v[k];
    }
    double t = s[0];
    if (count > 32) t = (t + s[1]) + (s[2] + s[3]);
    t = warp_sum(t);
    if (threadIdx.x == 0) out = f(t);
  }
  __syncthreads();
  return out;
}

// ---------------------------------------------------------------------------
// V-cycle kernels of the levels above the tail.  Every kernel of an iteration is a programmatic
// dependent launch: its blocks start as the kernel before runs out, load what does not change
// during a solve, and wait for that kernel before they read or write a vector (an iteration, with
// the sums below: 277 -> 229 us at 1M unknowns, 235 -> 190 us elasticity at 320k, 57 -> 51 us at 4k).  (So vectors are
// read by plain loads: the read-only path is for data that is constant while a kernel lives.)
enum { kPre = 0, kStep = 1, kRes = 2, kLast = 3 };

// kPre:  two Chebyshev steps from x = 0: x1 = b / theta gathered from b, then step 2
// kStep: one step: d <- c1 d + c2 (b - A x), out = x + d (c1 index < 0: first step, d unread)
// kRes:  out = b - A x
// kLast: kStep whose d is not needed again; on level 0 (partials) also the products b.out, r.z
template <int NB, bool D16, int LPR, int MODE>
__global__ void __launch_bounds__(kT) k_mg_sweep(MgLev L, const float* x, float* out, int c1, int c2, int keep_d,
                                                 double* partials) {
  pdl_trigger();
  double dot = 0.0;
  const float th = MODE == kPre ? __ldg(L.coef) : 0.0f;
  const float a1 = c1 >= 0 ? __ldg(L.coef + c1) : 0.0f, a2 = c2 >= 0 ? __ldg(L.coef + c2) : 0.0f;
  const int64_t rows = (int64_t)L.n * LPR;
  const int64_t lim = LPR == 1 ? rows : (rows + 31) / 32 * 32;  // (whole warps stay together in lane_sum)
  int64_t t = gtid();
  RowHead<NB, D16, LPR> row;
  if (t < lim) row.load(L, min((int)(t / LPR), L.n - 1), (int)(t % LPR));
  pdl_wait();
  for (; t < lim;) {
    const int r0 = (int)(t / LPR), lane = (int)(t % LPR);
    const int r = r0 < L.n ? r0 : L.n - 1;
    const Vec<NB> bi = load_vec<NB>(L.b, r);
    const Vec<NB> xi = MODE == kPre ? bi : load_vec<NB>(x, r);
    Vec<NB> di;
    if ((MODE == kStep || MODE == kLast) && c1 >= 0) di = load_vec<NB>(L.d, r);
    const Vec<NB> ax = row.product(L, r, lane, MODE == kPre ? L.b : x);
    Vec<NB> o, d;
#pragma unroll
    for (int c = 0; c < NB; c++) {
      if (MODE == kRes) {
        o.v[c] = bi.v[c] - ax.v[c];
      } else if (MODE == kPre) {
        const float x1 = th * bi.v[c];
        d.v[c] = fmaf(a1, x1, a2 * (bi.v[c] - th * ax.v[c]));
        o.v[c] = x1 + d.v[c];
      } else {
        const float res = bi.v[c] - ax.v[c];
        d.v[c] = c1 >= 0 ? fmaf(a1, di.v[c], a2 * res) : a2 * res;
        o.v[c] = xi.v[c] + d.v[c];
      }
    }
    if (lane == 0 && r0 < L.n) {
      store_vec<NB>(out, r, o);
      if ((MODE == kPre || MODE == kStep) && keep_d) store_vec<NB>(L.d, r, d);
      if (MODE == kLast)
#pragma unroll
        for (int c = 0; c < NB; c++) dot = fma((double)bi.v[c], (double)o.v[c], dot);
    }
    if (MODE != kLast) break;  // (the other modes have a lane group per row)
    t += gstride();
    if (t < lim) row.load(L, min((int)(t / LPR), L.n - 1), (int)(t % LPR));
  }
  if (MODE == kLast && partials) block_partial(dot, partials);
}

// The sweeps of level 0 of a scalar system whose rows have at most 8 entries (P1: 7), on the
// system's own pattern: straight-line code with 32-bit indices, all loads of a step issued
// together (4M DOF: 23.2 -> 18.8 ms a solve against the generic form's loop; 2 or 3 rows per
// thread with their loads side by side were no faster, the blocks' occupancy falls as the loads
// in flight per thread rise).  32 registers, so that eight blocks are resident: 530 instead of
// 568 us an iteration at 4M DOF with 36 to 38.
template <int MODE>
__global__ void __launch_bounds__(kT, MODE == kLast ? 6 : 8) k_mg_fine(MgLev L, const float* x, float* out, int c1, int c2,
                                                double* partials) {
  pdl_trigger();
  constexpr int W = 8;
  const float th = MODE == kPre ? __ldg(L.coef) : 0.0f;
  const float a1 = c1 >= 0 ? __ldg(L.coef + c1) : 0.0f, a2 = c2 >= 0 ? __ldg(L.coef + c2) : 0.0f;
  const float* g = MODE == kPre ? L.b : x;
  double dot = 0.0;
  int j[W];
  float v[W];
  auto load = [&](int r) {
    const int sl = r >> 5, s0 = __ldg(L.sptr + sl), w = (__ldg(L.sptr + sl + 1) - s0) >> 5, so = __ldg(L.spat + sl);
    const int idx = s0 + (r & 31);
#pragma unroll
    for (int e = 0; e < W; e++) {
      j[e] = r;
      if (e < w)
        j[e] += so >= 0 ? __ldg(L.pat + so + e) : __ldg(reinterpret_cast<const int16_t*>(L.col) + idx + 32 * e);
      v[e] = e < w ? __ldcs(L.val + idx + 32 * e) : 0.0f;
      if (!ADFEM_DCHECK(j[e] >= 0 && j[e] < L.n)) j[e] = r;
    }
  };
  int r = blockIdx.x * kT + threadIdx.x;
  if (r < L.n) load(r);
  pdl_wait();
  while (r < L.n) {
    const float bi = L.b[r], xi = MODE == kPre ? bi : x[r];
    const float di = (MODE == kStep || MODE == kLast) && c1 >= 0 ? L.d[r] : 0.0f;
    float gx[W], ax = 0.0f;
#pragma unroll
    for (int e = 0; e < W; e++) gx[e] = g[j[e]];
#pragma unroll
    for (int e = 0; e < W; e++) ax = fmaf(v[e], gx[e], ax);
    float o;
    if (MODE == kRes) {
      o = bi - ax;
    } else if (MODE == kPre) {
      const float x1 = th * bi;
      o = x1 + fmaf(a1, x1, a2 * (bi - th * ax));
    } else {
      const float d = fmaf(a1, di, a2 * (bi - ax));
      o = xi + d;
      if (MODE == kStep) L.d[r] = d;
      if (MODE == kLast) dot = fma((double)bi, (double)o, dot);
    }
    out[r] = o;
    if (MODE != kLast) break;  // (the other modes have a thread per row)
    r += gridDim.x * kT;
    if (r < L.n) load(r);
  }
  if (MODE == kLast) block_partial(dot, partials);
}

// out_J = sum_i P_iJ^T r_i
template <int NB, int NC, int LPR>
__global__ void __launch_bounds__(kT) k_mg_restrict(MgLev L, const float* r, float* out) {
  pdl_trigger();
  const int64_t t = gtid();
  const int J0 = (int)(t / LPR), lane = (int)(t % LPR);
  const int J = J0 < L.nc ? J0 : L.nc - 1;
  Vec<NC> acc;
#pragma unroll
  for (int c = 0; c < NC; c++) acc.v[c] = 0.0f;
  const int s0 = __ldg(L.pt_sptr + (J >> 5)), w = (__ldg(L.pt_sptr + (J >> 5) + 1) - s0) >> 5, base = s0 + (J & 31);
  constexpr int U = LPR == 1 ? 8 : 4;
  int i[U];
  auto cols = [&](int k0) {
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int k = k0 + u * LPR;
      i[u] = k < w ? __ldg(L.pt_col + base + 32 * k) : 0;
    }
  };
  cols(lane);
  // (the values of the first group, too)
  float v[U][NB * NC];
#pragma unroll
  for (int u = 0; u < U; u++)
    if (lane + u * LPR < w) load_block<NC, NB>(L.pt_val, base + 32 * (lane + u * LPR), L.npt, v[u]);
  pdl_wait();
#pragma unroll
  for (int u = 0; u < U; u++)
    if (lane + u * LPR < w) {
      const Vec<NB> x = load_vec<NB>(r, i[u]);
#pragma unroll
      for (int a = 0; a < NC; a++)
#pragma unroll
        for (int c = 0; c < NB; c++) acc.v[a] = fmaf(v[u][a * NB + c], x.v[c], acc.v[a]);
    }
  for (int k0 = lane + U * LPR; k0 < w; k0 += U * LPR) {
    cols(k0);
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int k = k0 + u * LPR;
      if (k < w) block_fma<NC, NB>(L.pt_val, base + 32 * k, L.npt, load_vec<NB>(r, i[u]), acc);
    }
  }
  if (LPR > 1) lane_sum<NC, LPR>(acc);
  if (lane == 0 && J0 < L.nc) store_vec<NC>(out, J, acc);
}

// x_i += sum_J P_iJ xc_J
template <int NB, int NC>
__global__ void __launch_bounds__(kT) k_mg_prolong(MgLev L, const float* xc, float* x) {
  pdl_trigger();
  const int64_t t = gtid();
  const int i = (int)min(t, (int64_t)L.n - 1);
  const int s0 = __ldg(L.p_sptr + (i >> 5)), w = (__ldg(L.p_sptr + (i >> 5) + 1) - s0) >> 5, base = s0 + (i & 31);
  constexpr int U = 4;
  int J[U];
  float v[U][NB * NC];
#pragma unroll
  for (int u = 0; u < U; u++) {
    J[u] = u < w ? __ldg(L.p_col + base + 32 * u) : 0;
    if (u < w) load_block<NB, NC>(L.p_val, base + 32 * u, L.np, v[u]);
  }
  pdl_wait();
  Vec<NB> acc = load_vec<NB>(x, i);
#pragma unroll
  for (int u = 0; u < U; u++)
    if (u < w) {
      const Vec<NC> y = load_vec<NC>(xc, J[u]);
#pragma unroll
      for (int a = 0; a < NB; a++)
#pragma unroll
        for (int c = 0; c < NC; c++) acc.v[a] = fmaf(v[u][a * NC + c], y.v[c], acc.v[a]);
    }
  for (int k0 = U; k0 < w; k0 += U) {
#pragma unroll
    for (int u = 0; u < U; u++) J[u] = k0 + u < w ? __ldg(L.p_col + base + 32 * (k0 + u)) : 0;
#pragma unroll
    for (int u = 0; u < U; u++)
      if (k0 + u < w) block_fma<NB, NC>(L.p_val, base + 32 * (k0 + u), L.np, load_vec<NC>(xc, J[u]), acc);
  }
  if (t < L.n) store_vec<NB>(x, i, acc);
}

// ---------------------------------------------------------------------------
// The residual decides: converged, at its attainable floor, out of iterations, or go on (the
// rules of replacement_step64, whose direction scalars do not apply here).
// rn: the recurrence's residual (its square, as rr)
__device__ __forceinline__ void mg_residual_step(CgState* st, double rr, double rn, bool first) {
  const double prev = st->last_rr64;
  st->rr64 = rr;
  st->last_rr64 = rr;
  if (!isfinite(rr)) {
    st->done = 2;
    return;
  }
  if (rr <= st->stop2) {
    st->done = 1;
    return;
  }
  if (!first) {
    const bool dropped = rn <= st->delta2 * prev;
    if (prev > 0.0 && rr > 0.0625 * prev && (dropped || st->final_seen)) {
      st->floor_hit = 1;
      st->done = 1;
      return;
    }
  }
  if (st->iters >= st->max_iter) {
    st->done = 4;
    return;
  }
  if (!first && rn <= st->stop2) st->final_seen = 1;
  if (!first) st->updates += 1;
  // A residual that is not the recurrence's (near the attainable floor it can be many times
  // larger) has nothing to do with the directions so far: keeping them made the iteration
  // stagnate (elasticity, 320k DOF: over 200 iterations to the floor instead of 10).
  if (first || rr > 1.21 * rn) st->ap = 1.0;
  st->fold = 1;
  st->ru2 = st->delta2 * rr;
  st->done = 0;
}

// ---------------------------------------------------------------------------
// The levels from Mg::tail on in one launch, `reps` cycles (two below three larger levels, where
// the tail costs little beside them and its coarse problem is then solved nearly exactly: 35
// instead of 44 iterations and 27.8 instead of 32.6 ms at 4M DOF; one below fewer levels: 41.1
// instead of 46.0 ms for elasticity at 320k DOF).  Two forms:
//  * one block (first level of at most kTailLocal unknowns): every level's vectors in shared
//    memory, a barrier of the block per sweep;
//  * a cluster of kTailC blocks (EX): each block owns a contiguous range of the first level's
//    rows and keeps both iterates of that level whole in its shared memory (gathers are local);
//    a row's new value goes to the blocks whose rows refer to it (MgLev::to; one or two of
//    eight, as the numbering is banded) by asynchronous stores that count on the receiver's
//    mbarrier, and a block goes on when what it needs has arrived.  (A cluster barrier instead
//    would also drop the operator's rows from L1, where they stay from sweep to sweep.)  Every
//    block sends every other one word per exchange, after it has read its operands, so that a
//    block is at most one exchange ahead of another: two mbarriers in turn suffice, and nothing
//    is overwritten before it has been read.  The smaller levels are computed by every block
//    for itself, which costs no exchange.
// What bounds it is latency and instruction issue: a thread owns one unknown's row and keeps its
// entries in registers over the steps of a smoother, and the operators of the levels that a
// block runs alone are copied to shared memory in bulk while it is busy with the first level.
// The coarsest operator is applied as its dense inverse.
struct TailArgs {
  MgLev L[kMgMaxTail];
  int nl;
  const float* dense;
  int N;         // unknowns of the coarsest level
  // patterns and values of the levels a block runs alone, each one range of device memory
  // (bytes 0: they do not fit and are read through L1)
  const char *pat, *vals;
  int pat_bytes, val_bytes;
  const float* b;
  float* x;
  int reps;
  int spin;      // tries of a wait
  // a whole solve (k_mg_tail's SOLVE): the system's operator, right-hand side and iterate
  const int32_t* sptr;
  const void* col;  // (int16 differences: a system of that size has no others)
  const double *val, *rowsum, *rhs;
  const float* s;
  double* y;
  CgState* st;
};
struct TailVecs {
  float *x, *y;  // whole: current iterate, other iterate (or right-hand side, residual)
  float *b, *d;  // own rows
  int r0, r1;    // own rows of the level
  int floats;    // EX: values an exchange of the level brings here
};

__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// shared-memory address p of this block, in the block of the given rank
__device__ __forceinline__ unsigned rank_addr(const void* p, int rank) {
  unsigned m;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(m) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
  return m;
}

// Whether the given phase of an mbarrier has completed, after at most `spin` tries.
__device__ __forceinline__ bool mbar_wait(const void* bar, unsigned parity, int spin) {
  unsigned ok = 0;
  for (int i = 0; i < spin && !ok; i++)
    asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
                 : "=r"(ok)
                 : "r"((unsigned)__cvta_generic_to_shared(bar)), "r"(parity)
                 : "memory");
  return ok;
}

// The exchanges of a block, numbered: exchange k counts on bar[k & 1] in its (k >> 1)-th phase.
//
// Waits are bounded (`spin` tries).  A block whose wait gives up is dead: it takes part in no further
// exchange (an arrival in a phase that has not completed would corrupt the barrier) and uses no
// indices that it waited for, so the blocks that wait for it give up as well, one exchange later at
// most.  The launch then ends with st->done set, and the solve is left to the Jacobi iteration.  A dead
// block stays until every block has ended its sends (a barrier of the cluster, in which blocks that
// have left count as arrived) and what was on its way to it has had time to arrive.  A block that is
// not dead at the end has received the last word of every other one, and may leave.
// (us an iteration at 4225 unknowns: 42.4; 43.9 with a barrier that also votes in place of the shared
// word and a look at the bulk copies in every cycle; 40.5 where waits that gave up were not looked at.)
struct TailSync {
  unsigned long long* bar;
  float* tok;    // kTailC words
  int rank;
  CgState* st;
  int spin;
  volatile int* gave; // (shared) a wait of this block has given up
  bool dead = false;  // the same in all threads
  int k = 0;
  __device__ __forceinline__ void give_up() {
    if (threadIdx.x == 0) st->done = 5;
    dead = true;
  }
  // this exchange brings `floats` values here
  __device__ __forceinline__ void expect(int floats) {
    if (threadIdx.x == 0)
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(
                       (unsigned)__cvta_generic_to_shared(bar + (k & 1))),
                   "r"(4 * (floats + kTailC))
                   : "memory");
  }
  __device__ __forceinline__ void send(const float* p, int rk, float v) const {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0], %1, [%2];" ::"r"(rank_addr(p, rk)),
                 "f"(v), "r"(rank_addr(bar + (k & 1), rk))
                 : "memory");
  }
  // the block has sent its rows: tell every block, and wait for what it needs itself
  __device__ __forceinline__ void exchange() {
    __syncthreads();
    bool ok = true;
    if (threadIdx.x < 32) {
      if (threadIdx.x < kTailC) send(tok + rank, threadIdx.x, 0.0f);
      ok = mbar_wait(bar + (k & 1), (k >> 1) & 1, spin);
    }
    if (!ok) *gave = 1;
    __syncthreads();
    k++;
    if (*gave) give_up();
  }
  // dead, and no block sends any more: some 0.2 ms for what is on its way to this one
  __device__ __forceinline__ void drain() const {
    for (int i = 0; i < 200; i++) __nanosleep(1000);
  }
};

// The level as the tail's threads see it (pointers into shared memory where it was copied).
struct TailLev {
  const int32_t *sptr, *col, *p_sptr, *p_col, *pt_sptr, *pt_col;
  const float *val, *p_val, *pt_val, *coef;
  const uint8_t* to;
  int n, nv, np, npt;
};

// Row of one unknown (component c of node r): the first E entries in registers.
template <int NB>
struct RowCache {
  static constexpr int E = NB == 1 ? 14 : (NB == 2 ? 8 : 6);
  float v[E][NB];
  int j[E];
  int base, w, c;
  __device__ __forceinline__ void load(const TailLev& L, int r, int comp) {
    const int s0 = L.sptr[r >> 5];
    w = (L.sptr[(r >> 5) + 1] - s0) >> 5;
    base = s0 + (r & 31);
    c = comp;
#pragma unroll
    for (int e = 0; e < E; e++) {
      if (e >= w) continue;
      j[e] = NB * L.col[base + 32 * e];
      if (!ADFEM_DCHECK(j[e] >= 0 && j[e] < NB * L.n)) j[e] = NB * r;
#pragma unroll
      for (int q = 0; q < NB; q++) v[e][q] = L.val[block_at<NB, NB>(c * NB + q, base + 32 * e, L.nv)];
    }
  }
  __device__ __forceinline__ float product(const TailLev& L, const float* x) const {
    float acc = 0.0f;
#pragma unroll
    for (int e = 0; e < E; e++) {
      if (e >= w) continue;
#pragma unroll
      for (int q = 0; q < NB; q++) acc = fmaf(v[e][q], x[j[e] + q], acc);
    }
    for (int e = E; e < w; e++) {
      const int k = base + 32 * e, jj = NB * L.col[k];
#pragma unroll
      for (int q = 0; q < NB; q++) acc = fmaf(L.val[block_at<NB, NB>(c * NB + q, k, L.nv)], x[jj + q], acc);
    }
    return acc;
  }
};

// Sum of a double per thread over the cluster, in a fixed order, in thread 0 of every block (sh: one
// double per thread, slot: two sets of kTailC; the sets alternate, and the barrier of a sum has every
// block past its reading of the one before).
template <bool EX, int T>
__device__ __forceinline__ double cluster_total(double x, double* sh, double* slot, int rank, int& phase) {
  sh[threadIdx.x] = x;
  __syncthreads();
  double* set = slot + (phase & 1) * kTailC;
  phase++;
  double s = 0.0;
  if (threadIdx.x < 32) {
    double v[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int k = 0; k < T / 32; k++) v[k & 3] += sh[threadIdx.x + 32 * k];
    s = warp_sum((v[0] + v[1]) + (v[2] + v[3]));
    if (EX && threadIdx.x < kTailC)
      asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(rank_addr(set + rank, threadIdx.x)), "d"(s) : "memory");
  }
  if (EX) {
    cluster_barrier();
    if (threadIdx.x == 0) {
      static_assert(kTailC == 8, "pairs of pairs of pairs");
      s = ((set[0] + set[1]) + (set[2] + set[3])) + ((set[4] + set[5]) + (set[6] + set[7]));
    }
  }
  return s;
}

constexpr int kTailT = kMgTailDofs / kTailC;  // threads of a tail block: one per own unknown

// publish unknown u (of a row that the ranks in the bit mask need): out[u] here or there
template <bool EX>
__device__ __forceinline__ void tail_put(const TailSync& sync, unsigned ranks, float* out, int u, float v) {
  if (EX) {
    for (; ranks; ranks &= ranks - 1) sync.send(out + u, __ffs(ranks) - 1, v);
  } else {
    out[u] = v;
  }
}
template <bool EX>
__device__ __forceinline__ void tail_end(TailSync& sync) {
  if (EX) sync.exchange();
  else __syncthreads();
}

// Chebyshev steps on (b, x) -> x, then (res) the residual into y.  fresh: x = 0 and the right-hand
// side stands whole in y; the first two steps are one sweep (as kPre).
template <bool EX, int NB, int T>
__device__ __forceinline__ void tail_smooth(TailSync& sync, const TailLev& L, TailVecs& v, int deg, bool fresh,
                                            bool res) {
  TailVecs f = v;
  const int m = (f.r1 - f.r0) * NB, u0 = f.r0 * NB;
  const bool one = m <= T;  // at most one row per thread: its entries stay in registers
  RowCache<NB> rc;
  unsigned ranks = 0;
  if (one && (int)threadIdx.x < m) {
    const int r = f.r0 + threadIdx.x / NB;
    rc.load(L, r, threadIdx.x % NB);
    if (EX) ranks = L.to[r];
  }
  const float th = L.coef[0];
  const int k1 = res ? deg + 1 : deg;
  for (int k = fresh ? 1 : 0; k < k1; k++) {
    if (EX && sync.dead) break;
    const bool pre = fresh && k == 1, last = k == deg;
    const float a1 = k > 0 && !last ? L.coef[2 * k] : 0.0f;
    const float a2 = k > 0 && !last ? L.coef[2 * k + 1] : th;
    const float* x = pre ? f.y : f.x;
    float* out = pre ? f.x : f.y;
    if (EX) sync.expect(f.floats);
    for (int q = threadIdx.x; q < m; q += T) {
      if (!one) {
        const int r = f.r0 + q / NB;
        rc.load(L, r, q % NB);
        if (EX) ranks = L.to[r];
      }
      const float ax = rc.product(L, x), bi = f.b[q];
      float o;
      if (last) {
        o = bi - ax;
      } else {
        const float x1 = pre ? th * bi : f.x[u0 + q];
        const float d0 = pre ? x1 : (a1 != 0.0f ? f.d[q] : 0.0f);
        const float d = fmaf(a1, d0, a2 * (bi - (pre ? th : 1.0f) * ax));
        f.d[q] = d;
        o = x1 + d;
      }
      tail_put<EX>(sync, ranks, out, u0 + q, o);
    }
    tail_end<EX>(sync);
    if (!pre && !last) {
      float* s = f.x;
      f.x = f.y;
      f.y = s;
    }
  }
  v.x = f.x;
  v.y = f.y;
}

// out = M x (+ add) for the rows [r0, r1) of a rectangular M with R unknowns per row, X per column.
// `to`: EX, the ranks that need a row (null: all); own: a second copy.
template <bool EX, int R, int X, int T>
__device__ __forceinline__ void tail_transfer(TailSync& sync, const int32_t* sp, const int32_t* col, const float* val,
                                              int nent, const uint8_t* to, int r0, int r1, int lg, const float* x,
                                              const float* add, float* out, float* own) {
  if (EX && sync.dead) return;
  const int lane = threadIdx.x & ((1 << lg) - 1), rows = (r1 - r0) * R;
  for (int q0 = 0; q0 < rows; q0 += T >> lg) {
    if (q0 + ((int)(threadIdx.x & ~31u) >> lg) >= rows) break;  // (whole warps without a row)
    const int q = q0 + ((int)threadIdx.x >> lg);
    const bool live = q < rows;
    const int u = r0 * R + (live ? q : rows - 1), r = u / R, c = u % R;
    const int s0 = sp[r >> 5], w = (sp[(r >> 5) + 1] - s0) >> 5, base = s0 + (r & 31);
    float acc = 0.0f;
    for (int k = lane; k < w; k += 1 << lg) {
      const int j = X * col[base + 32 * k];
#pragma unroll
      for (int e = 0; e < X; e++) acc = fmaf(val[block_at<R, X>(c * X + e, base + 32 * k, nent)], x[j + e], acc);
    }
    for (int o = (1 << lg) >> 1; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (!live || lane) continue;
    if (add) acc += add[u];
    if (own) own[u] = acc;
    tail_put<EX>(sync, EX ? (to ? to[r] : (1u << kTailC) - 1u) : 0u, out, u, acc);
  }
  tail_end<EX>(sync);
}

// log2 of the lanes per row of a transfer with that many rows
__device__ __forceinline__ int tail_lanes(int rows, int T) {
  int lg = 0;
  while (lg < 4 && (rows << (lg + 1)) <= T) lg++;
  return lg;
}

// the levels from l on, each whole in this block: (b in y and b) -> x
template <int NB, int T>
__device__ __noinline__ void tail_local(const TailLev* L, TailVecs* v, int l0, int last, int deg0,
                                        bool fresh0, const float* dense, int N) {
  TailSync sync{};  // (no exchange below)
  for (int l = l0; l < last; l++) {
    tail_smooth<false, NB, T>(sync, L[l], v[l], l == l0 ? deg0 : kMgDeg, l > l0 || fresh0, true);
    TailVecs& c = v[l + 1];
    tail_transfer<false, NB, NB, T>(sync, L[l].pt_sptr, L[l].pt_col, L[l].pt_val, L[l].npt, nullptr, 0, c.r1,
                                    tail_lanes(c.r1 * NB, T), v[l].y, nullptr, c.y, c.b);
  }
  {
    // coarsest: some lanes per row of the dense inverse
    const int lg = tail_lanes(N, T), lane = threadIdx.x & ((1 << lg) - 1);
    const float* bb = v[last].y;
    for (int q0 = 0; q0 < N; q0 += T >> lg) {
      if (q0 + ((int)(threadIdx.x & ~31u) >> lg) >= N) break;
      const int q = q0 + ((int)threadIdx.x >> lg), r = min(q, N - 1);
      float s = 0.0f;
      for (int k = lane; k < N; k += 1 << lg) s = fmaf(dense[r + k * N], bb[k], s);  // (symmetric)
      for (int o = (1 << lg) >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0 && q < N) v[last].x[q] = s;
    }
    __syncthreads();
  }
  for (int l = last - 1; l >= l0; l--) {
    tail_transfer<false, NB, NB, T>(sync, L[l].p_sptr, L[l].p_col, L[l].p_val, L[l].np, nullptr, 0, v[l].r1, 0,
                                    v[l + 1].x, v[l].x, v[l].x, nullptr);
    tail_smooth<false, NB, T>(sync, L[l], v[l], l == l0 ? deg0 : kMgDeg, false, false);
  }
}

__host__ __device__ inline int pad4(int n) { return (n + 3) & ~3; }
__host__ __device__ inline int tail_chunk(int n) { return (n + kTailC - 1) / kTailC; }
// floats of one level: two whole vectors and two of the block's own rows
__host__ __device__ inline int tail_floats(int n, int nb, bool ex) {
  return 2 * pad4(n * nb) + 2 * pad4((ex ? tail_chunk(n) : n) * nb);
}

// NT: unknowns per node of the tail's first level, NC: of the others
// SOLVE (level 0 is in the tail): the whole of the conjugate gradients around the cycle as well, one
// unknown per thread.  A block keeps the direction of every row that its own rows refer to and
// advances it from the cycle's result, which has reached it, so the direction needs no exchange; the
// cycle's right-hand side needs one, and the three sums a barrier of the cluster each.  (As five
// launches an iteration the same took 52.7 us at 4225 unknowns, here 40.0, of which the cycle 25.)
template <int NT, int NC, bool EX, bool SOLVE>
__global__ void __launch_bounds__(kTailT, 1) k_mg_tail(const __grid_constant__ TailArgs a) {
  constexpr int T = kTailT;
  extern __shared__ float4 tail_sm4[];
  __shared__ float tokens[kTailC];
  __shared__ unsigned long long bars[3];
  __shared__ int gave;
  __shared__ TailLev lev[kMgMaxTail];
  float* sm = reinterpret_cast<float*>(tail_sm4);
  const int rank = EX ? (int)cluster_rank() : 0;
  char* pat = reinterpret_cast<char*>(sm);
  char* vals = pat + a.pat_bytes;
  const bool copy = a.pat_bytes > 0;
  const unsigned fill = (unsigned)__cvta_generic_to_shared(bars + 2);
  if (threadIdx.x == 0) {
    gave = 0;
    for (int k = 0; k < 3; k++)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"((unsigned)__cvta_generic_to_shared(bars + k)));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    if (copy) {
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(fill),
                   "r"(a.pat_bytes + a.val_bytes)
                   : "memory");
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                       (unsigned)__cvta_generic_to_shared(pat)),
                   "l"(a.pat), "r"(a.pat_bytes), "r"(fill)
                   : "memory");
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                       (unsigned)__cvta_generic_to_shared(vals)),
                   "l"(a.vals), "r"(a.val_bytes), "r"(fill)
                   : "memory");
    }
  }
  sm += (a.pat_bytes + a.val_bytes) / sizeof(float);
  // where the copies of a level's arrays stand (level 0 of a cluster is read through L1)
  if (threadIdx.x < a.nl) {
    const int l = threadIdx.x;
    const MgLev& G = a.L[l];
    const bool in = copy && !(EX && l == 0);
    auto ip = [&](const void* p) {
      return reinterpret_cast<const int32_t*>(in && p ? pat + (reinterpret_cast<const char*>(p) - a.pat) : p);
    };
    auto fp = [&](const float* p) {
      return in && p ? reinterpret_cast<const float*>(vals + (reinterpret_cast<const char*>(p) - a.vals)) : p;
    };
    TailLev& S = lev[l];
    S.sptr = ip(G.sptr);
    S.col = ip(G.col);
    S.p_sptr = ip(G.p_sptr);
    S.p_col = ip(G.p_col);
    S.pt_sptr = ip(G.pt_sptr);
    S.pt_col = ip(G.pt_col);
    S.val = fp(G.val);
    S.p_val = fp(G.p_val);
    S.pt_val = fp(G.pt_val);
    S.coef = fp(G.coef);
    S.to = G.to;
    S.n = G.n;
    S.nv = G.nv;
    S.np = G.np;
    S.npt = G.npt;
  }
  const float* dense =
      copy ? reinterpret_cast<const float*>(vals + (reinterpret_cast<const char*>(a.dense) - a.vals)) : a.dense;
  TailVecs v[kMgMaxTail];
  for (int l = 0; l < a.nl; l++) {
    const bool ex = EX && l == 0;
    const int nb = l == 0 ? NT : NC, n = a.L[l].n, own = ex ? tail_chunk(n) : n;
    v[l].x = sm;
    v[l].y = sm + pad4(n * nb);
    v[l].b = sm + 2 * pad4(n * nb);
    v[l].d = v[l].b + pad4(own * nb);
    v[l].r0 = ex ? min(n, rank * own) : 0;
    v[l].r1 = ex ? min(n, rank * own + own) : n;
    v[l].floats = ex ? nb * __ldg(a.L[l].cnt + rank) : 0;
    sm += tail_floats(n, nb, ex);
  }
  TailSync sync{bars, tokens, rank, a.st, a.spin, &gave};
  pdl_wait();
  const int n0 = a.L[0].n * NT, own0 = (v[0].r1 - v[0].r0) * NT, off0 = v[0].r0 * NT;
  if (!SOLVE) {
    for (int t = threadIdx.x; t < n0; t += T) v[0].y[t] = a.b[t];
    for (int t = threadIdx.x; t < own0; t += T) v[0].b[t] = a.b[off0 + t];
  }
  // (EX also: no block stores to another's shared memory before that block runs and has its barriers)
  if (EX) cluster_barrier();
  else __syncthreads();
  // (also before the block leaves: a solve whose start has converged never ran a cycle, and the copies
  // may still be on their way into its shared memory)
  bool full = !copy;
  auto filled = [&](int spin) {
    if (full) return;
    full = __syncthreads_and(mbar_wait(bars + 2, 0, spin));
    if (!full) sync.give_up();
  };
  const int last = a.nl - 1;
  constexpr int deg0 = SOLVE ? kMgDeg0 : kMgDeg;
  // SOLVE: the directions, scales and own vectors behind the levels' in shared memory
  double* dir = reinterpret_cast<double*>(sm);
  double* res = dir + n0;
  double* cor = res + T;
  double* sh = cor + T;
  double* slot = sh + T;
  float* sc = reinterpret_cast<float*>(slot + 2 * kTailC);
  __shared__ CgState loc;
  __shared__ double bc[2];
  __shared__ int range[2], due;
  const int t = threadIdx.x, u = off0 + t;
  const bool live = t < own0;
  constexpr int U = 8;  // entries of a row whose loads are in flight together
  int64_t base = 0;
  int w = 0, phase = 0;
  unsigned ranks = 0;
  auto column = [&](int k) {
    const int64_t idx = base + 32 * (int64_t)k;
    int j = colof<true>(a.col, idx, u);
    if (!ADFEM_DCHECK(j >= 0 && j < n0)) j = u;
    return j;
  };
  if constexpr (SOLVE) {
    if (t == 0) {
      loc = *a.st;
      range[0] = n0;
      range[1] = 0;
      due = 1;
    }
    cor[t] = 0.0;
    __syncthreads();
    if (live) {
      sell_row(a.sptr, u, base, w);
      int lo = u, hi = u;
      for (int k = 0; k < w; k++) {
        const int j = column(k);
        lo = min(lo, j);
        hi = max(hi, j);
      }
      atomicMin(&range[0], lo);
      atomicMax(&range[1], hi + 1);
      if (EX) ranks = lev[0].to[u / NT];
    }
    __syncthreads();
    for (int i = range[0] + t; i < range[1]; i += T) sc[i] = __ldg(a.s + i);
    __syncthreads();
    sync.st = &loc;
  }
  bool start = true;
  double rn = 0.0;
  float bn = 0.0f;
  for (;;) {
    if constexpr (SOLVE) {
      const double g = loc.ar;
      if (due) {
        // r = b - K y in difference form, as k_mg_residual does; before it y += z, z = 0
        if (live && !start) {
          a.y[u] += cor[t];
          cor[t] = 0.0;
        }
        if (EX) cluster_barrier();
        else __syncthreads();
        double rr = 0.0;
        if (live) {
          double yo[NT], s = 0.0;
#pragma unroll
          for (int q = 0; q < NT; q++) {
            yo[q] = __ldcg(a.y + u / NT * NT + q);
            s = fma(__ldg(a.rowsum + NT * u + q), yo[q], s);
          }
          for (int k0 = 0; k0 < w; k0 += U) {
            double vv[U], x[U];
#pragma unroll
            for (int e = 0; e < U; e++) {
              vv[e] = k0 + e < w ? __ldg(a.val + base + 32 * (k0 + e)) : 0.0;
              x[e] = __ldcg(a.y + (k0 + e < w ? column(k0 + e) : u));
            }
#pragma unroll
            for (int e = 0; e < U; e++)
              if (k0 + e < w) s = fma(vv[e], x[e] - (e & 1 ? yo[NT - 1] : yo[0]), s);
          }
          const double ri = a.rhs[u] - s, tr = (double)sc[u] * ri;
          res[t] = ri;
          bn = (float)(tr * g);
          rr = tr * tr;
        }
        rr = cluster_total<EX, T>(rr, sh, slot, rank, phase);
        if (t == 0) {
          loc.iters = loc.it;
          mg_residual_step(&loc, rr, rn, start);
        }
        start = false;
        __syncthreads();
        if (loc.done) break;
        filled(a.spin);
        if (!EX && sync.dead) break;
      }
      // the cycle's right-hand side
      if (live) v[0].b[t] = bn;
      if (EX) sync.expect(v[0].floats);
      if (live) tail_put<EX>(sync, ranks, v[0].y, u, bn);
      tail_end<EX>(sync);
    }
    for (int rep = 0; rep < (SOLVE ? 1 : a.reps); rep++) {
      const bool first = rep == 0;
      if constexpr (!EX && NT == NC) {
        if (!SOLVE && first) filled(a.spin);
        if (!SOLVE && sync.dead) break;
        tail_local<NC, T>(lev, v, 0, last, deg0, first, dense, a.N);
      } else {
        const TailLev& L = lev[0];
        if (!SOLVE && !EX && first) filled(a.spin);
        if ((EX || !SOLVE) && sync.dead) break;
        tail_smooth<EX, NT, T>(sync, L, v[0], deg0, first, true);
        TailVecs& c = v[1];
        const int nc = lev[1].n;
        if (EX) {
          // coarse right-hand side: rows dealt in ranges, whole to every block
          const int ch = tail_chunk(nc), c0 = min(nc, rank * ch), c1 = min(nc, c0 + ch);
          if (!sync.dead) sync.expect(nc * NC);
          tail_transfer<true, NC, NT, T>(sync, L.pt_sptr, L.pt_col, L.pt_val, L.npt, nullptr, c0, c1,
                                         tail_lanes(ch * NC, T), v[0].y, nullptr, c.y, nullptr);
          for (int q = threadIdx.x; q < nc * NC; q += T) c.b[q] = c.y[q];
          if (!SOLVE && first) filled(a.spin);
          __syncthreads();
          if (sync.dead) break;
        } else {
          tail_transfer<false, NC, NT, T>(sync, L.pt_sptr, L.pt_col, L.pt_val, L.npt, nullptr, 0, c.r1,
                                          tail_lanes(c.r1 * NC, T), v[0].y, nullptr, c.y, c.b);
        }
        tail_local<NC, T>(lev, v, 1, last, kMgDeg, true, dense, a.N);
        if (EX) sync.expect(v[0].floats);
        tail_transfer<EX, NT, NC, T>(sync, L.p_sptr, L.p_col, L.p_val, L.np, L.to, v[0].r0, v[0].r1, 0, v[1].x,
                                     v[0].x, v[0].y, nullptr);
        float* s = v[0].x;
        v[0].x = v[0].y;
        v[0].y = s;
        tail_smooth<EX, NT, T>(sync, L, v[0], deg0, false, false);
      }
    }
    if constexpr (!SOLVE) break;
    if constexpr (SOLVE) {
      const float* x = v[0].x;
      // (a wait that gave up in any block ends the solve in all of them)
      double zb = live ? (double)x[u] * (double)v[0].b[t] : 0.0;
      if (EX && sync.dead) zb = nan("");
      double d = cluster_total<EX, T>(zb, sh, slot, rank, phase);
      if (t == 0) {
        const double rz = d * loc.iar;
        if (!(rz > 0.0) || !isfinite(rz)) loc.done = 2;
        bc[0] = loc.ap != 0.0 ? 0.0 : rz * loc.irz;
        loc.rz = rz;
        loc.ap = 0.0;
      }
      __syncthreads();
      if (loc.done) break;
      const double bt = bc[0];
      for (int i = range[0] + t; i < range[1]; i += T) {
        const double zi = (double)(sc[i] * x[i]);
        dir[i] = bt == 0.0 ? zi : fma(bt, dir[i], zi);
      }
      __syncthreads();
      if (t == T - 1) loc.irz = 1.0 / loc.rz;  // (beside the product: the division is read an iteration later)
      double q = 0.0, pu = 0.0;
      if (live) {
        for (int k0 = 0; k0 < w; k0 += U) {
          double vv[U];
          int j[U];
#pragma unroll
          for (int e = 0; e < U; e++) {
            vv[e] = k0 + e < w ? __ldg(a.val + base + 32 * (k0 + e)) : 0.0;
            j[e] = k0 + e < w ? column(k0 + e) : u;
          }
#pragma unroll
          for (int e = 0; e < U; e++)
            if (k0 + e < w) q = fma(vv[e], dir[j[e]], q);
        }
        pu = dir[u];
      }
      d = cluster_total<EX, T>(pu * q, sh, slot, rank, phase);
      if (t == 0) {
        if (!(d > 0.0) || !isfinite(d)) loc.done = 2;
        bc[1] = loc.rz / d;
        loc.it += 1;
      }
      __syncthreads();
      if (loc.done) break;
      const double al = bc[1], g = loc.ar;
      double tn = 0.0;
      if (live) {
        cor[t] = fma(al, pu, cor[t]);
        const double ri = fma(-al, q, res[t]);
        res[t] = ri;
        tn = ri * g * (double)sc[u];
        bn = (float)tn;
      }
      d = cluster_total<EX, T>(tn * tn, sh, slot, rank, phase);
      if (t == 0) {
        rn = d * loc.iar * loc.iar;
        loc.rho_new = rn;
        loc.iters = loc.it;
        if (!isfinite(rn)) loc.done = 2;
        due = rn <= loc.stop2 || rn <= loc.ru2 || loc.it >= loc.max_iter;
      }
      __syncthreads();
      if (loc.done) break;
    }
  }
  if (EX && sync.dead) {
    cluster_barrier();
    sync.drain();
  }
  filled(kTailSpin);
  if constexpr (SOLVE) {
    if (rank == 0 && t == 0) *a.st = loc;
  } else {
    pdl_trigger();  // (not before: blocks that wait would keep other solves' kernels off the SMs)
    for (int q = threadIdx.x; q < own0; q += T) a.x[off0 + q] = v[0].x[off0 + q];
  }
}

// ---------------------------------------------------------------------------
// values of the hierarchy (once per assembly)

// Level 0 from the assembled operator: FP32 copy scaled to unit diagonal, scale per unknown (0
// on Dirichlet rows: no interpolation there) and the FP64 row sums (per component of the
// column) of the difference form of the residual.
template <int NB, bool D16>
__global__ void __launch_bounds__(kT) k_mg_vals0(int64_t n, const int32_t* __restrict__ sptr,
                                                 const void* __restrict__ col, const double* __restrict__ val,
                                                 const float* __restrict__ s, const uint8_t* __restrict__ isbd,
                                                 MgLev L, double* __restrict__ rowsum) {
  const int64_t r = gtid();  // unknown
  if (r >= n) return;
  int64_t base;
  int w;
  sell_row(sptr, r, base, w);
  const float si = s[r];
  const int i = (int)(r / NB), c = (int)(r % NB);
  int64_t nbase = base;
  if (NB > 1) {
    int nw;
    slice_row(L.sptr, i, nbase, nw);
  }
  double rs[NB];
#pragma unroll
  for (int q = 0; q < NB; q++) rs[q] = 0.0;
  for (int k = 0; k < w; k++) {
    const int64_t idx = base + 32 * (int64_t)k;
    const double v = val[idx];
    int j = colof<D16>(col, idx, r);
    if (!ADFEM_DCHECK(j >= 0 && j < n)) j = (int)r;
    const float f = (float)v * (si * s[j]);
    if (NB == 1) {
      rs[0] += v;
      L.val[idx] = f;
    } else {
      // slot k = 2 (neighbour) + component
#pragma unroll
      for (int q = 0; q < NB; q++)
        if (k % NB == q) rs[q] += v;
      L.val[block_at<NB, NB>(c * NB + k % NB, nbase + 32 * (int64_t)(k / NB), L.nv)] = f;
    }
  }
#pragma unroll
  for (int q = 0; q < NB; q++) rowsum[NB * r + q] = rs[q];
  L.s[r] = isbd[r] == 1 ? 0.0f : si;
}

// P0 of node j: its NB x NC block
template <int NB, int NC>
__device__ __forceinline__ void tentative(const MgLev& L, int j, float (&T)[NB * NC], float (&t)[NB]) {
#pragma unroll
  for (int c = 0; c < NB; c++) {
    const float s = __ldg(L.s + (int64_t)NB * j + c);
    t[c] = s > 0.0f ? 1.0f / s : 0.0f;
  }
#pragma unroll
  for (int q = 0; q < NB * NC; q++) T[q] = 0.0f;
#pragma unroll
  for (int c = 0; c < NB; c++) T[c * NC + c] = t[c];
  if constexpr (NC == 3) {
    const float2 d = __ldg(L.dpos + j);
    T[2] = -d.y * t[0];
    T[NC + 2] = d.x * t[1];
  }
}

// P = P0 - (smooth / q) A P0 and the level's eigenvalue bound max q.  q: absolute row sums,
// weighted by P0 for scalar operators (then exactly 2 where the row sums to zero with
// non-positive off-diagonals, whatever the coefficients' jumps).  One thread per node; the
// loads of U neighbours are issued together (the kernel is a chain of dependent loads).
template <int NB, int NC, bool D16, int BT>
__global__ void __launch_bounds__(BT) k_mg_p(MgLev L, float smooth) {
  __shared__ float acc[kMgMaxP * NB * NC][BT];
  __shared__ int pc[kMgMaxP][BT];
  const int t = threadIdx.x;
  const int64_t i64 = gtid();
  float qmax = 0.0f;
  if (i64 < L.n) {
    const int i = (int)i64;
    int64_t pb, base;
    int pw, w;
    slice_row(L.p_sptr, i, pb, pw);
    slice_row(L.sptr, i, base, w);
    if (pw > kMgMaxP) pw = kMgMaxP;
    for (int s = 0; s < pw; s++) pc[s][t] = __ldg(L.p_col + pb + 32 * (int64_t)s);
    for (int e = 0; e < pw * NB * NC; e++) acc[e][t] = 0.0f;
    float ti[NB], Ti[NB * NC], q[NB];
    tentative<NB, NC>(L, i, Ti, ti);
#pragma unroll
    for (int c = 0; c < NB; c++) q[c] = 0.0f;
    const Cols<D16> cols(L, i);
    constexpr int U = NB == 1 ? 8 : 2;
    for (int k0 = 0; k0 < w; k0 += U) {
      int j[U], J[U];
      float a[U][NB * NB], T[U][NB * NC], tj[U][NB];
#pragma unroll
      for (int u = 0; u < U; u++) {
        j[u] = k0 + u < w ? cols.at(k0 + u, base + 32 * (int64_t)(k0 + u)) : i;
        if (!ADFEM_DCHECK(j[u] >= 0 && j[u] < L.n)) j[u] = i;
      }
#pragma unroll
      for (int u = 0; u < U; u++) {
        J[u] = __ldg(L.agg + j[u]);
        tentative<NB, NC>(L, j[u], T[u], tj[u]);
        if (k0 + u < w) load_block<NB, NB>(L.val, base + 32 * (int64_t)(k0 + u), L.nv, a[u]);
        else
#pragma unroll
          for (int e = 0; e < NB * NB; e++) a[u][e] = 0.0f;
      }
#pragma unroll
      for (int u = 0; u < U; u++) {
        int s = 0;
        while (s < pw && pc[s][t] != J[u]) s++;
#pragma unroll
        for (int c = 0; c < NB; c++) {
#pragma unroll
          for (int e = 0; e < NB; e++) q[c] += NB == 1 ? fabsf(a[u][0]) * tj[u][0] : fabsf(a[u][c * NB + e]);
          if (s < pw)
#pragma unroll
            for (int m = 0; m < NC; m++) {
              float v = 0.0f;
#pragma unroll
              for (int e = 0; e < NB; e++) v = fmaf(a[u][c * NB + e], T[u][e * NC + m], v);
              acc[s * NB * NC + c * NC + m][t] -= v;
            }
        }
      }
    }
#pragma unroll
    for (int c = 0; c < NB; c++) {
      if (NB == 1) q[0] = ti[0] > 0.0f ? q[0] / ti[0] : 1.0f;
      q[c] = fmaxf(q[c], 1.0f);
      qmax = fmaxf(qmax, q[c]);
    }
    // (padding repeats the first column behind the row's entries: the first match is the own aggregate)
    const int Ji = __ldg(L.agg + i);
    int own = 0;
    while (own < pw && pc[own][t] != Ji) own++;
    for (int s = 0; s < pw; s++)
#pragma unroll
      for (int c = 0; c < NB; c++) {
        const float f = ti[c] > 0.0f ? smooth / q[c] : 0.0f;
#pragma unroll
        for (int m = 0; m < NC; m++)
          L.p_val[block_at<NB, NC>(c * NC + m, pb + 32 * (int64_t)s, L.np)] =
              f * acc[s * NB * NC + c * NC + m][t] + (s == own ? Ti[c * NC + m] : 0.0f);
      }
  }
  // (positive floats order as their bits; a maximum does not depend on the order of arrival)
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) qmax = fmaxf(qmax, __shfl_xor_sync(0xffffffffu, qmax, o));
  if ((t & 31) == 0) atomicMax(L.lam, __float_as_int(qmax));
}

// rows of A P, one thread per node: the P rows of U neighbours are walked side by side
template <int NB, int NC, bool D16, int BT>
__global__ void __launch_bounds__(BT) k_mg_ap(MgLev L) {
  __shared__ float acc[kMgMaxAP * NB * NC][BT];
  __shared__ int ac[kMgMaxAP][BT];
  const int t = threadIdx.x;
  const int64_t i64 = gtid();
  if (i64 >= L.n) return;
  const int i = (int)i64;
  int64_t ab, base;
  int aw, w;
  slice_row(L.ap_sptr, i, ab, aw);
  slice_row(L.sptr, i, base, w);
  if (aw > kMgMaxAP) aw = kMgMaxAP;
  for (int s = 0; s < aw; s++) ac[s][t] = __ldg(L.ap_col + ab + 32 * (int64_t)s);
  for (int e = 0; e < aw * NB * NC; e++) acc[e][t] = 0.0f;
  const Cols<D16> cols(L, i);
  constexpr int U = NB == 1 ? 8 : 2;
  for (int k0 = 0; k0 < w; k0 += U) {
    int j[U], pw[U], pm = 0;
    int64_t pb[U];
    float a[U][NB * NB];
#pragma unroll
    for (int u = 0; u < U; u++) {
      j[u] = k0 + u < w ? cols.at(k0 + u, base + 32 * (int64_t)(k0 + u)) : i;
      if (!ADFEM_DCHECK(j[u] >= 0 && j[u] < L.n)) j[u] = i;
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      slice_row(L.p_sptr, j[u], pb[u], pw[u]);
      if (k0 + u < w) load_block<NB, NB>(L.val, base + 32 * (int64_t)(k0 + u), L.nv, a[u]);
      else
#pragma unroll
        for (int e = 0; e < NB * NB; e++) a[u][e] = 0.0f;
      bool any = false;
#pragma unroll
      for (int e = 0; e < NB * NB; e++) any |= a[u][e] != 0.0f;
      if (!any) pw[u] = 0;
      pm = max(pm, pw[u]);
    }
    for (int p = 0; p < pm; p++) {
      int K[U];
      float v[U][NB * NC];
#pragma unroll
      for (int u = 0; u < U; u++) {
        K[u] = -1;
        if (p < pw[u]) {
          const int64_t pe = pb[u] + 32 * (int64_t)p;
          K[u] = __ldg(L.p_col + pe);
          load_block<NB, NC>(L.p_val, pe, L.np, v[u]);
        }
      }
#pragma unroll
      for (int u = 0; u < U; u++) {
        if (K[u] < 0) continue;
        int s = 0;
        while (s < aw && ac[s][t] != K[u]) s++;
        if (s == aw) continue;
#pragma unroll
        for (int c = 0; c < NB; c++)
#pragma unroll
          for (int m = 0; m < NC; m++) {
            float x = acc[s * NB * NC + c * NC + m][t];
#pragma unroll
            for (int e = 0; e < NB; e++) x = fmaf(a[u][c * NB + e], v[u][e * NC + m], x);
            acc[s * NB * NC + c * NC + m][t] = x;
          }
      }
    }
  }
  for (int s = 0; s < aw; s++)
#pragma unroll
    for (int e = 0; e < NB * NC; e++)
      L.ap_val[block_at<NB, NC>(e, ab + 32 * (int64_t)s, L.nap)] = acc[s * NB * NC + e][t];
}

// Coarse rows P^T (A P) of a scalar level, one warp per row, one lane per node of the row's column
// of P.  Each lane adds its node's terms to its own column of a table in shared memory, whose rows
// are the entries of the coarse row (found through a small hash of the column, checked, by search
// where two entries share a word of it); then each entry is summed over the lanes by four of them, in
// a fixed order.  (One search and one shuffle tree per entry and lane, as k_mg_ac does: 803
// instead of 342 us at 4M rows, 137 instead of 78 at 446k, 22 instead of 7 at 484.)
// W: entries of a coarse row, at most (wider levels take k_mg_ac).
template <int W>
__global__ void __launch_bounds__(128) k_mg_ac1(MgLev L, MgLev C) {
  __shared__ float part[4][W][33];
  __shared__ int kc[4][W];
  __shared__ uint8_t tab[4][64];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t J64 = gtid() >> 5;
  if (J64 >= L.nc) return;
  const int J = (int)J64;
  int64_t cb, tb;
  int cw, tw;
  slice_row(C.sptr, J, cb, cw);
  slice_row(L.pt_sptr, J, tb, tw);
  if (cw > W) cw = W;  // (the host checks the widths)
  const int32_t* ccol = reinterpret_cast<const int32_t*>(C.col);
  int K = -1;
  if (lane < cw) {
    K = __ldg(ccol + cb + 32 * (int64_t)lane);
    // (padding repeats the first column behind the row's entries: the first match owns the sum)
    if (lane > 0 && K == __ldg(ccol + cb)) K = -1;
    kc[wid][lane] = K;
  }
  tab[wid][lane] = tab[wid][lane + 32] = 0;
  __syncwarp();
  if (K >= 0) tab[wid][K & 63] = (uint8_t)lane;
  for (int k = 0; k < cw; k++) part[wid][k][lane] = 0.0f;
  __syncwarp();
  for (int q = lane; q < tw; q += 32) {
    const int src = __ldg(L.pt_src + tb + 32 * (int64_t)q);
    if (src < 0) continue;
    int64_t ab;
    int aw;
    slice_row(L.ap_sptr, __ldg(L.pt_col + tb + 32 * (int64_t)q), ab, aw);
    const float p = L.p_val[src];
    constexpr int U = 4;
    for (int s0 = 0; s0 < aw; s0 += U) {
      int c[U];
      float v[U];
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int64_t idx = ab + 32 * (int64_t)(s0 + u);
        c[u] = s0 + u < aw ? __ldg(L.ap_col + idx) : -1;
        v[u] = s0 + u < aw ? L.ap_val[idx] : 0.0f;
      }
#pragma unroll
      for (int u = 0; u < U; u++) {
        if (c[u] < 0) continue;
        int k = tab[wid][c[u] & 63];
        if (kc[wid][k] != c[u])
          for (k = 0; k < cw && kc[wid][k] != c[u]; k++) {
          }
        if (!ADFEM_DCHECK(k < cw) || k >= cw) continue;
        part[wid][k][lane] = fmaf(p, v[u], part[wid][k][lane]);
      }
    }
  }
  __syncwarp();
  for (int k0 = 0; k0 < cw; k0 += 8) {
    const int k = k0 + (lane >> 2), h = lane & 3;
    float x = 0.0f;
    if (k < cw)
#pragma unroll
      for (int q = 0; q < 8; q++) x += part[wid][k][8 * h + q];
    x += __shfl_xor_sync(0xffffffffu, x, 1);
    x += __shfl_xor_sync(0xffffffffu, x, 2);
    if (k < cw && h == 0) {
      const int col = kc[wid][k];
      C.val[cb + 32 * (int64_t)k] = col >= 0 ? x : 0.0f;
      if (col == J) C.s[J] = x > 0.0f && isfinite(x) ? rsqrtf(x) : 0.0f;
    }
  }
}

// Coarse rows P^T (A P), one warp per row, one lane per node of the row's column of P: the
// lanes load their nodes' rows of A P together, then each entry of the coarse row is the sum
// over the lanes of the one term (if any) that each contributes, by a fixed shuffle tree.
template <int NB, int NC>
__global__ void __launch_bounds__(128) k_mg_ac(MgLev L, MgLev C) {
  __shared__ int kk[4][kMgMaxAP][32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t J64 = gtid() >> 5;
  if (J64 >= L.nc) return;
  const int J = (int)J64;
  int64_t cb, tb;
  int cw, tw;
  slice_row(C.sptr, J, cb, cw);
  slice_row(L.pt_sptr, J, tb, tw);
  const int32_t* ccol = reinterpret_cast<const int32_t*>(C.col);
  int K[2];
  float acc[2][NC * NC];
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const int k = lane + 32 * h;
    K[h] = k < cw ? __ldg(ccol + cb + 32 * (int64_t)k) : -1;
    // (padding repeats the first column behind the row's entries: the first match owns the sum)
    if (k > 0 && K[h] == __ldg(ccol + cb)) K[h] = -1;
#pragma unroll
    for (int e = 0; e < NC * NC; e++) acc[h][e] = 0.0f;
  }
  for (int q0 = 0; q0 < tw; q0 += 32) {
    const int q = q0 + lane;
    const int src = q < tw ? __ldg(L.pt_src + tb + 32 * (int64_t)q) : -1;
    int64_t ab = 0;
    int aw = 0;
    float p[NB * NC];
    if (src >= 0) {
      slice_row(L.ap_sptr, __ldg(L.pt_col + tb + 32 * (int64_t)q), ab, aw);
      if (aw > kMgMaxAP) aw = kMgMaxAP;
      load_block<NB, NC>(L.p_val, src, L.np, p);
#pragma unroll 4
      for (int s = 0; s < aw; s++) kk[wid][s][lane] = __ldg(L.ap_col + ab + 32 * (int64_t)s);
    }
    __syncwarp();
    for (int k = 0; k < cw; k++) {
      const int col = __shfl_sync(0xffffffffu, k < 32 ? K[0] : K[1], k & 31);
      if (col < 0) continue;
      float v[NB * NC], T[NC * NC];
      int s = 0;
      while (s < aw && kk[wid][s][lane] != col) s++;
      if (s < aw) load_block<NB, NC>(L.ap_val, ab + 32 * (int64_t)s, L.nap, v);
#pragma unroll
      for (int c = 0; c < NC; c++)
#pragma unroll
        for (int m = 0; m < NC; m++) {
          float x = 0.0f;
          if (s < aw)
#pragma unroll
            for (int e = 0; e < NB; e++) x = fmaf(p[e * NC + c], v[e * NC + m], x);
          T[c * NC + m] = x;
        }
#pragma unroll
      for (int e = 0; e < NC * NC; e++) {
        const float x = warp_sum(T[e]);
        if (lane == (k & 31)) {
          if (k < 32) acc[0][e] += x;
          else acc[1][e] += x;
        }
      }
    }
    __syncwarp();
  }
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const int k = lane + 32 * h;
    if (k >= cw) continue;
#pragma unroll
    for (int e = 0; e < NC * NC; e++)
      C.val[block_at<NC, NC>(e, cb + 32 * (int64_t)k, C.nv)] = K[h] >= 0 ? acc[h][e] : 0.0f;
    if (K[h] == J)
#pragma unroll
      for (int c = 0; c < NC; c++) {
        const float d = acc[h][c * NC + c];
        C.s[(int64_t)NC * J + c] = d > 0.0f && isfinite(d) ? rsqrtf(d) : 0.0f;
      }
  }
}

// Unit diagonal: A_JK <- s_J A_JK s_K (1 on the diagonal of unknowns without a scale), and
// the interpolation in those unknowns, P <- P S, with its transpose.  One warp per coarse row.
// The first thread also turns the level's eigenvalue bound into the Chebyshev coefficients:
// 1 / theta, then (c1, c2) of step k at 2k, 2k + 1.
template <int NB, int NC>
__global__ void __launch_bounds__(128) k_mg_scale(MgLev L, MgLev C, int deg, float frac) {
  const int lane = threadIdx.x & 31;
  const int64_t J64 = gtid() >> 5;
  if (gtid() == 0) {
    const float hi = __int_as_float(*L.lam), lo = frac * hi;
    const float th = 0.5f * (hi + lo), de = 0.5f * (hi - lo), s1 = th / de;
    float rho = 1.0f / s1;
    L.coef[0] = 1.0f / th;
    for (int k = 1; k < deg; k++) {
      const float rn = 1.0f / (2.0f * s1 - rho);
      L.coef[2 * k] = rn * rho;
      L.coef[2 * k + 1] = 2.0f * rn / de;
      rho = rn;
    }
  }
  if (J64 >= L.nc) return;
  const int J = (int)J64;
  float sJ[NC];
#pragma unroll
  for (int c = 0; c < NC; c++) sJ[c] = __ldg(C.s + (int64_t)NC * J + c);
  int64_t base;
  int w;
  slice_row(C.sptr, J, base, w);
  const int32_t* ccol = reinterpret_cast<const int32_t*>(C.col);
  for (int k = lane; k < w; k += 32) {
    const int64_t e = base + 32 * (int64_t)k;
    const int K = __ldg(ccol + e);
    const bool own = K == J && (k == 0 || K != __ldg(ccol + base));  // (padding repeats the first column)
#pragma unroll
    for (int c = 0; c < NC; c++)
#pragma unroll
      for (int m = 0; m < NC; m++) {
        float* v = C.val + block_at<NC, NC>(c * NC + m, e, C.nv);
        *v = own && c == m ? 1.0f : *v * (sJ[c] * __ldg(C.s + (int64_t)NC * K + m));
      }
  }
  slice_row(L.pt_sptr, J, base, w);
  for (int q = lane; q < w; q += 32) {
    const int64_t e = base + 32 * (int64_t)q;
    const int64_t src = __ldg(L.pt_src + e);
    if (src < 0) continue;
#pragma unroll
    for (int r = 0; r < NB; r++)
#pragma unroll
      for (int c = 0; c < NC; c++) {
        float* pv = L.p_val + block_at<NB, NC>(r * NC + c, src, L.np);
        const float v = *pv * sJ[c];
        *pv = v;
        L.pt_val[block_at<NC, NB>(c * NB + r, e, L.npt)] = v;
      }
  }
}

// Inverse of the coarsest operator (N <= kMgDense, unit diagonal) by Gauss-Jordan in one block
// of 32 x 32 threads, each holding the entries (ty + 32 a, tx + 32 b) in registers; a step
// exchanges the pivot row and column through shared memory (one barrier).  A pivot at rounding
// level (a near-null space the Dirichlet data leave in) drops its unknown from the inverse,
// which stays symmetric positive semi-definite.
template <int NC>
__global__ void __launch_bounds__(1024) k_mg_dense(MgLev C, float* __restrict__ inv) {
  constexpr int S = kMgDense / 32;
  static_assert(kMgDense % 32 == 0, "whole tiles");
  extern __shared__ float4 dense_sm4[];
  float* A = reinterpret_cast<float*>(dense_sm4);  // N x N, then two pivot rows and columns
  const int N = C.n * NC;
  float* piv = A + N * N;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  for (int t = threadIdx.x; t < N * N; t += blockDim.x) A[t] = 0.0f;
  __syncthreads();
  const int32_t* col = reinterpret_cast<const int32_t*>(C.col);
  for (int r = ty; r < C.n; r += 32) {
    int64_t base;
    int w;
    slice_row(C.sptr, r, base, w);
    for (int k = tx; k < w; k += 32) {
      const int64_t e = base + 32 * (int64_t)k;
      const int K = col[e];
      if (k > 0 && K == col[base]) continue;  // (padding)
      for (int c = 0; c < NC; c++)
        for (int m = 0; m < NC; m++)
          A[(r * NC + c) * N + K * NC + m] = C.val[block_at<NC, NC>(c * NC + m, e, C.nv)];
    }
  }
  __syncthreads();
  float x[S][S];
#pragma unroll
  for (int a = 0; a < S; a++)
#pragma unroll
    for (int b = 0; b < S; b++) {
      const int r = ty + 32 * a, c = tx + 32 * b;
      x[a][b] = r < N && c < N ? A[r * N + c] : 0.0f;
    }
  // Pivot k = 32 a0 + kk: its row and column are published, then x -= f s with s the scaled pivot
  // row; the pivot's own row and column fit the same formula once their x is 0 (f = -1, s = 1 / p).
  // The outer loops are unrolled, so that tiles and owners are compile-time and tiles beyond N are
  // skipped: bound by instruction issue, 25 FMAs and some 40 others per step at N = 160.  (Every
  // element looking whether it is the pivot's: 286 us instead of 95 at N = 160, 93 instead of 30 at 45.)
  const int tiles = (N + 31) / 32;
#pragma unroll
  for (int a0 = 0; a0 < S; a0++) {
    const int steps = min(32, N - 32 * a0);
    for (int kk = 0; kk < steps; kk++) {
      float* row = piv + (kk & 1) * 2 * kMgDense;
      float* cl = row + kMgDense;
      const bool mr = ty == kk, mc = tx == kk;
      if (mr) {
#pragma unroll
        for (int b = 0; b < S; b++) row[tx + 32 * b] = x[a0][b];
      }
      if (mc) {
#pragma unroll
        for (int a = 0; a < S; a++) cl[ty + 32 * a] = x[a][a0];
      }
      __syncthreads();
      const float p = row[32 * a0 + kk];
      const float ip = p > 1e-5f ? 1.0f / p : 0.0f;
      float s[S], f[S];
#pragma unroll
      for (int b = 0; b < S; b++) s[b] = b < tiles ? row[tx + 32 * b] * ip : 0.0f;
#pragma unroll
      for (int a = 0; a < S; a++) f[a] = a < tiles ? cl[ty + 32 * a] : 0.0f;
      if (mc) {
        s[a0] = ip;
#pragma unroll
        for (int a = 0; a < S; a++) x[a][a0] = 0.0f;
      }
      if (mr) {
        f[a0] = -1.0f;
#pragma unroll
        for (int b = 0; b < S; b++) x[a0][b] = 0.0f;
      }
#pragma unroll
      for (int a = 0; a < S; a++) {
        if (a >= tiles) break;
#pragma unroll
        for (int b = 0; b < S; b++) x[a][b] = fmaf(-f[a], s[b], x[a][b]);
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int a = 0; a < S; a++)
#pragma unroll
    for (int b = 0; b < S; b++) {
      const int r = ty + 32 * a, c = tx + 32 * b;
      if (r < N && c < N) A[r * N + c] = x[a][b];
    }
  __syncthreads();
  // (symmetrised: the cycle has to be symmetric)
  for (int r = ty; r < N; r += 32)
    for (int c = tx; c < N; c += 32) inv[r * N + c] = 0.5f * (A[r * N + c] + A[c * N + r]);
}

// ---------------------------------------------------------------------------
// FP64 CG around the cycle, in the physical unknowns; norms in the Jacobi-scaled ones.

// b = rhs (0 where zero_rows is tagged 1), y = u0, 0, or the prescribed value on Dirichlet rows
__global__ void __launch_bounds__(kT) k_mg_init(int64_t n, const double* __restrict__ rhs,
                                                const uint8_t* __restrict__ zero_rows,
                                                const uint8_t* __restrict__ fix, const double* __restrict__ fixval,
                                                const float* __restrict__ s, const double* __restrict__ u0,
                                                double* __restrict__ b, double* __restrict__ y,
                                                double* __restrict__ z, CgState* st, double* partials, double rtol2) {
  double acc = 0.0;
  for (int64_t i = gtid(); i < n; i += gstride()) {
    const double bi = (zero_rows && zero_rows[i] == 1) ? 0.0 : rhs[i];
    const double t = (double)s[i] * bi;
    b[i] = bi;
    y[i] = fix && fix[i] == 1 ? (fixval ? fixval[i] : 0.0) : (u0 ? u0[i] : 0.0);
    z[i] = 0.0;
    acc = fma(t, t, acc);
  }
  double v[1] = {acc}, tot[1];
  if (reduce_grid<double, 1>(v, partials, &st->counter[0], tot) && threadIdx.x == 0) {
    st->bnorm2 = tot[0];
    st->stop2 = rtol2 * tot[0];
    // scale of the FP32 right-hand sides of the cycle
    const double g = tot[0] > 0.0 ? rsqrt(tot[0]) : 1.0;
    st->ar = isfinite(g) ? g : 1.0;
    st->iar = 1.0 / st->ar;
  }
}

// r = b - K y in FP64, in difference form: row sums times the row's own unknowns plus entries
// times differences, so that it rounds with the differences of the solution.
// The iterate is y + z; the next direction kernel folds z into y (st->fold).
// mode 0: start, 1: the end of an iteration (evaluated when the recurrence has met the tolerance,
// has dropped far enough, or ends; sets the loop's condition), 2: final value only
template <bool D16, int NB>
__global__ void __launch_bounds__(kT) k_mg_residual(int64_t n, const int32_t* __restrict__ sptr,
                                                    const void* __restrict__ col, const double* __restrict__ val,
                                                    const double* __restrict__ rowsum, const float* __restrict__ sc,
                                                    const double* b, const double* y, const double* z,
                                                    double* r64, float* b32, CgState* st,
                                                    const double* rn_part, int rn_count,
                                                    double* partials, int mode, cudaGraphConditionalHandle loop) {
  pdl_trigger();
  pdl_wait();
  const bool lead = blockIdx.x == 0 && threadIdx.x == 0;
  double rn = 0.0;
  if (mode == 1) {
    const double2 v = grid_total(rn_part, rn_count, [&](double t) {
      return make_double2(t * st->iar * st->iar, st->done ? 1.0 : 0.0);
    });
    if (v.y != 0.0) {
      if (lead) cudaGraphSetConditional(loop, 0);
      return;
    }
    rn = v.x;
    const bool due = rn <= st->stop2 || rn <= st->ru2 || st->it >= st->max_iter;
    if (!isfinite(rn) || !due) {
      if (lead) {
        st->iters = st->it;
        st->rho_new = rn;
        if (!isfinite(rn)) st->done = 2;
        cudaGraphSetConditional(loop, isfinite(rn) ? 1 : 0);
      }
      return;
    }
  }
  const double g = st->ar;
  double a0 = 0.0;
  for (int64_t r = gtid(); r < n; r += gstride()) {
    int64_t base;
    int w;
    sell_row(sptr, r, base, w);
    double yo[NB], s = 0.0;
#pragma unroll
    for (int q = 0; q < NB; q++) {
      yo[q] = y[r / NB * NB + q] + z[r / NB * NB + q];
      s = fma(rowsum[NB * r + q], yo[q], s);
    }
    constexpr int U = 8;
    for (int k0 = 0; k0 < w; k0 += U) {
      double v[U], x[U];
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int64_t idx = base + 32 * (int64_t)(k0 + u);
        int j = (int)r;
        v[u] = 0.0;
        if (k0 + u < w) {
          v[u] = __ldg(val + idx);
          j = colof<D16>(col, idx, r);
          if (!ADFEM_DCHECK(j >= 0 && j < n)) j = (int)r;
        }
        x[u] = y[j] + z[j];
      }
#pragma unroll
      for (int u = 0; u < U; u++)
        if (k0 + u < w) s = fma(v[u], x[u] - (NB == 1 ? yo[0] : ((k0 + u) & 1 ? yo[NB - 1] : yo[0])), s);
    }
    const double ri = b[r] - s, t = (double)sc[r] * ri;
    a0 = fma(t, t, a0);
    if (mode != 2) {
      r64[r] = ri;
      b32[r] = (float)(t * g);
    }
  }
  double v[1] = {a0}, tot[1];
  if (reduce_grid<double, 1>(v, partials, &st->counter[1], tot) && threadIdx.x == 0) {
    if (mode == 2) {
      st->rr64 = tot[0];
      return;
    }
    st->iters = st->it;
    st->rho_new = rn;
    mg_residual_step(st, tot[0], rn, mode == 0);
    if (mode == 1) cudaGraphSetConditional(loop, st->done == 0 ? 1 : 0);
  }
}

// p = S c + beta p (c: the cycle's correction, its r.z in rz_part), and after a residual
// evaluation y += z, z = 0; two unknowns per thread
__global__ void __launch_bounds__(kT) k_mg_dir(int64_t n, const float* c, const float* __restrict__ s, double* p,
                                               double* y, double* z, CgState* st, const double* rz_part,
                                               int rz_count) {
  pdl_trigger();
  pdl_wait();
  const bool first = st->ap != 0.0;  // (the direction starts anew)
  const double2 v = grid_total(rz_part, rz_count, [&](double t) {
    const double rz = t * st->iar;  // (b carries the factor st->ar, and so does z)
    const bool ok = rz > 0.0 && isfinite(rz) && !st->done;
    if (blockIdx.x == 0 && !st->done) {
      if (ok) st->rz = rz;
      else st->done = 2;
    }
    return make_double2(ok ? 1.0 : 0.0, ok && !first ? rz * st->irz : 0.0);
  });
  if (v.x == 0.0) return;
  const double bt = v.y;
  const int64_t n2 = n >> 1;
#pragma unroll 4
  for (int64_t i = gtid(); i < n2; i += gstride()) {
    const float2 c2 = reinterpret_cast<const float2*>(c)[i], s2 = __ldg(reinterpret_cast<const float2*>(s) + i);
    double2 q = make_double2((double)(s2.x * c2.x), (double)(s2.y * c2.y));
    if (!first) {
      const double2 o = reinterpret_cast<const double2*>(p)[i];
      q.x = fma(bt, o.x, q.x);
      q.y = fma(bt, o.y, q.y);
    }
    reinterpret_cast<double2*>(p)[i] = q;
  }
  if ((n & 1) && gtid() == 0) {
    const double ci = (double)(s[n - 1] * c[n - 1]);
    p[n - 1] = first ? ci : fma(bt, p[n - 1], ci);
  }
  if (st->fold)
    for (int64_t i = gtid(); i < n; i += gstride()) {
      y[i] += z[i];
      z[i] = 0.0;
    }
}

// q = K p and p.q, one row per thread, entries in groups whose loads are in flight together, the
// first loaded ahead.  Rows of up to 8 entries are one group; longer ones (MORE: P2, elasticity) go in
// groups of 4, which leaves room for eight blocks on an SM: their scattered reads of p are what bounds
// them, and those overlap by warps rather than within a row (P2 4M DOF, ms a solve: groups of 12 and
// three blocks 79.3, 8 and five 73.2, 6 and six 71.1, 4 and eight 68.0).
template <bool D16, bool MORE>
__global__ void __launch_bounds__(kT, MORE ? 8 : 4) k_mg_spmv(int64_t n, const int32_t* __restrict__ sptr,
                                                   const void* __restrict__ col, const int32_t* __restrict__ spat,
                                                   const int16_t* __restrict__ pat, int period,
                                                   const double* __restrict__ val, const double* p, double* q,
                                                   CgState* st, double* partials) {
  constexpr int W = MORE ? 4 : 8;
  pdl_trigger();
  double v[W], acc = 0.0;
  int j[W], w = 0;
  int64_t base = 0;
  const int16_t* pp = nullptr;
  auto entries = [&](int r, int k0) {
#pragma unroll
    for (int u = 0; u < W; u++) {
      const int k = k0 + u;
      const int64_t idx = base + 32 * k;
      v[u] = k < w ? __ldg(val + idx) : 0.0;
      j[u] = r;
      if (k < w) j[u] = pp ? r + (int)__ldg(pp + k) : colof<D16>(col, idx, r);
      if (!ADFEM_DCHECK(j[u] >= 0 && j[u] < n)) j[u] = r;
    }
  };
  auto load = [&](int r) {
    sell_row(sptr, r, base, w);
    const int32_t so = __ldg(spat + (r >> 5));
    pp = so >= 0 ? pat + so + (period == 2 ? (r & 1) * w : 0) : nullptr;
    entries(r, 0);
  };
  int r = blockIdx.x * kT + threadIdx.x;
  const int rows = (int)n;
  if (r < rows) load(r);
  pdl_wait();
  if (st->done) return;
  // (state that the kernels before and after read and this one does not)
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    st->it += 1;
    st->irz = 1.0 / st->rz;
    st->ap = 0.0;
    st->fold = 0;
  }
  while (r < rows) {
    const double pr = p[r];
    double s = 0.0;
#pragma unroll
    for (int u = 0; u < W; u++)
      if (u < w) s = fma(v[u], p[j[u]], s);
    if (MORE)
      for (int k0 = W; k0 < w; k0 += W) {
        entries(r, k0);
#pragma unroll
        for (int u = 0; u < W; u++)
          if (k0 + u < w) s = fma(v[u], p[j[u]], s);
      }
    q[r] = s;
    acc = fma(pr, s, acc);
    r += gridDim.x * kT;
    if (r < rows) load(r);
  }
  block_partial(acc, partials);
}

// z += alpha p, r -= alpha q (z: the correction since the last residual evaluation), and the
// cycle's next right-hand side with its norm; two unknowns per thread
__global__ void __launch_bounds__(kT) k_mg_update(int64_t n, double* z, double* r, const double* p, const double* q,
                                                  const float* __restrict__ s, float* b32, CgState* st,
                                                  const double* pq_part, int pq_count, double* partials) {
  pdl_trigger();
  pdl_wait();
  const double2 v = grid_total(pq_part, pq_count, [&](double pq) {
    const bool ok = pq > 0.0 && isfinite(pq) && !st->done;
    if (!ok && blockIdx.x == 0 && !st->done) st->done = 2;
    return make_double2(ok ? 1.0 : 0.0, ok ? st->rz / pq : 0.0);
  });
  if (v.x == 0.0) return;
  const double a = v.y, g = st->ar;
  double acc = 0.0;
  const int64_t n2 = n >> 1;
  for (int64_t i = gtid(); i < n2; i += gstride()) {
    const double2 pp = reinterpret_cast<const double2*>(p)[i], qq = reinterpret_cast<const double2*>(q)[i];
    double2 zz = reinterpret_cast<const double2*>(z)[i], rr = reinterpret_cast<const double2*>(r)[i];
    const float2 ss = __ldg(reinterpret_cast<const float2*>(s) + i);
    zz.x = fma(a, pp.x, zz.x);
    zz.y = fma(a, pp.y, zz.y);
    rr.x = fma(-a, qq.x, rr.x);
    rr.y = fma(-a, qq.y, rr.y);
    reinterpret_cast<double2*>(z)[i] = zz;
    reinterpret_cast<double2*>(r)[i] = rr;
    const double tx = rr.x * g * (double)ss.x, ty = rr.y * g * (double)ss.y;
    reinterpret_cast<float2*>(b32)[i] = make_float2((float)tx, (float)ty);
    acc = fma(tx, tx, acc);
    acc = fma(ty, ty, acc);
  }
  if ((n & 1) && gtid() == 0) {
    const int64_t i = n - 1;
    z[i] = fma(a, p[i], z[i]);
    const double ri = fma(-a, q[i], r[i]);
    r[i] = ri;
    const double t = ri * g * (double)s[i];
    b32[i] = (float)t;
    acc = fma(t, t, acc);
  }
  block_partial(acc, partials);
}

__global__ void __launch_bounds__(kT) k_mg_out(int64_t n, const double* __restrict__ y,
                                               const uint8_t* __restrict__ fix, const double* __restrict__ fixval,
                                               double* __restrict__ u) {
  const int64_t i = gtid();
  if (i >= n) return;
  u[i] = fix && fix[i] == 1 ? (fixval ? fixval[i] : 0.0) : y[i];
}

// ---------------------------------------------------------------------------
// plan: one device slab with every pattern and work array
struct Slab {
  std::vector<char> host;  // the part that is uploaded
  size_t total = 0;
  std::vector<std::pair<void**, size_t>> fix;
  template <class T>
  void put(const T** p, const std::vector<T>& v) {
    const size_t off = (host.size() + 255) / 256 * 256;
    host.resize(off + sizeof(T) * std::max<size_t>(v.size(), 1));
    std::memcpy(host.data() + off, v.data(), sizeof(T) * v.size());
    fix.emplace_back((void**)p, off);
  }
  size_t mark() {
    host.resize((host.size() + 255) / 256 * 256);
    return host.size();
  }
  void seal() { total = (host.size() + 255) / 256 * 256; }
  template <class T>
  void room(T** p, size_t count) {
    fix.emplace_back((void**)p, total);
    total = (total + sizeof(T) * std::max<size_t>(count, 1) + 255) / 256 * 256;
  }
  void resolve(char* base) {
    for (auto& f : fix) *f.first = base + f.second;
  }
};

// slices of 32 rows with absolute columns (padding: the row's first column)
void slices(int64_t n, const MgPattern& P, std::vector<int32_t>& sptr, std::vector<int32_t>& col) {
  const int64_t ns = (n + 31) / 32;
  sptr.assign(ns + 1, 0);
  for (int64_t s = 0; s < ns; s++) {
    int32_t w = 0;
    for (int64_t r = 32 * s; r < std::min(n, 32 * s + 32); r++) w = std::max(w, P.rp[r + 1] - P.rp[r]);
    sptr[s + 1] = sptr[s] + 32 * w;
  }
  col.assign(std::max<int32_t>(sptr[ns], 1), 0);
  parallel_for(n, [&](int64_t lo, int64_t hi) {
    for (int64_t r = lo; r < hi; r++) {
      const int32_t len = P.rp[r + 1] - P.rp[r], w = (sptr[(r >> 5) + 1] - sptr[r >> 5]) / 32;
      for (int32_t k = 0; k < w; k++)
        col[sptr[r >> 5] + 32 * k + (r & 31)] = len ? P.ci[P.rp[r] + (k < len ? k : 0)] : 0;
    }
  });
}

// Tail blocks that need each row's value of the tail's first level: those that own a row that
// refers to it in A (sweeps) or a coarse row whose restriction reads it; cnt: how many rows each
// block needs.
void tail_targets(const MgHostLevel& H, int64_t nc, std::vector<uint8_t>& to, std::vector<int32_t>& cnt) {
  to.assign(H.n, 0);
  auto owner = [](int64_t r, int64_t n) { return (int)(r / tail_chunk((int)n)); };
  for (int64_t r = 0; r < H.n; r++)
    for (int32_t k = H.A.rp[r]; k < H.A.rp[r + 1]; k++) to[H.A.ci[k]] |= (uint8_t)(1 << owner(r, H.n));
  for (int64_t i = 0; i < H.n; i++)
    for (int32_t k = H.P.rp[i]; k < H.P.rp[i + 1]; k++) to[i] |= (uint8_t)(1 << owner(H.P.ci[k], nc));
  cnt.assign(kTailC, 0);
  for (uint8_t m : to)
    for (int k = 0; k < kTailC; k++) cnt[k] += (m >> k) & 1;
}

int lanes_per_row(int64_t n) {
  // one lane while the rows alone fill the chip (152 SMs x 2048 threads), more below
  return n >= 150000 ? 1 : (n >= 40000 ? 4 : 8);
}


}  // namespace

// the device has less than this left (a failed allocation is then no error of its own)
static bool short_of(size_t bytes) {
  size_t freeb = 0, total = 0;
  cudaGetLastError();
  return cudaMemGetInfo(&freeb, &total) == cudaSuccess && freeb < bytes + ((size_t)64 << 20);
}

static int plan(Solver& S) {
  const int nb0 = S.mg_nb, nbc = nb0 == 2 ? 3 : 1;
  std::vector<MgHostLevel> lv;
  // (a plan that ends in an error or an exception gives the graph back: the next solve tries again)
  struct GiveBack {
    Solver& S;
    std::vector<MgHostLevel>& lv;
    ~GiveBack() {
      if (S.mg || !S.mg_allowed || lv.empty()) return;
      S.mg_rp = std::move(lv[0].A.rp);
      S.mg_ci = std::move(lv[0].A.ci);
      S.mg_x = std::move(lv[0].x);
      S.mg_y = std::move(lv[0].y);
    }
  } give_back{S, lv};
  if (!mg_build_host((int64_t)S.mg_rp.size() - 1, std::move(S.mg_rp), std::move(S.mg_ci), nb0, nbc,
                     std::move(S.mg_x), std::move(S.mg_y), lv)) {
    S.mg_allowed = false;
    return ADFEM_OK;
  }
  std::unique_ptr<Mg> mg(new Mg());
  Mg& M = *mg;
  M.nlev = (int)lv.size();
  while (M.tail < M.nlev - 1 && lv[M.tail].n * (M.tail ? nbc : nb0) > kMgTailDofs) M.tail++;
  M.cluster = lv[M.tail].n * (M.tail ? nbc : nb0) > kTailLocal;
  if (M.nlev < 2 || M.nlev - M.tail > kMgMaxTail || M.tail + 1 >= M.nlev) {
    S.mg_allowed = false;
    return ADFEM_OK;
  }
  const Sell& A = *S.A;
  Slab sl;
  std::vector<int32_t> sptr, col, cnt;
  std::vector<uint8_t> to;
  std::vector<int64_t> vals(M.nlev);
  const int local = M.tail + (M.cluster ? 1 : 0);  // first level that a tail block runs alone
  for (int l = 0; l < M.nlev; l++) {
    MgLev& L = M.lev[l];
    MgHostLevel& H = lv[l];
    L.n = (int)H.n;
    L.nb = l ? nbc : nb0;
    L.nbc = nbc;
    const bool tail = l >= M.tail;
    L.lpr = l == 0 ? (nb0 == 1 || H.n >= 150000 ? 1 : 4) : lanes_per_row(H.n);
    if (l == M.tail && M.cluster) {
      tail_targets(lv[l], lv[l + 1].n, to, cnt);
      sl.put(&L.to, to);
      sl.put(&L.cnt, cnt);
    }
    if (l + 1 < M.nlev) {
      L.nc = (int)lv[l + 1].n;
      // (what only the value kernels read comes before the range that the tail copies)
      slices(H.n, H.AP, sptr, col);
      sl.put(&L.ap_sptr, sptr);
      sl.put(&L.ap_col, col);
      L.nap = sptr.back();
      slices(H.n, H.P, sptr, col);
      const std::vector<int32_t> psptr = sptr;
      slices(L.nc, H.PT, sptr, col);
      std::vector<int32_t> src(col.size(), -1);
      for (int64_t J = 0; J < L.nc; J++)
        for (int32_t k = H.PT.rp[J]; k < H.PT.rp[J + 1]; k++) {
          const int32_t i = H.PT.ci[k];
          src[sptr[J >> 5] + 32 * (k - H.PT.rp[J]) + (J & 31)] = psptr[i >> 5] + 32 * H.PTslot[k] + (i & 31);
        }
      sl.put(&L.pt_src, src);
      sl.put(&L.agg, H.agg);
      if (nbc == 3) {
        std::vector<float2> dp(H.n);
        for (int64_t i = 0; i < H.n; i++)
          dp[i] = make_float2((float)(H.x[i] - lv[l + 1].x[H.agg[i]]), (float)(H.y[i] - lv[l + 1].y[H.agg[i]]));
        sl.put(&L.dpos, dp);
      }
    }
    if (l == 0 && nb0 == 1 && !tail) {
      // the system's own pattern
      L.sptr = A.sptr.as<int32_t>();
      L.col = A.col.p;
      L.spat = A.spat.as<int32_t>();
      L.pat = A.pat.as<int16_t>();
      L.d16 = A.delta16 ? 1 : 0;
      vals[l] = A.nent;
    }
  }
  size_t pat0 = 0, val0 = 0;
  for (int l = 0; l < M.nlev; l++) {
    MgLev& L = M.lev[l];
    MgHostLevel& H = lv[l];
    if (l == local) pat0 = sl.mark();
    if (!(l == 0 && nb0 == 1 && M.tail > 0)) {
      slices(H.n, H.A, sptr, col);
      sl.put(&L.sptr, sptr);
      sl.put((const int32_t**)&L.col, col);
      vals[l] = sptr.back();
    }
    for (int64_t r = 0; r < H.n; r++) L.width = std::max<int>(L.width, H.A.rp[r + 1] - H.A.rp[r]);
    L.nv = (int)vals[l];
    if (l + 1 == M.nlev) continue;
    slices(H.n, H.P, sptr, col);
    sl.put(&L.p_sptr, sptr);
    sl.put(&L.p_col, col);
    L.np = sptr.back();
    slices(L.nc, H.PT, sptr, col);
    sl.put(&L.pt_sptr, sptr);
    sl.put(&L.pt_col, col);
    L.npt = sptr.back();
  }
  for (int l = 0; l < M.nlev; l++)
    if (vals[l] * M.lev[l].nb > INT32_MAX) {  // (entries are indexed with 32 bits)
      S.mg_allowed = false;
      return ADFEM_OK;
    }
  sl.seal();
  M.pat_bytes = (int)(sl.total - pat0);
  for (int l = 0; l < M.nlev; l++) {
    MgLev& L = M.lev[l];
    const size_t nb = L.nb, n = (size_t)L.n * nb;
    sl.room(&L.s, n);
    sl.room(&L.b, n);
    sl.room(&L.x, n);
    sl.room(&L.x2, n);
    sl.room(&L.d, n);
    if (l + 1 < M.nlev) sl.room(&L.ap_val, (size_t)L.nap * nb * nbc);
  }
  sl.room(&M.rowsum, (size_t)S.n * nb0);
  sl.room(&M.lam, kMgMaxLevels);
  sl.room(&M.part, 3 * kMgGrid);
  for (int l = 0; l < M.nlev; l++) {
    MgLev& L = M.lev[l];
    const size_t nb = L.nb;
    if (l == local) val0 = sl.total;
    sl.room(&L.val, (size_t)vals[l] * nb * nb);
    sl.room(&L.coef, kCoef + 2);
    if (l + 1 == M.nlev) continue;
    sl.room(&L.p_val, (size_t)L.np * nb * nbc);
    sl.room(&L.pt_val, (size_t)L.npt * nb * nbc);
  }
  M.ndense = M.lev[M.nlev - 1].n * M.lev[M.nlev - 1].nb;
  int dev = 0;
  ADFEM_CUDA(cudaGetDevice(&dev));
  ADFEM_CUDA(cudaDeviceGetAttribute(&M.sms, cudaDevAttrMultiProcessorCount, dev));
  sl.room(&M.dense, (size_t)M.ndense * M.ndense);
  M.val_bytes = (int)(sl.total - val0);
  S.mg_need = sl.total;
  if (S.mg_need > S.mg_limit) return ADFEM_OK;
  const int got = M.slab.alloc(sl.total);
  if (got == ADFEM_ERR_NOMEM && short_of(sl.total)) return ADFEM_OK;
  ADFEM_TRY(got);
  sl.resolve(M.slab.as<char>());
  for (int l = 0; l < M.nlev; l++) M.lev[l].lam = M.lam + l;
  ADFEM_CUDA(cudaMemcpy(M.slab.p, sl.host.data(), sl.host.size(), cudaMemcpyHostToDevice));
  ADFEM_CUDA(cudaMemset(M.slab.as<char>() + sl.host.size(), 0, sl.total - sl.host.size()));
  // (legacy-stream sync, not a device-wide one: other threads may be capturing graphs)
  ADFEM_CUDA(cudaStreamSynchronize(0));
  size_t fl = 0;
  for (int l = M.tail; l < M.nlev; l++) fl += (size_t)tail_floats(M.lev[l].n, M.lev[l].nb, M.cluster && l == M.tail);
  M.tail_smem = sizeof(float) * fl;
  if (M.tail == 0) {
    const size_t n0 = (size_t)M.lev[0].n * M.lev[0].nb;
    M.tail_smem += sizeof(double) * (n0 + 3 * kTailT + 2 * kTailC) + sizeof(float) * n0;
  }
  M.pat = M.slab.as<char>() + pat0;
  M.vals = M.slab.as<char>() + val0;
  if (M.tail_smem + M.pat_bytes + M.val_bytes > kTailSmem) M.pat_bytes = M.val_bytes = 0;  // read through L1
  M.tail_smem += M.pat_bytes + M.val_bytes;
  {
    // (once per process: changing a kernel attribute while another thread captures that
    // kernel would invalidate the capture)
    static std::once_flag once;
    static cudaError_t err = cudaSuccess;
    std::call_once(once, [] {
      const int tmax = (int)kTailSmem;
      const int dmax = (int)(sizeof(float) * (kMgDense * kMgDense + 4 * kMgDense));
      const auto a = cudaFuncAttributeMaxDynamicSharedMemorySize;
      for (cudaError_t e :
           {cudaFuncSetAttribute(k_mg_tail<1, 1, false, false>, a, tmax),
            cudaFuncSetAttribute(k_mg_tail<2, 3, false, false>, a, tmax),
            cudaFuncSetAttribute(k_mg_tail<3, 3, false, false>, a, tmax),
            cudaFuncSetAttribute(k_mg_tail<1, 1, true, false>, a, tmax),
            cudaFuncSetAttribute(k_mg_tail<2, 3, true, false>, a, tmax),
            cudaFuncSetAttribute(k_mg_tail<3, 3, true, false>, a, tmax),
            cudaFuncSetAttribute(k_mg_tail<1, 1, false, true>, a, tmax),
            cudaFuncSetAttribute(k_mg_tail<2, 3, false, true>, a, tmax),
            cudaFuncSetAttribute(k_mg_tail<1, 1, true, true>, a, tmax),
            cudaFuncSetAttribute(k_mg_tail<2, 3, true, true>, a, tmax),
            cudaFuncSetAttribute(k_mg_dense<1>, a, dmax), cudaFuncSetAttribute(k_mg_dense<3>, a, dmax)})
        if (e != cudaSuccess) err = e;
    });
    if (err != cudaSuccess) return cuda_fail(err, "cudaFuncSetAttribute (multigrid)");
    if (M.tail_smem > kTailSmem) {
      S.mg_allowed = false;
      return ADFEM_OK;
    }
  }
  S.mg = std::move(mg);
  return ADFEM_OK;
}

int mg_plan(Solver& S) {
  if (S.mg || !S.mg_allowed) return ADFEM_OK;
  // (a hierarchy that did not fit before: the patterns are not made again to find that out)
  if (!S.mg_room || S.mg_limit == 0 || S.mg_need > S.mg_limit || (S.mg_need > 0 && short_of(S.mg_need))) return ADFEM_OK;
  try {
    return plan(S);
  } catch (const std::bad_alloc&) {
    return ADFEM_OK;  // (no host memory for the patterns: this solve takes the Jacobi iteration)
  }
}

// ---------------------------------------------------------------------------
namespace {

unsigned blocks(int64_t n, int b) { return (unsigned)std::max<int64_t>(1, (n + b - 1) / b); }

template <int NB, int NC, bool D16>
void level_values(const MgLev& L, const MgLev& C, bool top, cudaStream_t st) {
  constexpr int BP = 64, BA = NB * NC == 1 ? 128 : 32;
  const int deg = top ? kMgDeg0 : kMgDeg;
  const float frac = top ? kFrac0 : kFrac;
  const float smooth = NC == 1 ? (top ? 1.6f : 1.8f) : (top ? 1.8f : 2.2f);
  k_mg_p<NB, NC, D16, BP><<<blocks(L.n, BP), BP, 0, st>>>(L, smooth);
  k_mg_ap<NB, NC, D16, BA><<<blocks(L.n, BA), BA, 0, st>>>(L);
  const unsigned gc = blocks(32 * (int64_t)L.nc, 128);
  if (NC == 1 && C.width <= 16) k_mg_ac1<16><<<gc, 128, 0, st>>>(L, C);
  else if (NC == 1 && C.width <= 32) k_mg_ac1<32><<<gc, 128, 0, st>>>(L, C);
  else k_mg_ac<NB, NC><<<gc, 128, 0, st>>>(L, C);
  k_mg_scale<NB, NC><<<blocks(32 * (int64_t)L.nc, 128), 128, 0, st>>>(L, C, deg, frac);
}

}  // namespace

// Enqueue the values of the hierarchy for the current assembly (s32 is current): level 0 with the row
// sums, which the residual needs, and the rest.  They count as made (Mg::current) once the host has
// seen the stream past them, in mg_solve: on a stream that is being captured nothing runs, and a call
// that fails before then leaves them to the next.
static int mg_values0(Solver& S, cudaStream_t st) {
  Mg& M = *S.mg;
  const Sell& A = *S.A;
  const MgLev& L0 = M.lev[0];
  const unsigned nb = blocks(S.n, kT);
  ADFEM_CUDA(cudaMemsetAsync(M.lam, 0, sizeof(int) * kMgMaxLevels, st));
  auto vals0 = [&](auto nbt, auto d16) {
    k_mg_vals0<decltype(nbt)::value, decltype(d16)::value><<<nb, kT, 0, st>>>(
        S.n, A.sptr.as<int32_t>(), A.col.p, A.val64.as<double>(), S.s32.as<float>(), S.mg_isbd, L0, M.rowsum);
  };
  using std::integral_constant;
  if (L0.nb == 2) {
    if (A.delta16) vals0(integral_constant<int, 2>{}, std::true_type{});
    else vals0(integral_constant<int, 2>{}, std::false_type{});
  } else {
    if (A.delta16) vals0(integral_constant<int, 1>{}, std::true_type{});
    else vals0(integral_constant<int, 1>{}, std::false_type{});
  }
  ADFEM_CUDA(cudaGetLastError());
  return ADFEM_OK;
}

static int mg_values_below(Solver& S, cudaStream_t st) {
  Mg& M = *S.mg;
  for (int l = 0; l + 1 < M.nlev; l++) {
    const MgLev &L = M.lev[l], &C = M.lev[l + 1];
    if (L.nb == 1) {
      if (L.d16) level_values<1, 1, true>(L, C, l == 0, st);
      else level_values<1, 1, false>(L, C, l == 0, st);
    } else if (L.nb == 2) {
      level_values<2, 3, false>(L, C, l == 0, st);
    } else {
      level_values<3, 3, false>(L, C, l == 0, st);
    }
  }
  const MgLev& C = M.lev[M.nlev - 1];
  const size_t dsm = sizeof(float) * ((size_t)M.ndense * M.ndense + 4 * kMgDense);
  if (C.nb == 1) k_mg_dense<1><<<1, 1024, dsm, st>>>(C, M.dense);
  else k_mg_dense<3><<<1, 1024, dsm, st>>>(C, M.dense);
  ADFEM_CUDA(cudaGetLastError());
  return ADFEM_OK;
}

namespace {

// Launch of a kernel of an iteration (programmatic dependent launch unless ADFEM_ZCG_PDL=0).
template <class... P, class... A>
void mg_launch(const Solver& S, cudaStream_t st, void (*kern)(P...), unsigned grid, unsigned block, size_t smem,
               unsigned cluster, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  int na = 0;
  if (S.zpdl) {
    at[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[na++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (cluster > 1) {
    at[na].id = cudaLaunchAttributeClusterDimension;
    at[na].val.clusterDim.x = cluster;
    at[na].val.clusterDim.y = at[na].val.clusterDim.z = 1;
    na++;
  }
  cfg.attrs = at;
  cfg.numAttrs = na;
  cudaLaunchKernelEx(&cfg, kern, P(args)...);  // (an error is reported by the caller's cudaGetLastError)
}

// Blocks of a kernel that sums over its grid or needs such a sum: at most one resident wave (every
// block reads all partial sums of the kernel before).
template <class K>
unsigned sum_grid(const Solver& S, K kern, int64_t threads) {
  int per = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, kT, 0) != cudaSuccess || per < 1) per = 1;
  return std::min(blocks(threads, kT), (unsigned)std::min(per * S.mg->sms, kMgGrid));
}

template <int MODE>
void sweep(const Solver& S, const MgLev& L, const float* x, float* out, int c1, int c2, int keep, double* part,
           cudaStream_t st) {
  const int64_t threads = (int64_t)L.n * L.lpr;
  auto grid = [&](auto kern) {
    if (MODE != kLast || !part) return blocks(threads, kT);
    const unsigned g = sum_grid(S, kern, threads);
    S.mg->nrz = (int)g;
    return g;
  };
#define ADFEM_SWEEP(NB, D16, LPR)                                                                 \
  mg_launch(S, st, k_mg_sweep<NB, D16, LPR, MODE>, grid(k_mg_sweep<NB, D16, LPR, MODE>), kT, 0, 1, L, x, out, c1, c2, \
            keep, part)
  if (L.d16 && S.A->maxw <= 8) {
    mg_launch(S, st, k_mg_fine<MODE>, grid(k_mg_fine<MODE>), kT, 0, 1, L, x, out, c1, c2, part);
    return;
  }
  if (L.nb == 1) {
    if (L.d16) ADFEM_SWEEP(1, true, 1);
    else if (L.lpr == 1) ADFEM_SWEEP(1, false, 1);
    else if (L.lpr == 4) ADFEM_SWEEP(1, false, 4);
    else ADFEM_SWEEP(1, false, 8);
  } else if (L.nb == 2) {
    if (L.lpr == 1) ADFEM_SWEEP(2, false, 1);
    else ADFEM_SWEEP(2, false, 4);
  } else {
    if (L.lpr == 1) ADFEM_SWEEP(3, false, 1);
    else if (L.lpr == 4) ADFEM_SWEEP(3, false, 4);
    else ADFEM_SWEEP(3, false, 8);
  }
#undef ADFEM_SWEEP
}

void restrict_to(const Solver& S, const MgLev& L, const float* r, float* out, cudaStream_t st) {
  const int lpr = L.nc >= 150000 ? 1 : 8;
  const unsigned g = blocks((int64_t)L.nc * lpr, kT);
#define ADFEM_RES(NB, NC)                                                \
  do {                                                                   \
    if (lpr == 1) mg_launch(S, st, k_mg_restrict<NB, NC, 1>, g, kT, 0, 1, L, r, out); \
    else mg_launch(S, st, k_mg_restrict<NB, NC, 8>, g, kT, 0, 1, L, r, out);          \
  } while (0)
  if (L.nb == 1) ADFEM_RES(1, 1);
  else if (L.nb == 2) ADFEM_RES(2, 3);
  else ADFEM_RES(3, 3);
#undef ADFEM_RES
}
void prolong_from(const Solver& S, const MgLev& L, const float* xc, float* x, cudaStream_t st) {
  const unsigned g = blocks(L.n, kT);
  if (L.nb == 1) mg_launch(S, st, k_mg_prolong<1, 1>, g, kT, 0, 1, L, xc, x);
  else if (L.nb == 2) mg_launch(S, st, k_mg_prolong<2, 3>, g, kT, 0, 1, L, xc, x);
  else mg_launch(S, st, k_mg_prolong<3, 3>, g, kT, 0, 1, L, xc, x);
}

template <int NT, int NC, bool SOLVE>
void launch_tail(const Solver& S, const TailArgs& a, cudaStream_t st) {
  const Mg& M = *S.mg;
  if (M.cluster) mg_launch(S, st, k_mg_tail<NT, NC, true, SOLVE>, kTailC, kTailT, M.tail_smem, kTailC, a);
  else mg_launch(S, st, k_mg_tail<NT, NC, false, SOLVE>, 1, kTailT, M.tail_smem, 1, a);
}

TailArgs tail_args(Solver& S) {
  const Mg& M = *S.mg;
  const Sell& A = *S.A;
  TailArgs a;
  a.nl = M.nlev - M.tail;
  for (int l = 0; l < a.nl; l++) a.L[l] = M.lev[M.tail + l];
  a.dense = M.dense;
  a.N = M.ndense;
  a.pat = M.pat;
  a.vals = M.vals;
  a.pat_bytes = M.pat_bytes;
  a.val_bytes = M.val_bytes;
  a.b = M.lev[M.tail].b;
  a.x = M.lev[M.tail].x;
  a.reps = M.tail >= 3 ? 2 : 1;
  a.st = S.state.as<CgState>();
  a.spin = S.mg_spin;
  a.sptr = A.sptr.as<int32_t>();
  a.col = A.col.p;
  a.val = A.val64.as<double>();
  a.rowsum = M.rowsum;
  a.rhs = S.b.as<double>();
  a.s = S.s32.as<float>();
  a.y = S.y64.as<double>();
  return a;
}

// One cycle: lev[0].b -> the vector returned; returns the launches through *count.
const float* enqueue_cycle(Solver& S, cudaStream_t st, int* count) {
  Mg& M = *S.mg;
  int nl = 0;
  float* xs[kMgMaxLevels];
  for (int l = 0; l < M.tail; l++) {
    const MgLev& L = M.lev[l];
    const int deg = l == 0 ? kMgDeg0 : kMgDeg;
    float *x = L.x, *y = L.x2;
    sweep<kPre>(S, L, nullptr, x, 2, 3, deg > 2, nullptr, st);
    nl++;
    for (int k = 2; k < deg; k++) {
      sweep<kStep>(S, L, x, y, 2 * k, 2 * k + 1, k + 1 < deg, nullptr, st);
      std::swap(x, y);
      nl++;
    }
    // (d is free between the smoothers: the residual goes there)
    sweep<kRes>(S, L, x, L.d, -1, -1, 0, nullptr, st);
    restrict_to(S, L, L.d, M.lev[l + 1].b, st);
    nl += 2;
    xs[l] = x;
  }
  {
    const TailArgs a = tail_args(S);
    const int nt = a.L[0].nb;
    if (nt == 1) launch_tail<1, 1, false>(S, a, st);
    else if (nt == 2) launch_tail<2, 3, false>(S, a, st);
    else launch_tail<3, 3, false>(S, a, st);
    xs[M.tail] = M.lev[M.tail].x;
    nl++;
  }
  for (int l = M.tail - 1; l >= 0; l--) {
    const MgLev& L = M.lev[l];
    const int deg = l == 0 ? kMgDeg0 : kMgDeg;
    float *x = xs[l], *y = x == L.x ? L.x2 : L.x;
    prolong_from(S, L, xs[l + 1], x, st);
    nl++;
    for (int k = 0; k < deg; k++) {
      const int c1 = k ? 2 * k : -1, c2 = k ? 2 * k + 1 : 0;
      if (k + 1 < deg) sweep<kStep>(S, L, x, y, c1, c2, 1, nullptr, st);
      else sweep<kLast>(S, L, x, y, c1, c2, 0, l == 0 ? M.part : nullptr, st);
      std::swap(x, y);
      nl++;
    }
    xs[l] = x;
  }
  *count = nl;
  return xs[0];
}

void enqueue_residual(Solver& S, int mode, cudaGraphConditionalHandle loop, cudaStream_t st) {
  Mg& M = *S.mg;
  const Sell& A = *S.A;
  auto go = [&](auto d16, auto nb) {
    auto k = k_mg_residual<decltype(d16)::value, decltype(nb)::value>;
    mg_launch(S, st, k, (unsigned)S.grid, kT, 0, 1, S.n, A.sptr.as<int32_t>(), A.col.p, A.val64.as<double>(), M.rowsum,
              S.s32.as<float>(), S.b.as<double>(), S.y64.as<double>(), S.z64.as<double>(), S.r64.as<double>(),
              M.lev[0].b, S.state.as<CgState>(), M.part + 2 * kMgGrid, M.nrn, S.partials.as<double>(), mode, loop);
  };
  using std::integral_constant;
  if (M.lev[0].nb == 2) {
    if (A.delta16) go(std::true_type{}, integral_constant<int, 2>{});
    else go(std::false_type{}, integral_constant<int, 2>{});
  } else {
    if (A.delta16) go(std::true_type{}, integral_constant<int, 1>{});
    else go(std::false_type{}, integral_constant<int, 1>{});
  }
}

// The body of the loop: cycle, direction, K p, update, and the residual when it is due.
void enqueue_body(Solver& S, cudaGraphConditionalHandle loop, cudaStream_t st) {
  Mg& M = *S.mg;
  CgState* cs = S.state.as<CgState>();
  int nl = 0;
  const float* z = enqueue_cycle(S, st, &nl);
  const Sell& A = *S.A;
  const int64_t n2 = (S.n + 1) / 2;
  double *rz = M.part, *pq = rz + kMgGrid, *rn = pq + kMgGrid;
  mg_launch(S, st, k_mg_dir, sum_grid(S, k_mg_dir, n2), kT, 0, 1, S.n, z, S.s32.as<float>(), S.p64.as<double>(),
            S.y64.as<double>(), S.z64.as<double>(), cs, rz, M.nrz);
  int npq = 0;
  auto spmv = [&](auto d16, auto more) {
    auto k = k_mg_spmv<decltype(d16)::value, decltype(more)::value>;
    npq = (int)sum_grid(S, k, S.n);
    mg_launch(S, st, k, (unsigned)npq, kT, 0, 1, S.n, A.sptr.as<int32_t>(), A.col.p, A.spat.as<int32_t>(),
              A.pat.as<int16_t>(), A.pat_period, A.val64.as<double>(), S.p64.as<double>(), S.q64.as<double>(), cs, pq);
  };
  if (A.maxw <= 8) {
    if (A.delta16) spmv(std::true_type{}, std::false_type{});
    else spmv(std::false_type{}, std::false_type{});
  } else {
    if (A.delta16) spmv(std::true_type{}, std::true_type{});
    else spmv(std::false_type{}, std::true_type{});
  }
  const unsigned gu = sum_grid(S, k_mg_update, n2);
  mg_launch(S, st, k_mg_update, gu, kT, 0, 1, S.n, S.z64.as<double>(), S.r64.as<double>(), S.p64.as<double>(),
            S.q64.as<double>(), S.s32.as<float>(), M.lev[0].b, cs, pq, npq, rn);
  M.nrn = (int)gu;
  enqueue_residual(S, 1, loop, st);
  M.body_launches = nl + 4;
}

int capture_solve(Solver& S) {
  Mg& M = *S.mg;
  if (M.solve) return ADFEM_OK;
  cudaError_t e = cudaSuccess;
  // (a capture can be invalidated by another thread's device-wide synchronisation: retried)
  for (int attempt = 0; attempt < 8; attempt++) {
    cudaGraph_t g = nullptr, body = nullptr;
    cudaGraphConditionalHandle loop;
    ADFEM_CUDA(cudaGraphCreate(&g, 0));
    struct Guard {
      cudaGraph_t g;
      ~Guard() { cudaGraphDestroy(g); }
    } guard{g};
    ADFEM_CUDA(cudaGraphConditionalHandleCreate(&loop, g, 1, cudaGraphCondAssignDefault));
    cudaGraphNodeParams p = {};
    p.type = cudaGraphNodeTypeConditional;
    p.conditional.handle = loop;
    p.conditional.type = cudaGraphCondTypeWhile;
    p.conditional.size = 1;
    cudaGraphNode_t node;
    ADFEM_CUDA(cudaGraphAddNode(&node, g, nullptr, nullptr, 0, &p));
    body = p.conditional.phGraph_out[0];
    {
      std::lock_guard<std::mutex> lk(device_alloc_mutex());
      ADFEM_CUDA(cudaStreamBeginCaptureToGraph(S.stream, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
      enqueue_body(S, loop, S.stream);
      e = cudaStreamEndCapture(S.stream, &body);
    }
    if (e == cudaErrorStreamCaptureInvalidated || e == cudaErrorStreamCaptureUnjoined) {
      cudaGetLastError();
      std::this_thread::yield();
      continue;
    }
    if (e != cudaSuccess) return cuda_fail(e, "cudaStreamEndCapture (multigrid)");
    e = cudaGraphInstantiate(&M.solve, g, 0);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGraphInstantiate (multigrid)");
    return ADFEM_OK;
  }
  return cuda_fail(e, "cudaStreamEndCapture (multigrid, retried)");
}

}  // namespace

int mg_solve(Solver& S, const double* rhs, double* u, const uint8_t* zero_rows, const uint8_t* fix_rows,
             const double* fix_vals, const adfem_solver_opts& o, adfem_solver_stats* stats, cudaStream_t user,
             bool* gave_up) {
  *gave_up = false;
  Mg& M = *S.mg;
  const bool one = M.tail == 0;  // the whole solve in one launch
  if (!one) ADFEM_TRY(capture_solve(S));
  // a warm start may have converged: its residual is looked at before the hierarchy's values are made
  // (ms of an assembly and a solve that is there already, 90k and 1M unknowns: 0.44 -> 0.19, 1.16 -> 0.45)
  const bool look = !one && o.warm_start && !M.current;
  if (!M.current) {
    ADFEM_TRY(mg_values0(S, user));
    if (!look) ADFEM_TRY(mg_values_below(S, user));
  }
  cudaStream_t st = S.stream;
  ADFEM_CUDA(cudaEventRecord(S.ev[0], user));
  ADFEM_CUDA(cudaStreamWaitEvent(st, S.ev[0], 0));
  ADFEM_CUDA(cudaEventRecord(S.ev[1], st));
  CgState init;
  std::memset(&init, 0, sizeof(init));
  init.max_iter = std::min(o.max_iter, S.mg_cap);
  init.delta2 = 1e-6;  // residual evaluated in FP64 after each drop of the recurrence by 1e-3
  S.h_state[1] = init;
  ADFEM_CUDA(cudaMemcpyAsync(S.state.p, &S.h_state[1], sizeof(CgState), cudaMemcpyHostToDevice, st));
  k_mg_init<<<S.grid, kT, 0, st>>>(S.n, rhs, zero_rows, fix_rows, fix_vals, S.s32.as<float>(),
                                   o.warm_start ? u : nullptr, S.b.as<double>(), S.y64.as<double>(),
                                   S.z64.as<double>(), S.state.as<CgState>(), S.partials.as<double>(),
                                   o.rtol * o.rtol);
  bool there = false;  // no iteration needed (and the values below level 0 not made)
  if (one) {
    const TailArgs a = tail_args(S);
    if (M.lev[0].nb == 1) launch_tail<1, 1, true>(S, a, st);
    else launch_tail<2, 3, true>(S, a, st);
  } else {
    const cudaGraphConditionalHandle none{};
    enqueue_residual(S, 0, none, st);
    ADFEM_CUDA(cudaGetLastError());
    if (look) {
      ADFEM_CUDA(cudaMemcpyAsync(&S.h_state[0], S.state.p, sizeof(CgState), cudaMemcpyDeviceToHost, st));
      ADFEM_CUDA(cudaStreamSynchronize(st));
      there = S.h_state[0].done != 0;
      if (!there) {
        ADFEM_TRY(mg_values_below(S, user));
        ADFEM_CUDA(cudaEventRecord(S.ev[0], user));
        ADFEM_CUDA(cudaStreamWaitEvent(st, S.ev[0], 0));
      }
    }
    if (!there) ADFEM_CUDA(cudaGraphLaunch(M.solve, st));
    solver_enqueue_fold64(S, 1, st);
    enqueue_residual(S, 2, none, st);
  }
  // (the caller's vector is written after the outcome is known to be usable: a solve that gives
  // up leaves it as the other iteration's start)
  ADFEM_CUDA(cudaMemcpyAsync(&S.h_state[0], S.state.p, sizeof(CgState), cudaMemcpyDeviceToHost, st));
  ADFEM_CUDA(cudaEventRecord(S.ev[2], st));
  ADFEM_CUDA(cudaGetLastError());
  ADFEM_CUDA(cudaEventSynchronize(S.ev[2]));
  if (!there) M.current = true;
  const CgState fin = S.h_state[0];
  if (fin.done != 1 && !(fin.done == 4 && fin.iters >= o.max_iter)) {
    *gave_up = true;
    ADFEM_CUDA(cudaStreamWaitEvent(user, S.ev[2], 0));
    return ADFEM_OK;
  }
  k_mg_out<<<blocks(S.n, kT), kT, 0, st>>>(S.n, S.y64.as<double>(), fix_rows, fix_vals, u);
  ADFEM_CUDA(cudaGetLastError());
  ADFEM_CUDA(cudaEventRecord(S.ev[3], st));
  ADFEM_CUDA(cudaEventSynchronize(S.ev[3]));  // (u is written when the call returns, on any stream)
  ADFEM_CUDA(cudaStreamWaitEvent(user, S.ev[3], 0));
  const int status = fin.done == 1 ? ADFEM_OK : ADFEM_ERR_NOT_CONVERGED;
  const double relres = fin.bnorm2 > 0.0 ? std::sqrt(fin.rr64 / fin.bnorm2) : 0.0;
  if (stats) {
    float ms = 0.0f;
    cudaEventElapsedTime(&ms, S.ev[1], S.ev[3]);
    stats->iterations = fin.iters;
    stats->updates = fin.updates;
    stats->relres = relres;
    stats->ms = ms;
    stats->status = status;
    stats->launches = one ? 3 : (long long)std::max(fin.iters, 1) * M.body_launches + 5;
  }
  if (status == ADFEM_ERR_NOT_CONVERGED)
    return fail(status, "CG did not reach rtol within max_iter (relres " + std::to_string(relres) + ")");
  return ADFEM_OK;
}

size_t mg_device_bytes(const Solver& S) { return S.mg ? S.mg->slab.bytes : 0; }

ADFEM_CHECK_READER(check_line_mg)

}  // namespace adfem
