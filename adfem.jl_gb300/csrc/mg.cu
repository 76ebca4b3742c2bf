// Multigrid-preconditioned CG of the resident systems (sm_103a).
//
// Jacobi-CG needs 5,000 to 16,000 iterations at 1M to 4M unknowns, each near the memory
// bound already, so the time of a solve is their number.  Here the preconditioner is one
// V-cycle of smoothed aggregation in FP32 and the CG around it is FP64 throughout (iterate,
// residual, direction, products), which needs 20 to 90 iterations at every size.
//  * Patterns (aggregates, interpolation, A P, coarse operators) are made once per system on
//    the host (mg_setup.cpp); after an assembly the kernels below fill in the values.
//  * Level 0 is S K S, S = diag(K_ii^-1/2) as in the Jacobi iterations, so the stopping
//    quantity is unchanged; the coarse operators are scaled to unit diagonal as well.
//  * Interpolation: P = P0 - (1.6 / q_i) A P0, q_i the weighted absolute row sum (2 for a row
//    of an M-matrix with zero sum); P0 is piecewise constant on the aggregates, plus the
//    rotation about the aggregate's centre for 2-D elasticity.
//  * Smoother: Chebyshev of degree 2 on level 0 and 4 below (the coarse levels are cheap and
//    the V-cycle gains most there), on [fr lam, lam] with lam = max q_i, an upper bound of the
//    spectrum, so the cycle is symmetric positive definite for every input.
//  * Every sum is formed by one thread or a fixed shuffle tree: results repeat bit for bit.
//  * A solve is one CUDA graph: a while node around one iteration, left when a residual
//    evaluated in FP64 from the iterate meets the tolerance (or the iteration ends otherwise);
//    the host waits once.
#include <cmath>
#include <cstring>
#include <mutex>
#include <thread>
#include <type_traits>

#include "cg_common.cuh"
#include "checks.cuh"

namespace adfem {

Mg::~Mg() {
  if (solve) cudaGraphExecDestroy(solve);
}

namespace {

constexpr float kSmoothP = 1.6f;
constexpr float kFrac0 = 0.125f, kFrac = 0.06f;  // lower end of the Chebyshev interval over lam
constexpr int kCoef = 2 * kMgDeg;
constexpr int kTailT = 1024;
constexpr int kMgIterations = 300;  // a solve that needs more is left to the Jacobi iteration

template <int NB>
struct Vec {
  float v[NB];
};
template <int NB>
__device__ __forceinline__ Vec<NB> load_vec(const float* __restrict__ p, int64_t i) {
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
// acc += M x, M an R x C block
template <int R, int C>
__device__ __forceinline__ void block_fma(const float* __restrict__ m, const Vec<C>& x, Vec<R>& acc) {
  if constexpr (R == 2 && C == 2) {
    const float4 t = *reinterpret_cast<const float4*>(m);
    acc.v[0] = fmaf(t.x, x.v[0], fmaf(t.y, x.v[1], acc.v[0]));
    acc.v[1] = fmaf(t.z, x.v[0], fmaf(t.w, x.v[1], acc.v[1]));
  } else {
#pragma unroll
    for (int r = 0; r < R; r++)
#pragma unroll
      for (int c = 0; c < C; c++) acc.v[r] = fmaf(m[r * C + c], x.v[c], acc.v[r]);
  }
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
  __device__ __forceinline__ int at(int k, int64_t idx) const {
    if (D16) return r + (int)(so >= 0 ? __ldg(L.pat + so + k) : __ldg(reinterpret_cast<const int16_t*>(L.col) + idx));
    return __ldg(reinterpret_cast<const int32_t*>(L.col) + idx);
  }
};

// (A x)_r over the LPR lanes of row r (every lane gets the sum)
template <int NB, bool D16, int LPR>
__device__ __forceinline__ Vec<NB> row_product(const MgLev& L, int r, int lane, const float* __restrict__ x) {
  Vec<NB> acc;
#pragma unroll
  for (int c = 0; c < NB; c++) acc.v[c] = 0.0f;
  int64_t base;
  int w;
  slice_row(L.sptr, r, base, w);
  const Cols<D16> cols(L, r);
  // entries in groups whose loads are all in flight at once
  constexpr int U = LPR == 1 ? (NB == 1 ? 8 : 4) : 2;
  for (int k0 = lane; k0 < w; k0 += U * LPR) {
    int j[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int k = k0 + u * LPR;
      j[u] = k < w ? cols.at(k, base + 32 * (int64_t)k) : r;
      if (!ADFEM_DCHECK(j[u] >= 0 && j[u] < L.n)) j[u] = r;
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int k = k0 + u * LPR;
      if (k < w) block_fma<NB, NB>(L.val + (base + 32 * (int64_t)k) * (NB * NB), load_vec<NB>(x, j[u]), acc);
    }
  }
  if (LPR > 1) lane_sum<NB, LPR>(acc);
  return acc;
}

// ---------------------------------------------------------------------------
// V-cycle kernels of the levels above the tail.
enum { kPre = 0, kStep = 1, kRes = 2, kLast = 3 };

// kPre:  two Chebyshev steps from x = 0: x1 = b / theta gathered from b, then step 2
// kStep: one step: d <- c1 d + c2 (b - A x), out = x + d (c1 index < 0: first step, d unread)
// kRes:  out = b - A x
// kLast: kStep whose d is not needed again; on level 0 the products b.out give r.z
template <int NB, bool D16, int LPR, int MODE>
__global__ void __launch_bounds__(kT) k_mg_sweep(MgLev L, const float* __restrict__ x, float* __restrict__ out,
                                                 int c1, int c2, int keep_d, CgState* st, double* partials) {
  float dot = 0.0f;
  const float th = MODE == kPre ? __ldg(L.coef) : 0.0f;
  const float a1 = c1 >= 0 ? __ldg(L.coef + c1) : 0.0f, a2 = c2 >= 0 ? __ldg(L.coef + c2) : 0.0f;
  const int64_t rows = (int64_t)L.n * LPR;
  const int64_t lim = LPR == 1 ? rows : (rows + 31) / 32 * 32;  // (whole warps stay together in lane_sum)
  for (int64_t t = gtid(); t < lim; t += gstride()) {
    const int r0 = (int)(t / LPR), lane = (int)(t % LPR);
    const int r = r0 < L.n ? r0 : L.n - 1;
    const Vec<NB> bi = load_vec<NB>(L.b, r);
    const Vec<NB> xi = MODE == kPre ? bi : load_vec<NB>(x, r);
    Vec<NB> di;
    if ((MODE == kStep || MODE == kLast) && c1 >= 0) di = load_vec<NB>(L.d, r);
    const Vec<NB> ax = row_product<NB, D16, LPR>(L, r, lane, MODE == kPre ? L.b : x);
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
    if (lane != 0 || r0 >= L.n) continue;
    store_vec<NB>(out, r, o);
    if ((MODE == kPre || MODE == kStep) && keep_d) store_vec<NB>(L.d, r, d);
    if (MODE == kLast)
#pragma unroll
      for (int c = 0; c < NB; c++) dot = fmaf(bi.v[c], o.v[c], dot);
  }
  if (MODE == kLast && st) {
    float v[1] = {dot};
    double tot[1];
    if (reduce_grid_w<1, kT, true>(v, partials, &st->counter[0], tot) && threadIdx.x == 0 && !st->done) {
      const double rz = tot[0] / st->ar;  // (b carries the factor st->ar, and so does z)
      if (!(rz > 0.0) || !isfinite(rz)) {
        st->done = 2;
      } else {
        st->beta = st->iters == 0 ? 0.0 : rz / st->rho;
        st->rho = rz;
      }
    }
  }
}

// out_J = sum_i P_iJ^T r_i
template <int NB, int NC, int LPR>
__global__ void __launch_bounds__(kT) k_mg_restrict(MgLev L, const float* __restrict__ r, float* __restrict__ out) {
  const int64_t t = gtid();
  const int J0 = (int)(t / LPR), lane = (int)(t % LPR);
  const int J = J0 < L.nc ? J0 : L.nc - 1;
  Vec<NC> acc;
#pragma unroll
  for (int c = 0; c < NC; c++) acc.v[c] = 0.0f;
  int64_t base;
  int w;
  slice_row(L.pt_sptr, J, base, w);
  constexpr int U = 4;
  for (int k0 = lane; k0 < w; k0 += U * LPR) {
    int i[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int k = k0 + u * LPR;
      i[u] = k < w ? __ldg(L.pt_col + base + 32 * (int64_t)k) : 0;
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int k = k0 + u * LPR;
      if (k < w) block_fma<NC, NB>(L.pt_val + (base + 32 * (int64_t)k) * (NB * NC), load_vec<NB>(r, i[u]), acc);
    }
  }
  if (LPR > 1) lane_sum<NC, LPR>(acc);
  if (lane == 0 && J0 < L.nc) store_vec<NC>(out, J, acc);
}

// x_i += sum_J P_iJ xc_J
template <int NB, int NC>
__global__ void __launch_bounds__(kT) k_mg_prolong(MgLev L, const float* __restrict__ xc, float* __restrict__ x) {
  const int64_t t = gtid();
  if (t >= L.n) return;
  const int i = (int)t;
  Vec<NB> acc = load_vec<NB>(x, i);
  int64_t base;
  int w;
  slice_row(L.p_sptr, i, base, w);
  constexpr int U = 4;
  for (int k0 = 0; k0 < w; k0 += U) {
    int J[U];
#pragma unroll
    for (int u = 0; u < U; u++) J[u] = k0 + u < w ? __ldg(L.p_col + base + 32 * (int64_t)(k0 + u)) : 0;
#pragma unroll
    for (int u = 0; u < U; u++)
      if (k0 + u < w)
        block_fma<NB, NC>(L.p_val + (base + 32 * (int64_t)(k0 + u)) * (NB * NC), load_vec<NC>(xc, J[u]), acc);
  }
  store_vec<NB>(x, i, acc);
}

// ---------------------------------------------------------------------------
// The levels from Mg::tail on in one block: all vectors in shared memory, the operators read
// through L1/L2; `reps` cycles (two cycles below a larger level: its coarse problem is then
// solved nearly exactly).  The coarsest operator is applied as its dense inverse.
struct TailArgs {
  MgLev L[kMgMaxTail];
  int nl;
  const float* dense;
  int N;         // unknowns of the coarsest level
  const float* b;
  float* x;
  int reps;
  CgState* st;   // level 0 in the tail: r.z from here
};
struct TailVecs {
  float *b, *x, *y, *d;
};

template <int NB, class Body>
__device__ __forceinline__ void tail_rows(const MgLev& L, const float* x, Body body) {
  const int lpr = L.lpr, lane = threadIdx.x & (lpr - 1);
  const int rows = (L.n + (kTailT / lpr) - 1) / (kTailT / lpr) * (kTailT / lpr);
  for (int r0 = threadIdx.x / lpr; r0 < rows; r0 += kTailT / lpr) {
    const int r = r0 < L.n ? r0 : L.n - 1;
    Vec<NB> acc;
#pragma unroll
    for (int c = 0; c < NB; c++) acc.v[c] = 0.0f;
    int64_t base;
    int w;
    slice_row(L.sptr, r, base, w);
    const int32_t* col = reinterpret_cast<const int32_t*>(L.col);
    constexpr int U = 4;
    for (int k0 = lane; k0 < w; k0 += U * lpr) {
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int k = k0 + u * lpr;
        if (k < w) {
          int j = __ldg(col + base + 32 * (int64_t)k);
          if (!ADFEM_DCHECK(j >= 0 && j < L.n)) j = r;
          block_fma<NB, NB>(L.val + (base + 32 * (int64_t)k) * (NB * NB), load_vec<NB>(x, j), acc);
        }
      }
    }
    for (int o = lpr >> 1; o > 0; o >>= 1)
#pragma unroll
      for (int c = 0; c < NB; c++) acc.v[c] += __shfl_xor_sync(0xffffffffu, acc.v[c], o);
    if (lane == 0 && r0 < L.n) body(r, acc);
  }
  __syncthreads();
}

// Chebyshev of the level's degree on (b, x) -> x; zero: x = 0 on entry.  v.y: the other iterate.
template <int NB>
__device__ void tail_smooth(const MgLev& L, TailVecs& v, int deg, bool zero) {
  const float th = L.coef[0];
  if (zero) {
    for (int t = threadIdx.x; t < L.n * NB; t += kTailT) {
      const float x1 = th * v.b[t];
      v.d[t] = x1;
      v.x[t] = x1;
    }
    __syncthreads();
  }
  for (int k = zero ? 1 : 0; k < deg; k++) {
    const float a1 = k > 0 ? L.coef[2 * k] : 0.0f, a2 = k > 0 ? L.coef[2 * k + 1] : th;
    tail_rows<NB>(L, v.x, [&](int r, const Vec<NB>& ax) {
#pragma unroll
      for (int c = 0; c < NB; c++) {
        const int t = NB * r + c;
        const float res = v.b[t] - ax.v[c];
        const float d = k > 0 ? fmaf(a1, v.d[t], a2 * res) : a2 * res;
        v.d[t] = d;
        v.y[t] = v.x[t] + d;
      }
    });
    float* s = v.x;
    v.x = v.y;
    v.y = s;
  }
}

template <int NB, int NC>
__device__ void tail_down(const MgLev& L, TailVecs& f, TailVecs& c, int deg, bool zero) {
  tail_smooth<NB>(L, f, deg, zero);
  tail_rows<NB>(L, f.x, [&](int r, const Vec<NB>& ax) {
#pragma unroll
    for (int q = 0; q < NB; q++) f.d[NB * r + q] = f.b[NB * r + q] - ax.v[q];
  });
  const int J8 = threadIdx.x >> 3, lane = threadIdx.x & 7;
  for (int J0 = J8; J0 < (L.nc + 127) / 128 * 128; J0 += kTailT / 8) {
    const int J = J0 < L.nc ? J0 : L.nc - 1;
    Vec<NC> acc;
#pragma unroll
    for (int q = 0; q < NC; q++) acc.v[q] = 0.0f;
    int64_t base;
    int w;
    slice_row(L.pt_sptr, J, base, w);
    for (int k = lane; k < w; k += 8)
      block_fma<NC, NB>(L.pt_val + (base + 32 * (int64_t)k) * (NB * NC),
                        load_vec<NB>(f.d, __ldg(L.pt_col + base + 32 * (int64_t)k)), acc);
    lane_sum<NC, 8>(acc);
    if (lane == 0 && J0 < L.nc) store_vec<NC>(c.b, J, acc);
  }
  __syncthreads();
}
template <int NB, int NC>
__device__ void tail_up(const MgLev& L, TailVecs& f, const TailVecs& c, int deg) {
  for (int i = threadIdx.x; i < L.n; i += kTailT) {
    Vec<NB> acc = load_vec<NB>(f.x, i);
    int64_t base;
    int w;
    slice_row(L.p_sptr, i, base, w);
    for (int k = 0; k < w; k++)
      block_fma<NB, NC>(L.p_val + (base + 32 * (int64_t)k) * (NB * NC),
                        load_vec<NC>(c.x, __ldg(L.p_col + base + 32 * (int64_t)k)), acc);
    store_vec<NB>(f.x, i, acc);
  }
  __syncthreads();
  tail_smooth<NB>(L, f, deg, false);
}

// NT: unknowns per node of the tail's first level, NC: of the others
template <int NT, int NC>
__global__ void __launch_bounds__(kTailT) k_mg_tail(TailArgs a) {
  extern __shared__ float4 tail_sm4[];
  float* sm = reinterpret_cast<float*>(tail_sm4);
  TailVecs v[kMgMaxTail];
  {
    float* p = sm;
    for (int l = 0; l < a.nl; l++) {
      const int m = (a.L[l].n * (l == 0 ? NT : NC) + 3) & ~3;
      v[l].b = p;
      v[l].x = p + m;
      v[l].y = p + 2 * m;
      v[l].d = p + 3 * m;
      p += 4 * m;
    }
  }
  const int n0 = a.L[0].n * NT;
  for (int t = threadIdx.x; t < n0; t += kTailT) v[0].b[t] = a.b[t];
  __syncthreads();
  const int last = a.nl - 1;
  for (int rep = 0; rep < a.reps; rep++) {
    for (int l = 0; l < last; l++) {
      const int deg = a.st && l == 0 ? kMgDeg0 : kMgDeg;
      if (l == 0) tail_down<NT, NC>(a.L[0], v[0], v[1], deg, rep == 0);
      else tail_down<NC, NC>(a.L[l], v[l], v[l + 1], deg, true);
    }
    {
      // coarsest: one warp per row of the dense inverse
      const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
      const float* bb = v[last].b;
      for (int r = wid; r < a.N; r += kTailT / 32) {
        float s = 0.0f;
        for (int k = lane; k < a.N; k += 32) s = fmaf(__ldg(a.dense + (int64_t)r * a.N + k), bb[k], s);
        s = warp_sum(s);
        if (lane == 0) v[last].x[r] = s;
      }
      __syncthreads();
    }
    for (int l = last - 1; l >= 0; l--) {
      const int deg = a.st && l == 0 ? kMgDeg0 : kMgDeg;
      if (l == 0) tail_up<NT, NC>(a.L[0], v[0], v[1], deg);
      else tail_up<NC, NC>(a.L[l], v[l], v[l + 1], deg);
    }
  }
  float dot = 0.0f;
  for (int t = threadIdx.x; t < n0; t += kTailT) {
    a.x[t] = v[0].x[t];
    dot = fmaf(v[0].x[t], v[0].b[t], dot);
  }
  if (a.st) {
    float w[1] = {dot};
    block_sum<float, 1, kTailT>(w);
    if (threadIdx.x == 0 && !a.st->done) {
      const double rz = (double)w[0] / a.st->ar;
      if (!(rz > 0.0) || !isfinite(rz)) {
        a.st->done = 2;
      } else {
        a.st->beta = a.st->iters == 0 ? 0.0 : rz / a.st->rho;
        a.st->rho = rz;
      }
    }
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
      L.val[(nbase + 32 * (int64_t)(k / NB)) * (NB * NB) + c * NB + k % NB] = f;
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

// P = P0 - (1.6 / q) A P0 and the level's eigenvalue bound max q.  q: absolute row sums,
// weighted by P0 for scalar operators (then exactly 2 where the row sums to zero with
// non-positive off-diagonals, whatever the coefficients' jumps).
template <int NB, int NC, bool D16, int BT>
__global__ void __launch_bounds__(BT) k_mg_p(MgLev L) {
  __shared__ float acc[kMgMaxP * NB * NC][BT];
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
    for (int e = 0; e < pw * NB * NC; e++) acc[e][t] = 0.0f;
    float ti[NB], Ti[NB * NC], q[NB];
    tentative<NB, NC>(L, i, Ti, ti);
#pragma unroll
    for (int c = 0; c < NB; c++) q[c] = 0.0f;
    const Cols<D16> cols(L, i);
    for (int k = 0; k < w; k++) {
      const int64_t idx = base + 32 * (int64_t)k;
      int j = cols.at(k, idx);
      if (!ADFEM_DCHECK(j >= 0 && j < L.n)) j = i;
      const float* a = L.val + idx * (NB * NB);
      float T[NB * NC], tj[NB];
      tentative<NB, NC>(L, j, T, tj);
      const int J = __ldg(L.agg + j);
      int s = 0;
      while (s < pw && __ldg(L.p_col + pb + 32 * (int64_t)s) != J) s++;
#pragma unroll
      for (int c = 0; c < NB; c++) {
#pragma unroll
        for (int e = 0; e < NB; e++) q[c] += NB == 1 ? fabsf(a[0]) * tj[0] : fabsf(a[c * NB + e]);
        if (s < pw)
#pragma unroll
          for (int m = 0; m < NC; m++) {
            float v = 0.0f;
#pragma unroll
            for (int e = 0; e < NB; e++) v = fmaf(a[c * NB + e], T[e * NC + m], v);
            acc[s * NB * NC + c * NC + m][t] -= v;
          }
      }
    }
#pragma unroll
    for (int c = 0; c < NB; c++) {
      if (NB == 1) q[0] = ti[0] > 0.0f ? q[0] / ti[0] : 1.0f;
      q[c] = fmaxf(q[c], 1.0f);
      qmax = fmaxf(qmax, q[c]);
    }
    // (padding repeats column 0 behind the row's entries: the first match is the own aggregate)
    const int Ji = __ldg(L.agg + i);
    int own = 0;
    while (own < pw && __ldg(L.p_col + pb + 32 * (int64_t)own) != Ji) own++;
    for (int s = 0; s < pw; s++)
#pragma unroll
      for (int c = 0; c < NB; c++) {
        const float f = ti[c] > 0.0f ? kSmoothP / q[c] : 0.0f;
#pragma unroll
        for (int m = 0; m < NC; m++)
          L.p_val[(pb + 32 * (int64_t)s) * (NB * NC) + c * NC + m] =
              f * acc[s * NB * NC + c * NC + m][t] + (s == own ? Ti[c * NC + m] : 0.0f);
      }
  }
  // (positive floats order as their bits; a maximum does not depend on the order of arrival)
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) qmax = fmaxf(qmax, __shfl_xor_sync(0xffffffffu, qmax, o));
  if ((t & 31) == 0) atomicMax(L.lam, __float_as_int(qmax));
}

// rows of A P
template <int NB, int NC, bool D16, int BT>
__global__ void __launch_bounds__(BT) k_mg_ap(MgLev L) {
  __shared__ float acc[kMgMaxAP * NB * NC][BT];
  const int t = threadIdx.x;
  const int64_t i64 = gtid();
  if (i64 >= L.n) return;
  const int i = (int)i64;
  int64_t ab, base;
  int aw, w;
  slice_row(L.ap_sptr, i, ab, aw);
  slice_row(L.sptr, i, base, w);
  if (aw > kMgMaxAP) aw = kMgMaxAP;
  for (int e = 0; e < aw * NB * NC; e++) acc[e][t] = 0.0f;
  const Cols<D16> cols(L, i);
  for (int k = 0; k < w; k++) {
    const int64_t idx = base + 32 * (int64_t)k;
    int j = cols.at(k, idx);
    if (!ADFEM_DCHECK(j >= 0 && j < L.n)) j = i;
    float a[NB * NB];
    bool any = false;
#pragma unroll
    for (int e = 0; e < NB * NB; e++) {
      a[e] = L.val[idx * (NB * NB) + e];
      any |= a[e] != 0.0f;
    }
    if (!any) continue;
    int64_t pb;
    int pw;
    slice_row(L.p_sptr, j, pb, pw);
    for (int p = 0; p < pw; p++) {
      const int64_t pe = pb + 32 * (int64_t)p;
      const int K = __ldg(L.p_col + pe);
      int s = 0;
      while (s < aw && __ldg(L.ap_col + ab + 32 * (int64_t)s) != K) s++;
      if (s == aw) continue;
      float v[NB * NC];
#pragma unroll
      for (int e = 0; e < NB * NC; e++) v[e] = L.p_val[pe * (NB * NC) + e];
#pragma unroll
      for (int c = 0; c < NB; c++)
#pragma unroll
        for (int m = 0; m < NC; m++) {
          float x = acc[s * NB * NC + c * NC + m][t];
#pragma unroll
          for (int e = 0; e < NB; e++) x = fmaf(a[c * NB + e], v[e * NC + m], x);
          acc[s * NB * NC + c * NC + m][t] = x;
        }
    }
  }
  for (int s = 0; s < aw; s++)
#pragma unroll
    for (int e = 0; e < NB * NC; e++)
      L.ap_val[(ab + 32 * (int64_t)s) * (NB * NC) + e] = acc[s * NB * NC + e][t];
}

// Coarse rows P^T (A P), one warp per row: lane k owns entries k and k + 32 of the row and
// picks its terms from the walk over the row's nodes (in ascending order).
template <int NB, int NC>
__global__ void __launch_bounds__(128) k_mg_ac(MgLev L, MgLev C) {
  const int lane = threadIdx.x & 31;
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
    // (padding repeats column 0 behind the row's entries: the first match owns the sum)
    if (k > 0 && K[h] == 0) K[h] = -1;
#pragma unroll
    for (int e = 0; e < NC * NC; e++) acc[h][e] = 0.0f;
  }
  for (int q = 0; q < tw; q++) {
    const int src = __ldg(L.pt_src + tb + 32 * (int64_t)q);
    if (src < 0) continue;
    const int i = __ldg(L.pt_col + tb + 32 * (int64_t)q);
    float p[NB * NC];
#pragma unroll
    for (int e = 0; e < NB * NC; e++) p[e] = L.p_val[(int64_t)src * (NB * NC) + e];
    int64_t ab;
    int aw;
    slice_row(L.ap_sptr, i, ab, aw);
    for (int s = 0; s < aw; s++) {
      const int64_t ae = ab + 32 * (int64_t)s;
      const int k = __ldg(L.ap_col + ae);
#pragma unroll
      for (int h = 0; h < 2; h++)
        if (k == K[h]) {
#pragma unroll
          for (int e = 0; e < NB; e++)
#pragma unroll
            for (int m = 0; m < NC; m++) {
              const float v = L.ap_val[ae * (NB * NC) + e * NC + m];
#pragma unroll
              for (int c = 0; c < NC; c++) acc[h][c * NC + m] = fmaf(p[e * NC + c], v, acc[h][c * NC + m]);
            }
        }
    }
  }
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const int k = lane + 32 * h;
    if (k >= cw) continue;
#pragma unroll
    for (int e = 0; e < NC * NC; e++)
      C.val[(cb + 32 * (int64_t)k) * (NC * NC) + e] = K[h] >= 0 ? acc[h][e] : 0.0f;
    if (K[h] == J)
#pragma unroll
      for (int c = 0; c < NC; c++) {
        const float d = acc[h][c * NC + c];
        C.s[(int64_t)NC * J + c] = d > 0.0f && isfinite(d) ? rsqrtf(d) : 0.0f;
      }
  }
}

// unit diagonal: A_JK <- s_J A_JK s_K (1 on the diagonal of unknowns without a scale), and
// the interpolation in those unknowns, P <- P S, with its transpose
template <int NB, int NC>
__global__ void __launch_bounds__(128) k_mg_scale(MgLev L, MgLev C) {
  const int64_t J64 = gtid();
  if (J64 >= L.nc) return;
  const int J = (int)J64;
  float sJ[NC];
#pragma unroll
  for (int c = 0; c < NC; c++) sJ[c] = C.s[(int64_t)NC * J + c];
  int64_t base;
  int w;
  slice_row(C.sptr, J, base, w);
  const int32_t* ccol = reinterpret_cast<const int32_t*>(C.col);
  bool diag = false;
  for (int k = 0; k < w; k++) {
    const int64_t e = base + 32 * (int64_t)k;
    const int K = __ldg(ccol + e);
    const bool own = K == J && !diag;
    diag |= own;
#pragma unroll
    for (int c = 0; c < NC; c++)
#pragma unroll
      for (int m = 0; m < NC; m++) {
        float* v = C.val + e * (NC * NC) + c * NC + m;
        const float sk = C.s[(int64_t)NC * K + m];
        *v = own && c == m ? 1.0f : *v * (sJ[c] * sk);
      }
  }
  slice_row(L.pt_sptr, J, base, w);
  for (int q = 0; q < w; q++) {
    const int64_t e = base + 32 * (int64_t)q;
    const int64_t src = __ldg(L.pt_src + e);
    if (src < 0) continue;
#pragma unroll
    for (int r = 0; r < NB; r++)
#pragma unroll
      for (int c = 0; c < NC; c++) {
        const float v = L.p_val[src * (NB * NC) + r * NC + c] * sJ[c];
        L.p_val[src * (NB * NC) + r * NC + c] = v;
        L.pt_val[e * (NB * NC) + c * NB + r] = v;
      }
  }
}

// Chebyshev coefficients of one level: 1 / theta, then (c1, c2) of step k at 2k, 2k + 1
__global__ void k_mg_coef(MgLev L, int deg, float frac) {
  if (threadIdx.x || blockIdx.x) return;
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

// Inverse of the coarsest operator (N <= kMgDense, unit diagonal) by Gauss-Jordan in shared
// memory; a pivot at rounding level (a near-null space the Dirichlet data leave in) drops its
// unknown from the inverse, which stays symmetric positive semi-definite.
template <int NC>
__global__ void __launch_bounds__(kTailT) k_mg_dense(MgLev C, float* __restrict__ inv) {
  extern __shared__ float4 dense_sm4[];
  float* A = reinterpret_cast<float*>(dense_sm4);
  const int N = C.n * NC;
  float* f = A + N * N;  // the pivot column
  for (int t = threadIdx.x; t < N * N; t += blockDim.x) A[t] = 0.0f;
  __syncthreads();
  const int32_t* col = reinterpret_cast<const int32_t*>(C.col);
  for (int t = threadIdx.x; t < C.n; t += blockDim.x) {
    int64_t base;
    int w;
    slice_row(C.sptr, t, base, w);
    for (int k = 0; k < w; k++) {
      const int64_t e = base + 32 * (int64_t)k;
      const int K = col[e];
      for (int c = 0; c < NC; c++)
        for (int m = 0; m < NC; m++) A[(t * NC + c) * N + K * NC + m] += C.val[e * (NC * NC) + c * NC + m];
    }
  }
  __syncthreads();
  for (int k = 0; k < N; k++) {
    const float p = A[k * N + k];
    const float ip = p > 1e-5f ? 1.0f / p : 0.0f;
    for (int t = threadIdx.x; t < N; t += blockDim.x) f[t] = A[t * N + k];
    __syncthreads();
    for (int t = threadIdx.x; t < N; t += blockDim.x) A[k * N + t] = t == k ? ip : A[k * N + t] * ip;
    __syncthreads();
    for (int t = threadIdx.x; t < N * N; t += blockDim.x) {
      const int r = t / N, c = t - r * N;
      if (r == k) continue;
      A[t] = c == k ? -f[r] * ip : fmaf(-f[r], A[k * N + c], A[t]);
    }
    __syncthreads();
  }
  // (symmetrised: the cycle has to be symmetric)
  for (int t = threadIdx.x; t < N * N; t += blockDim.x) {
    const int r = t / N, c = t - r * N;
    inv[t] = 0.5f * (A[t] + A[c * N + r]);
  }
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
  }
}

// The residual decides: converged, at its attainable floor, out of iterations, or go on (the
// rules of replacement_step64, whose direction scalars do not apply here).
__device__ __forceinline__ void mg_residual_step(CgState* st, double rr, bool first) {
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
    const bool dropped = st->rho_new <= st->delta2 * prev;
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
  if (st->final_req) st->final_seen = 1;
  st->final_req = 0;
  if (!first) st->updates += 1;
  st->ru2 = st->delta2 * rr;
  st->done = 0;
}

// r = b - K y in FP64, in difference form: row sums times the row's own unknowns plus entries
// times differences, so that it rounds with the differences of the solution.
// mode 0: start, 1: when due (st->done == 3), also the end of an iteration (sets the loop's
// condition), 2: final value only
template <bool D16, int NB>
__global__ void __launch_bounds__(kT) k_mg_residual(int64_t n, const int32_t* __restrict__ sptr,
                                                    const void* __restrict__ col, const double* __restrict__ val,
                                                    const double* __restrict__ rowsum, const float* __restrict__ sc,
                                                    const double* __restrict__ b, const double* __restrict__ y,
                                                    double* __restrict__ r64, float* __restrict__ b32, CgState* st,
                                                    double* partials, int mode, cudaGraphConditionalHandle loop) {
  if (mode == 1 && st->done != 3) {
    if (blockIdx.x == 0 && threadIdx.x == 0) cudaGraphSetConditional(loop, st->done == 0 ? 1 : 0);
    return;
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
      yo[q] = y[r / NB * NB + q];
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
        x[u] = __ldg(y + j);
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
    if (mode == 2) st->rr64 = tot[0];
    else mg_residual_step(st, tot[0], mode == 0);
    if (mode == 1) cudaGraphSetConditional(loop, st->done == 0 ? 1 : 0);
  }
}

// p = S z + beta p
__global__ void __launch_bounds__(kT) k_mg_dir(int64_t n, const float* __restrict__ z, const float* __restrict__ s,
                                               double* __restrict__ p, const CgState* st) {
  if (st->done) return;
  const double bt = st->beta;
  const bool first = bt == 0.0;
  for (int64_t i = gtid(); i < n; i += gstride()) {
    const double zi = (double)(s[i] * z[i]);
    p[i] = first ? zi : fma(bt, p[i], zi);
  }
}

// z += alpha p, r -= alpha q (z: the correction since the last residual evaluation), and the
// cycle's next right-hand side with its norm
__global__ void __launch_bounds__(kT) k_mg_update(int64_t n, double* __restrict__ z, double* __restrict__ r,
                                                  const double* __restrict__ p, const double* __restrict__ q,
                                                  const float* __restrict__ s, float* __restrict__ b32, CgState* st,
                                                  double* partials) {
  if (st->done) return;
  const double a = st->alpha, g = st->ar;
  float acc = 0.0f;
  for (int64_t i = gtid(); i < n; i += gstride()) {
    z[i] = fma(a, p[i], z[i]);
    const double ri = fma(-a, q[i], r[i]);
    r[i] = ri;
    const float t = (float)(ri * g) * s[i];
    b32[i] = t;
    acc = fmaf(t, t, acc);
  }
  float v[1] = {acc};
  double tot[1];
  if (reduce_grid_w<1, kT, true>(v, partials + gridDim.x, &st->counter[2], tot) && threadIdx.x == 0) {
    const double rn = tot[0] / (g * g);
    st->iters += 1;
    st->rho_new = rn;
    if (!isfinite(rn)) {
      st->done = 2;
    } else if (rn <= st->stop2) {
      st->final_req = 1;
      st->done = 3;
    } else if (rn <= st->ru2 || st->iters >= st->max_iter) {
      st->done = 3;
    }
  }
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

// slices of 32 rows with absolute columns (padding: column 0)
void slices(int64_t n, const MgPattern& P, std::vector<int32_t>& sptr, std::vector<int32_t>& col) {
  const int64_t ns = (n + 31) / 32;
  sptr.assign(ns + 1, 0);
  for (int64_t s = 0; s < ns; s++) {
    int32_t w = 0;
    for (int64_t r = 32 * s; r < std::min(n, 32 * s + 32); r++) w = std::max(w, P.rp[r + 1] - P.rp[r]);
    sptr[s + 1] = sptr[s] + 32 * w;
  }
  col.assign(std::max<int32_t>(sptr[ns], 1), 0);
  for (int64_t r = 0; r < n; r++)
    for (int32_t k = P.rp[r]; k < P.rp[r + 1]; k++) col[sptr[r >> 5] + 32 * (k - P.rp[r]) + (r & 31)] = P.ci[k];
}

int lanes_per_row(int64_t n) {
  // one lane while the rows alone fill the chip (152 SMs x 2048 threads), more below
  return n >= 150000 ? 1 : (n >= 40000 ? 4 : 8);
}
int tail_lanes(int64_t n) {
  int l = 1;
  while (l < 8 && 2 * l * n <= kTailT) l *= 2;
  return l;
}

}  // namespace

int mg_plan(Solver& S) {
  if (S.mg || !S.mg_allowed) return ADFEM_OK;
  const int nb0 = S.mg_nb, nbc = nb0 == 2 ? 3 : 1;
  std::vector<MgHostLevel> lv;
  if (!mg_build_host((int64_t)S.mg_rp.size() - 1, std::move(S.mg_rp), std::move(S.mg_ci), nb0, nbc,
                     std::move(S.mg_x), std::move(S.mg_y), lv)) {
    S.mg_allowed = false;
    return ADFEM_OK;
  }
  // (a plan that ends in an error gives the graph back: the next solve tries again)
  struct GiveBack {
    Solver& S;
    std::vector<MgHostLevel>& lv;
    ~GiveBack() {
      if (S.mg || !S.mg_allowed) return;
      S.mg_rp = std::move(lv[0].A.rp);
      S.mg_ci = std::move(lv[0].A.ci);
      S.mg_x = std::move(lv[0].x);
      S.mg_y = std::move(lv[0].y);
    }
  } give_back{S, lv};
  std::unique_ptr<Mg> mg(new Mg());
  Mg& M = *mg;
  M.nlev = (int)lv.size();
  while (M.tail < M.nlev - 1 && lv[M.tail].n * (M.tail ? nbc : nb0) > kMgTailDofs) M.tail++;
  if (M.nlev < 2 || M.nlev - M.tail > kMgMaxTail) {
    S.mg_allowed = false;
    return ADFEM_OK;
  }
  const Sell& A = *S.A;
  Slab sl;
  std::vector<int32_t> sptr, col;
  std::vector<int64_t> vals(M.nlev), pv(M.nlev), apv(M.nlev), ptv(M.nlev);
  for (int l = 0; l < M.nlev; l++) {
    MgLev& L = M.lev[l];
    MgHostLevel& H = lv[l];
    L.n = (int)H.n;
    L.nb = l ? nbc : nb0;
    L.nbc = nbc;
    const bool tail = l >= M.tail;
    L.lpr = tail ? tail_lanes(H.n) : lanes_per_row(H.n);
    if (l == 0) L.lpr = tail ? L.lpr : (nb0 == 1 ? 1 : (H.n >= 150000 ? 1 : 4));
    if (l == 0 && nb0 == 1 && !tail) {
      // the system's own pattern
      L.sptr = A.sptr.as<int32_t>();
      L.col = A.col.p;
      L.spat = A.spat.as<int32_t>();
      L.pat = A.pat.as<int16_t>();
      L.d16 = A.delta16 ? 1 : 0;
      vals[l] = A.nent;
    } else {
      slices(H.n, H.A, sptr, col);
      sl.put(&L.sptr, sptr);
      sl.put((const int32_t**)&L.col, col);
      vals[l] = sptr.back();
    }
    if (l + 1 == M.nlev) continue;
    L.nc = (int)lv[l + 1].n;
    slices(H.n, H.P, sptr, col);
    sl.put(&L.p_sptr, sptr);
    sl.put(&L.p_col, col);
    pv[l] = sptr.back();
    const std::vector<int32_t> psptr = sptr;
    slices(H.n, H.AP, sptr, col);
    sl.put(&L.ap_sptr, sptr);
    sl.put(&L.ap_col, col);
    apv[l] = sptr.back();
    slices(L.nc, H.PT, sptr, col);
    sl.put(&L.pt_sptr, sptr);
    sl.put(&L.pt_col, col);
    ptv[l] = sptr.back();
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
  sl.seal();
  for (int l = 0; l < M.nlev; l++) {
    MgLev& L = M.lev[l];
    const size_t nb = L.nb, n = (size_t)L.n * nb;
    sl.room(&L.val, (size_t)vals[l] * nb * nb);
    sl.room(&L.s, n);
    sl.room(&L.b, n);
    sl.room(&L.x, n);
    sl.room(&L.x2, n);
    sl.room(&L.d, n);
    sl.room(&L.coef, kCoef + 2);
    sl.room(&L.lam, 1);
    if (l + 1 == M.nlev) continue;
    sl.room(&L.p_val, (size_t)pv[l] * nb * nbc);
    sl.room(&L.ap_val, (size_t)apv[l] * nb * nbc);
    sl.room(&L.pt_val, (size_t)ptv[l] * nb * nbc);
  }
  M.ndense = M.lev[M.nlev - 1].n * M.lev[M.nlev - 1].nb;
  sl.room(&M.dense, (size_t)M.ndense * M.ndense);
  sl.room(&M.rowsum, (size_t)S.n * nb0);
  ADFEM_TRY(M.slab.alloc(sl.total));
  sl.resolve(M.slab.as<char>());
  ADFEM_CUDA(cudaMemcpy(M.slab.p, sl.host.data(), sl.host.size(), cudaMemcpyHostToDevice));
  ADFEM_CUDA(cudaMemset(M.slab.as<char>() + sl.host.size(), 0, sl.total - sl.host.size()));
  // (legacy-stream sync, not a device-wide one: other threads may be capturing graphs)
  ADFEM_CUDA(cudaStreamSynchronize(0));
  size_t fl = 0;
  for (int l = M.tail; l < M.nlev; l++) fl += 4 * (((size_t)M.lev[l].n * M.lev[l].nb + 3) / 4 * 4);
  M.tail_smem = sizeof(float) * fl;
  {
    // (once per process: changing a kernel attribute while another thread captures that
    // kernel would invalidate the capture)
    static std::once_flag once;
    static cudaError_t err = cudaSuccess;
    std::call_once(once, [] {
      const int tmax = (int)(sizeof(float) * 4 * (2 * kMgTailDofs + 64));
      const int dmax = (int)(sizeof(float) * (kMgDense * kMgDense + kMgDense));
      const auto a = cudaFuncAttributeMaxDynamicSharedMemorySize;
      for (cudaError_t e : {cudaFuncSetAttribute(k_mg_tail<1, 1>, a, tmax), cudaFuncSetAttribute(k_mg_tail<2, 3>, a, tmax),
                            cudaFuncSetAttribute(k_mg_tail<3, 3>, a, tmax), cudaFuncSetAttribute(k_mg_dense<1>, a, dmax),
                            cudaFuncSetAttribute(k_mg_dense<3>, a, dmax)})
        if (e != cudaSuccess) err = e;
    });
    if (err != cudaSuccess) return cuda_fail(err, "cudaFuncSetAttribute (multigrid)");
    if (M.tail_smem > sizeof(float) * 4 * (2 * kMgTailDofs + 64)) {
      S.mg_allowed = false;
      return ADFEM_OK;
    }
  }
  S.mg = std::move(mg);
  return ADFEM_OK;
}

// ---------------------------------------------------------------------------
namespace {

unsigned blocks(int64_t n, int b) { return (unsigned)std::max<int64_t>(1, (n + b - 1) / b); }

template <int NB, int NC, bool D16>
void level_values(const MgLev& L, const MgLev& C, cudaStream_t st) {
  constexpr int BP = 64, BA = NB * NC == 1 ? 128 : 32;
  k_mg_p<NB, NC, D16, BP><<<blocks(L.n, BP), BP, 0, st>>>(L);
  k_mg_ap<NB, NC, D16, BA><<<blocks(L.n, BA), BA, 0, st>>>(L);
  k_mg_ac<NB, NC><<<blocks(32 * (int64_t)L.nc, 128), 128, 0, st>>>(L, C);
  k_mg_scale<NB, NC><<<blocks(L.nc, 128), 128, 0, st>>>(L, C);
}

}  // namespace

// values of the hierarchy for the current assembly (s32 is current)
int mg_values(Solver& S, cudaStream_t st) {
  Mg& M = *S.mg;
  if (M.current) return ADFEM_OK;
  const Sell& A = *S.A;
  const MgLev& L0 = M.lev[0];
  const unsigned nb = blocks(S.n, kT);
  for (int l = 0; l < M.nlev; l++) ADFEM_CUDA(cudaMemsetAsync(M.lev[l].lam, 0, sizeof(int), st));
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
  for (int l = 0; l + 1 < M.nlev; l++) {
    const MgLev &L = M.lev[l], &C = M.lev[l + 1];
    if (L.nb == 1) {
      if (L.d16) level_values<1, 1, true>(L, C, st);
      else level_values<1, 1, false>(L, C, st);
    } else if (L.nb == 2) {
      level_values<2, 3, false>(L, C, st);
    } else {
      level_values<3, 3, false>(L, C, st);
    }
    k_mg_coef<<<1, 32, 0, st>>>(L, l == 0 ? kMgDeg0 : kMgDeg, l == 0 ? kFrac0 : kFrac);
  }
  const MgLev& C = M.lev[M.nlev - 1];
  const size_t dsm = sizeof(float) * ((size_t)M.ndense * M.ndense + M.ndense);
  if (C.nb == 1) k_mg_dense<1><<<1, kTailT, dsm, st>>>(C, M.dense);
  else k_mg_dense<3><<<1, kTailT, dsm, st>>>(C, M.dense);
  ADFEM_CUDA(cudaGetLastError());
  M.current = true;
  return ADFEM_OK;
}

namespace {

template <int MODE>
void sweep(const Solver& S, const MgLev& L, const float* x, float* out, int c1, int c2, int keep, CgState* cs,
           cudaStream_t st) {
  double* part = S.partials.as<double>();
  // (the kernel with the dot product keeps to the solver's grid: its partials have that size)
  const unsigned g = MODE == kLast && cs ? (unsigned)S.grid : blocks((int64_t)L.n * L.lpr, kT);
#define ADFEM_SWEEP(NB, D16, LPR) k_mg_sweep<NB, D16, LPR, MODE><<<g, kT, 0, st>>>(L, x, out, c1, c2, keep, cs, part)
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

void restrict_to(const MgLev& L, const float* r, float* out, cudaStream_t st) {
  const int lpr = L.nc >= 150000 ? 1 : 8;
  const unsigned g = blocks((int64_t)L.nc * lpr, kT);
#define ADFEM_RES(NB, NC)                                                \
  do {                                                                   \
    if (lpr == 1) k_mg_restrict<NB, NC, 1><<<g, kT, 0, st>>>(L, r, out); \
    else k_mg_restrict<NB, NC, 8><<<g, kT, 0, st>>>(L, r, out);          \
  } while (0)
  if (L.nb == 1) ADFEM_RES(1, 1);
  else if (L.nb == 2) ADFEM_RES(2, 3);
  else ADFEM_RES(3, 3);
#undef ADFEM_RES
}
void prolong_from(const MgLev& L, const float* xc, float* x, cudaStream_t st) {
  const unsigned g = blocks(L.n, kT);
  if (L.nb == 1) k_mg_prolong<1, 1><<<g, kT, 0, st>>>(L, xc, x);
  else if (L.nb == 2) k_mg_prolong<2, 3><<<g, kT, 0, st>>>(L, xc, x);
  else k_mg_prolong<3, 3><<<g, kT, 0, st>>>(L, xc, x);
}

// One cycle: lev[0].b -> the vector returned; returns the launches through *count.
const float* enqueue_cycle(Solver& S, cudaStream_t st, int* count) {
  Mg& M = *S.mg;
  CgState* cs = S.state.as<CgState>();
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
    restrict_to(L, L.d, M.lev[l + 1].b, st);
    nl += 2;
    xs[l] = x;
  }
  {
    TailArgs a;
    a.nl = M.nlev - M.tail;
    for (int l = 0; l < a.nl; l++) a.L[l] = M.lev[M.tail + l];
    a.dense = M.dense;
    a.N = M.ndense;
    a.b = M.lev[M.tail].b;
    a.x = M.lev[M.tail].x;
    a.reps = M.tail == 0 ? 1 : 2;
    a.st = M.tail == 0 ? cs : nullptr;
    const int nt = a.L[0].nb, nc = a.L[0].nbc;
    if (nt == 1) k_mg_tail<1, 1><<<1, kTailT, M.tail_smem, st>>>(a);
    else if (nt == 2 && nc == 3) k_mg_tail<2, 3><<<1, kTailT, M.tail_smem, st>>>(a);
    else k_mg_tail<3, 3><<<1, kTailT, M.tail_smem, st>>>(a);
    xs[M.tail] = M.lev[M.tail].x;
    nl++;
  }
  for (int l = M.tail - 1; l >= 0; l--) {
    const MgLev& L = M.lev[l];
    const int deg = l == 0 ? kMgDeg0 : kMgDeg;
    float *x = xs[l], *y = x == L.x ? L.x2 : L.x;
    prolong_from(L, xs[l + 1], x, st);
    nl++;
    for (int k = 0; k < deg; k++) {
      const int c1 = k ? 2 * k : -1, c2 = k ? 2 * k + 1 : 0;
      if (k + 1 < deg) sweep<kStep>(S, L, x, y, c1, c2, 1, nullptr, st);
      else sweep<kLast>(S, L, x, y, c1, c2, 0, l == 0 ? cs : nullptr, st);
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
    k_mg_residual<decltype(d16)::value, decltype(nb)::value><<<S.grid, kT, 0, st>>>(
        S.n, A.sptr.as<int32_t>(), A.col.p, A.val64.as<double>(), M.rowsum, S.s32.as<float>(), S.b.as<double>(),
        S.y64.as<double>(), S.r64.as<double>(), M.lev[0].b, S.state.as<CgState>(), S.partials.as<double>(), mode, loop);
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
  k_mg_dir<<<S.grid, kT, 0, st>>>(S.n, z, S.s32.as<float>(), S.p64.as<double>(), cs);
  solver_enqueue_spmv64(S, S.A->val64.as<double>(), st);
  k_mg_update<<<S.grid, kT, 0, st>>>(S.n, S.z64.as<double>(), S.r64.as<double>(), S.p64.as<double>(),
                                     S.q64.as<double>(), S.s32.as<float>(), M.lev[0].b, cs, S.partials.as<double>());
  solver_enqueue_fold64(S, 0, st);
  enqueue_residual(S, 1, loop, st);
  M.body_launches = nl + 5;
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
  ADFEM_TRY(mg_values(S, user));
  ADFEM_TRY(capture_solve(S));
  Mg& M = *S.mg;
  cudaStream_t st = S.stream;
  ADFEM_CUDA(cudaEventRecord(S.ev[0], user));
  ADFEM_CUDA(cudaStreamWaitEvent(st, S.ev[0], 0));
  ADFEM_CUDA(cudaEventRecord(S.ev[1], st));
  CgState init;
  std::memset(&init, 0, sizeof(init));
  init.max_iter = std::min(o.max_iter, kMgIterations);
  init.delta2 = 1e-6;  // residual evaluated in FP64 after each drop of the recurrence by 1e-3
  S.h_state[1] = init;
  ADFEM_CUDA(cudaMemcpyAsync(S.state.p, &S.h_state[1], sizeof(CgState), cudaMemcpyHostToDevice, st));
  k_mg_init<<<S.grid, kT, 0, st>>>(S.n, rhs, zero_rows, fix_rows, fix_vals, S.s32.as<float>(),
                                   o.warm_start ? u : nullptr, S.b.as<double>(), S.y64.as<double>(),
                                   S.z64.as<double>(), S.state.as<CgState>(), S.partials.as<double>(),
                                   o.rtol * o.rtol);
  const cudaGraphConditionalHandle none{};
  enqueue_residual(S, 0, none, st);
  ADFEM_CUDA(cudaGetLastError());
  ADFEM_CUDA(cudaGraphLaunch(M.solve, st));
  solver_enqueue_fold64(S, 1, st);
  enqueue_residual(S, 2, none, st);
  // (the caller's vector is written after the outcome is known to be usable: a solve that gives
  // up leaves it as the other iteration's start)
  ADFEM_CUDA(cudaMemcpyAsync(&S.h_state[0], S.state.p, sizeof(CgState), cudaMemcpyDeviceToHost, st));
  ADFEM_CUDA(cudaEventRecord(S.ev[2], st));
  ADFEM_CUDA(cudaGetLastError());
  ADFEM_CUDA(cudaEventSynchronize(S.ev[2]));
  const CgState fin = S.h_state[0];
  if (fin.done != 1 && !(fin.done == 4 && fin.iters >= o.max_iter)) {
    *gave_up = true;
    ADFEM_CUDA(cudaStreamWaitEvent(user, S.ev[2], 0));
    return ADFEM_OK;
  }
  k_mg_out<<<blocks(S.n, kT), kT, 0, st>>>(S.n, S.y64.as<double>(), fix_rows, fix_vals, u);
  ADFEM_CUDA(cudaGetLastError());
  ADFEM_CUDA(cudaEventRecord(S.ev[3], st));
  ADFEM_CUDA(cudaStreamWaitEvent(user, S.ev[3], 0));
  const int status = fin.done == 1 ? ADFEM_OK : ADFEM_ERR_NOT_CONVERGED;
  const double relres = fin.bnorm2 > 0.0 ? std::sqrt(fin.rr64 / fin.bnorm2) : 0.0;
  if (stats) {
    float ms = 0.0f;
    ADFEM_CUDA(cudaEventSynchronize(S.ev[3]));
    cudaEventElapsedTime(&ms, S.ev[1], S.ev[3]);
    stats->iterations = fin.iters;
    stats->updates = fin.updates;
    stats->relres = relres;
    stats->ms = ms;
    stats->status = status;
    stats->launches = (long long)std::max(fin.iters, 1) * M.body_launches + 5;
  }
  if (status == ADFEM_ERR_NOT_CONVERGED)
    return fail(status, "CG did not reach rtol within max_iter (relres " + std::to_string(relres) + ")");
  return ADFEM_OK;
}

size_t mg_device_bytes(const Solver& S) { return S.mg ? S.mg->slab.bytes : 0; }

ADFEM_CHECK_READER(check_line_mg)

}  // namespace adfem
