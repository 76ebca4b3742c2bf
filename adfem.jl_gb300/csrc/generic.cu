// Degree-generic element kernels for P1 and P2 Lagrange triangles: the reference's
// element loops written over elem_ndof and the per-point tables h, hx, hy, w
// (deps/MFEM/Common.cpp:46-126), for
//   FemLaplaceScalar forward/backward   deps/MFEM/FemLaplace1/FemLaplaceScalar.h:3-54
//   ComputeFemMassMatrix1 fwd/bwd       deps/MFEM/ComputeFemMassMatrix1/ComputeFemMassMatrixMfem.h:4-55
//   FemSourceScalar forward/backward    deps/MFEM/FemSource1/FemSourceScalar.h:4-32
//   ComputeFemStiffnessMatrixMfem       deps/MFEM/ComputeFemStiffnessMatrixMfem/ComputeFemStiffnessMatrixMfem.h:4-81
//   FemToGaussPoints / DofToGaussPoints deps/MFEM/FemToGaussPoints/FemToGaussPointsMfem.h:5-34,
//                                       deps/MFEM/DofToGaussPoints/DofToGaussPointsMfem.h:5-35
// and the summed (SparseMatrixCSC) operators of the Laplace, mass and elasticity
// matrices.  The P1 Laplace/source/stiffness path of P1 meshes has its own fused
// kernels (assemble.cu, elastic.cu); these serve P2 meshes and the mass and
// interpolation ops of both degrees.
//
// Layout: one thread per (Gauss point, local row) for the unsummed COO outputs, so a
// warp writes one contiguous stretch of entries; one thread per DOF row for every
// scatter (load vector, summed operators, interpolation transposes), walking the
// DOF->element incidence in ascending element order, so results are deterministic
// and no atomics are needed.  The per-point basis tables of the degree are built in
// shared memory by every block (formed from the rule by the compiler).
#include <mutex>

#include "adfem_internal.h"
#include "cg_common.cuh"
#include "checks.cuh"

namespace adfem {
namespace {

constexpr int kGT = 256;
constexpr int kRowBTs = 128;  // rows per block of the resident-system row kernel

// rule points (xi, eta, weight) on the reference triangle: order 2 (3 points, P1) and
// order 4 (6 points, P2: the published Strang-Fix/Dunavant rule); same constants as
// the host tables of mesh.cpp
constexpr double c_rule[2][6][3] = {
    {{1.0 / 6.0, 1.0 / 6.0, 1.0 / 6.0},
     {1.0 / 6.0, 2.0 / 3.0, 1.0 / 6.0},
     {2.0 / 3.0, 1.0 / 6.0, 1.0 / 6.0},
     {0.0, 0.0, 0.0},
     {0.0, 0.0, 0.0},
     {0.0, 0.0, 0.0}},
    {{0.091576213509770743460, 0.091576213509770743460, 0.054975871827660933819},
     {0.091576213509770743460, 0.81684757298045851308, 0.054975871827660933819},
     {0.81684757298045851308, 0.091576213509770743460, 0.054975871827660933819},
     {0.44594849091596488632, 0.44594849091596488632, 0.11169079483900573285},
     {0.44594849091596488632, 0.10810301816807022736, 0.11169079483900573285},
     {0.10810301816807022736, 0.44594849091596488632, 0.11169079483900573285}}};

template <int DEG>
struct Tab {
  static constexpr int ND = DEG == 2 ? 6 : 3;  // DOFs per element
  static constexpr int NG = DEG == 2 ? 6 : 3;  // Gauss points per element
  double h[NG][ND];     // phi_r at point k
  double t[NG][ND][3];  // d phi_r / d l_c at point k
  double l[NG][3];      // barycentric coordinates of point k
  double w[NG];         // rule weight of point k
  double hw[NG][ND];    // phi_r w / 0.5 at point k
};

// Lagrange basis in barycentric coordinates.  P1: phi_r = l_r.  P2 (nodes at the
// vertices and edge midpoints, vertex functions first, then edges (0,1), (1,2),
// (2,0)): phi_a = l_a (2 l_a - 1), phi_ab = 4 l_a l_b.
template <int DEG>
constexpr Tab<DEG> make_tab() {
  constexpr int ND = Tab<DEG>::ND, NG = Tab<DEG>::NG;
  Tab<DEG> T{};
  for (int k = 0; k < NG; k++) {
    const double xi = c_rule[DEG - 1][k][0], eta = c_rule[DEG - 1][k][1];
    const double l[3] = {1.0 - xi - eta, xi, eta};
    T.w[k] = c_rule[DEG - 1][k][2];
    for (int c = 0; c < 3; c++) T.l[k][c] = l[c];
    if (DEG == 1) {
      for (int r = 0; r < 3; r++) {
        T.h[k][r] = l[r];
        T.t[k][r][r] = 1.0;
      }
    } else {
      for (int a = 0; a < 3; a++) {
        T.h[k][a] = l[a] * (2.0 * l[a] - 1.0);
        T.t[k][a][a] = 4.0 * l[a] - 1.0;
      }
      for (int j = 0; j < 3; j++) {
        const int a = j, b = (j + 1) % 3;
        T.h[k][3 + j] = 4.0 * l[a] * l[b];
        T.t[k][3 + j][a] = 4.0 * l[b];
        T.t[k][3 + j][b] = 4.0 * l[a];
      }
    }
    for (int r = 0; r < ND; r++) T.hw[k][r] = T.h[k][r] * T.w[k] / 0.5;
  }
  return T;
}
__device__ constexpr Tab<1> c_tab1 = make_tab<1>();
__device__ constexpr Tab<2> c_tab2 = make_tab<2>();

// The table in shared memory.  (Copied from memory: formed by a block's first threads, its chain of
// FP64 operations held every block back: interpolation transpose 41 instead of 33 us at 641k rows.)
template <int DEG>
__device__ __forceinline__ void tab_init(Tab<DEG>& T) {
  const double* src;
  if constexpr (DEG == 1) src = reinterpret_cast<const double*>(&c_tab1);
  else src = reinterpret_cast<const double*>(&c_tab2);
  for (int i = threadIdx.x; i < (int)(sizeof(Tab<DEG>) / sizeof(double)); i += blockDim.x)
    reinterpret_cast<double*>(&T)[i] = __ldg(src + i);
  __syncthreads();
}

// physical gradient of basis r at point k: sum_c (d phi_r / d l_c) grad l_c
template <int DEG>
__device__ __forceinline__ void grad_at(const Tab<DEG>& T, int k, int r, const double2 (&g)[3], double& hx,
                                        double& hy) {
  const double t0 = T.t[k][r][0], t1 = T.t[k][r][1], t2 = T.t[k][r][2];
  hx = t0 * g[0].x + t1 * g[1].x + t2 * g[2].x;
  hy = t0 * g[0].y + t1 * g[1].y + t2 * g[2].y;
}

__device__ __forceinline__ void load_grad(const double2* __restrict__ grad, int64_t e, double2 (&g)[3]) {
  g[0] = grad[3 * e];
  g[1] = grad[3 * e + 1];
  g[2] = grad[3 * e + 2];
}

// w_k = ip.weight * area / 0.5 (Common.cpp:116)
template <int DEG>
__device__ __forceinline__ double weight_at(const Tab<DEG>& T, int k, double area) {
  return T.w[k] * area / 0.5;
}

// Callers' arrays are 8-byte aligned at least; 16-byte accesses only where they are 16-byte
// aligned (an element's six values keep the array's alignment).
__device__ __forceinline__ bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
__device__ __forceinline__ void load6(const double* __restrict__ p, double (&v)[6]) {
  if (aligned16(p)) {
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const double2 x = __ldg(reinterpret_cast<const double2*>(p) + k);
      v[2 * k] = x.x;
      v[2 * k + 1] = x.y;
    }
  } else {
#pragma unroll
    for (int k = 0; k < 6; k++) v[k] = __ldg(p + k);
  }
}

// sum_k f_k t(k) over an element's points
template <int NG, class F>
__device__ __forceinline__ double point_sum(const double* __restrict__ f, F t) {
  double v[NG];
  if constexpr (NG == 6) {
    load6(f, v);
  } else {
#pragma unroll
    for (int k = 0; k < NG; k++) v[k] = __ldg(f + k);
  }
  double s = v[0] * t(0);
#pragma unroll
  for (int k = 1; k < NG; k++) s = fma(v[k], t(k), s);
  return s;
}

int grid_for(int64_t n, int bt = kGT) {
  int64_t b = (n + bt - 1) / bt;
  return (int)std::max<int64_t>(1, std::min<int64_t>(b, 152 * 32));
}

// ---------------------------------------------------------------- P2 by orbits
// The order-4 rule has two orbits of three points; at the point with special vertex i the
// barycentric coordinates are b at i and a at the other two.  A sum over an orbit of a
// coefficient times a product of basis values (or of their derivatives' factors) is therefore
// base * (c_0 + c_1 + c_2) + alpha * c_i (+ beta * c_j), so the sums that an element matrix, a
// load or an interpolation needs cost one or two FP64 operations each instead of six, which is
// what bounds these kernels (FP64 issues at 1/64 of FP32 here).  Laplace: the basis gradients
// are combinations of the barycentric ones, so the matrix is a contraction of the moments
//   VV_ab = sum c w t_a t_b, Q_ab = sum c w t_a 4 l_b, R_ab = sum c w 16 l_a l_b  (t = 4 l - 1)
// with the three products g_ab of the P1 geometry record, the diagonal from the zero row sums.  ~125
// FP64 operations per element against ~500 with gradients formed at every point.
namespace p2 {
__device__ constexpr double A[2] = {0.091576213509770743460, 0.44594849091596488632};
__device__ constexpr double B[2] = {0.81684757298045851308, 0.10810301816807022736};
__device__ constexpr double W[2] = {0.054975871827660933819, 0.11169079483900573285};
// point k of an orbit -> its special vertex: (a, a), (a, b), (b, a) in (xi, eta)
__host__ __device__ constexpr int special(int k) { return k == 0 ? 0 : 3 - k; }
// local edge opposite to vertex m: edges (0,1), (1,2), (2,0) are DOFs 3, 4, 5
__host__ __device__ constexpr int edge_opp(int m) { return m == 0 ? 4 : (m == 1 ? 5 : 3); }
__host__ __device__ constexpr int third(int i, int j) { return 3 - i - j; }

// the six values of an element by orbit and special vertex
__device__ __forceinline__ void by_special(const double* __restrict__ c6, double (&c)[2][3]) {
  double v[6];
  load6(c6, v);
#pragma unroll
  for (int k = 0; k < 6; k++) c[k / 3][special(k % 3)] = v[k];
}

// symmetric family: D[i] (both factors at i) and O[k] (factors at i, j with third vertex k) of
// sum c x_i x_j, x = xs at the special vertex, xo elsewhere
__device__ __forceinline__ void sym_sums(const double (&c)[2][3], const double (&cs)[2], const double (&xs)[2],
                                         const double (&xo)[2], const double (&w)[2], double (&D)[3], double (&O)[3]) {
  const double d = fma(w[1] * xo[1] * xo[1], cs[1], w[0] * xo[0] * xo[0] * cs[0]);
  const double o = fma(w[1] * xs[1] * xo[1], cs[1], w[0] * xs[0] * xo[0] * cs[0]);
#pragma unroll
  for (int i = 0; i < 3; i++) {
    D[i] = fma(w[1] * (xs[1] * xs[1] - xo[1] * xo[1]), c[1][i], fma(w[0] * (xs[0] * xs[0] - xo[0] * xo[0]), c[0][i], d));
    O[i] = fma(w[1] * (xo[1] * xo[1] - xs[1] * xo[1]), c[1][i], fma(w[0] * (xo[0] * xo[0] - xs[0] * xo[0]), c[0][i], o));
  }
}
// mixed family: M[i][j] of sum c x_i y_j
__device__ __forceinline__ void mixed_sums(const double (&c)[2][3], const double (&cs)[2], const double (&xs)[2],
                                           const double (&xo)[2], const double (&ys)[2], const double (&yo)[2],
                                           const double (&w)[2], double (&M)[3][3]) {
  const double m = fma(w[1] * xo[1] * yo[1], cs[1], w[0] * xo[0] * yo[0] * cs[0]);
#pragma unroll
  for (int i = 0; i < 3; i++) {
    M[i][i] = fma(w[1] * (xs[1] * ys[1] - xo[1] * yo[1]), c[1][i],
                  fma(w[0] * (xs[0] * ys[0] - xo[0] * yo[0]), c[0][i], m));
    const double mi = fma(w[1] * (xs[1] * yo[1] - xo[1] * yo[1]), c[1][i],
                          fma(w[0] * (xs[0] * yo[0] - xo[0] * yo[0]), c[0][i], m));
#pragma unroll
    for (int j = 0; j < 3; j++)
      if (j != i)
        M[i][j] = fma(w[1] * (xo[1] * ys[1] - xo[1] * yo[1]), c[1][j],
                      fma(w[0] * (xo[0] * ys[0] - xo[0] * yo[0]), c[0][j], mi));
  }
}
// values of a P2 function at the six points: sums over vertices and edges, then two operations
// per point (f: the point weights, 1 for plain values)
template <class F>
__device__ __forceinline__ void at_points(const double (&u)[6], F put, const double (&f)[2]) {
  const double U = u[0] + u[1] + u[2], E = u[3] + u[4] + u[5];
#pragma unroll
  for (int o = 0; o < 2; o++) {
    const double hs = B[o] * (2 * B[o] - 1), ho = A[o] * (2 * A[o] - 1), es = 4 * A[o] * A[o], eo = 4 * A[o] * B[o];
    const double base = fma(f[o] * eo, E, f[o] * ho * U);
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const int i = special(k);
      put(3 * o + k, fma(f[o] * (es - eo), u[edge_opp(i)], fma(f[o] * (hs - ho), u[i], base)));
    }
  }
}
}  // namespace p2

// P2 element matrices, one thread per element, stored as the full 6 x 6 matrix (a row gather
// reads one contiguous row)
template <int OP>
__global__ void __launch_bounds__(kGT) k_p2_ke(int64_t ne, const double4* __restrict__ geo,
                                               const double* __restrict__ area, const double* __restrict__ coef,
                                               double* __restrict__ ke) {
  for (int64_t e = gtid(); e < ne; e += gstride()) {
    double c[2][3];
    p2::by_special(coef + 6 * e, c);
    const double cs[2] = {c[0][0] + c[0][1] + c[0][2], c[1][0] + c[1][1] + c[1][2]};
    double K[6][6];
    if (OP == (int)GenOp::LAPLACE) {
      // 2 area grad_a.grad_b = 6 g_ab of the record (whose weight is area / 3)
      constexpr double w6[2] = {6 * p2::W[0], 6 * p2::W[1]}, w16[2] = {96 * p2::W[0], 96 * p2::W[1]},
                       w4[2] = {24 * p2::W[0], 24 * p2::W[1]};
      constexpr double ts[2] = {4 * p2::B[0] - 1, 4 * p2::B[1] - 1}, to[2] = {4 * p2::A[0] - 1, 4 * p2::A[1] - 1};
      const double4 gr = geo[e];
      const double g[3][3] = {{-(gr.x + gr.y), gr.x, gr.y}, {gr.x, -(gr.x + gr.z), gr.z}, {gr.y, gr.z, -(gr.y + gr.z)}};
      double D[3], O[3], Q[3][3], RD[3], RO[3];
      p2::sym_sums(c, cs, ts, to, w6, D, O);
      p2::mixed_sums(c, cs, ts, to, p2::B, p2::A, w4, Q);
      p2::sym_sums(c, cs, p2::B, p2::A, w16, RD, RO);
      auto R = [&](int i, int j) { return i == j ? RD[i] : RO[p2::third(i, j)]; };
#pragma unroll
      for (int i = 0; i < 3; i++) {
#pragma unroll
        for (int j = 0; j < i; j++) K[i][j] = K[j][i] = O[p2::third(i, j)] * g[i][j];
#pragma unroll
        for (int j = 0; j < 3; j++) {
          const int q = (j + 1) % 3;  // edge j joins j and q
          K[i][3 + j] = K[3 + j][i] = fma(Q[i][q], g[i][j], Q[i][j] * g[i][q]);
        }
      }
#pragma unroll
      for (int i = 0; i < 3; i++) {
        const int q = (i + 1) % 3;
#pragma unroll
        for (int j = 0; j < i; j++) {
          const int s = (j + 1) % 3;
          K[3 + i][3 + j] = K[3 + j][3 + i] =
              fma(R(q, s), g[i][j], fma(R(q, j), g[i][s], fma(R(i, s), g[q][j], R(i, j) * g[q][s])));
        }
      }
      // The basis functions sum to one, so a row does to zero.  The factors of the orbit sums are
      // rounded the same way in every element, and a row sum that is off by them adds up over the mesh
      // (P2 solves 241 x 251: 2.5e-12 of the solution; 1.1e-13 with an entry's points summed one by one).
#pragma unroll
      for (int i = 0; i < 6; i++) {
        double d = K[i][(i + 1) % 6];
#pragma unroll
        for (int j = 2; j < 6; j++) d += K[i][(i + j) % 6];
        K[i][i] = -d;
      }
    } else {
      constexpr double w2[2] = {2 * p2::W[0], 2 * p2::W[1]};
      constexpr double hs[2] = {p2::B[0] * (2 * p2::B[0] - 1), p2::B[1] * (2 * p2::B[1] - 1)};
      constexpr double ho[2] = {p2::A[0] * (2 * p2::A[0] - 1), p2::A[1] * (2 * p2::A[1] - 1)};
      constexpr double es[2] = {4 * p2::A[0] * p2::A[0], 4 * p2::A[1] * p2::A[1]};
      constexpr double eo[2] = {4 * p2::A[0] * p2::B[0], 4 * p2::A[1] * p2::B[1]};
      const double ar = area[e];
      double D[3], O[3], M[3][3], ED[3], EO[3];
      p2::sym_sums(c, cs, hs, ho, w2, D, O);
      p2::mixed_sums(c, cs, hs, ho, es, eo, w2, M);
      p2::sym_sums(c, cs, es, eo, w2, ED, EO);
#pragma unroll
      for (int i = 0; i < 3; i++) {
        K[i][i] = ar * D[i];
        K[p2::edge_opp(i)][p2::edge_opp(i)] = ar * ED[i];
#pragma unroll
        for (int j = 0; j < i; j++) {
          K[i][j] = K[j][i] = ar * O[p2::third(i, j)];
          K[p2::edge_opp(i)][p2::edge_opp(j)] = K[p2::edge_opp(j)][p2::edge_opp(i)] = ar * EO[p2::third(i, j)];
        }
#pragma unroll
        for (int j = 0; j < 3; j++) K[i][p2::edge_opp(j)] = K[p2::edge_opp(j)][i] = ar * M[i][j];
      }
    }
    double2* out = reinterpret_cast<double2*>(ke + 36 * e);
#pragma unroll
    for (int a = 0; a < 6; a++)
#pragma unroll
      for (int b = 0; b < 3; b++) out[3 * a + b] = make_double2(K[a][2 * b], K[a][2 * b + 1]);
  }
}

// Gradient factors of the P2 basis at point k of the rule: t[a] = 4 l_a - 1 (vertex a), l4[a] = 4 l_a
// (edge (p, q) has 4 l_q grad_p + 4 l_p grad_q)
__device__ __forceinline__ void p2_factors(int k, double (&t)[3], double (&l4)[3]) {
  const int o = k >= 3 ? 1 : 0, i = p2::special(k - 3 * o);
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const double l = a == i ? (o ? p2::B[1] : p2::B[0]) : (o ? p2::A[1] : p2::A[0]);
    l4[a] = 4 * l;
    t[a] = 4 * l - 1;
  }
}

// Gradients of the six basis functions at point k
__device__ __forceinline__ void p2_gradients(int k, const double2 (&g)[3], double (&hx)[6], double (&hy)[6]) {
  double t[3], l4[3];
  p2_factors(k, t, l4);
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const int b = (a + 1) % 3;
    hx[a] = t[a] * g[a].x;
    hy[a] = t[a] * g[a].y;
    hx[3 + a] = fma(l4[b], g[a].x, l4[a] * g[b].x);
    hy[3 + a] = fma(l4[b], g[a].y, l4[a] * g[b].y);
  }
}

// Unsummed P2 Laplace COO: a block takes kCooPts Gauss points; one thread per point forms the 21
// distinct entries from the gradients there (75 FP64 operations; recomputing the gradients per row
// took ~400), all threads write values and indices in order through shared memory.  (From the three
// g_ab of the P1 geometry record they take 51, but the products with a vertex of small gradient lose
// digits to cancellation: 3 of 16 in elements of aspect 10^4.)
// (The points fill every warp of the block: two warps of eight left half of the SM's FP64 pipes
// idle, 54 instead of 40 us at 39k elements.)
constexpr int kCooPts = 126, kCooT = 128;  // whole elements
__global__ void __launch_bounds__(kCooT) k_p2_coo(int64_t ne, const int32_t* __restrict__ dof,
                                                const double* __restrict__ area, const double2* __restrict__ grad,
                                                const double* __restrict__ coef, longlong2* __restrict__ idx,
                                                double* __restrict__ vv) {
  __shared__ double sv[kCooPts][37];
  __shared__ int32_t sd[kCooPts / 6][6];
  const int64_t ngp = 6 * ne;
  for (int64_t g0 = (int64_t)blockIdx.x * kCooPts; g0 < ngp; g0 += (int64_t)gridDim.x * kCooPts) {
    const int np = (int)std::min<int64_t>(kCooPts, ngp - g0);
    const int64_t e0 = g0 / 6;
    const int nel = np / 6;
    __syncthreads();  // the previous tile has been written
    for (int t = threadIdx.x; t < 6 * nel; t += kCooT) sd[t / 6][t % 6] = dof[6 * e0 + t];
    if ((int)threadIdx.x < np) {
      const int64_t gp = g0 + threadIdx.x, e = gp / 6;
      const int k = (int)(gp - 6 * e);
      double2 g[3];
      load_grad(grad, e, g);
      const double cw = coef[gp] * (2 * p2::W[k >= 3 ? 1 : 0] * area[e]);
      double hx[6], hy[6];
      p2_gradients(k, g, hx, hy);
      double* K = sv[threadIdx.x];
#pragma unroll
      for (int i = 0; i < 6; i++) {
        const double x = cw * hx[i], y = cw * hy[i];
#pragma unroll
        for (int j = 0; j <= i; j++) K[6 * i + j] = K[6 * j + i] = fma(x, hx[j], y * hy[j]);
      }
    }
    __syncthreads();
    for (int q = threadIdx.x; q < 36 * np; q += kCooT) {
      const int p = q / 36, m = q - 36 * p, r = m / 6, c = m - 6 * r;
      const int le = p / 6;
      __stcs(vv + 36 * g0 + q, sv[p][m]);
      idx[36 * g0 + q] = make_longlong2(sd[le][r], sd[le][c]);
    }
  }
}

// Its transpose: grad_coef[gp] = sum_pq grad_vv[gp, p, q] (d N_pq / d coef).  The block reads its
// points' entries in order into shared memory, one thread per point multiplies them with the
// gradients from both sides (104 operations).
__global__ void __launch_bounds__(kCooT) k_p2_coo_backward(int64_t ne, const double* __restrict__ area,
                                                         const double2* __restrict__ grad,
                                                         const double* __restrict__ gv, double* __restrict__ out) {
  __shared__ double sv[kCooPts][37];
  const int64_t ngp = 6 * ne;
  for (int64_t g0 = (int64_t)blockIdx.x * kCooPts; g0 < ngp; g0 += (int64_t)gridDim.x * kCooPts) {
    const int np = (int)std::min<int64_t>(kCooPts, ngp - g0);
    __syncthreads();
    if (aligned16(gv)) {
      for (int q = threadIdx.x; q < 18 * np; q += kCooT) {
        const double2 v = __ldcs(reinterpret_cast<const double2*>(gv + 36 * g0) + q);
        const int p = q / 18, m = 2 * (q - 18 * p);
        sv[p][m] = v.x;
        sv[p][m + 1] = v.y;
      }
    } else {
      for (int q = threadIdx.x; q < 36 * np; q += kCooT) sv[q / 36][q % 36] = __ldcs(gv + 36 * g0 + q);
    }
    __syncthreads();
    if ((int)threadIdx.x < np) {
      const int64_t gp = g0 + threadIdx.x, e = gp / 6;
      const int k = (int)(gp - 6 * e);
      double2 g[3];
      load_grad(grad, e, g);
      double hx[6], hy[6], v = 0.0;
      p2_gradients(k, g, hx, hy);
      const double* G = sv[threadIdx.x];
#pragma unroll
      for (int p = 0; p < 6; p++) {
        double x = G[6 * p] * hx[0], y = G[6 * p] * hy[0];
#pragma unroll
        for (int q = 1; q < 6; q++) {
          x = fma(G[6 * p + q], hx[q], x);
          y = fma(G[6 * p + q], hy[q], y);
        }
        v = fma(hx[p], x, fma(hy[p], y, v));
      }
      out[gp] = v * (2 * p2::W[k >= 3 ? 1 : 0] * area[e]);
    }
  }
}

// P2 values at the Gauss points, one thread per element (SRC: the load's transpose, times w_k)
template <bool SRC>
__global__ void __launch_bounds__(kGT) k_p2_to_gauss(int64_t ne, const int32_t* __restrict__ dof,
                                                     const double* __restrict__ area, const double* __restrict__ u,
                                                     double* __restrict__ out) {
  for (int64_t e = gtid(); e < ne; e += gstride()) {
    const int2* d = reinterpret_cast<const int2*>(dof + 6 * e);
    const int2 a = __ldg(d), b = __ldg(d + 1), c = __ldg(d + 2);
    const double v[6] = {__ldg(u + a.x), __ldg(u + a.y), __ldg(u + b.x), __ldg(u + b.y), __ldg(u + c.x), __ldg(u + c.y)};
    double o[6];
    if (SRC) {
      constexpr double w[2] = {2 * p2::W[0], 2 * p2::W[1]};
      const double ar = area[e];
      p2::at_points(v, [&](int k, double x) { o[k] = ar * x; }, w);
    } else {
      constexpr double one[2] = {1.0, 1.0};
      p2::at_points(v, [&](int k, double x) { o[k] = x; }, one);
    }
    if (aligned16(out)) {
      double2* q = reinterpret_cast<double2*>(out + 6 * e);
#pragma unroll
      for (int k = 0; k < 3; k++) q[k] = make_double2(o[2 * k], o[2 * k + 1]);
    } else {
#pragma unroll
      for (int k = 0; k < 6; k++) out[6 * e + k] = o[k];
    }
  }
}

// ---------------------------------------------------------------- unsummed COO
template <int DEG, int OP>
__global__ void __launch_bounds__(kGT) k_gen_coo(int64_t ne, const int32_t* __restrict__ dof,
                                                 const double* __restrict__ area, const double2* __restrict__ grad,
                                                 const double* __restrict__ coef, long long* __restrict__ idx,
                                                 double* __restrict__ vv) {
  constexpr int ND = Tab<DEG>::ND, NG = Tab<DEG>::NG;
  __shared__ Tab<DEG> T;
  tab_init(T);
  const int64_t n = ne * NG * ND;
  for (int64_t t = gtid(); t < n; t += gstride()) {
    const int64_t gp = t / ND;
    const int p = (int)(t - gp * ND);
    const int64_t e = gp / NG;
    const int k = (int)(gp - e * NG);
    const double w = weight_at(T, k, area[e]);
    const double c = coef[gp];
    int32_t d[ND];
#pragma unroll
    for (int q = 0; q < ND; q++) d[q] = dof[ND * e + q];
    const int32_t dp = dof[ND * e + p];
    double2 g[3];
    double px = 0.0, py = 0.0;
    if (OP == (int)GenOp::LAPLACE) {
      load_grad(grad, e, g);
      grad_at(T, k, p, g, px, py);
    }
    const int64_t base = t * ND;
#pragma unroll
    for (int q = 0; q < ND; q++) {
      double v;
      if (OP == (int)GenOp::LAPLACE) {
        double qx, qy;
        grad_at(T, k, q, g, qx, qy);
        v = (px * qx + py * qy) * c * w;
      } else {
        v = T.h[k][p] * T.h[k][q] * c * w;
      }
      reinterpret_cast<longlong2*>(idx)[base + q] = make_longlong2(dp, d[q]);
      vv[base + q] = v;
    }
  }
}

// grad_coef[gp] = sum_pq grad_vv[gp, p, q] * (d N_pq / d coef): threads (gp, p) form
// the row sums, the gp's first thread adds the rows in order
template <int DEG, int OP>
__global__ void __launch_bounds__(64 * Tab<DEG>::ND) k_gen_coo_backward(int64_t ne, const double* __restrict__ area,
                                                                      const double2* __restrict__ grad,
                                                                      const double* __restrict__ gv,
                                                                      double* __restrict__ out) {
  constexpr int ND = Tab<DEG>::ND, NG = Tab<DEG>::NG;
  __shared__ Tab<DEG> T;
  __shared__ double part[64 * ND];
  tab_init(T);
  const int64_t ngp = ne * NG;
  const int64_t gp = (int64_t)blockIdx.x * 64 + threadIdx.x / ND;
  const int p = threadIdx.x % ND;
  double s = 0.0;
  if (gp < ngp) {
    const int64_t e = gp / NG;
    const int k = (int)(gp - e * NG);
    const double w = weight_at(T, k, area[e]);
    const double* row = gv + (gp * ND + p) * ND;
    if (OP == (int)GenOp::LAPLACE) {
      double2 g[3];
      load_grad(grad, e, g);
      double px, py;
      grad_at(T, k, p, g, px, py);
#pragma unroll
      for (int q = 0; q < ND; q++) {
        double qx, qy;
        grad_at(T, k, q, g, qx, qy);
        s += row[q] * ((px * qx + py * qy) * w);
      }
    } else {
#pragma unroll
      for (int q = 0; q < ND; q++) s += T.h[k][p] * T.h[k][q] * w * row[q];
    }
  }
  part[threadIdx.x] = s;
  __syncthreads();
  if (p == 0 && gp < ngp) {
    double v = 0.0;
#pragma unroll
    for (int r = 0; r < ND; r++) v += part[threadIdx.x + r];
    out[gp] = v;
  }
}

// B = [hx 0; 0 hy; hy hx] (3 x 2 nd), ComputeFemStiffnessMatrixMfem.h:18-23: column l
template <int ND>
__device__ __forceinline__ void bcol(const double (&hx)[ND], const double (&hy)[ND], int l, double& b0, double& b1,
                                     double& b2) {
  if (l < ND) {
    b0 = hx[l];
    b1 = 0.0;
    b2 = hy[l];
  } else {
    b0 = 0.0;
    b1 = hy[l - ND];
    b2 = hx[l - ND];
  }
}

// elasticity COO: thread (gp, l) writes row l of B^T K B w (2 nd entries)
template <int DEG>
__global__ void __launch_bounds__(kGT) k_gen_stiffness_coo(int64_t ne, int64_t ndof, const int32_t* __restrict__ dof,
                                                           const double* __restrict__ area,
                                                           const double2* __restrict__ grad,
                                                           const double* __restrict__ D, long long* __restrict__ idx,
                                                           double* __restrict__ vv) {
  constexpr int ND = Tab<DEG>::ND, NG = Tab<DEG>::NG, N2 = 2 * ND;
  __shared__ Tab<DEG> T;
  tab_init(T);
  const int64_t n = ne * NG * N2;
  for (int64_t t = gtid(); t < n; t += gstride()) {
    const int64_t gp = t / N2;
    const int l = (int)(t - gp * N2);
    const int64_t e = gp / NG;
    const int k = (int)(gp - e * NG);
    const double w = weight_at(T, k, area[e]);
    double2 g[3];
    load_grad(grad, e, g);
    double hx[ND], hy[ND];
#pragma unroll
    for (int r = 0; r < ND; r++) grad_at(T, k, r, g, hx[r], hy[r]);
    const double* K = D + 9 * gp;
    double b0, b1, b2;
    bcol<ND>(hx, hy, l, b0, b1, b2);
    double tq[3];
#pragma unroll
    for (int q = 0; q < 3; q++) tq[q] = b0 * K[q] + b1 * K[3 + q] + b2 * K[6 + q];
    const long long dl = (long long)dof[ND * e + (l % ND)] + (l >= ND ? ndof : 0);
    const int64_t base = t * N2;
#pragma unroll
    for (int c = 0; c < N2; c++) {
      double c0, c1, c2;
      bcol<ND>(hx, hy, c, c0, c1, c2);
      const long long dc = (long long)dof[ND * e + (c % ND)] + (c >= ND ? ndof : 0);
      reinterpret_cast<longlong2*>(idx)[base + c] = make_longlong2(dl, dc);
      vv[base + c] = (tq[0] * c0 + tq[1] * c1 + tq[2] * c2) * w;
    }
  }
}

// grad_D[gp] = w B G B^T: thread (gp, l) reads row l of G and contributes
// B[:, l] (G[l, :] B^T); the gp's threads then add the 2 nd rows, in order, for each of the nine entries
template <int DEG>
__global__ void __launch_bounds__(32 * 2 * Tab<DEG>::ND) k_gen_stiffness_coo_backward(
    int64_t ne, const double* __restrict__ area, const double2* __restrict__ grad, const double* __restrict__ gv,
    double* __restrict__ out) {
  constexpr int ND = Tab<DEG>::ND, NG = Tab<DEG>::NG, N2 = 2 * ND;
  __shared__ Tab<DEG> T;
  __shared__ double part[32 * N2][9];
  tab_init(T);
  const int64_t ngp = ne * NG;
  const int slot = threadIdx.x / N2;
  const int64_t gp = (int64_t)blockIdx.x * 32 + slot;
  const int l = threadIdx.x % N2;
  double acc[9];
#pragma unroll
  for (int j = 0; j < 9; j++) acc[j] = 0.0;
  double w = 0.0;
  if (gp < ngp) {
    const int64_t e = gp / NG;
    const int k = (int)(gp - e * NG);
    w = weight_at(T, k, area[e]);
    double2 g[3];
    load_grad(grad, e, g);
    double hx[ND], hy[ND];
#pragma unroll
    for (int r = 0; r < ND; r++) grad_at(T, k, r, g, hx[r], hy[r]);
    const double* row = gv + (gp * N2 + l) * N2;
    double u[3] = {0.0, 0.0, 0.0};  // G[l, :] B^T
#pragma unroll
    for (int c = 0; c < N2; c++) {
      double c0, c1, c2;
      bcol<ND>(hx, hy, c, c0, c1, c2);
      const double gl = row[c];
      u[0] += gl * c0;
      u[1] += gl * c1;
      u[2] += gl * c2;
    }
    double b[3];
    bcol<ND>(hx, hy, l, b[0], b[1], b[2]);
#pragma unroll
    for (int a = 0; a < 3; a++)
#pragma unroll
      for (int q = 0; q < 3; q++) acc[3 * a + q] = b[a] * u[q];
  }
#pragma unroll
  for (int j = 0; j < 9; j++) part[threadIdx.x][j] = acc[j];
  __syncthreads();
  if (gp < ngp)
    for (int j = l; j < 9; j += N2) {  // 2 nd threads per point write its 9 entries
      double v = 0.0;
      for (int r = 0; r < N2; r++) v += part[slot * N2 + r][j];
      out[9 * gp + j] = v * w;
    }
}

// ---------------------------------------------------------------- summed operators
// Gradients of every basis function at point k with compile-time indices (the P2
// vertex functions depend on one barycentric gradient, the edge functions on two).
template <int DEG>
__device__ __forceinline__ void grads_all(const Tab<DEG>& T, int k, const double2 (&g)[3],
                                          double (&hx)[Tab<DEG>::ND], double (&hy)[Tab<DEG>::ND]) {
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const double t = T.t[k][a][a];
    hx[a] = t * g[a].x;
    hy[a] = t * g[a].y;
  }
  if constexpr (DEG == 2) {
#pragma unroll
    for (int j = 0; j < 3; j++) {
      const int a = j, b = (j + 1) % 3;
      const double ta = T.t[k][3 + j][a], tb = T.t[k][3 + j][b];
      hx[3 + j] = ta * g[a].x + tb * g[b].x;
      hy[3 + j] = ta * g[a].y + tb * g[b].y;
    }
  }
}

// packed index of (a, b), a <= b, in the upper triangle of an nd x nd matrix
__host__ __device__ constexpr int sym_idx(int nd, int a, int b) { return a * nd - a * (a - 1) / 2 + (b - a); }

// Laplace / mass element matrices, one thread per element: the nd (nd + 1) / 2 distinct
// entries of sum_k coef_k w_k N_k, stored as the full nd x nd matrix of the element
// (row-major, ke[(e * nd + a) * nd + b]) so that a row gather reads one contiguous row.
template <int DEG, int OP>
__global__ void __launch_bounds__(kGT) k_gen_ke(int64_t ne, const double* __restrict__ area,
                                                const double2* __restrict__ grad, const double* __restrict__ coef,
                                                double* __restrict__ ke) {
  constexpr int ND = Tab<DEG>::ND, NG = Tab<DEG>::NG, NS = ND * (ND + 1) / 2;
  __shared__ Tab<DEG> T;
  tab_init(T);
  for (int64_t e = gtid(); e < ne; e += gstride()) {
    const double ar = area[e];
    double2 g[3];
    if (OP == (int)GenOp::LAPLACE) load_grad(grad, e, g);
    double acc[NS];
#pragma unroll
    for (int j = 0; j < NS; j++) acc[j] = 0.0;
#pragma unroll 1
    for (int k = 0; k < NG; k++) {
      const double cw = coef[NG * e + k] * weight_at(T, k, ar);
      if (OP == (int)GenOp::LAPLACE) {
        double hx[ND], hy[ND];
        grads_all(T, k, g, hx, hy);
#pragma unroll
        for (int a = 0; a < ND; a++)
#pragma unroll
          for (int b = a; b < ND; b++) acc[sym_idx(ND, a, b)] += (hx[a] * hx[b] + hy[a] * hy[b]) * cw;
      } else {
#pragma unroll
        for (int a = 0; a < ND; a++)
#pragma unroll
          for (int b = a; b < ND; b++) acc[sym_idx(ND, a, b)] += T.h[k][a] * T.h[k][b] * cw;
      }
    }
    double* out = ke + e * ND * ND;
#pragma unroll
    for (int a = 0; a < ND; a++)
#pragma unroll
      for (int b = 0; b < ND; b++) out[a * ND + b] = acc[a <= b ? sym_idx(ND, a, b) : sym_idx(ND, b, a)];
  }
}

// elasticity element matrices (2 nd x 2 nd, not symmetric for a general D): thread
// (l, e) forms row l of sum_k w_k B_k^T D_k B_k, elements fastest so that a warp shares
// l; stored row-major per element, ke[(e * 2nd + l) * 2nd + c]
template <int DEG>
__global__ void __launch_bounds__(kGT) k_gen_ke_stiffness(int64_t ne, const double* __restrict__ area,
                                                          const double2* __restrict__ grad,
                                                          const double* __restrict__ D, double* __restrict__ ke) {
  constexpr int ND = Tab<DEG>::ND, NG = Tab<DEG>::NG, N2 = 2 * ND;
  __shared__ Tab<DEG> T;
  tab_init(T);
  const int64_t n = ne * N2;
  for (int64_t t = gtid(); t < n; t += gstride()) {
    const int l = (int)(t / ne);
    const int64_t e = t - (int64_t)l * ne;
    const int r = l < ND ? l : l - ND;
    const double ar = area[e];
    double2 g[3];
    load_grad(grad, e, g);
    double row[N2];
#pragma unroll
    for (int c = 0; c < N2; c++) row[c] = 0.0;
#pragma unroll 1
    for (int k = 0; k < NG; k++) {
      const double w = weight_at(T, k, ar);
      double hx[ND], hy[ND];
      grads_all(T, k, g, hx, hy);
      double rx, ry;  // gradient of the row's own basis function
      grad_at(T, k, r, g, rx, ry);
      const double* K = D + 9 * (NG * e + k);
      // column l of B: (rx, 0, ry) for an x row, (0, ry, rx) for a y row
      const double b0 = l < ND ? rx : 0.0, b1 = l < ND ? 0.0 : ry, b2 = l < ND ? ry : rx;
      double tq[3];
#pragma unroll
      for (int q = 0; q < 3; q++) tq[q] = (b0 * K[q] + b1 * K[3 + q] + b2 * K[6 + q]) * w;
#pragma unroll
      for (int c = 0; c < ND; c++) {
        row[c] += tq[0] * hx[c] + tq[2] * hy[c];       // column (c, x): B[:, c] = (hx, 0, hy)
        row[ND + c] += tq[1] * hy[c] + tq[2] * hx[c];  // column (c, y): B[:, c + nd] = (0, hy, hx)
      }
    }
    double* out = ke + (e * N2 + l) * N2;
#pragma unroll
    for (int c = 0; c < N2; c++) out[c] = row[c];
  }
}

// Summed rows of [x; y] elasticity blocks, one thread per scalar DOF row (every FP64 add of a warp
// does 32 rows' work): the thread owns the x row at 2 rowptr[i] and the y row at 2 nnz + 2 rowptr[i],
// each with the x columns, then the y columns, of the scalar row, accumulated in a per-thread
// shared-memory buffer of CAP entries in ascending element order; transpose gives the CSC values.
// The block's rows occupy one contiguous range of each half of vals, written by the whole block in
// order.  Rows longer than the buffer are summed in place in global memory.
template <int DEG, int BT, int CAP>
__global__ void __launch_bounds__(BT) k_gen_rows(int64_t ndof, int64_t nnz, const int32_t* __restrict__ rowptr,
                                                 const int32_t* __restrict__ inc_ptr, const uint4* __restrict__ inc,
                                                 const double* __restrict__ ke, double* __restrict__ vals,
                                                 bool transpose) {
  constexpr int NB = 2, ND = Tab<DEG>::ND, KN = NB * ND;  // element matrix is KN x KN
  extern __shared__ double buf[];                 // [NB][CAP][BT]
  __shared__ int32_t srp[BT + 1];
  const int tid = threadIdx.x;
  for (int64_t i0 = (int64_t)blockIdx.x * BT; i0 < ndof; i0 += (int64_t)gridDim.x * BT) {
    const int nrow = (int)std::min<int64_t>(BT, ndof - i0);
    __syncthreads();  // previous tile's write-out done with buf / srp
    if (tid < nrow) srp[tid] = rowptr[i0 + tid];
    if (tid == 0) srp[nrow] = rowptr[i0 + nrow];
    const int64_t i = i0 + tid;
    int len = 0;
    if (tid < nrow) {
      len = rowptr[i + 1] - rowptr[i];
      const int rl = NB * len;  // entries of each of the thread's NB rows
      const bool fits = rl <= CAP;
      const int64_t gb[2] = {NB * (int64_t)rowptr[i], 2 * nnz + 2 * (int64_t)rowptr[i]};
#pragma unroll
      for (int rc = 0; rc < NB; rc++)
        for (int j = 0; j < rl; j++) {
          if (fits) buf[(rc * CAP + j) * BT + tid] = 0.0;
          else vals[gb[rc] + j] = 0.0;
        }
      for (int32_t s = inc_ptr[i]; s < inc_ptr[i + 1]; s++) {
        const uint4 r = inc[s];
        const double* K = ke + (int64_t)r.x * KN * KN;
#pragma unroll
        for (int rc = 0; rc < NB; rc++) {
          const int li = (int)r.y + rc * ND;
#pragma unroll
          for (int cb = 0; cb < NB; cb++)
#pragma unroll
            for (int b = 0; b < ND; b++) {
              const int lj = b + cb * ND;
              const double v = transpose ? K[lj * KN + li] : K[li * KN + lj];
              const int j = (int)space_off(r, b) + cb * len;
              if (fits) buf[(rc * CAP + j) * BT + tid] += v;
              else vals[gb[rc] + j] += v;
            }
        }
      }
      if (!fits) len = -1;  // written in place
    }
    __syncthreads();
    // write-out: the tile's rows of each block are contiguous in vals
    const int64_t b0 = srp[0], b1 = srp[nrow];
    for (int rc = 0; rc < NB; rc++) {
      const int64_t out0 = rc == 0 ? NB * b0 : 2 * nnz + 2 * b0;
      const int64_t total = NB * (b1 - b0);
      for (int64_t q = tid; q < total; q += BT) {
        // row of entry q: the last row whose start (in this block's entries) is <= q
        int lo = 0, hi = nrow - 1;
        while (lo < hi) {
          const int mid = (lo + hi + 1) >> 1;
          if ((int64_t)NB * (srp[mid] - b0) <= q) lo = mid;
          else hi = mid - 1;
        }
        const int rlen = NB * (srp[lo + 1] - srp[lo]);
        if (rlen > CAP) continue;  // that row was summed in place
        const int j = (int)(q - (int64_t)NB * (srp[lo] - b0));
        vals[out0 + q] = buf[(rc * CAP + j) * BT + lo];
      }
    }
  }
}

// Summed rows of a scalar operator, one thread per DOF row as above.  The rows of the element
// matrices of four incident elements are loaded before they are added (the walk is a chain of
// dependent loads), and the write-out finds the row of an entry in a table of bytes that the
// rows' threads fill, instead of a search per entry.
template <int DEG, int BT, int CAP>
__global__ void __launch_bounds__(BT) k_gen_scalar_rows(int64_t ndof, const int32_t* __restrict__ rowptr,
                                                        const int32_t* __restrict__ inc_ptr,
                                                        const uint4* __restrict__ inc, const double* __restrict__ ke,
                                                        double* __restrict__ vals) {
  constexpr int ND = Tab<DEG>::ND;
  static_assert(BT <= 256, "a row of the tile is a byte");
  __shared__ double buf[CAP][BT];
  __shared__ uint8_t owner[CAP * BT];
  const int tid = threadIdx.x;
  const int64_t i0 = (int64_t)blockIdx.x * BT, i = i0 + tid;
  const int nrow = (int)std::min<int64_t>(BT, ndof - i0);
  const int32_t b0 = rowptr[i0], total = rowptr[i0 + nrow] - b0;
  if (tid < nrow) {
    const int32_t p0 = rowptr[i], len = rowptr[i + 1] - p0;
    const bool fits = len <= CAP;
    const int32_t s0 = inc_ptr[i], s1 = inc_ptr[i + 1];
    double* row = vals + p0;
    for (int j = 0; j < len; j++) {
      if (fits) buf[j][tid] = 0.0;
      else row[j] = 0.0;
      if (p0 - b0 + j < CAP * BT) owner[p0 - b0 + j] = (uint8_t)tid;
    }
    auto load = [&](const uint4& r, double (&v)[ND]) {
      const double* K = ke + ((int64_t)r.x * ND + r.y) * ND;
      if constexpr (ND == 6) {
        load6(K, v);
      } else {
#pragma unroll
        for (int b = 0; b < ND; b++) v[b] = __ldg(K + b);
      }
    };
    auto add = [&](const uint4& r, const double (&v)[ND]) {
      // (an element's entries go to different slots: all are read before any is written, so that
      // their FP64 additions do not wait for one another: 90 -> 73 us at 641k rows of P2)
      if (fits) {
        double a[ND];
#pragma unroll
        for (int b = 0; b < ND; b++) a[b] = buf[space_off(r, b)][tid];
#pragma unroll
        for (int b = 0; b < ND; b++) buf[space_off(r, b)][tid] = a[b] + v[b];
      } else {
#pragma unroll
        for (int b = 0; b < ND; b++) row[space_off(r, b)] += v[b];
      }
    };
    constexpr int U = 4;
    for (int32_t s = s0; s < s1; s += U) {
      uint4 r[U];
      double v[U][ND];
#pragma unroll
      for (int u = 0; u < U; u++) r[u] = s + u < s1 ? inc[s + u] : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
      for (int u = 0; u < U; u++)
        if (s + u < s1) load(r[u], v[u]);
#pragma unroll
      for (int u = 0; u < U; u++)
        if (s + u < s1) add(r[u], v[u]);
    }
  }
  __syncthreads();
  for (int32_t q = tid; q < total; q += BT) {
    int r = nrow - 1;
    if (q < CAP * BT) {
      r = owner[q];
    } else {  // (only where rows longer than the buffer make the tile longer than the table)
      while (r > 0 && rowptr[i0 + r] - b0 > q) r--;
    }
    const int32_t p0 = rowptr[i0 + r];
    if (rowptr[i0 + r + 1] - p0 > CAP) continue;  // that row was summed in place
    vals[b0 + q] = buf[q - (p0 - b0)][r];
  }
}

// ---------------------------------------------------------------- load vector
template <int DEG>
__global__ void __launch_bounds__(kGT) k_gen_source(int64_t ndof, const int32_t* __restrict__ inc_ptr,
                                                    const uint4* __restrict__ inc, const double* __restrict__ area,
                                                    const double* __restrict__ f, double* __restrict__ rhs,
                                                    bool accumulate) {
  constexpr int NG = Tab<DEG>::NG;
  __shared__ Tab<DEG> T;
  tab_init(T);
  for (int64_t i = gtid(); i < ndof; i += gstride()) {
    double acc = accumulate ? rhs[i] : 0.0;
    for (int32_t s = inc_ptr[i]; s < inc_ptr[i + 1]; s++) {
      const uint4 r = inc[s];
      acc = fma(area[r.x], point_sum<NG>(f + (int64_t)r.x * NG, [&](int k) { return T.hw[k][r.y]; }), acc);
    }
    rhs[i] = acc;
  }
}

template <int DEG>
__global__ void __launch_bounds__(kGT) k_gen_source_backward(int64_t ne, const int32_t* __restrict__ dof,
                                                             const double* __restrict__ area,
                                                             const double* __restrict__ grhs,
                                                             double* __restrict__ gf) {
  constexpr int ND = Tab<DEG>::ND, NG = Tab<DEG>::NG;
  __shared__ Tab<DEG> T;
  tab_init(T);
  for (int64_t gp = gtid(); gp < ne * NG; gp += gstride()) {
    const int64_t e = gp / NG;
    const int k = (int)(gp - e * NG);
    const double w = weight_at(T, k, area[e]);
    double v = 0.0;
#pragma unroll
    for (int r = 0; r < ND; r++) v += T.h[k][r] * w * grhs[dof[ND * e + r]];
    gf[gp] = v;
  }
}

// ---------------------------------------------------------------- interpolation
template <int DEG, bool VERT>
__global__ void __launch_bounds__(kGT) k_gen_to_gauss(int64_t ne, const int4* __restrict__ conn,
                                                      const int32_t* __restrict__ dof, const double* __restrict__ u,
                                                      double* __restrict__ out) {
  constexpr int ND = Tab<DEG>::ND, NG = Tab<DEG>::NG;
  __shared__ Tab<DEG> T;
  tab_init(T);
  for (int64_t gp = gtid(); gp < ne * NG; gp += gstride()) {
    const int64_t e = gp / NG;
    const int k = (int)(gp - e * NG);
    double v;
    if (VERT) {
      const int4 c = conn[e];
      v = u[c.x] * T.l[k][0] + u[c.y] * T.l[k][1] + u[c.z] * T.l[k][2];
    } else {
      v = 0.0;
#pragma unroll
      for (int r = 0; r < ND; r++) v += u[dof[ND * e + r]] * T.h[k][r];
    }
    out[gp] = v;
  }
}

// transposes: VERT walks the vertex->element incidence of the mesh (local vertex in
// the low bits of the record), else the space's DOF->element incidence
template <int DEG, bool VERT>
__global__ void __launch_bounds__(kGT) k_gen_to_gauss_backward(int64_t nrow, const int32_t* __restrict__ inc_ptr,
                                                               const void* __restrict__ incp,
                                                               const double* __restrict__ gout,
                                                               double* __restrict__ gu, bool accumulate) {
  constexpr int NG = Tab<DEG>::NG;
  __shared__ Tab<DEG> T;
  tab_init(T);
  for (int64_t i = gtid(); i < nrow; i += gstride()) {
    double acc = accumulate ? gu[i] : 0.0;
    for (int32_t s = inc_ptr[i]; s < inc_ptr[i + 1]; s++) {
      int64_t e;
      int a;
      if (VERT) {
        const uint2 r = reinterpret_cast<const uint2*>(incp)[s];
        e = r.x;
        a = (int)inc_a(r.y);
      } else {
        const uint4 r = reinterpret_cast<const uint4*>(incp)[s];
        e = r.x;
        a = (int)r.y;
      }
      acc += point_sum<NG>(gout + e * NG, [&](int k) { return VERT ? T.l[k][a] : T.h[k][a]; });
    }
    gu[i] = acc;
  }
}

// ---------------------------------------------------------------- resident P2 systems
// Poisson system rows of a degree-DEG space: one thread per DOF row i (space order), the
// row summed from the element matrices ke in ascending element order, the load
// sum_e sum_k f_k phi_a(x_k) w_k over the same incidence, and the Dirichlet condition
// applied as by the P1 system kernel: a Dirichlet row (tag 1) becomes the identity row
// with rhs = bdval; a row next to Dirichlet DOFs (tag 2) moves those columns into the
// right-hand side lift.  Values go to the system's sliced-ELL operator: row nperm[i],
// slot kperm[rowptr[i] + k] (identity without renumbering); isbd, bdval, rhs in solver
// order.  Deterministic: every value is summed by one thread in a fixed order.
template <int DEG, int MAXW>
__global__ void __launch_bounds__(kRowBTs) k_gen_poisson_rows(
    int64_t ndof, const int32_t* __restrict__ rowptr, const int32_t* __restrict__ colind,
    const int32_t* __restrict__ inc_ptr, const uint4* __restrict__ inc, const double* __restrict__ area,
    const double* __restrict__ ke, const double* __restrict__ f, const int32_t* __restrict__ sptr,
    const uint8_t* __restrict__ isbd, const double* __restrict__ bdval, double* __restrict__ vals,
    double* __restrict__ rhs, const int32_t* __restrict__ nperm, const uint8_t* __restrict__ kperm,
    const int32_t* __restrict__ diagpos) {
  constexpr int ND = Tab<DEG>::ND, NG = Tab<DEG>::NG;
  __shared__ Tab<DEG> T;
  __shared__ double acc[MAXW][kRowBTs];
  tab_init(T);
  const int t = threadIdx.x;
  const int64_t i = (int64_t)blockIdx.x * kRowBTs + t;
  if (i >= ndof) return;
  const int32_t r0 = rowptr[i];
  const int w = rowptr[i + 1] - r0;
  const int64_t ri = nperm ? (int64_t)nperm[i] : i;
  const int64_t base = (int64_t)sptr[ri >> 5] + (ri & 31);
  const uint8_t tag = isbd[ri];
  auto slot = [&](int k) -> int64_t { return base + 32 * (int64_t)(kperm ? (int)kperm[r0 + k] : k); };
  if (tag == 1) {
    const int dp = diagpos[i];
    for (int k = 0; k < w; k++) vals[slot(k)] = (k == dp) ? 1.0 : 0.0;
    rhs[ri] = bdval[ri];
    return;
  }
  for (int k = 0; k < w; k++) acc[k][t] = 0.0;
  double r = 0.0;
  for (int32_t s = inc_ptr[i]; s < inc_ptr[i + 1]; s++) {
    const uint4 rec = inc[s];
    const int a = (int)rec.y;
    double K[ND];
    if constexpr (ND == 6) {
      load6(ke + ((int64_t)rec.x * ND + a) * ND, K);
    } else {
#pragma unroll
      for (int b = 0; b < ND; b++) K[b] = __ldg(ke + ((int64_t)rec.x * ND + a) * ND + b);
    }
    // (different slots: read before any is written)
    double old[ND];
    bool in = true;
#pragma unroll
    for (int b = 0; b < ND; b++) {
      const unsigned o = space_off(rec, b);
      in &= ADFEM_DCHECK(o < (unsigned)w && o < (unsigned)MAXW);
    }
    if (in) {
#pragma unroll
      for (int b = 0; b < ND; b++) old[b] = acc[space_off(rec, b)][t];
#pragma unroll
      for (int b = 0; b < ND; b++) acc[space_off(rec, b)][t] = old[b] + K[b];
    }
    r = fma(area[rec.x], point_sum<NG>(f + (int64_t)rec.x * NG, [&](int k) { return T.hw[k][a]; }), r);
  }
  if (tag == 2) {
    for (int k = 0; k < w; k++) {
      const int64_t j = nperm ? (int64_t)nperm[colind[r0 + k]] : (int64_t)colind[r0 + k];
      if (isbd[j] == 1) {
        r = fma(-acc[k][t], bdval[j], r);
        acc[k][t] = 0.0;
      }
    }
  }
  rhs[ri] = r;
  for (int k = 0; k < w; k++) vals[slot(k)] = acc[k][t];
}

// dL/dkappa at Gauss point k of element e for the resident system: -w_k grad(lam).grad(u)
// at x_k, lam zero on the Dirichlet DOFs (isbd_ref in space order) -- the composition of
// the sparse-solve gradient (-lam_i u_j per entry), the Dirichlet backward and the
// FemLaplaceScalar backward, with the element matrix's rank-one structure per point.
template <int DEG>
__global__ void __launch_bounds__(kGT) k_gen_kappa_grad(int64_t ne, const int32_t* __restrict__ dof,
                                                        const double* __restrict__ area,
                                                        const double2* __restrict__ grad,
                                                        const double* __restrict__ u, const double* __restrict__ lam,
                                                        const uint8_t* __restrict__ isbd, double* __restrict__ gk) {
  constexpr int ND = Tab<DEG>::ND, NG = Tab<DEG>::NG;
  __shared__ Tab<DEG> T;
  tab_init(T);
  for (int64_t gp = gtid(); gp < ne * NG; gp += gstride()) {
    const int64_t e = gp / NG;
    const int k = (int)(gp - e * NG);
    double2 g[3];
    load_grad(grad, e, g);
    double hx[ND], hy[ND];
    grads_all(T, k, g, hx, hy);
    double ux = 0.0, uy = 0.0, lx = 0.0, ly = 0.0;
#pragma unroll
    for (int b = 0; b < ND; b++) {
      const int32_t d = dof[ND * e + b];
      const double ub = u[d];
      const double lb = isbd[d] == 1 ? 0.0 : lam[d];
      ux = fma(hx[b], ub, ux);
      uy = fma(hy[b], ub, uy);
      lx = fma(hx[b], lb, lx);
      ly = fma(hy[b], lb, ly);
    }
    gk[gp] = -weight_at(T, k, area[e]) * fma(lx, ux, ly * uy);
  }
}

// ---------------------------------------------------------------- PCL
__global__ void __launch_bounds__(kGT) k_fill(int64_t n, double v, double* __restrict__ out) {
  for (int64_t i = gtid(); i < n; i += gstride()) out[i] = v;
}

// H[gp + nz * ng] = vv[nz] for the nd^2 entries nz of Gauss point gp (column-major
// ngauss x nd^2 ngauss, pcl_FemLaplaceScalar_Jacobian, FemLaplaceScalar.h:63-91)
__global__ void __launch_bounds__(kGT) k_pcl_scatter(int64_t N, int nd2, int64_t ng, const double* __restrict__ vv,
                                                     double* __restrict__ H) {
  for (int64_t nz = gtid(); nz < N; nz += gstride()) H[nz / nd2 + nz * ng] = vv[nz];
}

}  // namespace

cudaError_t launch_fill(int64_t n, double v, double* out, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  k_fill<<<grid_for(n), kGT, 0, st>>>(n, v, out);
  return cudaGetLastError();
}

cudaError_t launch_pcl_scatter(int64_t N, int nd2, int64_t ng, const double* vv, double* H, cudaStream_t st) {
  if (N <= 0) return cudaSuccess;
  k_pcl_scatter<<<grid_for(N), kGT, 0, st>>>(N, nd2, ng, vv, H);
  return cudaGetLastError();
}

// ---------------------------------------------------------------- launchers
#define GEN_DISPATCH(sp, KERNEL_CALL1, KERNEL_CALL2) \
  do {                                               \
    if ((sp).degree == 2) {                          \
      KERNEL_CALL2;                                  \
    } else {                                         \
      KERNEL_CALL1;                                  \
    }                                                \
  } while (0)

cudaError_t launch_gen_coo(const Mesh& m, const Space& sp, GenOp op, const double* coef, long long* indices,
                           double* vv, cudaStream_t st) {
  const int64_t n = m.ne * sp.ng * sp.nd;
  const int g = grid_for(n);
  const int32_t* dof = sp.d_dof.as<int32_t>();
  const double* area = sp.d_area.as<double>();
  const double2* grad = m.d_grad.as<double2>();
  if (op == GenOp::LAPLACE)
    GEN_DISPATCH(sp, (k_gen_coo<1, 0><<<g, kGT, 0, st>>>(m.ne, dof, area, grad, coef, indices, vv)),
                 (k_p2_coo<<<grid_for(6 * m.ne, kCooPts), kCooT, 0, st>>>(m.ne, dof, area, grad, coef,
                                                                       reinterpret_cast<longlong2*>(indices), vv)));
  else
    GEN_DISPATCH(sp, (k_gen_coo<1, 1><<<g, kGT, 0, st>>>(m.ne, dof, area, grad, coef, indices, vv)),
                 (k_gen_coo<2, 1><<<g, kGT, 0, st>>>(m.ne, dof, area, grad, coef, indices, vv)));
  return cudaGetLastError();
}

cudaError_t launch_gen_coo_backward(const Mesh& m, const Space& sp, GenOp op, const double* grad_vv, double* grad_coef,
                                    cudaStream_t st) {
  const int64_t ngp = m.ne * sp.ng;
  if (ngp == 0) return cudaSuccess;
  const int g = (int)((ngp + 63) / 64);
  const double* area = sp.d_area.as<double>();
  const double2* grad = m.d_grad.as<double2>();
  if (op == GenOp::LAPLACE)
    GEN_DISPATCH(sp, (k_gen_coo_backward<1, 0><<<g, 64 * 3, 0, st>>>(m.ne, area, grad, grad_vv, grad_coef)),
                 (k_p2_coo_backward<<<grid_for(ngp, kCooPts), kCooT, 0, st>>>(m.ne, area, grad, grad_vv, grad_coef)));
  else
    GEN_DISPATCH(sp, (k_gen_coo_backward<1, 1><<<g, 64 * 3, 0, st>>>(m.ne, area, grad, grad_vv, grad_coef)),
                 (k_gen_coo_backward<2, 1><<<g, 64 * 6, 0, st>>>(m.ne, area, grad, grad_vv, grad_coef)));
  return cudaGetLastError();
}

cudaError_t launch_gen_stiffness_coo(const Mesh& m, const Space& sp, const double* D, long long* indices, double* vv,
                                     cudaStream_t st) {
  const int g = grid_for(m.ne * sp.ng * 2 * sp.nd);
  const int32_t* dof = sp.d_dof.as<int32_t>();
  const double* area = sp.d_area.as<double>();
  const double2* grad = m.d_grad.as<double2>();
  GEN_DISPATCH(sp, (k_gen_stiffness_coo<1><<<g, kGT, 0, st>>>(m.ne, sp.ndof, dof, area, grad, D, indices, vv)),
               (k_gen_stiffness_coo<2><<<g, kGT, 0, st>>>(m.ne, sp.ndof, dof, area, grad, D, indices, vv)));
  return cudaGetLastError();
}

cudaError_t launch_gen_stiffness_coo_backward(const Mesh& m, const Space& sp, const double* grad_vv, double* grad_D,
                                              cudaStream_t st) {
  const int64_t ngp = m.ne * sp.ng;
  if (ngp == 0) return cudaSuccess;
  const int g = (int)((ngp + 31) / 32);
  const double* area = sp.d_area.as<double>();
  const double2* grad = m.d_grad.as<double2>();
  GEN_DISPATCH(sp, (k_gen_stiffness_coo_backward<1><<<g, 32 * 6, 0, st>>>(m.ne, area, grad, grad_vv, grad_D)),
               (k_gen_stiffness_coo_backward<2><<<g, 32 * 12, 0, st>>>(m.ne, area, grad, grad_vv, grad_D)));
  return cudaGetLastError();
}

constexpr int kRowBT = 128;     // rows per block of the row gathers
constexpr int kRowCap0 = 20;    // buffered entries per scalar row (P2 vertices of valence up to 6: 19)
constexpr int kRowCap1 = 32;    // the same for longer rows
constexpr int kRowCap2 = 48;    // buffered entries per elasticity row (x and y columns)

// element matrices of the space's operator
static void launch_ke(const Mesh& m, const Space& sp, GenOp op, const double* coef, double* ke, cudaStream_t st) {
  const int g = grid_for(m.ne);
  const double* area = sp.d_area.as<double>();
  const double2* grad = m.d_grad.as<double2>();
  const double4* geo = m.d_geo.as<double4>();
  if (op == GenOp::LAPLACE)
    GEN_DISPATCH(sp, (k_gen_ke<1, 0><<<g, kGT, 0, st>>>(m.ne, area, grad, coef, ke)),
                 (k_p2_ke<0><<<g, kGT, 0, st>>>(m.ne, geo, area, coef, ke)));
  else
    GEN_DISPATCH(sp, (k_gen_ke<1, 1><<<g, kGT, 0, st>>>(m.ne, area, grad, coef, ke)),
                 (k_p2_ke<1><<<g, kGT, 0, st>>>(m.ne, geo, area, coef, ke)));
}

cudaError_t launch_gen_matrix(const Mesh& m, const Space& sp, GenOp op, const double* coef, double* ke, double* vals,
                              bool transpose, cudaStream_t st) {
  (void)transpose;  // Laplace and mass element matrices are symmetric: CSR and CSC values agree
  launch_ke(m, sp, op, coef, ke, st);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  const int32_t* rp = sp.d_rowptr.as<int32_t>();
  const int32_t* ip = sp.d_inc_ptr.as<int32_t>();
  const uint4* inc = sp.d_inc.as<uint4>();
  const unsigned gr = (unsigned)((sp.ndof + kRowBT - 1) / kRowBT);
  // (the smaller buffer where it holds every row: a third more blocks fit an SM)
  if (sp.maxrow <= kRowCap0)
    GEN_DISPATCH(sp, (k_gen_scalar_rows<1, kRowBT, kRowCap0><<<gr, kRowBT, 0, st>>>(sp.ndof, rp, ip, inc, ke, vals)),
                 (k_gen_scalar_rows<2, kRowBT, kRowCap0><<<gr, kRowBT, 0, st>>>(sp.ndof, rp, ip, inc, ke, vals)));
  else
    GEN_DISPATCH(sp, (k_gen_scalar_rows<1, kRowBT, kRowCap1><<<gr, kRowBT, 0, st>>>(sp.ndof, rp, ip, inc, ke, vals)),
                 (k_gen_scalar_rows<2, kRowBT, kRowCap1><<<gr, kRowBT, 0, st>>>(sp.ndof, rp, ip, inc, ke, vals)));
  return cudaGetLastError();
}

cudaError_t launch_gen_poisson_system(const Mesh& m, const Space& sp, const double* kappa, const double* f, double* ke,
                                      const uint8_t* isbd, const double* bdval, double* sell_vals, double* rhs,
                                      const int32_t* sptr, const int32_t* diagpos_space, const int32_t* nperm,
                                      const uint8_t* kperm, cudaStream_t st) {
  const double* area = sp.d_area.as<double>();
  launch_ke(m, sp, GenOp::LAPLACE, kappa, ke, st);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  // (P2 rows of a triangle mesh: 19 entries for a vertex of valence 6, 25 for valence 8)
  if (sp.maxrow > 32) return cudaErrorNotSupported;
  const unsigned gr = (unsigned)((sp.ndof + kRowBTs - 1) / kRowBTs);
  const int32_t* rp = sp.d_rowptr.as<int32_t>();
  const int32_t* ci = sp.d_colind.as<int32_t>();
  const int32_t* ip = sp.d_inc_ptr.as<int32_t>();
  const uint4* inc = sp.d_inc.as<uint4>();
#define ADFEM_GPR(DEG, W)                                                                                        \
  k_gen_poisson_rows<DEG, W><<<gr, kRowBTs, 0, st>>>(sp.ndof, rp, ci, ip, inc, area, ke, f, sptr, isbd, bdval, \
                                                     sell_vals, rhs, nperm, kperm, diagpos_space)
  if (sp.maxrow <= 24) GEN_DISPATCH(sp, (ADFEM_GPR(1, 24)), (ADFEM_GPR(2, 24)));
  else GEN_DISPATCH(sp, (ADFEM_GPR(1, 32)), (ADFEM_GPR(2, 32)));
#undef ADFEM_GPR
  return cudaGetLastError();
}

cudaError_t launch_gen_kappa_grad(const Mesh& m, const Space& sp, const double* u, const double* lam,
                                  const uint8_t* isbd_space, double* grad_kappa, cudaStream_t st) {
  const int g = grid_for(m.ne * sp.ng);
  const int32_t* dof = sp.d_dof.as<int32_t>();
  const double* area = sp.d_area.as<double>();
  const double2* grad = m.d_grad.as<double2>();
  GEN_DISPATCH(sp, (k_gen_kappa_grad<1><<<g, kGT, 0, st>>>(m.ne, dof, area, grad, u, lam, isbd_space, grad_kappa)),
               (k_gen_kappa_grad<2><<<g, kGT, 0, st>>>(m.ne, dof, area, grad, u, lam, isbd_space, grad_kappa)));
  return cudaGetLastError();
}

cudaError_t launch_gen_stiffness_matrix(const Mesh& m, const Space& sp, const double* D, double* ke, double* vals,
                                        bool transpose, cudaStream_t st) {
  const int g = grid_for(m.ne * 2 * sp.nd);
  const double* area = sp.d_area.as<double>();
  const double2* grad = m.d_grad.as<double2>();
  GEN_DISPATCH(sp, (k_gen_ke_stiffness<1><<<g, kGT, 0, st>>>(m.ne, area, grad, D, ke)),
               (k_gen_ke_stiffness<2><<<g, kGT, 0, st>>>(m.ne, area, grad, D, ke)));
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  static std::once_flag once;
  std::call_once(once, [] {
    const int bytes = (int)(sizeof(double) * 2 * kRowCap2 * kRowBT);
    cudaFuncSetAttribute(k_gen_rows<1, kRowBT, kRowCap2>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    cudaFuncSetAttribute(k_gen_rows<2, kRowBT, kRowCap2>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  });
  const int gr = grid_for(sp.ndof, kRowBT);
  const size_t smem = sizeof(double) * 2 * kRowCap2 * kRowBT;
  const int32_t* rp = sp.d_rowptr.as<int32_t>();
  const int32_t* ip = sp.d_inc_ptr.as<int32_t>();
  const uint4* inc = sp.d_inc.as<uint4>();
  GEN_DISPATCH(sp,
               (k_gen_rows<1, kRowBT, kRowCap2><<<gr, kRowBT, smem, st>>>(sp.ndof, sp.nnz, rp, ip, inc, ke, vals,
                                                                              transpose)),
               (k_gen_rows<2, kRowBT, kRowCap2><<<gr, kRowBT, smem, st>>>(sp.ndof, sp.nnz, rp, ip, inc, ke, vals,
                                                                              transpose)));
  return cudaGetLastError();
}

cudaError_t launch_gen_source(const Mesh& m, const Space& sp, const double* f, double* rhs, bool accumulate,
                              cudaStream_t st) {
  const int g = grid_for(sp.ndof);
  const int32_t* ip = sp.d_inc_ptr.as<int32_t>();
  const uint4* inc = sp.d_inc.as<uint4>();
  const double* area = sp.d_area.as<double>();
  GEN_DISPATCH(sp, (k_gen_source<1><<<g, kGT, 0, st>>>(sp.ndof, ip, inc, area, f, rhs, accumulate)),
               (k_gen_source<2><<<g, kGT, 0, st>>>(sp.ndof, ip, inc, area, f, rhs, accumulate)));
  return cudaGetLastError();
}

cudaError_t launch_gen_source_backward(const Mesh& m, const Space& sp, const double* grad_rhs, double* grad_f,
                                       cudaStream_t st) {
  const int g = grid_for(m.ne * sp.ng);
  const int32_t* dof = sp.d_dof.as<int32_t>();
  const double* area = sp.d_area.as<double>();
  GEN_DISPATCH(sp, (k_gen_source_backward<1><<<g, kGT, 0, st>>>(m.ne, dof, area, grad_rhs, grad_f)),
               (k_p2_to_gauss<true><<<grid_for(m.ne), kGT, 0, st>>>(m.ne, dof, area, grad_rhs, grad_f)));
  return cudaGetLastError();
}

cudaError_t launch_gen_to_gauss(const Mesh& m, const Space& sp, bool vertex_only, const double* u, double* out,
                                cudaStream_t st) {
  const int g = grid_for(m.ne * sp.ng);
  const int4* conn = m.d_conn.as<int4>();
  const int32_t* dof = sp.d_dof.as<int32_t>();
  if (vertex_only)
    GEN_DISPATCH(sp, (k_gen_to_gauss<1, true><<<g, kGT, 0, st>>>(m.ne, conn, dof, u, out)),
                 (k_gen_to_gauss<2, true><<<g, kGT, 0, st>>>(m.ne, conn, dof, u, out)));
  else
    GEN_DISPATCH(sp, (k_gen_to_gauss<1, false><<<g, kGT, 0, st>>>(m.ne, conn, dof, u, out)),
                 (k_p2_to_gauss<false><<<grid_for(m.ne), kGT, 0, st>>>(m.ne, dof, nullptr, u, out)));
  return cudaGetLastError();
}

cudaError_t launch_gen_to_gauss_backward(const Mesh& m, const Space& sp, bool vertex_only, const double* grad_out,
                                         double* grad_u, bool accumulate, cudaStream_t st) {
  if (vertex_only) {
    const int g = grid_for(m.nv);
    const int32_t* ip = m.d_inc_ptr.as<int32_t>();
    const void* inc = m.d_inc.p;
    GEN_DISPATCH(sp, (k_gen_to_gauss_backward<1, true><<<g, kGT, 0, st>>>(m.nv, ip, inc, grad_out, grad_u, accumulate)),
                 (k_gen_to_gauss_backward<2, true><<<g, kGT, 0, st>>>(m.nv, ip, inc, grad_out, grad_u, accumulate)));
  } else {
    const int g = grid_for(sp.ndof);
    const int32_t* ip = sp.d_inc_ptr.as<int32_t>();
    const void* inc = sp.d_inc.p;
    GEN_DISPATCH(sp,
                 (k_gen_to_gauss_backward<1, false><<<g, kGT, 0, st>>>(sp.ndof, ip, inc, grad_out, grad_u, accumulate)),
                 (k_gen_to_gauss_backward<2, false><<<g, kGT, 0, st>>>(sp.ndof, ip, inc, grad_out, grad_u, accumulate)));
  }
  return cudaGetLastError();
}

ADFEM_CHECK_READER(check_line_generic)

}  // namespace adfem
