// Plane-strain material and 2-D linear-elasticity assembly for P1 triangles (sm_103a).
//
// Element matrix (ComputeFemStiffnessMatrixMfem.h:4-48): K_e = sum_k w B^T D_k B with
// B = [hx 0; 0 hy; hy hx] (3 x 6) and DOFs [u_x of the 3 vertices; u_y of the 3].
// For P1 B is constant over the element, so K_e = B^T Dbar_e B with
// Dbar_e = w sum_k D_k, formed once per element by a prepass.  Rows are then
// assembled like the scalar operator: one thread per matrix row walks the
// elements around its node in ascending element order, so each value is summed
// by one thread in a fixed order (bit-reproducible, no atomics).
#include "adfem_internal.h"
#include "elastic.cuh"

namespace adfem {

static constexpr int kB = 128;
__device__ __forceinline__ int64_t gtid() { return (int64_t)blockIdx.x * blockDim.x + threadIdx.x; }
static inline unsigned nblk(int64_t n, int b) { return (unsigned)((n + b - 1) / b); }

// ---------------------------------------------------------------------------
// PlaneStrainAndStress.h:5-78.  FP64 divisions (about ten operations each) bound these kernels:
// one reciprocal per point instead of two to four quotients; the nine entries of a point are
// written (read) in order by the whole block.
__global__ void __launch_bounds__(256) k_plane_strain(int mode, int64_t n, const double* __restrict__ E,
                                                      const double* __restrict__ nu, double* __restrict__ D) {
  __shared__ double sv[256][3];  // diagonal, off-diagonal, last entry
  const int64_t i0 = (int64_t)blockIdx.x * 256;
  const int np = (int)min((int64_t)256, n - i0);
  if ((int)threadIdx.x < np) {
    const double e = E[i0 + threadIdx.x], v = nu[i0 + threadIdx.x];
    const double d = 1 - 2 * v, s = e / ((1 + v) * d);
    sv[threadIdx.x][0] = s * (1 - v);
    sv[threadIdx.x][1] = s * v;
    sv[threadIdx.x][2] = mode == 0 ? s * (1 - v) : s * d / 2.0;
  }
  __syncthreads();
  for (int q = threadIdx.x; q < 9 * np; q += 256) {
    const int p = q / 9, m = q - 9 * p;
    double v = sv[p][m == 8 ? 2 : (m % 4 == 0 ? 0 : 1)];
    if (mode != 0 && (m == 2 || (m >= 5 && m <= 7))) v = 0.0;
    D[9 * i0 + q] = v;
  }
}

// derivative of the entries above (the reference obtains it with an AD tape)
__global__ void __launch_bounds__(256) k_plane_strain_backward(int mode, int64_t n, const double* __restrict__ g,
                                                               const double* __restrict__ E,
                                                               const double* __restrict__ nu, double* __restrict__ gE,
                                                               double* __restrict__ gnu) {
  __shared__ double sv[9 * 256];
  const int64_t i0 = (int64_t)blockIdx.x * 256;
  const int np = (int)min((int64_t)256, n - i0);
  for (int q = threadIdx.x; q < 9 * np; q += 256) sv[q] = __ldcs(g + 9 * i0 + q);
  __syncthreads();
  if ((int)threadIdx.x >= np) return;
  const int64_t i = i0 + threadIdx.x;
  const double* q = sv + 9 * threadIdx.x;
  const double v = nu[i], r = 1.0 / ((1 + v) * (1 - 2 * v)), er2 = E[i] * r * r;
  if (mode == 0) {
    const double gd = q[0] + q[4] + q[8];
    const double go = q[1] + q[2] + q[3] + q[5] + q[6] + q[7];
    gE[i] = (gd * (1 - v) + go * v) * r;
    gnu[i] = er2 * (gd * 2 * v * (2 - v) + go * (1 + 2 * v * v));
  } else {
    const double a = q[0] + q[4], b = q[1] + q[3], c = q[8], d = 1 - 2 * v;
    gE[i] = (a * (1 - v) + b * v + c * d / 2.0) * r;
    gnu[i] = er2 * (a * 2 * v * (2 - v) + b * (1 + 2 * v * v) - c * 0.5 * d * d);
  }
}

cudaError_t launch_plane_strain(int mode, int64_t n, const double* E, const double* nu, double* D, cudaStream_t st) {
  k_plane_strain<<<nblk(n, 256), 256, 0, st>>>(mode, n, E, nu, D);
  return cudaGetLastError();
}
cudaError_t launch_plane_strain_backward(int mode, int64_t n, const double* g, const double* E, const double* nu,
                                         double* gE, double* gnu, cudaStream_t st) {
  k_plane_strain_backward<<<nblk(n, 256), 256, 0, st>>>(mode, n, g, E, nu, gE, gnu);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Dbar_e = w * (D_0 + D_1 + D_2), 9 values per element
__global__ void k_stiffness_prepass(int64_t ne, const double* __restrict__ D, const double4* __restrict__ geo,
                                    double* __restrict__ Dbar) {
  const int64_t t = gtid();
  if (t >= 9 * ne) return;
  const int64_t e = t / 9;
  const int j = (int)(t - 9 * e);
  const double* d = D + 27 * e + j;
  Dbar[t] = geo[e].w * (d[0] + d[9] + d[18]);
}

// fused material: D_k = plane_strain(E_k, nu_k) (mode 0), Dbar as above
__global__ void k_stiffness_prepass_E(int64_t ne, const double* __restrict__ E, const double* __restrict__ nu,
                                      const double4* __restrict__ geo, double* __restrict__ Dbar) {
  const int64_t e = gtid();
  if (e >= ne) return;
  double sd = 0.0, so = 0.0;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const double ev = E[3 * e + k], v = nu[3 * e + k];
    const double s = ev * (1 - v) / (1 + v) / (1 - 2 * v);
    sd += s;
    so += s * v / (1 - v);
  }
  const double w = geo[e].w;
  sd *= w;
  so *= w;
  double* o = Dbar + 9 * e;
  o[0] = sd; o[1] = so; o[2] = so;
  o[3] = so; o[4] = sd; o[5] = so;
  o[6] = so; o[7] = so; o[8] = sd;
}

cudaError_t launch_stiffness_prepass(const Mesh& m, const double* D, double* Dbar, cudaStream_t st) {
  k_stiffness_prepass<<<nblk(9 * m.ne, 256), 256, 0, st>>>(m.ne, D, m.d_geo.as<double4>(), Dbar);
  return cudaGetLastError();
}
cudaError_t launch_stiffness_prepass_E(const Mesh& m, const double* E, const double* nu, double* Dbar,
                                       cudaStream_t st) {
  k_stiffness_prepass_E<<<nblk(m.ne, 256), 256, 0, st>>>(m.ne, E, nu, m.d_geo.as<double4>(), Dbar);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// One element's contribution to matrix row (c, a): local DOF l = a + 3c of element e,
// added to acc at slot offsets: x-column of vertex b -> ox(b), y-column -> oy(b).
// v = B(:,l)^T Dbar (or Dbar B(:,l) for the transpose), then entry(col) = v . B(:,col).
struct RowSlots {
  int x[3], y[3];
};

template <bool TRANSPOSE, int BT = kB>
__device__ __forceinline__ void elastic_row_add(const double* __restrict__ Db, const double2* __restrict__ gr, int a,
                                                int c, const RowSlots& sl, double (*acc)[BT], int t) {
  double d[9];
#pragma unroll
  for (int j = 0; j < 9; j++) d[j] = TRANSPOSE ? Db[(j % 3) * 3 + (j / 3)] : Db[j];
  const double2 ga = gr[a];
  double v0, v1, v2;
  if (c == 0) {  // B(:,a) = (hx_a, 0, hy_a)
    v0 = fma(ga.x, d[0], ga.y * d[6]);
    v1 = fma(ga.x, d[1], ga.y * d[7]);
    v2 = fma(ga.x, d[2], ga.y * d[8]);
  } else {  // B(:,a+3) = (0, hy_a, hx_a)
    v0 = fma(ga.y, d[3], ga.x * d[6]);
    v1 = fma(ga.y, d[4], ga.x * d[7]);
    v2 = fma(ga.y, d[5], ga.x * d[8]);
  }
  // (the six slots differ: read before any is written, their chains run side by side)
  double ax[3], ay[3];
#pragma unroll
  for (int b = 0; b < 3; b++) {
    ax[b] = acc[sl.x[b]][t];
    ay[b] = acc[sl.y[b]][t];
  }
#pragma unroll
  for (int b = 0; b < 3; b++) {
    const double2 gb = gr[b];
    acc[sl.x[b]][t] = fma(v0, gb.x, fma(v2, gb.y, ax[b]));
    acc[sl.y[b]][t] = fma(v1, gb.y, fma(v2, gb.x, ay[b]));
  }
}

// Reference [x-block; y-block] ordering, CSR rows r in [0, 2nv): node i = r mod nv,
// component c = r / nv.  Row r holds the scalar row of i twice: x columns then
// y columns.  Row pointer: x-rows at 2 rowptr[i], y-rows at 2 nnz + 2 rowptr[i].
// BT threads per block: kB for rows of up to 16 scalar entries; meshes with vertices of up
// to 63 neighbours (the most mesh_build accepts) take MAXW = 64 in blocks of 32 threads, so
// the accumulator stays at 32 KB of static shared memory.
template <int MAXW, bool TRANSPOSE, int BT = kB>
__global__ void __launch_bounds__(BT) k_stiffness_rows(int64_t nv, int64_t nnz, const int32_t* __restrict__ inc_ptr,
                                                       const uint2* __restrict__ inc,
                                                       const double2* __restrict__ grad,
                                                       const double* __restrict__ Dbar,
                                                       const int32_t* __restrict__ rowptr,
                                                       double* __restrict__ vals) {
  __shared__ double acc[2 * MAXW][BT];
  const int t = threadIdx.x;
  const int64_t r = gtid();
  if (r >= 2 * nv) return;
  const int c = r >= nv ? 1 : 0;
  const int64_t i = r - c * nv;
  const int w = rowptr[i + 1] - rowptr[i];
  for (int k = 0; k < 2 * w; k++) acc[k][t] = 0.0;
  for (int32_t s = inc_ptr[i]; s < inc_ptr[i + 1]; s++) {
    const uint2 rec = inc[s];
    const unsigned e = rec.x, y = rec.y, a = inc_a(y);
    RowSlots sl;
#pragma unroll
    for (int b = 0; b < 3; b++) {
      sl.x[b] = (int)inc_off(y, b);
      sl.y[b] = w + (int)inc_off(y, b);
    }
    elastic_row_add<TRANSPOSE, BT>(Dbar + 9 * (int64_t)e, grad + 3 * (int64_t)e, (int)a, c, sl, acc, t);
  }
  const int64_t base = c ? 2 * nnz + 2 * (int64_t)rowptr[i] : 2 * (int64_t)rowptr[i];
  for (int k = 0; k < 2 * w; k++) vals[base + k] = acc[k][t];
}

cudaError_t launch_stiffness_rows(const Mesh& m, const double* Dbar, double* vals, bool transpose, cudaStream_t st) {
  const auto* ip = m.d_inc_ptr.as<int32_t>();
  const auto* inc = m.d_inc.as<uint2>();
  const auto* gr = m.d_grad.as<double2>();
  const auto* rp = m.d_rowptr.as<int32_t>();
  const unsigned nb = nblk(2 * m.nv, kB);
  if (m.maxrow <= 8) {
    if (transpose) k_stiffness_rows<8, true><<<nb, kB, 0, st>>>(m.nv, m.nnz, ip, inc, gr, Dbar, rp, vals);
    else k_stiffness_rows<8, false><<<nb, kB, 0, st>>>(m.nv, m.nnz, ip, inc, gr, Dbar, rp, vals);
  } else if (m.maxrow <= 16) {
    if (transpose) k_stiffness_rows<16, true><<<nb, kB, 0, st>>>(m.nv, m.nnz, ip, inc, gr, Dbar, rp, vals);
    else k_stiffness_rows<16, false><<<nb, kB, 0, st>>>(m.nv, m.nnz, ip, inc, gr, Dbar, rp, vals);
  } else if (m.maxrow <= 64) {
    const unsigned nbw = nblk(2 * m.nv, 32);
    if (transpose) k_stiffness_rows<64, true, 32><<<nbw, 32, 0, st>>>(m.nv, m.nnz, ip, inc, gr, Dbar, rp, vals);
    else k_stiffness_rows<64, false, 32><<<nbw, 32, 0, st>>>(m.nv, m.nnz, ip, inc, gr, Dbar, rp, vals);
  } else {
    return cudaErrorNotSupported;
  }
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Fused elasticity system in the interleaved DOF order (2i = x, 2i+1 = y of node i),
// sliced-ELL.  Row 2i+c holds columns (2j, 2j+1) for each j of the scalar row of i:
// slot 2k is the x-column of the k-th neighbour, slot 2k+1 its y-column.
// isbd: 0 free, 1 Dirichlet DOF, 2 free with a Dirichlet neighbour (interleaved ids).
// rhs: body force [src(fx); src(fy)] interleaved, minus the Dirichlet lift.
// PERM: nodes renumbered (nperm[node]); row 2i+c goes to solver row 2 nperm[i] + c and
// slot 2k+cc to 2 kperm[rowptr[i] + k] + cc; isbd, bdval and rhs in solver order.
template <int MAXW, bool PERM>
__global__ void __launch_bounds__(kB) k_elastic_system(int64_t nv, const int32_t* __restrict__ inc_ptr,
                                                       const uint2* __restrict__ inc,
                                                       const double2* __restrict__ grad,
                                                       const double* __restrict__ Dbar,
                                                       const double* __restrict__ srcx,
                                                       const double* __restrict__ srcy,
                                                       const int32_t* __restrict__ rowptr,
                                                       const int32_t* __restrict__ colind,
                                                       const int32_t* __restrict__ sptr,
                                                       const uint8_t* __restrict__ isbd,
                                                       const double* __restrict__ bdval,
                                                       double* __restrict__ vals, double* __restrict__ rhs,
                                                       const int32_t* __restrict__ nperm,
                                                       const uint8_t* __restrict__ kperm) {
  __shared__ double acc[2 * MAXW][kB];
  const int t = threadIdx.x;
  const int64_t r = gtid();
  if (r >= 2 * nv) return;
  const int64_t i = r >> 1;
  const int c = (int)(r & 1);
  const int w = rowptr[i + 1] - rowptr[i];
  const int32_t r0 = rowptr[i];
  const int64_t rs = PERM ? 2 * (int64_t)nperm[i] + c : r;
  const int64_t base = (int64_t)sptr[rs >> 5] + (rs & 31);
  auto slot = [&](int k) { return PERM ? (int)kperm[r0 + k] : k; };
  const uint8_t tag = isbd[rs];
  if (tag == 1) {
    // diagonal: slot 2*diagpos + c
    const int32_t* row = colind + r0;
    int dk = 0;
    for (int k = 0; k < w; k++)
      if (row[k] == i) dk = k;
    const int ds = 2 * slot(dk) + c;
    for (int k = 0; k < 2 * w; k++) vals[base + 32 * k] = (k == ds) ? 1.0 : 0.0;
    rhs[rs] = bdval[rs];
    return;
  }
  for (int k = 0; k < 2 * w; k++) acc[k][t] = 0.0;
  double rr = 0.0;
  const double* src = c ? srcy : srcx;
  for (int32_t s = inc_ptr[i]; s < inc_ptr[i + 1]; s++) {
    const uint2 rec = inc[s];
    const unsigned e = rec.x, y = rec.y, a = inc_a(y);
    RowSlots sl;
#pragma unroll
    for (int b = 0; b < 3; b++) {
      sl.x[b] = 2 * (int)inc_off(y, b);
      sl.y[b] = 2 * (int)inc_off(y, b) + 1;
    }
    elastic_row_add<false>(Dbar + 9 * (int64_t)e, grad + 3 * (int64_t)e, (int)a, c, sl, acc, t);
    rr += src[3 * (int64_t)e + a];
  }
  if (tag == 2) {
    const int32_t* row = colind + r0;
    for (int k = 0; k < w; k++) {
      const int64_t j = PERM ? (int64_t)nperm[row[k]] : (int64_t)row[k];
#pragma unroll
      for (int cc = 0; cc < 2; cc++) {
        const int64_t dj = 2 * j + cc;
        if (isbd[dj] == 1) {
          rr = fma(-acc[2 * k + cc][t], bdval[dj], rr);
          acc[2 * k + cc][t] = 0.0;
        }
      }
    }
  }
  rhs[rs] = rr;
  for (int k = 0; k < w; k++) {
    const int sk = 2 * slot(k);
    vals[base + 32 * sk] = acc[2 * k][t];
    vals[base + 32 * (sk + 1)] = acc[2 * k + 1][t];
  }
}

cudaError_t launch_elastic_system(const Mesh& m, const double* Dbar, const double* srcx, const double* srcy,
                                  const int32_t* sptr2, const uint8_t* isbd2, const double* bdval2, double* vals,
                                  double* rhs, const int32_t* nperm, const uint8_t* kperm, cudaStream_t st) {
  const auto* ip = m.d_inc_ptr.as<int32_t>();
  const auto* inc = m.d_inc.as<uint2>();
  const auto* gr = m.d_grad.as<double2>();
  const auto* rp = m.d_rowptr.as<int32_t>();
  const auto* ci = m.d_colind.as<int32_t>();
  const unsigned nb = nblk(2 * m.nv, kB);
#define ADFEM_ES(W)                                                                                              \
  do {                                                                                                           \
    if (nperm)                                                                                                   \
      k_elastic_system<W, true><<<nb, kB, 0, st>>>(m.nv, ip, inc, gr, Dbar, srcx, srcy, rp, ci, sptr2, isbd2,    \
                                                   bdval2, vals, rhs, nperm, kperm);                            \
    else                                                                                                         \
      k_elastic_system<W, false><<<nb, kB, 0, st>>>(m.nv, ip, inc, gr, Dbar, srcx, srcy, rp, ci, sptr2, isbd2,   \
                                                    bdval2, vals, rhs, nullptr, nullptr);                       \
  } while (0)
  if (m.maxrow <= 8) ADFEM_ES(8);
  else if (m.maxrow <= 16) ADFEM_ES(16);
  else return cudaErrorNotSupported;
#undef ADFEM_ES
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Unsummed COO of ComputeFemStiffnessMatrixMfem_forward: entry 108 e + 36 k + 6 l + s of
// NN_k = w B^T D_k B.  FP64 issue bounds the kernel: one thread per Gauss point, the weight in the
// rows' gradients (114 operations); the block then writes values and indices in order through
// shared memory.  Every entry comes from the gradients of its own two vertices.  (Rows and columns of
// vertex 2 as negated sums of the others' take 80 operations, but lose digits to cancellation where
// that vertex' gradient is the small one: 6 of 16 in elements of aspect 1000.)
constexpr int kStiffPts = 126, kStiffT = 128;  // whole elements; every warp of the block has points
__global__ void __launch_bounds__(kStiffT) k_stiffness_coo(int64_t ne, int64_t ndof, const int4* __restrict__ conn,
                                                       const double2* __restrict__ grad,
                                                       const double4* __restrict__ geo, const double* __restrict__ D,
                                                       longlong2* __restrict__ idx, double* __restrict__ vv) {
  __shared__ double sv[kStiffPts][37];
  __shared__ int32_t sd[kStiffPts / 3][3];
  const int64_t e0 = (int64_t)blockIdx.x * (kStiffPts / 3);
  const int np = (int)min((int64_t)kStiffPts, 3 * (ne - e0));
  if ((int)threadIdx.x < np) {
    const int64_t e = e0 + threadIdx.x / 3;
    const double2 h[3] = {grad[3 * e], grad[3 * e + 1], grad[3 * e + 2]};
    const double w = geo[e].w;
    double d[9];
#pragma unroll
    for (int q = 0; q < 9; q++) d[q] = __ldg(D + 27 * e0 + 9 * threadIdx.x + q);
    double* N = sv[threadIdx.x];
    // row l: x of vertex l (B column (hx, 0, hy)), y of vertex l - 3 ((0, hy, hx))
#pragma unroll
    for (int l = 0; l < 6; l++) {
      const double a = w * h[l % 3].x, b = w * h[l % 3].y;
      double v[3];
#pragma unroll
      for (int q = 0; q < 3; q++) v[q] = l < 3 ? fma(a, d[q], b * d[6 + q]) : fma(b, d[3 + q], a * d[6 + q]);
#pragma unroll
      for (int c = 0; c < 3; c++) {
        N[6 * l + c] = fma(v[0], h[c].x, v[2] * h[c].y);
        N[6 * l + 3 + c] = fma(v[1], h[c].y, v[2] * h[c].x);
      }
    }
    if (threadIdx.x % 3 == 0) {
      const int4 cn = conn[e];
      sd[threadIdx.x / 3][0] = cn.x;
      sd[threadIdx.x / 3][1] = cn.y;
      sd[threadIdx.x / 3][2] = cn.z;
    }
  }
  __syncthreads();
  for (int q = threadIdx.x; q < 36 * np; q += kStiffT) {
    const int p = q / 36, m = q - 36 * p, r = m / 6, c = m - 6 * r;
    __stcs(vv + 108 * e0 + q, sv[p][m]);
    const int32_t* v = sd[p / 3];
    idx[108 * e0 + q] = make_longlong2(v[r % 3] + (r < 3 ? 0 : ndof), v[c % 3] + (c < 3 ? 0 : ndof));
  }
}

cudaError_t launch_stiffness_coo(const Mesh& m, const double* D, long long* indices, double* vv, cudaStream_t st) {
  k_stiffness_coo<<<nblk(m.ne, kStiffPts / 3), kStiffT, 0, st>>>(m.ne, m.nv, m.d_conn.as<int4>(), m.d_grad.as<double2>(),
                                                             m.d_geo.as<double4>(), D,
                                                             reinterpret_cast<longlong2*>(indices), vv);
  return cudaGetLastError();
}

// ComputeFemStiffnessMatrixMfem_backward: grad_D_k = w B G B^T, G = grad_vv block (6x6): 117
// operations (100 with G's differences to the rows and columns of vertex 2, at up to six times the
// error).  The block reads and writes its points' entries in order through shared memory.
__global__ void __launch_bounds__(kStiffT) k_stiffness_coo_backward(int64_t ne, const double2* __restrict__ grad,
                                                                const double4* __restrict__ geo,
                                                                const double* __restrict__ gvv,
                                                                double* __restrict__ gD) {
  __shared__ double sv[kStiffPts][37];
  const int64_t e0 = (int64_t)blockIdx.x * (kStiffPts / 3);
  const int np = (int)min((int64_t)kStiffPts, 3 * (ne - e0));
  const double* src = gvv + 108 * e0;
  if ((reinterpret_cast<uintptr_t>(gvv) & 15) == 0) {
    for (int q = threadIdx.x; q < 18 * np; q += kStiffT) {
      const double2 v = __ldcs(reinterpret_cast<const double2*>(src) + q);
      const int p = q / 18, m = 2 * (q - 18 * p);
      sv[p][m] = v.x;
      sv[p][m + 1] = v.y;
    }
  } else {
    for (int q = threadIdx.x; q < 36 * np; q += kStiffT) sv[q / 36][q % 36] = __ldcs(src + q);
  }
  __syncthreads();
  if ((int)threadIdx.x < np) {
    const int64_t e = e0 + threadIdx.x / 3;
    const double2 h[3] = {grad[3 * e], grad[3 * e + 1], grad[3 * e + 2]};
    const double w = geo[e].w;
    double* G = sv[threadIdx.x];
    double T[3][6];  // B G
#pragma unroll
    for (int c = 0; c < 6; c++) {
      T[0][c] = h[0].x * G[c];
      T[1][c] = h[0].y * G[18 + c];
      T[2][c] = h[0].y * G[c];
#pragma unroll
      for (int l = 1; l < 3; l++) {
        T[0][c] = fma(h[l].x, G[6 * l + c], T[0][c]);
        T[1][c] = fma(h[l].y, G[18 + 6 * l + c], T[1][c]);
        T[2][c] = fma(h[l].y, G[6 * l + c], T[2][c]);
      }
#pragma unroll
      for (int l = 0; l < 3; l++) T[2][c] = fma(h[l].x, G[18 + 6 * l + c], T[2][c]);
    }
#pragma unroll
    for (int p = 0; p < 3; p++) {
      double x = T[p][0] * h[0].x, y = T[p][3] * h[0].y, z = T[p][0] * h[0].y;
#pragma unroll
      for (int l = 1; l < 3; l++) {
        x = fma(T[p][l], h[l].x, x);
        y = fma(T[p][3 + l], h[l].y, y);
        z = fma(T[p][l], h[l].y, z);
      }
#pragma unroll
      for (int l = 0; l < 3; l++) z = fma(T[p][3 + l], h[l].x, z);
      G[3 * p] = x * w;
      G[3 * p + 1] = y * w;
      G[3 * p + 2] = z * w;
    }
  }
  __syncthreads();
  for (int q = threadIdx.x; q < 9 * np; q += kStiffT) gD[27 * e0 + q] = sv[q / 9][q % 9];
}

cudaError_t launch_stiffness_coo_backward(const Mesh& m, const double* grad_vv, double* grad_D, cudaStream_t st) {
  k_stiffness_coo_backward<<<nblk(m.ne, kStiffPts / 3), kStiffT, 0, st>>>(m.ne, m.d_grad.as<double2>(),
                                                                      m.d_geo.as<double4>(), grad_vv, grad_D);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// dL/dE at each Gauss point: -w (B lam_e)^T (dD/dE) (B u_e), plane strain with the
// reference formula, lam zero on Dirichlet DOFs.  u, lam interleaved.
__global__ void k_elastic_grad_E(int64_t ne, const int4* __restrict__ conn, const double2* __restrict__ grad,
                                 const double4* __restrict__ geo, const double* __restrict__ u,
                                 const double* __restrict__ lam, const uint8_t* __restrict__ isbd2,
                                 const double* __restrict__ nu, double* __restrict__ gE) {
  const int64_t e = gtid();
  if (e >= ne) return;
  const int4 cn = conn[e];
  const int vtx[3] = {cn.x, cn.y, cn.z};
  const double2* gr = grad + 3 * e;
  double eu[3] = {0, 0, 0}, el[3] = {0, 0, 0};
#pragma unroll
  for (int b = 0; b < 3; b++) {
    const int64_t dx = 2 * (int64_t)vtx[b], dy = dx + 1;
    const double ux = u[dx], uy = u[dy];
    const double lx = isbd2[dx] == 1 ? 0.0 : lam[dx], ly = isbd2[dy] == 1 ? 0.0 : lam[dy];
    const double2 g = gr[b];
    eu[0] = fma(g.x, ux, eu[0]);
    eu[1] = fma(g.y, uy, eu[1]);
    eu[2] = fma(g.y, ux, fma(g.x, uy, eu[2]));
    el[0] = fma(g.x, lx, el[0]);
    el[1] = fma(g.y, ly, el[1]);
    el[2] = fma(g.y, lx, fma(g.x, ly, el[2]));
  }
  const double dd = el[0] * eu[0] + el[1] * eu[1] + el[2] * eu[2];
  const double all = (el[0] + el[1] + el[2]) * (eu[0] + eu[1] + eu[2]);
  const double off = all - dd;  // sum over p != q of el_p eu_q
  const double w = geo[e].w;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const double v = nu[3 * e + k];
    const double den = (1 + v) * (1 - 2 * v);
    const double sp = (1 - v) / den, ap = v / den;  // dD/dE entries
    gE[3 * e + k] = -w * (sp * dd + ap * off);
  }
}

cudaError_t launch_elastic_grad_E(const Mesh& m, const double* u2, const double* lam2, const uint8_t* isbd2,
                                  const double* nu, double* gE, cudaStream_t st) {
  k_elastic_grad_E<<<nblk(m.ne, 256), 256, 0, st>>>(m.ne, m.d_conn.as<int4>(), m.d_grad.as<double2>(),
                                                    m.d_geo.as<double4>(), u2, lam2, isbd2, nu, gE);
  return cudaGetLastError();
}

// reference order <-> solver order through a DOF map: sol[map[d]] = ref[d]
__global__ void k_to_solver(int64_t n, const int32_t* __restrict__ map, const double* __restrict__ ref,
                            double* __restrict__ sol) {
  const int64_t d = gtid();
  if (d >= n) return;
  sol[map[d]] = ref[d];
}
__global__ void k_from_solver(int64_t n, const int32_t* __restrict__ map, const double* __restrict__ sol,
                              double* __restrict__ ref) {
  const int64_t d = gtid();
  if (d >= n) return;
  ref[d] = sol[map[d]];
}
cudaError_t launch_to_solver(int64_t n, const int32_t* map, const double* ref, double* sol, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  k_to_solver<<<nblk(n, 256), 256, 0, st>>>(n, map, ref, sol);
  return cudaGetLastError();
}
cudaError_t launch_from_solver(int64_t n, const int32_t* map, const double* sol, double* ref, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  k_from_solver<<<nblk(n, 256), 256, 0, st>>>(n, map, sol, ref);
  return cudaGetLastError();
}

// reference [x; y] <-> interleaved
__global__ void k_to_interleaved(int64_t nv, const double* __restrict__ ref, double* __restrict__ il) {
  const int64_t r = gtid();
  if (r >= 2 * nv) return;
  il[r] = ref[(r & 1) * nv + (r >> 1)];
}
__global__ void k_from_interleaved(int64_t nv, const double* __restrict__ il, double* __restrict__ ref) {
  const int64_t r = gtid();
  if (r >= 2 * nv) return;
  ref[(r & 1) * nv + (r >> 1)] = il[r];
}
cudaError_t launch_to_interleaved(int64_t nv, const double* ref, double* il, cudaStream_t st) {
  k_to_interleaved<<<nblk(2 * nv, 256), 256, 0, st>>>(nv, ref, il);
  return cudaGetLastError();
}
cudaError_t launch_from_interleaved(int64_t nv, const double* il, double* ref, cudaStream_t st) {
  k_from_interleaved<<<nblk(2 * nv, 256), 256, 0, st>>>(nv, il, ref);
  return cudaGetLastError();
}

}  // namespace adfem
