// Multigrid-preconditioned conjugate gradients of the resident systems (mg.cu, mg_setup.cpp).
//
// The preconditioner is one symmetric V-cycle of smoothed aggregation: the matrix graph is
// aggregated level by level once per system on the host (mg_setup.cpp: patterns only), and
// after every assembly the device forms the interpolation values P = P0 - c D^-1 A P0 and the
// coarse operators P^T A P on those fixed patterns (mg.cu).  Every level is scaled to unit
// diagonal, so its smoother (Chebyshev) needs no diagonal; levels of at most kMgTailDofs
// unknowns run in one launch (k_mg_tail).
#pragma once
#include <stdint.h>

#include <memory>
#include <vector>

#include "adfem_internal.h"

namespace adfem {

constexpr int kMgMaxLevels = 12;
constexpr int kMgMaxTail = 6;
constexpr int kMgMaxP = 16;       // entries per interpolation row
constexpr int kMgMaxAP = 32;      // entries per row of A P
constexpr int kMgMaxA = 64;       // entries per coarse row
constexpr int kMgDense = 160;     // unknowns of the directly solved coarsest level
constexpr int kMgTailDofs = 5120; // unknowns of the largest level of the one-launch tail
constexpr int kTailC = 8;         // blocks of the tail's cluster
constexpr int kTailSpin = 1 << 16;  // tries of a wait in the tail before it gives up
constexpr int kTailLocal = kMgTailDofs / kTailC;  // unknowns of a tail that one block runs alone
constexpr int kMgGrid = 1280;     // blocks of the kernels that sum over the grid, at most
constexpr int kMgIterations = 300;  // a solve that needs more is left to the Jacobi iteration
constexpr int kMgDeg0 = 2, kMgDeg = 4;  // Chebyshev degree: level 0, coarser levels

// Patterns of one level (host), rows in solver order at level 0.  Rows are in compressed
// form; the device keeps them in slices of 32 rows as Sell does, with absolute int32 columns.
struct MgPattern {
  std::vector<int32_t> rp, ci;
};
struct MgHostLevel {
  int64_t n = 0;
  MgPattern A;                 // graph of the level
  std::vector<int32_t> agg;    // aggregate of each node (empty on the coarsest level)
  MgPattern P, AP, PT;         // interpolation, A P, transpose of P
  std::vector<int32_t> PTslot; // position of each PT entry within its P row
  std::vector<double> x, y;    // node positions (2-D elasticity only)
};
// Hierarchy of a graph of n nodes with nb0 unknowns each on level 0 and nbc on the others;
// x, y (may be empty): node positions for the rotation mode.  false: the graph does not
// coarsen to a size the tail can hold, or a pattern has more than `limit` entries (they are
// numbered with 32 bits); the system keeps the Jacobi iteration.
bool mg_build_host(int64_t n, std::vector<int32_t>&& rp, std::vector<int32_t>&& ci, int nb0, int nbc,
                   std::vector<double>&& x, std::vector<double>&& y, std::vector<MgHostLevel>& lv,
                   int64_t limit = INT32_MAX);

// Device view of one level
struct MgLev {
  int n = 0, nc = 0, nb = 1, nbc = 1, lpr = 1;
  int nv = 0, np = 0, nap = 0, npt = 0;  // entries of val, p_val, ap_val, pt_val
  int width = 0;               // longest row of the operator
  int d16 = 0;                 // level 0 only: the system's own pattern (int16 deltas, slice patterns)
  const int32_t *sptr = nullptr, *spat = nullptr;
  const void* col = nullptr;
  const int16_t* pat = nullptr;
  float* val = nullptr;        // nb x nb per entry, unit diagonal
  const int32_t *p_sptr = nullptr, *p_col = nullptr;
  float* p_val = nullptr;      // nb x nbc per entry
  const int32_t *ap_sptr = nullptr, *ap_col = nullptr;
  float* ap_val = nullptr;
  const int32_t *pt_sptr = nullptr, *pt_col = nullptr, *pt_src = nullptr;
  float* pt_val = nullptr;     // nbc x nb per entry
  const int32_t* agg = nullptr;
  const float2* dpos = nullptr;  // position relative to the aggregate's centre (rotation mode)
  float* s = nullptr;          // scale of each unknown (0: unknown without a degree of freedom)
  float *b = nullptr, *x = nullptr, *x2 = nullptr, *d = nullptr;
  const uint8_t* to = nullptr;  // tail: the blocks that need each row's value (one bit each)
  const int32_t* cnt = nullptr; // tail: rows each block needs
  float* coef = nullptr;       // Chebyshev coefficients
  int* lam = nullptr;          // bound of the largest eigenvalue (float bits)
};

struct Mg {
  int nlev = 0, tail = 0;      // levels, first level of the one-launch tail
  MgLev lev[kMgMaxLevels];
  float* dense = nullptr;      // inverse of the coarsest operator
  int ndense = 0;
  int sms = 0;
  int nrz = 0, nrn = 0;        // partial sums of r.z and of the residual's square
  double* rowsum = nullptr;    // FP64 row sums of K per component of the column (nb per row)
  int* lam = nullptr;          // MgLev::lam of every level
  double* part = nullptr;      // partial sums of the iteration's three sums (kMgGrid each)
  DevBuf slab;                 // all of the above
  bool cluster = false;        // the tail's first level is shared by a cluster
  const char *pat = nullptr, *vals = nullptr;  // of the levels that a tail block runs alone
  int pat_bytes = 0, val_bytes = 0;            // (0: too large for its shared memory)
  size_t tail_smem = 0;
  bool current = false;        // values belong to the current assembly
  cudaGraphExec_t solve = nullptr;  // while (not finished) one iteration
  int body_launches = 0;
  ~Mg();
};

}  // namespace adfem
