"""K\\F of a user's matrix (adfem_csc_solve): the matrices that get a multigrid hierarchy for the one
solve and those that keep the Jacobi iteration, against the direct solve.

Bars: the iteration ends at a residual of 1e-12 |b| in the Jacobi-scaled norm, and the condition
numbers here are below 1e4 (64 x 64 cells: about (4 / pi^2) 64^2 times a coefficient ratio of 3), so
1e-8 relative (2-norm) holds for every one.
"""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from scipy import sparse as sp

from adfem_gpu import synth

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a) - b) / np.linalg.norm(b))


def poisson(oracle, m, n, seed=0):
    coords, elems = synth.jittered_square(m, n=n, seed=seed)
    O = oracle.OracleMesh(coords, elems)
    rng = np.random.default_rng(seed)
    ng = 3 * len(elems)
    K = O.laplace_csc(1.0 + 2.0 * rng.random(ng))
    bd = O.bcnode()
    bv = rng.random(bd.size)
    B, r = oracle.dirichlet_csc(K, O.source(rng.random(ng)), bd, bv)
    return sp.csc_matrix(B), r


def raw_solve(gpulib, K, F, order=None):
    """The entry point itself, with the columns' entries in a given order."""
    from adfem_gpu import _lib

    cp, rv, nz = K.indptr.astype(np.int64) + 1, K.indices.astype(np.int64) + 1, K.data.astype(np.float64).copy()
    if order == "reversed":
        for j in range(K.shape[0]):
            s = slice(K.indptr[j], K.indptr[j + 1])
            rv[s], nz[s] = rv[s][::-1].copy(), nz[s][::-1].copy()
    u, F = np.zeros(K.shape[0]), np.ascontiguousarray(F)
    o, st = gpulib.solver_opts(), gpulib.SolverStats()
    L = _lib.load()
    assert L.adfem_csc_solve(K.shape[0], _lib.ptr(cp), _lib.ptr(rv), _lib.ptr(nz), _lib.ptr(F), _lib.ptr(u),
                             ctypes.byref(o), ctypes.byref(st)) == 0
    return u, st


# cells: 11 x 11 is solved by the Jacobi iteration (144 unknowns), 12 x 12 is the first with a
# hierarchy; 31 x 20 one block, 64 x 64 a cluster, 90 x 80 a level above the one-launch cycle
@pytest.mark.parametrize("m,n", [(11, 11), (12, 12), (31, 20), (64, 64), (90, 80)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_poisson_matrices(oracle, gpulib, m, n, precision):
    K, F = poisson(oracle, m, n, seed=m)
    u, st = gpulib.solve(K, F, precision=precision, return_stats=True)
    assert rel(u, oracle.spsolve(K, F)) < 1e-8
    if (m + 1) * (n + 1) > 160 and precision == "fp64":
        assert st.iterations < 40
    w, st = gpulib.solve(K, F, precision=precision, u0=u, return_stats=True)  # warm start
    assert st.iterations <= 3 and rel(w, u) < 1e-8


def test_unsorted_columns_and_stored_zeros(oracle, gpulib):
    K, F = poisson(oracle, 40, 33)
    ref = oracle.spsolve(K, F)
    u, st = raw_solve(gpulib, K, F, order="reversed")  # (keeps the Jacobi iteration)
    assert rel(u, ref) < 1e-8 and st.iterations > 40
    # eliminated rows that still store zeros towards their neighbours
    Z = K.copy()
    i = int(np.flatnonzero(np.diff(K.indptr) == 1)[7])
    j = int(np.flatnonzero(np.diff(K.indptr) > 5)[20])
    Z = (Z + sp.coo_matrix(([1.0, 1.0], ([i, j], [j, i])), shape=K.shape).tocsc()).tocsc()
    Z.sort_indices()
    Z.data[[k for k in range(Z.indptr[i], Z.indptr[i + 1]) if Z.indices[k] == j]] = 0.0
    Z.data[[k for k in range(Z.indptr[j], Z.indptr[j + 1]) if Z.indices[k] == i]] = 0.0
    assert Z.nnz == K.nnz + 2
    u, st = raw_solve(gpulib, Z, F)
    assert rel(u, ref) < 1e-8 and st.iterations < 40


def test_matrices_that_keep_the_jacobi_iteration(oracle, gpulib):
    K, F = poisson(oracle, 30, 30)
    # no eliminated row: K + 1
    B = (K + sp.identity(K.shape[0], format="csc")).tocsc()
    free = np.flatnonzero(np.diff(K.indptr) > 1)
    B = B[free][:, free].tocsc()
    assert rel(gpulib.solve(B, F[free]), oracle.spsolve(B, F[free])) < 1e-8
    # two unknowns per node, numbered by component and by node
    A = K[free][:, free]
    for V in (sp.kron(np.array([[2.0, 0.5], [0.5, 2.0]]), A), sp.kron(A, np.array([[2.0, 0.5], [0.5, 2.0]]))):
        V = sp.block_diag([V, sp.identity(9)]).tocsc()
        f = np.random.default_rng(3).random(V.shape[0])
        u, st = gpulib.solve(V, f, return_stats=True)
        assert rel(u, oracle.spsolve(V, f)) < 1e-8
        assert st.iterations > 40
