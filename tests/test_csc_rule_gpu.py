"""K\\F in FP64: matrices whose diagonal preconditions them well keep the Jacobi iteration where a
hierarchy would cost more than it saves, and every choice gives the direct solution.

Bars: the solves end at a residual of 1e-12 |b| in the Jacobi-scaled norm and the condition numbers are
below 1e5 (200 x 200 cells: about (4 / pi^2) 200^2 times a coefficient ratio of 3), so 1e-7 relative.
"""
import numpy as np
import pytest

pytest.importorskip("torch")

from scipy import sparse as sp

from adfem_gpu import synth

pytestmark = pytest.mark.gpu


# c: M + c h^2 K of m x m cells (None: K); multigrid takes 10 to 19 iterations, Jacobi 25 and more on these
@pytest.mark.parametrize("m,c,multigrid", [(20, 0.0, True), (64, 1.0, True), (64, None, True), (200, 0.0, False),
                                           (200, 1.0, False), (200, 10.0, False), (200, 100.0, True), (200, None, True)])
def test_choice_of_preconditioner(oracle, gpulib, m, c, multigrid):
    coords, elems = synth.jittered_square(m, seed=1)
    O = oracle.OracleMesh(coords, elems)
    rng = np.random.default_rng(0)
    K = O.laplace_csc(1.0 + 2.0 * rng.random(O.ngauss))
    if c is not None:
        M = gpulib.compute_fem_mass_matrix1(np.ones(O.ngauss), gpulib.Mesh(coords, elems))
        K = sp.csc_matrix(M + c / m**2 * K)
    bd = O.bcnode()
    B, r = oracle.dirichlet_csc(K, rng.random(O.ndof), bd, rng.random(bd.size))
    u, st = gpulib.solve(sp.csc_matrix(B), r, rtol=1e-12, return_stats=True)
    ref = oracle.spsolve(B, r)
    assert st.status == 0 and np.linalg.norm(u - ref) < 1e-7 * np.linalg.norm(ref)
    assert (st.iterations < 22) == multigrid


@pytest.mark.parametrize("bad", [np.inf, np.nan, 0.0, -1.0])
@pytest.mark.parametrize("every", [1, 7])
def test_diagonal_that_is_not_positive_and_finite_is_refused(oracle, gpulib, bad, every):
    coords, elems = synth.jittered_square(20, seed=1)
    O = oracle.OracleMesh(coords, elems)
    K = sp.csc_matrix(O.laplace_csc(np.ones(O.ngauss)))
    bd = O.bcnode()
    B, r = oracle.dirichlet_csc(K, np.ones(O.ndof), bd, np.zeros(bd.size))
    B = sp.csc_matrix(B)
    d = np.flatnonzero(np.repeat(np.arange(O.ndof), np.diff(B.indptr)) == B.indices)
    B.data[d[::every]] = bad
    with pytest.raises(gpulib.AdFemError):
        gpulib.solve(B, r, rtol=1e-12)
