"""P2 solves at the precision of their matrix: rounding of the element matrices that is the same in every
element (of the quadrature's constants) must not leave row sums that add up over the mesh.

Reference: the oracle's matrix, whose entries are sums over the points one by one, and one step of
refinement from the solution under test with a sparse direct solve (its error enters the correction
only).  Bar: 1e-13 of the solution.  Independent roundings of the entries move it by some 1e-14 at this
size (50 roundings of 2^-53 each way, both matrices), row sums off by half a rounding the same way in
every element by 5e-13.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from adfem_gpu import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_p2_solution(oracle, gpulib, precision):
    import scipy.sparse.linalg as sl

    coords, elems = synth.jittered_square(120, n=110, seed=2)
    O = oracle.OracleSpace(coords, elems, 2)
    M = gpulib.Mesh(coords, elems, degree=2)
    g = O.gauss_nodes()
    kappa = np.exp(1.7 * np.sin(5 * g[:, 0] + 1) * np.cos(7 * g[:, 1]))
    f = np.ones(O.ngauss)
    bd = O.bcnode()
    S = gpulib.PoissonSystem(M)
    S.set_dirichlet(bd)
    S.assemble(torch.tensor(kappa, device="cuda"), torch.tensor(f, device="cuda"))
    u = S.solve(precision=precision, rtol=1e-13).cpu().numpy()
    inner = np.ones(O.ndof, bool)
    inner[bd - 1] = False
    K = O.laplace_csc(kappa).tocsr()
    A = K[inner]
    # (the residual in extended precision)
    row = np.repeat(np.arange(A.shape[0]), np.diff(A.indptr))
    r = O.source(f)[inner].astype(np.longdouble)
    np.add.at(r, row, -A.data.astype(np.longdouble) * u[A.indices])
    d = sl.spsolve(A[:, inner].tocsc(), r.astype(float))
    assert np.linalg.norm(d) / np.linalg.norm(u) < 1e-13
