"""Solves of small resident systems, which are one launch of one block (up to 640 unknowns) or of a
cluster (up to 5120): the sizes around those limits, few rows in the last block, warm starts, a zero
right-hand side, the adjoint and the iteration limit, against the direct solve.

Bars: 1e-9 relative (max norm), as for every solve of this suite.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from adfem_gpu import synth

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.max(np.abs(a.cpu().numpy() - b)) / np.max(np.abs(b)))


def t(a):
    return torch.tensor(np.asarray(a, dtype=np.float64), device="cuda")


def system(oracle, gpulib, m, n, elastic):
    coords, elems = synth.jittered_square(m, n=n, seed=m)
    O = oracle.OracleMesh(coords, elems)
    rng = np.random.default_rng(n)
    M = gpulib.Mesh(coords, elems)
    if elastic:
        E, nu, f = 1e3 * (1 + rng.random(O.ngauss)), np.full(O.ngauss, 0.3), rng.random(O.ngauss)
        left = synth.left_edge_nodes(coords) + 1
        bd = np.concatenate([left, left + O.ndof])
        B, r = oracle.dirichlet_csc(O.stiffness_csc(oracle.plane_strain(E, nu, 0)),
                                    np.concatenate([O.source(f), O.source(f)]), bd, np.zeros(bd.size))
        S = gpulib.ElasticitySystem(M)
        S.set_dirichlet(bd)
        S.assemble(t(E), t(nu), t(f), t(f))
    else:
        kappa, f = 1 + 9 * rng.random(O.ngauss), rng.random(O.ngauss)
        bd = O.bcnode()
        bv = rng.random(bd.size)
        B, r = oracle.dirichlet_csc(O.laplace_csc(kappa), O.source(f), bd, bv)
        S = gpulib.PoissonSystem(M)
        S.set_dirichlet(bd, bv)
        S.assemble(t(kappa), t(f))
    return S, B, r, bd - 1


# nodes: 640 (one block, full), 651 (cluster, 82 rows a block, 77 in the last), 648, 5112, 5120;
# elasticity: 320 (640 unknowns), 324, 2550, 2560
@pytest.mark.parametrize("m,n,elastic", [(31, 19, 0), (30, 20, 0), (26, 23, 0), (70, 71, 0), (79, 63, 0),
                                         (19, 15, 1), (17, 17, 1), (50, 49, 1), (63, 39, 1)])
def test_one_launch_solves(oracle, gpulib, m, n, elastic):
    S, B, r, bd = system(oracle, gpulib, m, n, elastic)
    ref = oracle.spsolve(B, r)
    u = S.solve(rtol=1e-12)
    st = S.last_stats
    assert rel(u, ref) < 1e-9 and 0 < st.iterations < 120
    assert (st.launches < 10) == (B.shape[0] <= 5120)
    assert torch.equal(S.solve(rtol=1e-12), u)
    w = S.solve(u=u.clone(), rtol=1e-12, warm=True)
    assert S.last_stats.iterations <= 3 and rel(w, ref) < 1e-9
    # adjoint: K is symmetric, eliminated rows of the right-hand side do not enter
    g = np.random.default_rng(1).random(B.shape[0])
    free = g.copy()
    free[bd] = 0.0
    lam = S.adjoint(t(g), rtol=1e-12)
    assert rel(lam, oracle.spsolve(B, free)) < 1e-9
    assert float(S.adjoint(t(0.0 * g), rtol=1e-12).abs().max()) == 0.0
    with pytest.raises(gpulib.AdFemError):
        S.solve(rtol=1e-12, max_iter=3)
    assert rel(S.solve(rtol=1e-12), ref) < 1e-9
