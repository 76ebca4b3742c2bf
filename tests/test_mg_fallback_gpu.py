"""Solves that the multigrid iteration gives up are finished by the Jacobi iteration.

Bars: 1e-9 relative (max norm) against the direct solve, as for every solve of this suite.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from adfem_gpu import synth

pytestmark = pytest.mark.gpu
JACOBI = 100  # iterations: the Jacobi iteration needs more on every case here, multigrid fewer


def rel(a, b):
    return float(np.max(np.abs(a.cpu().numpy() - b)) / np.max(np.abs(b)))


def t(a):
    return torch.tensor(np.asarray(a, dtype=np.float64), device="cuda")


def system(oracle, gpulib, m, elastic=False):
    """A system, its direct solution and its assembly's arguments."""
    coords, elems = synth.jittered_square(m, seed=m)
    O = oracle.OracleMesh(coords, elems)
    rng = np.random.default_rng(m)
    M = gpulib.Mesh(coords, elems)
    if elastic:
        E, nu, f = 1e3 * (1 + rng.random(O.ngauss)), np.full(O.ngauss, 0.3), rng.random(O.ngauss)
        left = synth.left_edge_nodes(coords) + 1
        bd = np.concatenate([left, left + O.ndof])
        B, r = oracle.dirichlet_csc(O.stiffness_csc(oracle.plane_strain(E, nu, 0)),
                                    np.concatenate([O.source(f), O.source(f)]), bd, np.zeros(bd.size))
        S, args = gpulib.ElasticitySystem(M), (t(E), t(nu), t(f), t(f))
        S.set_dirichlet(bd)
    else:
        kappa, f = 1 + 99 * rng.random(O.ngauss), rng.random(O.ngauss)
        bd = O.bcnode()
        bv = rng.random(bd.size)
        B, r = oracle.dirichlet_csc(O.laplace_csc(kappa), O.source(f), bd, bv)
        S, args = gpulib.PoissonSystem(M), (t(kappa), t(f))
        S.set_dirichlet(bd, bv)
    S.assemble(*args)
    return S, oracle.spsolve(B, r), args


# nodes: 576 (one block), 3721 (a cluster), 10201 (a graph with a tail); elasticity: 1352 unknowns (a
# cluster), 10082 (a graph)
@pytest.mark.parametrize("m,elastic", [(23, 0), (60, 0), (100, 0), (25, 1), (70, 1)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_waits_that_give_up(oracle, gpulib, monkeypatch, m, elastic, precision):
    monkeypatch.setenv("ADFEM_MG_SPIN", "0")
    S, ref, args = system(oracle, gpulib, m, elastic)
    monkeypatch.delenv("ADFEM_MG_SPIN")
    for _ in range(2):
        assert rel(S.solve(precision=precision, rtol=1e-12), ref) < 1e-9
        assert S.last_stats.status == 0 and S.last_stats.iterations > JACOBI
        S.assemble(*args)
    # the device is as it was for the systems that do wait
    S, ref, _ = system(oracle, gpulib, m, elastic)
    assert rel(S.solve(precision=precision, rtol=1e-12), ref) < 1e-9 and S.last_stats.iterations < JACOBI
