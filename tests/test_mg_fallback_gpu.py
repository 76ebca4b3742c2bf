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


@pytest.mark.parametrize("m,elastic", [(23, 0), (60, 0), (100, 0), (25, 1), (70, 1)])
def test_iteration_cap(oracle, gpulib, monkeypatch, m, elastic):
    cap = 25 if elastic else 8  # enough for a residual of 1e-2, too few for 1e-12
    monkeypatch.setenv("ADFEM_MG_MAX_ITER", str(cap))
    S, ref, args = system(oracle, gpulib, m, elastic)
    for precision in ("fp64", "mixed"):
        S.solve(precision=precision, rtol=1e-2)
        few = S.last_stats.iterations
        assert few < cap
        u = S.solve(precision=precision, rtol=1e-12)
        assert S.last_stats.iterations > JACOBI and rel(u, ref) < 1e-9
        # the start of a warm solve is the caller's vector, as before the multigrid iterations
        w = S.solve(t(ref), precision=precision, rtol=1e-8, warm=True)
        assert S.last_stats.iterations == 0 and rel(w, ref) < 1e-9
        # the assembly's later solves do not try again, the next assembly's do
        S.solve(precision=precision, rtol=1e-2)
        assert S.last_stats.iterations > few
        S.assemble(*args)
        S.solve(precision=precision, rtol=1e-2)
        assert S.last_stats.iterations == few
        S.assemble(*args)
        w = S.solve(t(ref * (1 + 1e-3 * np.sin(np.arange(ref.size)))), precision=precision, rtol=1e-12, warm=True)
        assert S.last_stats.iterations > JACOBI / 2 and rel(w, ref) < 1e-9
        S.assemble(*args)


def test_indefinite_operator_with_a_positive_diagonal(oracle, gpulib):
    coords, elems = synth.jittered_square(20, seed=1)
    O = oracle.OracleMesh(coords, elems)
    k = np.arange(len(elems))
    x, y = k // 2 % 20, k // 2 // 20
    kappa = np.repeat(np.where((x % 4 == 2) & (y % 4 == 2) & (k % 2 == 0), -0.6, 1.0 / 3), 3)
    f, bd = np.ones(O.ngauss), O.bcnode()
    B, _ = oracle.dirichlet_csc(O.laplace_csc(kappa), O.source(f), bd, np.zeros(bd.size))
    assert B.diagonal().min() > 0.01 and np.linalg.eigvalsh(B.toarray()).min() < -0.1
    S = gpulib.PoissonSystem(gpulib.Mesh(coords, elems))
    S.set_dirichlet(bd)
    for _ in range(2):
        S.assemble(t(kappa), t(f))
        for precision in ("fp64", "mixed", "fp64"):
            with pytest.raises(gpulib.AdFemError) as e:
                S.solve(precision=precision, rtol=1e-12)
            assert e.value.status == gpulib._lib.ERR_BREAKDOWN
    # the system is as before for an operator that is definite
    S.assemble(t(np.ones(O.ngauss)), t(f))
    B, r = oracle.dirichlet_csc(O.laplace_csc(np.ones(O.ngauss)), O.source(f), bd, np.zeros(bd.size))
    assert rel(S.solve(rtol=1e-12), oracle.spsolve(B, r)) < 1e-9 and S.last_stats.iterations < JACOBI


@pytest.mark.parametrize("m,elastic", [(23, 0), (100, 0), (25, 1)])
def test_hierarchy_without_room(oracle, gpulib, monkeypatch, m, elastic):
    monkeypatch.setenv("ADFEM_MG_MAX_BYTES", "10000")  # (these take 100 KB and more)
    S, ref, args = system(oracle, gpulib, m, elastic)
    monkeypatch.delenv("ADFEM_MG_MAX_BYTES")
    L = gpulib._lib.load()
    for _ in range(2):
        for precision in ("fp64", "mixed"):
            try:
                L.adfem_debug_fail_alloc(0)  # (nothing is allocated for the Jacobi iteration either)
                u = S.solve(precision=precision, rtol=1e-12)
            finally:
                L.adfem_debug_fail_alloc(-1)
            assert S.last_stats.iterations > JACOBI and rel(u, ref) < 1e-9
        S.assemble(*args)
    # with room, an allocation that fails although the device is not short is reported, and tried again
    S, ref, _ = system(oracle, gpulib, m, elastic)
    try:
        L.adfem_debug_fail_alloc(0)
        with pytest.raises(gpulib.AdFemError) as e:
            S.solve(rtol=1e-12)
    finally:
        L.adfem_debug_fail_alloc(-1)
    assert e.value.status == gpulib._lib.ERR_NOMEM
    assert rel(S.solve(rtol=1e-12), ref) < 1e-9 and S.last_stats.iterations < JACOBI


@pytest.mark.parametrize("m", [23, 60, 100])
def test_warm_start_far_from_the_solution(oracle, gpulib, m):
    # residuals of 1e20 |b| and more, whose squares are no FP32 numbers: the multigrid iteration takes
    # them (36 digits at some 0.7 of a digit an iteration), without the Jacobi iteration's help
    S, ref, _ = system(oracle, gpulib, m)
    u = 1e24 * np.random.default_rng(m).standard_normal(ref.size)
    w = S.solve(t(u), rtol=1e-12, warm=True)
    assert rel(w, ref) < 1e-9 and S.last_stats.iterations < JACOBI
