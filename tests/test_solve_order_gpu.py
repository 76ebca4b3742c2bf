"""When a solve's results are there, and what a refused one leaves behind.

* A solve on a stream that is being captured is refused and leaves the capture and the system as
  they were: the hierarchy values of a later solve belong to the last assembly.
* The solution is written when the call returns, with or without statistics asked for.
* Solves that end before their first iteration disturb none that follows.

Bars: 1e-9 relative (max norm) against the direct solve, as for every solve of this suite.
"""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from adfem_gpu import _lib, synth

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.max(np.abs(a.cpu().numpy() - b)) / np.max(np.abs(b)))


def t(a):
    return torch.tensor(np.asarray(a, dtype=np.float64), device="cuda")


# nodes: 169 (one block), 4225 (a cluster), 10201 (a graph)
@pytest.mark.parametrize("m", [12, 64, 100])
def test_refused_capture_leaves_the_system_as_it_was(oracle, gpulib, m):
    coords, elems = synth.jittered_square(m, seed=2)
    O = oracle.OracleMesh(coords, elems)
    rng = np.random.default_rng(m)
    bd = O.bcnode()
    bv = rng.random(bd.size)
    S = gpulib.PoissonSystem(gpulib.Mesh(coords, elems))
    S.set_dirichlet(bd, bv)
    f = rng.random(O.ngauss)
    S.assemble(t(1.0 + rng.random(O.ngauss)), t(f))
    S.solve(rtol=1e-12)  # (the hierarchy holds the values of this assembly)
    kappa = 1e3 * (1.0 + 9.0 * rng.random(O.ngauss))
    S.assemble(t(kappa), t(f))
    u = torch.zeros(O.ndof, dtype=torch.float64, device="cuda")
    o, st = gpulib.solver_opts(rtol=1e-12), _lib.SolverStats()
    s, g, x = torch.cuda.Stream(), torch.cuda.CUDAGraph(), torch.zeros(8, device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=s):
        x.add_(1.0)
        r = _lib.load().adfem_system_solve_d(S.handle, _lib.ptr(u), ctypes.byref(o), ctypes.byref(st),
                                             _lib.stream_ptr(s))
        x.add_(1.0)
    assert r == _lib.ERR_UNSUPPORTED and "captured" in _lib.load().adfem_last_error().decode()
    g.replay()
    torch.cuda.synchronize()
    assert float(x[0]) == 2.0
    B, b = oracle.dirichlet_csc(O.laplace_csc(kappa), O.source(f), bd, bv)
    assert rel(S.solve(rtol=1e-12), oracle.spsolve(B, b)) < 1e-9
    assert S.last_stats.iterations < 60  # (not the Jacobi iteration)


def test_solution_is_there_when_the_call_returns(gpulib):
    # the caller's vector is pinned host memory, which the device writes slower than its own and the
    # host can look at at once; natural numbering, so that the solver writes it itself
    M = gpulib.Mesh(*synth.jittered_square(1000, seed=1))
    S = gpulib.PoissonSystem(M)
    S.set_dirichlet(gpulib.bcnode(M))
    ng = gpulib.get_ngauss(M)
    S.assemble(t(np.ones(ng)), t(np.ones(ng)))
    assert S.solver_info()["renumbered"] == 0
    ref = S.solve(rtol=1e-3).cpu().numpy()
    u = torch.empty(ref.size, dtype=torch.float64).pin_memory()
    h, o = u.numpy(), gpulib.solver_opts(rtol=1e-3)
    solve = _lib.load().adfem_system_solve_d
    for stats in (None, _lib.SolverStats()):
        args = (S.handle, _lib.ptr(u), ctypes.byref(o), ctypes.byref(stats) if stats else None, _lib.stream_ptr(0))
        for _ in range(5):
            h[:] = np.nan
            r = solve(*args)
            last = h[-2000:].copy()
            torch.cuda.synchronize()
            assert r == 0 and np.array_equal(last, ref[-2000:]) and np.array_equal(h, ref)


@pytest.mark.parametrize("m", [24, 60])  # one block, a cluster
def test_solves_whose_start_has_converged(gpulib, m):
    # they end before the first cycle, which is what first waits for the block's bulk copies; other
    # solves take the same places on the device right behind them
    M = gpulib.Mesh(*synth.jittered_square(m, seed=1))
    ng, bd = gpulib.get_ngauss(M), gpulib.bcnode(M)
    A, B = gpulib.PoissonSystem(M), gpulib.PoissonSystem(M)
    for S in (A, B):
        S.set_dirichlet(bd)
        S.assemble(t(np.ones(ng)), t(np.ones(ng)))
    ref, zero = B.solve(rtol=1e-12), torch.zeros(M.nnode, dtype=torch.float64, device="cuda")
    for _ in range(100):
        assert not bool(A.adjoint(zero).any()) and A.last_stats.iterations == 0
        assert torch.equal(B.solve(rtol=1e-12), ref)


@pytest.mark.parametrize("m", [64, 100, 300])  # a cluster, graphs
def test_warm_start_that_is_there_right_after_an_assembly(oracle, gpulib, m):
    # (it is found by its residual, before the hierarchy has the assembly's values, which the solves
    # after it need)
    coords, elems = synth.jittered_square(m, seed=2)
    O = oracle.OracleMesh(coords, elems)
    rng = np.random.default_rng(m)
    bd = O.bcnode()
    bv = rng.random(bd.size)
    S = gpulib.PoissonSystem(gpulib.Mesh(coords, elems))
    S.set_dirichlet(bd, bv)
    f = rng.random(O.ngauss)
    for scale in (1.0, 1e3):
        kappa = scale * (1.0 + 9.0 * rng.random(O.ngauss))
        B, b = oracle.dirichlet_csc(O.laplace_csc(kappa), O.source(f), bd, bv)
        ref = oracle.spsolve(B, b)
        S.assemble(t(kappa), t(f))
        for precision in ("mixed", "fp64"):
            w = S.solve(t(ref), precision=precision, rtol=1e-8, warm=True)
            assert S.last_stats.iterations == 0 and rel(w, ref) < 1e-9
        w = S.solve(t(0.0 * ref), rtol=1e-12, warm=True)  # (far from there)
        assert 0 < S.last_stats.iterations < 60 and rel(w, ref) < 1e-9
        u = S.solve(rtol=1e-12)
        assert rel(u, ref) < 1e-9 and rel(S.solve(t(ref), rtol=1e-8, warm=True), ref) < 1e-9
        # a NaN start is no start: the solve ends with a status, and the next is as before
        with pytest.raises(gpulib.AdFemError):
            S.solve(torch.full_like(u, float("nan")), rtol=1e-12, warm=True)
        S.assemble(t(kappa), t(f))
        assert torch.equal(S.solve(rtol=1e-12), u)
