"""FP64 Jacobi solves of resident systems scale the operator in place: they need no memory beyond the
system's own, and what else reads the operator in the same assembly stays right.

Bars: 1e-7 relative (max norm) against the direct solve: the solves end at a residual of 1e-11 |b| and
the condition number is below 1e4 (40 x 40 cells: about (4 / pi^2) 40^2 times a coefficient ratio of 10);
1e-12 for products.
"""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from adfem_gpu import _lib, synth
from adfem_gpu import system as SY

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.max(np.abs(a.cpu().numpy() - b)) / np.max(np.abs(b)))


def t(a):
    return torch.tensor(np.asarray(a, dtype=np.float64), device="cuda")


# the iterations: banded and scaled mixed, banded and plain FP64; a system that multigrid does not solve
# because the variant was chosen (ADFEM_ZCG*), it was switched off, or nothing is fixed
@pytest.mark.parametrize("env", [{"ADFEM_MG": "0"}, {"ADFEM_ZCG": "0"}, {"ADFEM_ZCG64": "1"}, {}])
def test_fp64_solves_allocate_nothing_and_share_the_operator(oracle, gpulib, monkeypatch, env):
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    coords, elems = synth.jittered_square(40, seed=3)
    O = oracle.OracleMesh(coords, elems)
    rng = np.random.default_rng(1)
    kappa, f = 1 + 9 * rng.random(O.ngauss), rng.random(O.ngauss)
    S = gpulib.PoissonSystem(gpulib.Mesh(coords, elems))
    bd = O.bcnode() if env else np.zeros(0, dtype=np.int64)
    S.set_dirichlet(bd)
    x = rng.standard_normal(O.ndof)
    L, got = _lib.load(), []
    for rep in range(2):
        S.assemble(t(kappa), t(f))
        if env:
            B, r = oracle.dirichlet_csc(O.laplace_csc(kappa), O.source(f), bd, np.zeros(bd.size))
            ref = oracle.spsolve(B, r)
            solve = lambda p: S.solve(precision=p, rtol=1e-12 if p == "fp64" else 1e-11)  # noqa: E731
        else:
            B = O.laplace_csc(kappa)  # singular: a compatible load, the solution up to a constant
            r = O.source(f)
            r -= r.mean()
            ref = np.append(oracle.spsolve(B[:-1][:, :-1].tocsc(), r[:-1]), 0.0)
            ref -= ref.mean()

            def solve(p):
                u = S.adjoint(t(r), precision=p, rtol=1e-12 if p == "fp64" else 1e-11)
                return u - u.mean()

        assert rel(S.apply(t(x)), B @ x) < 1e-12
        try:
            L.adfem_debug_fail_alloc(0)  # (the next device allocation fails)
            u = solve("fp64")
            w = solve("mixed")
        finally:
            L.adfem_debug_fail_alloc(-1)
        assert rel(u, ref) < 1e-7 and rel(w, ref) < 1e-7
        assert rel(S.apply(t(x)), B @ x) < 1e-12
        if env:
            (p,), _ = SY.solve_packed([S], rtol=1e-11)
            assert rel(p, ref) < 1e-7
        assert torch.equal(solve("fp64"), u)
        got.append((u, w))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])


def test_profiled_fp64_solve_leaves_multigrid_its_operator(oracle, gpulib):
    coords, elems = synth.jittered_square(40, seed=3)
    O = oracle.OracleMesh(coords, elems)
    rng = np.random.default_rng(2)
    kappa, f = 1 + 9 * rng.random(O.ngauss), rng.random(O.ngauss)
    bd = O.bcnode()
    B, r = oracle.dirichlet_csc(O.laplace_csc(kappa), O.source(f), bd, np.zeros(bd.size))
    ref = oracle.spsolve(B, r)
    S = gpulib.PoissonSystem(gpulib.Mesh(coords, elems))
    S.set_dirichlet(bd)
    S.assemble(t(kappa), t(f))
    u0 = S.solve(rtol=1e-12)
    o, st, v = gpulib.solver_opts(rtol=1e-12), _lib.SolverStats(), torch.zeros_like(u0)
    ms, n = (ctypes.c_double * 4)(), (ctypes.c_longlong * 4)()
    for _ in range(2):
        assert _lib.load().adfem_system_solve_profiled_d(S.handle, _lib.ptr(v), ctypes.byref(o), ctypes.byref(st), ms,
                                                         n, None) == 0
        torch.cuda.synchronize()
        assert st.iterations > 60 and rel(v, ref) < 1e-7
        assert torch.equal(S.solve(rtol=1e-12), u0) and S.last_stats.iterations < 60
        S.assemble(t(kappa), t(f))
