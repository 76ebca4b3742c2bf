"""Multigrid-preconditioned CG of resident systems against the direct solve and the Jacobi
iterations: sizes around the edges of the hierarchy (no hierarchy at all, one-launch cycle only,
first level above the one-launch tail), wide rows, renumbered meshes, and the cases that keep or
fall back to the Jacobi iteration.

Bars: 1e-9 relative (max norm) against the direct solve, as for every solve of this suite.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from adfem_gpu import synth

pytestmark = pytest.mark.gpu


def rel(a, b):
    a = a.cpu().numpy() if hasattr(a, "cpu") else np.asarray(a)
    return float(np.max(np.abs(a - b)) / max(np.max(np.abs(b)), 1e-300))


def t(a):
    return torch.tensor(np.asarray(a, dtype=np.float64), device="cuda")


def poisson(gpulib, oracle, coords, elems, contrast=1e3, bv=None):
    O = oracle.OracleMesh(coords, elems)
    g = O.gauss_nodes()
    G = synth.fourier_field(g[:, 0], g[:, 1], seed=1)
    kappa = 1 + np.exp(synth.contrast_sigma(G, contrast) * G)
    f = 1e5 * (g[:, 0] + g[:, 1])
    bd = O.bcnode()
    bv = np.zeros(bd.size) if bv is None else bv(O.coords[bd - 1])
    S = gpulib.PoissonSystem(gpulib.Mesh(coords, elems))
    S.set_dirichlet(bd, bv)
    S.assemble(t(kappa), t(f))
    B, r = oracle.dirichlet_csc(O.laplace_csc(kappa), O.source(f), bd, bv)
    return S, oracle.spsolve(B, r), (O, kappa, f, bd, B, r)


# (m, n): 12 x 12 nodes stay below the directly solved size (no hierarchy), 13 x 13 are just above
# it; 80 x 64 nodes = 5120 unknowns are the largest one-launch cycle, 81 x 64 the first above it
@pytest.mark.parametrize("m,n", [(11, 11), (12, 12), (40, 3), (63, 63), (79, 63), (80, 63), (141, 97)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_poisson_sizes(oracle, gpulib, m, n, precision):
    S, u0, (O, *_) = poisson(gpulib, oracle, *synth.jittered_square(m, n=n, seed=3), bv=lambda x: np.sin(3 * x[:, 0]))
    u = S.solve(precision=precision, rtol=1e-12)
    assert S.last_stats.status == 0 and rel(u, u0) < 1e-9
    if (m + 1) * (n + 1) > 160:
        assert 0 < S.last_stats.iterations < 60  # (Jacobi-CG needs several times as many)
    assert torch.equal(S.solve(precision=precision, rtol=1e-12), u)


@pytest.mark.parametrize("m,n", [(8, 5), (36, 35), (63, 39), (64, 39), (90, 70)])
def test_elasticity_sizes(oracle, gpulib, m, n):
    coords, elems = synth.jittered_square(m, n=n, seed=2)
    O = oracle.OracleMesh(coords, elems)
    g = O.gauss_nodes()
    E, nu = 1e9 * np.exp(0.3 * synth.fourier_field(g[:, 0], g[:, 1], seed=2)), np.full(O.ngauss, 0.3)
    fx, fy = np.full(O.ngauss, 1e5), np.full(O.ngauss, -1e6)
    left = synth.left_edge_nodes(coords) + 1
    bd = np.concatenate([left, left + O.ndof])
    B, r = oracle.dirichlet_csc(O.stiffness_csc(oracle.plane_strain(E, nu, 0)),
                                np.concatenate([O.source(fx), O.source(fy)]), bd, np.zeros(bd.size))
    S = gpulib.ElasticitySystem(gpulib.Mesh(coords, elems))
    S.set_dirichlet(bd)
    S.assemble(t(E), t(nu), t(fx), t(fy))
    u = S.solve(precision="mixed", rtol=1e-12)
    assert S.last_stats.status == 0 and rel(u, oracle.spsolve(B, r)) < 1e-9
    if 2 * O.ndof > 160:
        assert S.last_stats.iterations < 120


def test_p2_and_fan_and_renumbered(oracle, gpulib):
    coords, elems = synth.jittered_square(40, seed=5)
    O = oracle.OracleSpace(coords, elems, 2)
    M = gpulib.Mesh(coords, elems, degree=2)
    g = gpulib.gauss_nodes(M)
    kappa, f = synth.poisson_c1_fields(g[:, 0], g[:, 1])
    bd = gpulib.bcnode(M)
    S = gpulib.PoissonSystem(M)
    S.set_dirichlet(bd)
    S.assemble(t(kappa), t(f))
    B, r = oracle.dirichlet_csc(O.laplace_csc(kappa), O.source(f), bd, np.zeros(bd.size))
    u = S.solve(precision="mixed", rtol=1e-12)
    assert rel(u, oracle.spsolve(B, r)) < 1e-9 and S.last_stats.iterations < 100
    for coords, elems in (synth.fan_mesh(40, rings=6), synth.fan_mesh(63, rings=4)):
        S, u0, _ = poisson(gpulib, oracle, coords, elems, contrast=10.0)
        assert rel(S.solve(rtol=1e-12), u0) < 1e-9
    coords, elems = synth.jittered_square(70, seed=6)
    perm = np.random.default_rng(5).permutation(coords.shape[0])
    inv = np.empty_like(perm)
    inv[perm] = np.arange(perm.size)
    S, u0, _ = poisson(gpulib, oracle, coords[perm], inv[elems - 1] + 1)
    assert rel(S.solve(rtol=1e-12), u0) < 1e-9 and S.last_stats.iterations < 60


def test_limits_warm_start_and_changed_data(oracle, gpulib):
    S, u0, (O, kappa, f, bd, B, r) = poisson(gpulib, oracle, *synth.jittered_square(80, seed=1))
    # an unattainable tolerance ends at the attainable residual, a small cap with the status
    u = S.solve(rtol=1e-18)
    assert S.last_stats.status == 0 and 1e-18 < S.last_stats.relres < 1e-11 and rel(u, u0) < 1e-9
    with pytest.raises(gpulib.AdFemError) as e:
        S.solve(rtol=1e-12, max_iter=3)
    assert e.value.status == gpulib._lib.ERR_NOT_CONVERGED and S.last_stats.iterations == 3
    # warm start from the solution, zero right-hand side
    w = S.solve(t(u0), rtol=1e-9, warm=True)
    assert S.last_stats.iterations == 0 and rel(w, u0) < 1e-9
    lam = S.adjoint(torch.zeros(O.ndof, dtype=torch.float64, device="cuda"))
    assert S.last_stats.iterations == 0 and not bool(lam.any())
    # other coefficients, other Dirichlet DOFs on the same system
    k2, bd2 = kappa[::-1].copy(), bd[: bd.size // 2]
    S.set_dirichlet(bd2, np.ones(bd2.size))
    S.assemble(t(k2), t(f))
    B2, r2 = oracle.dirichlet_csc(O.laplace_csc(k2), O.source(f), bd2, np.ones(bd2.size))
    assert rel(S.solve(rtol=1e-12), oracle.spsolve(B2, r2)) < 1e-9


def test_jacobi_iterations_stay_selectable_and_serve_what_multigrid_does_not(oracle, gpulib, monkeypatch):
    coords, elems = synth.jittered_square(50, seed=1)
    monkeypatch.setenv("ADFEM_MG", "0")
    S, u0, _ = poisson(gpulib, oracle, coords, elems)
    assert rel(S.solve(rtol=1e-12), u0) < 1e-9 and S.last_stats.iterations > 200
    out = {}
    for pdl in ("0", "1"):  # dependent launches of the banded iteration: same bits
        monkeypatch.setenv("ADFEM_ZCG_PDL", pdl)
        S, _, _ = poisson(gpulib, oracle, coords, elems)
        out[pdl] = S.solve(precision="mixed", rtol=1e-11)
    assert torch.equal(out["0"], out["1"])
    monkeypatch.delenv("ADFEM_ZCG_PDL")
    monkeypatch.delenv("ADFEM_MG")
    # an indefinite operator (negative coefficients in a corner) ends with the breakdown status
    O = oracle.OracleMesh(coords, elems)
    g = O.gauss_nodes()
    kappa = np.where((g[:, 0] < 0.2) & (g[:, 1] < 0.2), -0.05, 1.0)
    S = gpulib.PoissonSystem(gpulib.Mesh(coords, elems))
    S.set_dirichlet(O.bcnode())
    with pytest.raises(gpulib.AdFemError) as e:
        S.assemble(t(kappa), t(np.ones(O.ngauss)))
        S.solve(rtol=1e-12)
    assert e.value.status == gpulib._lib.ERR_BREAKDOWN
    # no Dirichlet DOFs: singular; a compatible load converges through the Jacobi iteration
    S = gpulib.PoissonSystem(gpulib.Mesh(coords, elems))
    f = np.sign(g[:, 0] - 0.5)
    S.assemble(t(np.ones(O.ngauss)), t(np.zeros(O.ngauss)))
    b = O.source(f)
    b -= b.mean()
    u = S.adjoint(t(b), rtol=1e-8).cpu().numpy()
    assert np.max(np.abs(O.laplace_csc(np.ones(O.ngauss)) @ u - b)) < 1e-6 * np.max(np.abs(b))
