"""Operator kernels that stage a tile of Gauss points in shared memory or walk elements by pairs,
against the oracle: meshes around the edges of the tiles (fewer elements than a tile, one tile,
remainders) and inputs that are only 8-byte aligned.

Bars: COO indices equal; values within 1e-12 of the output's largest entry (64-bit sums of at
most a few dozen terms of that size: the rounding of any order stays two orders below).
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from adfem_gpu import synth

pytestmark = pytest.mark.gpu
TOL = 1e-12


def rel(a, b):
    a = a.cpu().numpy() if hasattr(a, "cpu") else np.asarray(a)
    return float(np.max(np.abs(a - b)) / np.max(np.abs(b)))


def dev(a, shift):
    """a on the device, `shift` doubles past a 16-byte boundary."""
    a = np.ascontiguousarray(a, dtype=np.float64).ravel()
    t = torch.empty(a.size + 2, dtype=torch.float64, device="cuda")[shift:shift + a.size]
    t.copy_(torch.tensor(a))
    assert t.is_contiguous() and (t.data_ptr() % 16 == 0) == (shift == 0)
    return t


# elements: 2, 20 (less than a tile), 42 (an elasticity tile, two P2 tiles, a Laplace tile and 2),
# 40 (a Laplace tile), 130 (a backward block and 2)
@pytest.mark.parametrize("m,n", [(1, 1), (2, 5), (3, 7), (4, 5), (5, 13)])
@pytest.mark.parametrize("degree,shift", [(1, 0), (1, 1), (2, 0), (2, 1)])
def test_scalar_operators(oracle, gpulib, m, n, degree, shift):
    from adfem_gpu import system as S

    coords, elems = synth.jittered_square(m, n=n, seed=m + n)
    O = oracle.OracleSpace(coords, elems, degree)
    M = gpulib.Mesh(coords, elems, degree=degree)
    ng, ndof = gpulib.get_ngauss(M), M.ndof
    rng = np.random.default_rng(7)
    kappa, f = 1 + rng.random(ng), rng.standard_normal(ng)
    idx, vv = S.laplace_coo(M, dev(kappa, shift))
    oi, ov = O.laplace_coo(kappa)
    np.testing.assert_array_equal(idx.cpu().numpy(), oi)
    assert rel(vv, ov) < TOL
    g = rng.standard_normal(ov.size)
    assert rel(S.laplace_coo_backward(M, dev(g, shift)), O.laplace_coo_backward(g)) < TOL
    assert rel(S.laplace_csr(M, dev(kappa, shift)), O.laplace_csc(kappa).data) < TOL
    assert rel(S.mass_csr(M, dev(kappa, shift)), O.mass_csc(kappa).data) < TOL
    assert rel(S.source(M, dev(f, shift)), O.source(f)) < TOL
    gr = rng.standard_normal(ndof)
    assert rel(S.source_backward(M, dev(gr, shift)), O.source_backward(gr)) < TOL
    assert rel(S.dof_to_gauss(M, dev(gr, shift)), O.dof_to_gauss(gr)) < TOL
    assert rel(S.dof_to_gauss_backward(M, dev(f, shift)), O.dof_to_gauss_backward(f)) < TOL


@pytest.mark.parametrize("m,n", [(1, 1), (2, 5), (3, 7), (5, 13)])
@pytest.mark.parametrize("shift", [0, 1])
def test_elasticity_operators(oracle, gpulib, m, n, shift):
    from adfem_gpu import system as S

    coords, elems = synth.jittered_square(m, n=n, seed=m + n)
    O = oracle.OracleMesh(coords, elems)
    M = gpulib.Mesh(coords, elems)
    rng = np.random.default_rng(9)
    D = rng.standard_normal((O.ngauss, 3, 3))
    idx, vv = S.stiffness_coo(M, dev(D, shift))
    oi, ov = O.stiffness_coo(D)
    np.testing.assert_array_equal(idx.cpu().numpy(), oi)
    assert rel(vv, ov) < TOL
    g = rng.standard_normal(ov.size)
    assert rel(S.stiffness_coo_backward(M, dev(g, shift)), O.stiffness_coo_backward(g).ravel()) < TOL
    for mode in (0, 1):
        k = 9 * (m * n) + 1  # blocks of 256 points with a remainder
        E, nu = 1 + rng.random(k), 0.05 + 0.4 * rng.random(k)
        g9 = rng.standard_normal(9 * k)
        assert rel(S.plane_strain(dev(E, shift), dev(nu, shift), mode), oracle.plane_strain(E, nu, mode).ravel()) < TOL
        gE, gn = S.plane_strain_backward(dev(g9, shift), dev(E, shift), dev(nu, shift), mode)
        oE, on = oracle.plane_strain_backward(g9, E, nu, mode)
        assert rel(gE, oE) < TOL and rel(gn, on) < TOL
