"""Scalar matrix and load of small P1 meshes, whose rows are summed straight from the Gauss-point
inputs, next to the meshes beside that rule (wide rows, many nodes), against the oracle.

Bars: an entry is a sum of at most 16 terms, each a product of the geometry factor and a sum of three
inputs: within 64 roundings of the sum of magnitudes, taken as 1e-13 of the largest entry.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from adfem_gpu import synth, system

pytestmark = pytest.mark.gpu

MESHES = {
    "one cell": lambda: synth.jittered_square(1, seed=1),
    "3x5": lambda: synth.jittered_square(3, n=5, seed=2),
    "one block of rows": lambda: synth.jittered_square(7, n=7, seed=3),
    "one row more": lambda: synth.jittered_square(12, n=4, seed=4),
    "33x29": lambda: synth.jittered_square(33, n=29, seed=5),
    "rows of 9": lambda: synth.fan_mesh(8, rings=2),
    "rows of 16": lambda: synth.fan_mesh(15, rings=2),
    "rows of 17": lambda: synth.fan_mesh(16, rings=2),
    "rows of 41": lambda: synth.fan_mesh(40, rings=2),
    "below the limit": lambda: synth.jittered_square(315, n=315, seed=6),
    "above the limit": lambda: synth.jittered_square(316, n=316, seed=7),
}


@pytest.mark.parametrize("name", list(MESHES))
def test_rows_match_oracle(oracle, gpulib, name):
    coords, elems = MESHES[name]()
    O = oracle.OracleMesh(coords, elems)
    mesh = gpulib.Mesh(coords, elems)
    rng = np.random.default_rng(len(elems))
    kappa, f, r0 = 0.1 + rng.random(O.ngauss), rng.standard_normal(O.ngauss), rng.standard_normal(mesh.ndof)
    dev = lambda a: torch.tensor(a, device="cuda")
    K = O.laplace_csc(kappa)
    K.sort_indices()
    v = system.laplace_csr(mesh, dev(kappa)).cpu().numpy()
    assert np.array_equal(K.indices, mesh.pattern()[1] - 1)
    assert np.max(np.abs(v - K.data)) <= 1e-13 * np.max(np.abs(K.data))
    F = O.source(f)
    s = system.source(mesh, dev(f)).cpu().numpy()
    assert np.max(np.abs(s - F)) <= 1e-13 * np.max(np.abs(F))
    a = system.source(mesh, dev(f), rhs=dev(r0), accumulate=True).cpu().numpy()
    assert np.max(np.abs(a - (r0 + F))) <= 1e-13 * max(np.max(np.abs(F)), np.max(np.abs(r0)))
    z = system.source(mesh, dev(f), accumulate=True).cpu().numpy()
    assert np.array_equal(z, s)
