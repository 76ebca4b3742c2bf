"""K\\F of a matrix whose band is beyond 16-bit column differences: the multigrid solve and the Jacobi
iterations on 32-bit columns, against the direct solve.

Bars: the FP64 solve ends at a residual of 1e-12 |b| in the Jacobi-scaled norm, and the condition number
is below 1e5 (272 cells a side: about (4 / pi^2) 272^2 times a coefficient ratio of 3), so 1e-7 relative
(2-norm); the mixed solve ends at 1e-11: 1e-6.
"""
import numpy as np
import pytest

pytest.importorskip("torch")

from scipy import sparse as sp

from adfem_gpu import synth

pytestmark = pytest.mark.gpu


def test_randomly_numbered_matrix(oracle, gpulib):
    coords, elems = synth.jittered_square(256, n=272, seed=1)
    O = oracle.OracleMesh(coords, elems)
    rng = np.random.default_rng(1)
    bd = O.bcnode()
    B, r = oracle.dirichlet_csc(O.laplace_csc(1.0 + 2.0 * rng.random(O.ngauss)), O.source(rng.random(O.ngauss)), bd,
                                rng.random(bd.size))
    ref = oracle.spsolve(B, r)
    p = rng.permutation(O.ndof)
    K = sp.csc_matrix(B)[p][:, p].tocsc()
    K.sort_indices()
    C = K.tocoo()
    assert np.max(np.abs(C.row - C.col)) > 32767
    for precision, rtol, bar in (("fp64", 1e-12, 1e-7), ("mixed", 1e-11, 1e-6)):
        u, st = gpulib.solve(K, r[p], precision=precision, rtol=rtol, return_stats=True)
        assert st.status == 0 and np.linalg.norm(u - ref[p]) < bar * np.linalg.norm(ref)
        assert (st.iterations < 60) == (precision == "fp64")
        w, st = gpulib.solve(K, r[p], precision=precision, rtol=rtol, u0=u, return_stats=True)
        assert st.iterations <= 3 and np.linalg.norm(w - ref[p]) < bar * np.linalg.norm(ref)
