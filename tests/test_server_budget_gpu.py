"""The server's device-memory budget and the multigrid hierarchies, which a system gets in its first solve
outside a pack: they are booked before they are made, idle systems give way to them, and a request
that only its hierarchy keeps from fitting is solved without one.

Bars: 1e-9 relative (max norm) against the direct solve, as for every solve of this suite.
"""
import numpy as np
import pytest

pytest.importorskip("torch")

from adfem_gpu import synth

pytestmark = pytest.mark.gpu
JACOBI = 60  # iterations: the Jacobi iteration needs more on the cases here, multigrid fewer


def rel(a, b):
    return float(np.max(np.abs(np.asarray(a) - b)) / np.max(np.abs(b)))


class Case:
    def __init__(self, gpulib, oracle, m, seed):
        coords, elems = synth.jittered_square(m, seed=seed)
        O = oracle.OracleMesh(coords, elems)
        rng = np.random.default_rng(seed)
        self.mesh, self.kind = gpulib.Mesh(coords, elems), gpulib._lib.SYS_POISSON
        self.fields = (1 + 9 * rng.random(O.ngauss), rng.random(O.ngauss))
        self.bd = O.bcnode()
        B, r = oracle.dirichlet_csc(O.laplace_csc(self.fields[0]), O.source(self.fields[1]), self.bd,
                                    np.zeros(self.bd.size))
        self.ref = oracle.spsolve(B, r)

    def run(self, srv, **kw):
        resp, u, _ = srv.wait(srv.submit(self.mesh, self.kind, self.fields, self.bd, **kw))
        assert resp["status"] == 0 and rel(u, self.ref) < 1e-9
        return resp


def sizes(gpulib, case):
    """Booked bytes after a packed request and after an FP64 one on the same system."""
    with gpulib.Server(workers=1, precision="mixed", rtol=1e-12) as srv:
        assert case.run(srv)["packed"] == 1
        packed = srv.stats()["device_bytes"]
        r = case.run(srv, precision="fp64")
        assert r["packed"] == 0 and r["iterations"] < JACOBI
        both = srv.stats()["device_bytes"]
    assert both - packed > 100 * case.ref.size  # (the hierarchy)
    return packed, both


def accepted(gpulib, case, lo, hi):
    """The smallest budget in steps of 2 % from lo that takes the case's requests at all."""
    b = lo
    while True:
        assert b < hi
        with gpulib.Server(workers=1, hbm_budget_bytes=int(b), rtol=1e-12) as srv:
            try:
                case.run(srv)
                return int(b)
            except gpulib.AdFemError as e:
                assert e.status == gpulib._lib.ERR_BUSY
        b *= 1.02


def test_hierarchy_is_an_extra(gpulib, oracle):
    c = Case(gpulib, oracle, 48, 1)
    packed, both = sizes(gpulib, c)
    booked = 250 * c.ref.size + 65536
    # the smallest budget that takes the system and its buffers (as estimated, which is above what they
    # take): a first FP64 request has no room for a hierarchy beside the estimate and is solved without
    # one, the next has
    tight = accepted(gpulib, c, packed, packed + 2 * booked)
    with gpulib.Server(workers=1, precision="mixed", hbm_budget_bytes=tight, rtol=1e-12) as srv:
        assert c.run(srv, precision="fp64")["iterations"] > JACOBI
        assert srv.stats()["device_bytes"] <= tight
        assert c.run(srv)["packed"] == 1
        assert c.run(srv, precision="fp64")["iterations"] < JACOBI
        assert srv.stats()["device_bytes"] <= tight and srv.stats()["evictions"] == 0
        assert c.run(srv, precision="fp64")["iterations"] < JACOBI


def test_idle_systems_give_way_to_a_hierarchy(gpulib, oracle):
    a, b = Case(gpulib, oracle, 48, 1), Case(gpulib, oracle, 47, 2)
    with gpulib.Server(workers=1, precision="mixed", rtol=1e-12) as srv:
        a.run(srv)
        b.run(srv)
        two = srv.stats()["device_bytes"]
    # the smallest budget (in steps of 10 KB) that holds both systems at once, which is one that does not
    # hold a hierarchy beside them as it is booked
    budget, evictions = two, 1
    while evictions:
        budget += 10000
        assert budget < two + 250 * b.ref.size + 65536
        with gpulib.Server(workers=1, precision="mixed", hbm_budget_bytes=budget, rtol=1e-12) as srv:
            a.run(srv)
            b.run(srv)
            evictions = srv.stats()["evictions"]
            if evictions:
                continue
            assert b.run(srv, precision="fp64")["iterations"] < JACOBI
            st = srv.stats()
            assert st["evictions"] == 1 and st["device_bytes"] <= budget
            a.run(srv)
            assert srv.stats()["device_bytes"] <= budget
