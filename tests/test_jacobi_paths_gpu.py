"""The Jacobi iterations of resident systems, which serve what multigrid does not (no Dirichlet DOFs, no
hierarchy, profiled solves, solves that multigrid gives up): the checks of test_mixed_paths_gpu.py and
test_checks_build_gpu.py with multigrid switched off, so that it is these iterations that run.

The path that ran is identified by its launches: one (mixed) or three (FP64) an iteration, the checks and
the chunks in flight at the end beside them; multigrid takes three for a whole small solve and over 20
an iteration otherwise.
"""
import os
import subprocess
import sys

import pytest

import test_checks_build_gpu as C
import test_mixed_paths_gpu as P

pytestmark = pytest.mark.gpu


@pytest.fixture
def solves(gpulib, monkeypatch):
    """(precision, iterations, launches, banded) of every resident solve of a test, multigrid off."""
    monkeypatch.setenv("ADFEM_MG", "0")
    from adfem_gpu import system as SY

    seen, solve = [], SY._System.solve

    def recorded(self, *a, **kw):
        u = solve(self, *a, **kw)
        st = self.last_stats
        seen.append((kw["precision"], st.iterations, st.launches, self.solver_info()["banded"]))
        return u

    monkeypatch.setattr(SY._System, "solve", recorded)
    return seen


@pytest.mark.parametrize("name,args", [("test_randomly_renumbered_mesh", (40,)), ("test_randomly_renumbered_mesh", (80,)),
                                       ("test_renumbered_elasticity", ()), ("test_system_reports_banded_layout", ()),
                                       ("test_elasticity_block_form_super_tiles", ("",))])
def test_mixed_path_checks(oracle, gpulib, monkeypatch, solves, name, args):
    getattr(P, name)(oracle, gpulib, monkeypatch, *args)
    assert any(p == "mixed" for p, *_ in solves)
    for precision, its, launches, banded in solves:
        assert its > 60 and banded == 1  # (multigrid needs fewer on the scalar cases, and fewer launches)
        assert (1 if precision == "mixed" else 3) <= launches / its < 15, (precision, its, launches)


def test_dependent_launches(gpulib, monkeypatch, solves):
    P.test_dependent_launches_bit_identical(gpulib, monkeypatch)
    assert len(solves) == 2 and all(its > 500 and 1 <= n / its < 15 for _, its, n, _ in solves)


def test_checks_build_without_multigrid(gpulib):
    import build as B

    lib = B.build(checks=True)
    r = subprocess.run([sys.executable, "-c", C.SCRIPT, lib], cwd=C.ROOT, capture_output=True, text=True, timeout=900,
                       env=dict(os.environ, ADFEM_MG="0"))
    assert r.returncode == 0 and "checks build ok" in r.stdout, (r.stdout[-2000:], r.stderr[-4000:])
