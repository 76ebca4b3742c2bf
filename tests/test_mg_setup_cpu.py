"""The multigrid set-up on the host (adfem.jl_gb300/csrc/mg_setup.cpp) through mg_setup_harness.cpp,
with UndefinedBehaviorSanitizer where the compiler has it."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "adfem.jl_gb300", "csrc")


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    cuda_inc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    if not os.path.exists(os.path.join(cuda_inc, "cuda_runtime.h")):
        pytest.skip("CUDA headers not available")
    exe = str(tmp_path_factory.mktemp("mg") / "mg_setup")
    cmd = ["g++", "-std=c++17", "-O1", "-g", "-pthread", "-I", cuda_inc, "-I", CSRC, "-I", os.path.join(ROOT, "include"),
           "-o", exe, os.path.join(ROOT, "tests", "mg_setup_harness.cpp"), os.path.join(CSRC, "mg_setup.cpp")]
    if subprocess.run(cmd + ["-fsanitize=undefined", "-fno-sanitize-recover=all"], capture_output=True).returncode:
        subprocess.check_call(cmd)
    return exe


@pytest.mark.parametrize("what", ["limit", "exceptions"])
def test_mg_setup(harness, what):
    r = subprocess.run([harness, what], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "mg setup ok" in r.stdout, (r.stdout[-2000:], r.stderr[-2000:])
