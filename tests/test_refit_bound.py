"""The bound under which the searches take a refit from integer sums instead of the
reference's float steps (CPU only: the kernels' own header compiled for the host)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("g++ not available")
    exe = str(tmp_path_factory.mktemp("refit") / "refit_check")
    p = subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fno-strict-aliasing",
                        "-I", os.path.join(ROOT, "mptc_gb300", "csrc"),
                        os.path.join(ROOT, "tests", "c", "refit_check.cpp"), "-o", exe],
                       capture_output=True, text=True, timeout=120)
    assert p.returncode == 0, p.stderr[-3000:]
    return exe


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_sure_refits_are_the_float_steps(program, seed):
    r = subprocess.run([program, str(seed), "100000"], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
