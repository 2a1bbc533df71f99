"""CPU check of the rounding of composite register butterflies (fft_core.cuh):
forward and inverse of random data are as close to the data as with the
symmetric DFT of the same size (within 3 %, the scatter of 4000 draws being
below 1 %), and the mean gain, which repeated transforms such as the slices of
beam propagation add up, stays within 2e-8, a sixth of the spacing of
floats at 1."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "inverse_solver_b200", "csrc")


@pytest.fixture(scope="module")
def figures(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("bf") / "butterfly_host_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I" + os.environ.get("CUDA_HOME", "/usr/local/cuda") + "/include",
                    "-I" + CSRC, os.path.join(ROOT, "tests", "native", "butterfly_host_check.cpp"), "-o", exe],
                   check=True)
    out = subprocess.run([exe], capture_output=True, text=True, check=True).stdout
    return {int(l.split()[0]): [float(x) for x in l.split()[1:]] for l in out.splitlines()}


@pytest.mark.parametrize("r", [9, 15, 21, 25, 27])
def test_composite_butterfly_rounds_like_the_symmetric_one(figures, r):
    err, gain, err_sym, _ = figures[r]
    assert err <= 1.03 * err_sym
    assert abs(gain) <= 2e-8
