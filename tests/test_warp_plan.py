"""The points a round of the warp search evaluates (sq_warp_plan.cuh): whatever the damping, every trial
the round comes to, and the probes it takes from the same round, are points of the round."""
import ctypes as C
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
BUILD = os.path.join(HERE, "_build")


@pytest.fixture(scope="module")
def lib():
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc is needed to build the host copy")
    os.makedirs(BUILD, exist_ok=True)
    out = os.path.join(BUILD, "libwarp_plan_host.so")
    r = subprocess.run([nvcc, "-O1", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-o", out,
                        os.path.join(HERE, "warp_plan_host.cu")], stdout=subprocess.PIPE, stderr=subprocess.STDOUT)
    assert r.returncode == 0, r.stdout.decode(errors="replace")
    return C.CDLL(out)


@pytest.mark.parametrize("W", [1, 2])
@pytest.mark.parametrize("nu", [2, 4, 1 << 30])
@pytest.mark.parametrize("mu", [0.0, 5e-324, 1e-300, 0.34, 0.5, 0.51, 1.0, 1.01, 1e300, float("inf"), float("nan")])
@pytest.mark.parametrize("rejected", [0.0, 5e-324, 1.0, float("inf")])
def test_a_round_holds_what_it_is_read_for(lib, W, nu, mu, rejected):
    out = (C.c_int * 64)()
    lib.wph_plan(W, C.c_double(mu), C.c_double(rejected), nu, out)
    trials = out[1]
    groups = [(out[2 + 2 * g], out[3 + 2 * g]) for g in range(6 * W)]
    assert 0 < trials <= 6 * W
    for a in range(trials):
        g, probed = out[2 + 12 * W + 2 * a], out[3 + 12 * W + 2 * a]
        assert 0 <= g < 6 * W and groups[g] == (a, 0)
        if probed:
            assert g + 2 < 6 * W and groups[g + 1:g + 3] == [(a, 1), (a, 2)]
