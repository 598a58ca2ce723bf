"""The FP32 decision of the restart rule's isInside test (insideFast) against the FP64 expression.

A verdict has to be the FP64 expression's at every shape the engine accepts; where the value is near
1 there must be none (-1: the kernels then evaluate the FP64 expression)."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

import oracle
from oracle import OracleScene
from parity_util import oracle_state, restore_oracle, snapshot_into
from sudodem_gb300 import Engine, assemblies

HERE = os.path.dirname(os.path.abspath(__file__))
BUILD = os.path.join(HERE, "_build")
LIB = os.path.join(BUILD, "libinside_host.so")
SOURCES = [os.path.join(HERE, "inside_host.cu"), os.path.join(HERE, "..", "sudodem_gb300", "csrc", "sq_device.cuh")]
SMALL = [(a, b) for a in (0.01, 0.02, 0.03) for b in (1.0, 1.5, 1.9)]


@pytest.fixture(scope="module")
def lib():
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc is needed to build the host copy")
    if not os.path.exists(LIB) or any(os.path.getmtime(s) > os.path.getmtime(LIB) for s in SOURCES):
        os.makedirs(BUILD, exist_ok=True)
        cmd = [nvcc, "-O2", "-std=c++17", "-Xcompiler", "-fPIC", "-Xcompiler", "-ffp-contract=off", "--fmad=false",
               "-diag-suppress", "1444", "-shared", "-o", LIB + ".tmp", SOURCES[0]]
        r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT)
        assert r.returncode == 0, r.stdout.decode(errors="replace")
        os.replace(LIB + ".tmp", LIB)
    return C.CDLL(LIB)


def _verdicts(lib, rows):
    rows = np.ascontiguousarray(rows, dtype=np.float64)
    fast, exact = np.zeros(len(rows), np.int32), np.zeros(len(rows), np.int32)
    ip, dp = C.POINTER(C.c_int), C.POINTER(C.c_double)
    lib.inh_test(rows.ctypes.data_as(dp), C.c_long(len(rows)), fast.ctypes.data_as(ip), exact.ctypes.data_as(ip))
    return fast, exact


def _rows(rng, n, radii, eps, ratios):
    q = rng.standard_normal((n, 4))
    q /= np.linalg.norm(q, axis=1)[:, None]
    w, x, y, z = q.T
    R = np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y), 2 * (x * y + w * z),
                  1 - 2 * (x * x + z * z), 2 * (y * z - w * x), 2 * (x * z - w * y), 2 * (y * z + w * x),
                  1 - 2 * (x * x + y * y)], -1).reshape(-1, 3, 3)
    return np.hstack([radii, eps, q, np.einsum("nij,nj->ni", R, ratios * radii)])


@pytest.mark.parametrize("eps", SMALL + [(0.01, 0.01), (1.99, 0.01), (0.01, 1.99), (1.0, 1.0), None])
@pytest.mark.parametrize("size,aspect", [(1e-3, 1.5), (1e-3, 1000.0), (1e-17, 1.5), (1e4, 20.0)])
def test_verdict_is_the_fp64_expressions(lib, eps, size, aspect):
    """Points of log-uniform coordinates between 0.001 and 1 of the radii, and points scaled next to the
    surface, in turned and stretched shapes."""
    rng = np.random.default_rng(7)
    n = 200000
    radii = size * np.exp(rng.uniform(0, np.log(aspect), (n, 3)))
    e = rng.uniform(0.01, 1.99, (n, 2)) if eps is None else np.tile(eps, (n, 1))
    u = np.exp(rng.uniform(np.log(1e-3), 0, (n, 3)))
    # half of them: the largest coordinate moved so that no other alone decides, and up to 1.3
    near = rng.random(n) < 0.5
    k = rng.integers(0, 3, n)
    u[near, k[near]] = rng.uniform(0.3, 1.3, near.sum())
    fast, exact = _verdicts(lib, _rows(rng, n, radii, e, u * rng.choice([-1, 1], (n, 3))))
    said = fast >= 0
    assert np.array_equal(fast[said], exact[said])
    # the value as it is in exact arithmetic: a verdict wherever it is clear of the band
    m, t = np.maximum(u[:, 0], u[:, 1]), np.minimum(u[:, 0], u[:, 1]) / np.maximum(u[:, 0], u[:, 1])
    with np.errstate(under="ignore", over="ignore"):
        v = m ** (2 / e[:, 1]) * (1 + t ** (2 / e[:, 0])) ** (e[:, 0] / e[:, 1]) + u[:, 2] ** (2 / e[:, 1])
    assert np.all(fast[(v < 0.899) | (v > 1.101)] >= 0)
    assert np.all(fast[(v > 0.901) & (v < 1.099)] == -1)


def test_no_verdict_without_a_value(lib):
    """Exponents beyond the bound's range, radii outside FP32's, points that are no numbers."""
    def row(r=(1e-3, 1e-3, 1e-3), eps=(1.0, 1.0), p=(1e-4, 1e-4, 1e-4)):
        return [*r, *eps, 1, 0, 0, 0, *p]
    nan = float("nan")
    rows = [row(eps=(0.005, 1.0)), row(eps=(1.0, 0.005)), row(r=(1e-40, 1e-40, 1e-40), p=(1e-41,) * 3),
            row(r=(1e30, 1e30, 1e30), p=(1e29,) * 3), row(p=(nan, 0, 0)), row(p=(0, nan, 0)), row(p=(0, 0, nan))]
    fast, _ = _verdicts(lib, rows)
    assert np.all(fast == -1)
    fast, exact = _verdicts(lib, [row(p=(0, 0, 0)), row(p=(1e300, 0, 0))])
    assert list(fast) == [1, 0] and list(exact) == [1, 0]


def _pairs(eps1, eps2, n):
    """n pairs of particles, each pair deep in contact and far from the others."""
    rng = np.random.default_rng(11)
    b = assemblies._builder()
    for i in range(n):
        at = np.array([i % 20, i // 20 % 20, i // 400]) * 0.01
        sides = []
        for _ in range(2):
            q = rng.standard_normal(4)
            sides.append((rng.uniform(0.8e-3, 1.2e-3, 3), assemblies._quat_normalize(q)))
        u = rng.standard_normal(3)
        gap = rng.uniform(0.7, 1.1) * 1e-3
        assemblies._add_sq(b, sides[0][0], [eps1, eps2], sides[0][1], at, 2650.0)
        assemblies._add_sq(b, sides[1][0], [eps1, eps2], sides[1][1], at + gap * u / np.linalg.norm(u), 2650.0)
    params = {"dt": 1e-9, "gravity": (0.0, 0.0, 0.0), "damping": 0.0, "verletDist": 1e-4, "targetInterv": 50,
              "minSweepDistFactor": 0.1, "sortAxis": 0, "isSuperquadrics": 1, "exactAsphericalRot": 1}
    return assemblies._finish(b, assemblies.default_material(), params, {})


@pytest.mark.gpu
@pytest.mark.parametrize("eps1,eps2", SMALL)
def test_gpu_warm_deep_pairs_restart_as_the_oracle(gpu, eps1, eps2):
    """One step of 800 deep pairs from stored directions a little off: a search that ends far apart
    is run again from the centre line unless both points are inside the other particle.  Where the oracle's
    own answer does not move when its pow, sin, cos and atan2 results move by an ulp (six times, all
    directions within 1e-6), the GPU ends within 1e-5 of it, lmder2's last step."""
    spec = _pairs(eps1, eps2, 800)
    orc = OracleScene.from_spec(spec, threads=os.cpu_count())
    orc.step(1)
    recs = orc.interactions()
    rng = np.random.default_rng(3)
    recs[:, 5:7] += rng.uniform(-0.6, 0.6, (len(recs), 2))
    orc.set_interactions(recs)
    state = oracle_state(orc)
    eng = Engine(device=0)
    eng.load(spec)
    snapshot_into(eng, orc)
    eng.step(1)
    eng.sync()

    def direction(r):
        p = r[:, 5:7]
        return np.stack([np.cos(p[:, 0]) * np.cos(p[:, 1]), np.sin(p[:, 0]) * np.cos(p[:, 1]), np.sin(p[:, 1])], -1)

    def run():
        o = restore_oracle(spec, state, os.cpu_count())
        o.step(1)
        return direction(o.interactions()), o
    ref, o = run()
    steady = np.isfinite(ref).all(axis=1)
    inside = o.margins()[:, 6]
    steady &= ~(inside < 1e-6)
    try:
        for seed in range(1, 7):
            oracle.set_math_noise(seed, 0.0)
            steady &= np.linalg.norm(run()[0] - ref, axis=1) < 1e-6
    finally:
        oracle.set_math_noise(0)
    key = {(int(r[0]), int(r[1])): i for i, r in enumerate(recs)}
    got = eng.interactions(True)
    at = np.array([key[(int(r[0]), int(r[1]))] for r in got])
    off = np.linalg.norm(direction(got) - ref[at], axis=1)[steady[at]]
    print(f"eps ({eps1}, {eps2}): {len(off)} of {len(recs)} steady, {np.mean(inside[steady] < 1e300):.0%} of them "
          f"with an isInside test, furthest {off.max():.1e}")
    assert len(off) > 100
    assert np.all(off < 1e-5)
