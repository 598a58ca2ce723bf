"""Edge cases of the superellipsoid timestep on the GPU, through the C ABI, against the oracle:
a scene without particles, one particle on the floor (wall contact only), two particles with
coincident centres (the narrowphase meets NaN angles), and the host-side limits."""
import numpy as np
import pytest

from oracle import OracleScene
from sudodem_gb300 import Engine, SqdemError, assemblies
from sudodem_gb300._native import shape_props
from test_gpu_parity import canon_pairs

pytestmark = pytest.mark.gpu


def _params(dt=2e-6):
    return {"dt": dt, "gravity": (0.0, 0.0, -9.81), "damping": 0.3, "verletDist": 2e-4, "targetInterv": 50,
            "minSweepDistFactor": 0.1, "sortAxis": 0, "isSuperquadrics": 1, "exactAsphericalRot": 1}


def _box(b, side=10e-3, lid=0.2):
    assemblies._add_wall(b, [0, 0, 0], 0, +1)
    assemblies._add_wall(b, [side, 0, 0], 0, -1)
    assemblies._add_wall(b, [0, 0, 0], 1, +1)
    assemblies._add_wall(b, [0, side, 0], 1, -1)
    assemblies._add_wall(b, [0, 0, 0], 2, +1)
    assemblies._add_wall(b, [0, 0, lid], 2, -1)


def _engine(spec):
    e = Engine(device=0)
    e.load(spec)
    return e


def test_scene_without_particles_steps(gpu):
    b = assemblies._builder()
    _box(b)
    spec = assemblies._finish(b, assemblies.default_material(), _params(), {"box": 10e-3})
    spec.state[5, 7:10] = (0.0, 0.0, -0.5)   # the lid moves down at its prescribed velocity
    eng, orc = _engine(spec), OracleScene.from_spec(spec)
    eng.step(10); rep = eng.sync(); orc.step(10)
    assert int(eng.scalars()[0]) == 10
    assert rep["lm_calls"] == 0 and rep["nan_forces"] == 0
    assert len(eng.interactions(False)) == 0
    g, r = eng.body_state(), orc.bodies()
    assert np.array_equal(g[:, 0:3], r[:, 0:3])
    assert g[5, 2] < 0.2


def test_one_particle_resting_on_the_floor(gpu):
    b = assemblies._builder()
    _box(b)
    assemblies._add_sq(b, [1e-3, 0.8e-3, 0.7e-3], [0.8, 1.2], assemblies._quat_normalize([1, 0.2, 0.1, 0]),
                       [5e-3, 5e-3, 0.9e-3], 2650.0)
    spec = assemblies._finish(b, assemblies.default_material(), _params(), {"box": 10e-3})
    eng, orc = _engine(spec), OracleScene.from_spec(spec)
    for _ in range(4):
        eng.step(500); eng.sync(); orc.step(500)
        g, r = eng.body_state(), orc.bodies()
        assert np.allclose(g[6, 0:16], r[6, 0:16], rtol=1e-9, atol=1e-15)
    assert 0 < g[6, 2] < 1e-3
    recs = eng.interactions(False)
    assert len(recs) >= 1 and np.all(recs[:, 0] == 4)   # the floor, as id1 (wall first)


def test_coincident_centres_do_not_break_the_step(gpu):
    spec = assemblies.pair_scene([1e-3, 0.9e-3, 0.8e-3, 0.7, 1.3], [0.9e-3, 0.9e-3, 0.9e-3, 1.1, 0.9],
                                 [0, 0, 0], [0, 0, 0], [1, 0, 0, 0], [0.9, 0.1, 0.3, 0.2])
    eng, orc = _engine(spec), OracleScene.from_spec(spec)
    eng.step(3); rep = eng.sync(); orc.step(3)
    g, r = eng.body_state(), orc.bodies()
    assert np.array_equal(np.isfinite(g[:, 0:16]), np.isfinite(r[:, 0:16]))
    assert np.all(np.isfinite(g[:, 0:3]))
    st = orc.stats()
    assert rep["nan_normals"] == st["nan_normals"]


def test_host_limits(gpu):
    b = assemblies._builder()
    for k in range(65):
        assemblies._add_wall(b, [0, 0, -1.0 - k], 2, +1)
    assemblies._add_sq(b, [1e-3, 1e-3, 1e-3], [1.0, 1.0], [1, 0, 0, 0], [0, 0, 0], 2650.0)
    spec = assemblies._finish(b, assemblies.default_material(), _params(), {})
    e = Engine(device=0)
    with pytest.raises(SqdemError) as ei:
        e.load(spec)
    assert ei.value.status == 3   # SQDEM_ERR_CAPACITY: at most 64 walls
    e2 = Engine(device=0)
    with pytest.raises(SqdemError):
        e2.step(1)                # bodies and materials first


@pytest.mark.parametrize("size", [1e-3, 1.0, 1e-17])
@pytest.mark.parametrize("off", [-2e-5, -3e-6, -1e-15, 0.0, 1e-15, 3e-6, 2e-5])
def test_bounding_sphere_rejection_near_its_threshold(gpu, size, off):
    """Pairs whose centres are at the summed bounding radii times (1 + off).  A pair beyond them is
    rejected without a start point (contactAngle (0, 0)), any other gets the centre line's.  The FP32
    test decides outside a band around the threshold only, so the answer is FP64's at every size."""
    s1, s2 = [size, 0.9 * size, 0.8 * size, 0.7, 1.3], [0.9 * size, 0.8 * size, size, 1.1, 0.9]
    rsum = shape_props(*s1)[4] + shape_props(*s2)[4]
    gap = rsum * (1 + off)
    spec = assemblies.pair_scene(s1, s2, [0, 0, 0], [gap, 0, 0], [1, 0, 0, 0], [1, 0, 0, 0], walls=False)
    spec.params["verletDist"] = size
    eng = _engine(spec)
    eng.step(1); eng.sync()
    recs = eng.interactions(True)
    assert len(recs) == 1
    assert np.all(recs[0, 5:7] == 0) == (gap > rsum)


@pytest.mark.parametrize("n,periodic", [(1, False), (1594, False), (1595, False), (1600, True), (1601, True)])
def test_collider_pass_in_one_launch_and_in_kernels(gpu, n, periodic):
    """Scenes of up to 1,600 bodies run the collider pass as one thread-block cluster, larger ones as
    one kernel per pass: either way the pairs and their orientation are the oracle's."""
    if periodic:
        spec = assemblies.periodic_cell(n, seed=3, solid_fraction=0.5)
    else:
        spec = assemblies.cubic_specimen(n, seed=3, eps_range=(0.6, 1.4), spacing=2.1e-3, wall_gap=0.0)
    eng, orc = _engine(spec), OracleScene.from_spec(spec)
    for steps in (1,) if periodic else (1, 4):   # the first pass sorts all bounds, later ones insert
        eng.step(steps); eng.sync(); orc.step(steps)
        G, R = eng.interactions(True), orc.interactions()
        assert canon_pairs(G, spec.kind) == canon_pairs(R, spec.kind)
        assert canon_pairs(G[G[:, 2] == 1], spec.kind) == canon_pairs(R[R[:, 2] == 1], spec.kind)
        if steps == 1:   # bounds, reference positions, sweep lengths: bit for bit
            assert np.array_equal(eng.body_state()[:, 22:33], orc.bodies()[:, 22:33])
