"""GPU engine (libsqdem_gpu.so, through the C ABI) against the CPU oracle.

Bit-exact: bounds (BoundDispatcher + Bo1_*), the potential-pair set with its (id1, id2)
orientation after every collider pass, and the real/potential state of each pair.

Floating point (narrowphase, forces, integration): the reference's Levenberg-Marquardt
search is ill-conditioned (its own result moves by up to ~1e-7 relative when an input is
perturbed by one ulp), and CUDA's pow/atan2/sin/cos differ from glibc's in the last ulp.
The tolerance is therefore stated against the oracle's own one-ulp sensitivity measured in
the same test: the GPU-vs-oracle error quantiles must stay within a factor of the
oracle-vs-perturbed-oracle quantiles, and the median error must be at the 1e-10 level.
"""
import numpy as np
import pytest

from oracle import OracleScene
from sudodem_gb300 import Engine, SqdemError, assemblies

pytestmark = pytest.mark.gpu


def canon_pairs(recs, kind):
    out = set()
    for r in recs:
        a, b = int(r[0]), int(r[1])
        if kind[a] == 1 and kind[b] == 1:
            a, b = min(a, b), max(a, b)
        out.add((a, b))
    return out


def by_pair(recs):
    return {(int(r[0]), int(r[1])): r for r in recs}


def engine_for(spec, **kw):
    e = Engine(device=0, **kw)
    e.load(spec)
    return e


def snapshot_into(eng, orc, force_collider=False):
    eng.put_body_state(orc.bodies())
    eng.put_interactions(orc.interactions())
    s = orc.scalars()
    if force_collider:
        s = s.copy()
        s[1] = 2.0
        orc.set_scalars(s)
    eng.put_scalars(s)


def dense_spec(seed=5, n=400):
    return assemblies.walled_lattice(n, seed=seed, box=14e-3, per_side=5, spacing=2.1e-3)


def rel_force_errors(G, R):
    fg = G[:, 26:29] + G[:, 29:32]
    fr = R[:, 26:29] + R[:, 29:32]
    den = np.linalg.norm(fr, axis=1)
    return np.linalg.norm(fg - fr, axis=1) / np.where(den > 0, den, 1)


def touching_common(gi, ri):
    G, R = by_pair(gi), by_pair(ri)
    keys = [k for k, r in R.items() if k in G and r[4] > 0 and r[2] == 1]
    return np.array([G[k] for k in keys]), np.array([R[k] for k in keys])


def test_first_step_bounds_and_pair_set_bitexact(gpu):
    spec = assemblies.config0(seed=11)
    eng = engine_for(spec)
    orc = OracleScene.from_spec(spec)
    for _ in range(3):
        eng.step(1); eng.sync(); orc.step(1)
        g, r = eng.body_state(), orc.bodies()
        assert np.array_equal(g[:, 22:33], r[:, 22:33])  # bmin bmax refPos sweepLength lastUpdateIter
        gi, ri = eng.interactions(True), orc.interactions()
        assert canon_pairs(gi, spec.kind) == canon_pairs(ri, spec.kind)
        G, R = by_pair(gi), by_pair(ri)
        assert all(G[k][2] == R[k][2] for k in R if k in G)


@pytest.mark.parametrize("steps_before", [150, 400])
def test_incremental_collider_pair_set_bitexact(gpu, steps_before):
    spec = dense_spec(seed=6)
    orc = OracleScene.from_spec(spec, threads=4)
    orc.step(steps_before)
    eng = engine_for(spec)
    snapshot_into(eng, orc, force_collider=True)
    eng.step(1); eng.sync(); orc.step(1)
    assert orc.last_step_collided()
    g, r = eng.body_state(), orc.bodies()
    assert np.array_equal(g[:, 22:33], r[:, 22:33])
    gi, ri = eng.interactions(True), orc.interactions()
    assert canon_pairs(gi, spec.kind) == canon_pairs(ri, spec.kind)
    G, R = by_pair(gi), by_pair(ri)
    assert all(G[k][2] == R[k][2] for k in R if k in G)


def oracle_self_sensitivity(spec, orc_state):
    """Force errors of the oracle against itself with positions perturbed by one ulp."""
    a = OracleScene.from_spec(spec)
    b = OracleScene.from_spec(spec)
    bodies, intr, sc = orc_state
    rng = np.random.default_rng(0)
    pert = bodies.copy()
    sgn = rng.choice([-1.0, 1.0], size=pert[:, 0:3].shape)
    pert[:, 0:3] = np.nextafter(pert[:, 0:3], pert[:, 0:3] + sgn * np.inf)
    for o, bb in ((a, bodies), (b, pert)):
        o.set_bodies(bb); o.set_interactions(intr); o.set_scalars(sc); o.rebuild_sorted_bounds()
        o.step(1)
    G, R = touching_common(b.interactions(), a.interactions())
    return rel_force_errors(G, R)


def test_single_step_contacts_within_oracle_conditioning(gpu):
    spec = dense_spec(seed=5)
    orc = OracleScene.from_spec(spec, threads=4)
    orc.step(3)
    state = (orc.bodies(), orc.interactions(), orc.scalars())
    eng = engine_for(spec)
    eng.set_record_full(True)
    snapshot_into(eng, orc)
    eng.step(1); eng.sync(); orc.step(1)
    G, R = touching_common(eng.interactions(True), orc.interactions())
    assert len(G) > 50
    e = rel_force_errors(G, R)
    depth = np.abs(G[:, 4] - R[:, 4]) / R[:, 4]
    selfe = oracle_self_sensitivity(spec, state)
    q = lambda x, p: float(np.quantile(x, p))
    print(f"touching={len(e)} gpu-vs-oracle force err: median {q(e, .5):.2e} p90 {q(e, .9):.2e} max {e.max():.2e}; "
          f"oracle 1-ulp self: median {q(selfe, .5):.2e} p90 {q(selfe, .9):.2e} max {selfe.max():.2e}; "
          f"depth median {q(depth, .5):.2e}")
    assert q(e, 0.5) < 1e-9
    assert q(e, 0.9) < max(100 * q(selfe, 0.9), 1e-8)
    assert np.mean(e < 1e-6) > 0.97


def test_wall_contacts_tight(gpu):
    spec = dense_spec(seed=8)
    orc = OracleScene.from_spec(spec, threads=4)
    orc.step(60)   # the lattice's initial overlaps throw particles against the walls
    eng = engine_for(spec)
    snapshot_into(eng, orc)
    eng.step(1); eng.sync(); orc.step(1)
    G, R = touching_common(eng.interactions(True), orc.interactions())
    wall = (G[:, 0] < 6)
    assert wall.sum() > 5
    e = rel_force_errors(G[wall], R[wall])
    assert e.max() < 1e-11


def test_body_update_parity(gpu):
    spec = dense_spec(seed=12)
    orc = OracleScene.from_spec(spec, threads=4)
    orc.step(25)
    eng = engine_for(spec)
    snapshot_into(eng, orc)
    x0 = orc.bodies()
    eng.step(1); eng.sync(); orc.step(1)
    g, r = eng.body_state(), orc.bodies()
    p = 6
    fr = np.linalg.norm(r[p:, 16:19], axis=1)
    ef = np.linalg.norm(g[p:, 16:19] - r[p:, 16:19], axis=1) / np.where(fr > 0, fr, 1)
    assert np.median(ef) < 1e-9 and np.mean(ef < 1e-6) > 0.97
    dv = np.linalg.norm(r[p:, 7:10] - x0[p:, 7:10], axis=1)
    ev = np.linalg.norm(g[p:, 7:10] - r[p:, 7:10], axis=1) / np.where(dv > 0, dv, 1)
    assert np.median(ev) < 1e-9
    assert np.max(np.abs(g[:, 0:3] - r[:, 0:3])) < 1e-13
    qn = np.linalg.norm(g[:, 3:7], axis=1)
    assert np.allclose(qn, 1.0, atol=1e-14)


def test_graph_replay_equals_eager_launches(gpu):
    spec = dense_spec(seed=3, n=200)
    a = engine_for(spec, use_graph=True)
    b = engine_for(spec, use_graph=False)
    a.step(30); b.step(30)
    a.sync(); b.sync()
    assert np.array_equal(a.body_state(), b.body_state())


def test_deterministic(gpu):
    spec = dense_spec(seed=4, n=200)
    a, b = engine_for(spec), engine_for(spec)
    a.step(60); b.step(60)
    a.sync(); b.sync()
    assert np.array_equal(a.body_state(), b.body_state())
    assert np.array_equal(a.interactions(True), b.interactions(True))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("kind", ["walled", "periodic"])
def test_lm_spread_rounds_equal_one_point_rounds(gpu, kind, precision):
    """Spare lanes evaluating the points running searches ask for next changes nothing."""
    spec = dense_spec(seed=7, n=400) if kind == "walled" else periodic_spec(seed=4, n=400)
    a, b = engine_for(spec, precision=precision), engine_for(spec, precision=precision)
    b.set_lm_spread(False)
    a.step(40); b.step(40)
    ra, rb = a.sync(), b.sync()
    assert np.array_equal(a.body_state(), b.body_state())
    assert np.array_equal(a.interactions(True), b.interactions(True))
    for k in ("lm_calls", "lm_iterations", "lm_maxiter", "nan_normals", "nan_forces", "fallback_fp64"):
        assert ra[k] == rb[k], k
    # the spare lanes' evaluations are counted with the searches' own
    key = "evals_fp32" if precision == "mixed" else "evals_fp64"
    assert ra[key] >= rb[key] > 0


def test_capacity_overflow_is_reported_not_faulted(gpu):
    spec = dense_spec(seed=2, n=200)
    eng = engine_for(spec, contacts_per_body=1)
    eng.step(2)
    with pytest.raises(SqdemError) as ei:
        eng.sync()
    assert ei.value.status == 3
    g = eng.body_state()
    assert np.all(np.isfinite(g[:, :16]))


def test_nonfinite_input_rejected_on_host(gpu):
    spec = dense_spec(seed=2, n=50)
    eng = engine_for(spec)
    st = eng.body_state()
    st[10, 0] = np.nan
    with pytest.raises(SqdemError) as ei:
        eng.put_body_state(st)
    assert ei.value.status == 1


def test_deposition_statistics_match_oracle(gpu):
    spec = assemblies.config0(seed=21)
    eng = engine_for(spec)
    orc = OracleScene.from_spec(spec, threads=8)
    eng.step(2000); eng.sync(); orc.step(2000)
    g, r = eng.body_state(), orc.bodies()
    p = 6
    assert abs(g[p:, 2].mean() - r[p:, 2].mean()) < 1e-3 * abs(r[p:, 2].mean())
    ke = lambda b: 0.5 * np.sum(b[p:, 33] * np.sum(b[p:, 7:10] ** 2, axis=1))
    assert abs(ke(g) - ke(r)) <= 0.05 * ke(r)
    ng = np.sum(eng.interactions(False)[:, 4] > 0)
    nr = np.sum(orc.interactions()[:, 4] > 0)
    assert abs(int(ng) - int(nr)) <= max(3, 0.05 * nr)


def brute_periodic(b, L):
    from test_oracle import _brute_pairs_periodic
    return _brute_pairs_periodic(b, L)


def test_periodic_pair_set_equals_image_overlaps(gpu):
    """GPU periodic collider: after each pass the table holds exactly the pairs whose bounds
    overlap under a periodic image, plus real pairs the law has not yet erased."""
    spec = assemblies.periodic_cell(300, seed=9, solid_fraction=0.38, strain_rate=3.0)
    eng = engine_for(spec)
    checked = 0
    for _ in range(80):
        before = eng.scalars()[7]
        eng.step(1); eng.sync()
        if eng.scalars()[7] == before:   # bounds and cell size must be those of this pass
            continue
        b = eng.body_state()
        L = eng.cell()[27:30]
        I = eng.interactions(True)
        have = {tuple(sorted(map(int, r[:2]))) for r in I}
        nonreal = {tuple(sorted(map(int, r[:2]))) for r in I if r[2] == 0}
        brute = brute_periodic(b, L)
        assert brute <= have
        assert have - brute <= nonreal
        checked += 1
    assert checked >= 2


def periodic_spec(seed=3, n=400):
    return assemblies.periodic_cell(n, seed=seed, solid_fraction=0.42, strain_rate=3.0)


def test_periodic_first_steps_pair_set_celldist_bitexact(gpu):
    """From identical states: full-sort pass (step 0) and incremental passes (snapshots of the
    oracle with the collider forced) give bit-identical bounds, cell, pair set, orientation
    and cellDist."""
    spec = periodic_spec()
    eng = engine_for(spec)
    orc = OracleScene.from_spec(spec, threads=1)   # one thread: the same force sums every run
    eng.step(1); eng.sync(); orc.step(1)
    assert np.array_equal(eng.cell(), orc.cell())
    assert np.array_equal(eng.body_state()[:, 22:33], orc.bodies()[:, 22:33])
    gi, ri = eng.interactions(True), orc.interactions()
    G, R = by_pair(gi), by_pair(ri)
    assert set(G) == set(R)
    assert all(np.array_equal(G[k][44:47], R[k][44:47]) for k in R)
    for nsteps in (20, 60):
        orc.step(nsteps)
        e2 = engine_for(spec)
        snapshot_into(e2, orc, force_collider=True)
        e2.put_cell(orc.cell())
        e2.step(1); e2.sync(); orc.step(1)
        assert orc.last_step_collided()
        assert np.array_equal(e2.cell(), orc.cell())
        assert np.array_equal(e2.body_state()[:, 22:33], orc.bodies()[:, 22:33])
        G, R = by_pair(e2.interactions(True)), by_pair(orc.interactions())
        # the GPU holds every image-overlapping pair; the oracle's circular insertion sort may
        # transiently miss one (a bound that wrapped down and moved back below the cell size is
        # not compared with the other body's wrapped bound), so compare on the oracle's pairs
        missing = set(R) - set(G)
        assert not missing, [(k, R[k][2], R[k][4], R[k][44:47]) for k in missing]
        assert all(np.array_equal(G[k][44:47], R[k][44:47]) for k in R)
        assert all(G[k][2] == R[k][2] for k in R)


def test_periodic_single_step_within_oracle_conditioning(gpu):
    spec = periodic_spec(seed=4)
    orc = OracleScene.from_spec(spec, threads=4)
    orc.step(40)
    eng = engine_for(spec)
    snapshot_into(eng, orc)
    eng.put_cell(orc.cell())
    x0 = orc.bodies()
    eng.step(1); eng.sync(); orc.step(1)
    assert np.array_equal(eng.cell(), orc.cell())
    G, R = touching_common(eng.interactions(True), orc.interactions())
    assert len(G) > 30
    e = rel_force_errors(G, R)
    assert np.median(e) < 1e-9 and np.mean(e < 1e-6) > 0.97
    g, r = eng.body_state(), orc.bodies()
    fr = np.linalg.norm(r[:, 16:19], axis=1)
    ef = np.linalg.norm(g[:, 16:19] - r[:, 16:19], axis=1) / np.where(fr > 0, fr, 1)
    assert np.median(ef) < 1e-9 and np.mean(ef < 1e-6) > 0.97
    dv = np.linalg.norm(r[:, 7:10] - x0[:, 7:10], axis=1)
    ev = np.linalg.norm(g[:, 7:10] - r[:, 7:10], axis=1) / np.where(dv > 0, dv, 1)
    assert np.median(ev) < 1e-9 and np.mean(ev < 1e-6) > 0.97


@pytest.mark.gpu
def test_autotuned_launch_shapes_change_nothing(gpu):
    """The autotuner's steps are ordinary timesteps and the shape it picks changes no result."""
    spec = dense_spec(seed=10, n=300)
    a, b = engine_for(spec), engine_for(spec)
    t = a.autotune(steps=2)
    assert 1 <= t["search_blocks_per_sm"] and t["pass1_blocks_per_sm"] in (4, 8, 16, 32)
    n_tuned = int(a.scalars()[0])
    assert n_tuned == t["candidates"] * (2 * 2 + 1)
    b.step(n_tuned)
    a.step(20); b.step(20)
    a.sync(); b.sync()
    assert np.array_equal(a.body_state(), b.body_state())
    assert np.array_equal(a.interactions(True), b.interactions(True))
    for sb, p1 in ((1, 4), (2, 32)):
        c = engine_for(spec)
        c.set_launch_shape(sb, p1)
        c.step(n_tuned + 20); c.sync()
        assert np.array_equal(c.body_state(), b.body_state())


@pytest.mark.gpu
@pytest.mark.parametrize("precision,model,swept", [("fp64", "linear", False), ("fp64", "hertz_mindlin", False),
                                                   ("mixed", "linear", True)])
def test_autotuner_times_only_shapes_that_are_read(gpu, precision, model, swept):
    """A scene whose searches all have a warp reads no search blocks: four shapes of pass 1 are timed, and the
    search blocks the caller set stay set.  The mixed form's search kernels read them."""
    spec = assemblies.walled_lattice(64, seed=3, box=12e-3, per_side=4, spacing=2.2e-3)
    e = Engine(device=0, precision=precision)
    e.load(spec)
    if model == "hertz_mindlin":
        e.set_material_moduli([1e6] * len(spec.materials["Kn"]), [0.3] * len(spec.materials["Kn"]))
        e.set_contact_model(model)
    e.set_launch_shape(1, 0)
    t = e.autotune(steps=1)
    assert t["candidates"] > 4 if swept else (t["candidates"], t["search_blocks_per_sm"]) == (4, 1)
    assert t["candidates"] % 4 == 0 and int(e.scalars()[0]) == 3 * t["candidates"]


def _bed_statistics(spec, bodies, recs, slab=10e-3):
    """Packing fraction of the bottom slab (Superquadrics::Initial volumes of the particles
    whose centres lie in it, over the slab volume), coordination number (touching
    particle-particle contacts per particle) and floor stress (normal force on the floor wall
    over the box area)."""
    from sudodem_gb300 import shape_props
    p = spec.kind == 0
    vol = np.array([shape_props(*s)[0] for s in spec.shape5[p]])
    z = bodies[p, 2]
    box = spec.info["box"]
    phi = float(np.sum(vol[z < slab]) / (box * box * slab))
    touch = recs[(recs[:, 4] > 0) & (recs[:, 0] > 5) & (recs[:, 2] == 1)]
    coord = 2.0 * len(touch) / int(np.sum(p))
    floor = abs(bodies[4, 18]) / (box * box)   # force z of the floor wall (body 4)
    return np.array([phi, coord, floor])


def test_long_run_statistics_over_five_seeds(gpu):
    """Granular dynamics are chaotic, so long runs are compared statistically: the config-0
    deposition (1,000 superellipsoids, 30,000 steps: the lower layers have landed and
    packed) on the GPU and on the oracle for five
    seeds; the mean over seeds of packing fraction, coordination number and floor stress
    must agree within three standard errors of the per-seed differences plus 2%."""
    import os
    thr = max(1, min(16, os.cpu_count() or 1))
    G, R = [], []
    for seed in (31, 32, 33, 34, 35):
        spec = assemblies.config0(seed=seed)
        eng = engine_for(spec)
        orc = OracleScene.from_spec(spec, threads=thr)
        eng.step(30000); eng.sync(); orc.step(30000)
        G.append(_bed_statistics(spec, eng.body_state(), eng.interactions(False)))
        R.append(_bed_statistics(spec, orc.bodies(), orc.interactions()))
    G, R = np.array(G), np.array(R)
    d = G - R
    se = d.std(axis=0, ddof=1) / np.sqrt(len(d))
    print("gpu mean", G.mean(axis=0), "oracle mean", R.mean(axis=0), "diff", d.mean(axis=0), "se", se)
    assert np.all(R.mean(axis=0) > 0)
    assert np.all(np.abs(d.mean(axis=0)) <= 3 * se + 0.02 * np.abs(R.mean(axis=0)))
