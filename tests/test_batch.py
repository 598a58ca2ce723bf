"""Batches of specimens: one graph launch steps every scene; each scene's results are those of
its context stepped alone (bitwise), in both precision forms, with the CompressionEngine."""
import ctypes as C
import os

import numpy as np
import pytest

from sudodem_gb300 import Batch, Engine, SqdemError, assemblies
from sudodem_gb300.servo import servo_config

pytestmark = pytest.mark.gpu

SERVO = servo_config(z_servo=0, shearMode=1, goalx=1e5, goaly=1e5, goalz=0.05, max_vel=1.0,
                     ramp_interval=30, ramp_chunks=3, iterate_num_max=10)


def specs(k=4, seed=11):
    sizes = [60, 150, 90, 220, 40, 130][:k]
    return [assemblies.cubic_specimen(n, seed=seed + i, friction=0.2 + 0.1 * i) for i, n in enumerate(sizes)]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_batch_scenes_equal_independent_runs(gpu, precision):
    ss = specs()
    b = Batch(len(ss), precision=precision)
    b.load(ss, servo=SERVO)
    b.scenes[2].set_servo(servo_config(enabled=0))   # one scene without the engine
    b.step(25)
    b.sync()
    for i, spec in enumerate(ss):
        e = Engine(precision=precision)
        e.load(spec)
        if i != 2:
            e.set_servo(SERVO)
        e.step(25)
        e.sync()
        assert np.array_equal(b.scenes[i].body_state(), e.body_state()), i
        assert np.array_equal(b.scenes[i].interactions(True), e.interactions(True)), i
        assert np.array_equal(b.scenes[i].servo_state(), e.servo_state(), equal_nan=True), i
    b.close()


def test_batch_graph_rebuilt_after_a_scene_changes(gpu):
    ss = specs(3, seed=21)
    b = Batch(3)
    b.load(ss)
    b.step(10)
    b.scenes[1].set_servo(SERVO)   # the step's kernel sequence of scene 1 changes
    b.step(10)
    b.sync()
    e = Engine()
    e.load(ss[1])
    e.step(10)
    e.set_servo(SERVO)
    e.step(10)
    e.sync()
    assert np.array_equal(b.scenes[1].body_state(), e.body_state())
    assert b.launch_count() > 0
    b.close()


def test_batch_sync_reports_a_scene_overflow(gpu):
    ss = specs(2, seed=31)
    b = Batch(2, contacts_per_body=1)
    b.load(ss)
    b.step(3)
    with pytest.raises(SqdemError) as ei:
        b.sync()
    assert ei.value.status == 3
    b.close()


def test_batch_time_e2e_round_trips_kinematics(gpu):
    ss = specs(3, seed=41)
    b = Batch(3)
    b.load(ss, servo=SERVO)
    b.step(2)
    b.sync()
    kin = np.concatenate([e.kinematics() for e in b.scenes])
    a, c = kin.copy(), np.zeros_like(kin)
    ms = b.time_e2e(2, a.ctypes.data, c.ctypes.data)     # in -> out -> in
    assert ms > 0
    b.sync()
    now = np.concatenate([e.kinematics() for e in b.scenes])
    assert np.array_equal(a, now)
    # the same two steps from the same state on independent contexts
    ref = []
    for i, spec in enumerate(ss):
        e = Engine()
        e.load(spec)
        e.set_servo(SERVO)
        e.step(4)
        e.sync()
        ref.append(e.kinematics())
    assert np.array_equal(now, np.concatenate(ref))
    b.close()


@pytest.mark.parametrize("precision,sizes", [("fp64", (1, 17, 33, 250, 15800)), ("fp64", (2, 16400)),
                                             ("mixed", (1, 17, 33, 250, 7800)), ("mixed", (2, 8100))])
def test_searches_in_rounds_equal_searches_by_warps(gpu, precision, sizes):
    """Scenes of up to 16,000 particles (8,000 in the mixed form) are searched one contact per warp,
    larger ones, and the scenes of a larger batch, in rounds over compact lists: the same operations
    per contact, so the same bits, whatever share of the lists' last warps is filled."""
    ss = [assemblies.cubic_specimen(n, seed=31 + i, eps_range=(0.3, 1.7), spacing=2.1e-3, wall_gap=0.0)
          for i, n in enumerate(sizes)]
    b = Batch(len(ss), precision=precision)
    b.load(ss)
    b.step(6)
    b.sync()
    for i, spec in enumerate(ss):
        e = Engine(precision=precision)
        e.load(spec)
        e.step(6)
        e.sync()
        assert np.array_equal(b.scenes[i].interactions(True), e.interactions(True)), i
        assert np.array_equal(b.scenes[i].body_state(), e.body_state()), i
    b.close()


def test_more_long_searches_than_warps_take_at_once(gpu):
    """The second step of a freshly loaded dense cell has some 23,000 searches that ran 8 iterations or
    more: the FP64 form gives the longest and 6,000 others a warp, the rest goes to the rounds.  In a
    batch the line is 16 iterations (some 6,000 searches, all of which take a warp): the same bits."""
    tile = os.path.join(os.path.dirname(__file__), "golden", "config1_tile.npz")
    spec = assemblies.config1_dense(tile, tiles=3)
    e = Engine()
    e.load(spec)
    e.step(1)
    e.sync()
    e.step(1)
    assert e.sync()["long_queue"] > 6000
    e.step(1)
    b = Batch(1)
    b.load([spec])
    b.step(3)
    b.sync()
    assert np.array_equal(b.scenes[0].interactions(True), e.interactions(True))
    assert np.array_equal(b.scenes[0].body_state(), e.body_state())
    b.close()


@pytest.mark.parametrize("precision,small,large", [("fp64", 250, 15800), ("mixed", 250, 7800)])
def test_report_counts_the_rounds_of_every_search(gpu, precision, small, large):
    """The report's longest search counts what was run in rounds over lists as well as what a warp ran.
    Alone, both scenes give each search a warp, several evaluations a round; in the batch the first four (FP64)
    or three rounds, a trial and two probes each, run over lists, one evaluation a round, which takes a
    search no fewer rounds."""
    ss = [assemblies.cubic_specimen(n, seed=41 + i, eps_range=(0.3, 1.7), spacing=2.1e-3, wall_gap=0.0)
          for i, n in enumerate((small, large))]
    word = "lm_rounds_max" if precision == "fp64" else "lm_rounds_max_ff"
    alone = []
    for spec in ss:
        e = Engine(precision=precision)
        e.load(spec)
        e.step(1)
        alone.append(e.sync()[word])
    b = Batch(2, precision=precision)
    b.load(ss)
    b.step(1)
    rep = b.sync()
    b.close()
    # a search that goes on to the warps has been through all of the lists' rounds
    lists = 3 * (4 if precision == "fp64" else 3)
    assert max(alone) > lists
    assert rep[word] >= max(alone)


@pytest.mark.parametrize("precision,sizes", [("fp64", (700, 15400)), ("mixed", (700, 7400))])
def test_few_searches_take_warps_in_large_scenes(gpu, precision, sizes):
    """Loose scenes with a hundred touching pairs, in a batch above the particle line of the rounds: each search
    takes a warp as it does in the scenes alone, so the longest takes as many rounds, with the same bits.  A
    jammed scene beside them in the batch keeps its rounds, with the same bits too."""
    per = 30
    ss = [assemblies.walled_lattice(n, seed=51 + i, spacing=2.6e-3, r_range=(0.9e-3, 1.2e-3), per_side=per,
                                    box=(per + 0.7) * 2.6e-3) for i, n in enumerate(sizes)]
    word = "lm_rounds_max" if precision == "fp64" else "lm_rounds_max_ff"

    def alone(spec, steps):
        e = Engine(precision=precision)
        e.load(spec)
        e.step(steps)
        return e.sync(), e

    def together(specs, steps):
        b = Batch(len(specs), precision=precision)
        b.load(specs)
        b.step(steps)
        return b.sync(), b
    rep, b = together(ss, 1)
    b.close()
    longest = max(alone(s, 1)[0][word] for s in ss)
    assert longest > 0 and rep[word] == longest
    ss.append(assemblies.cubic_specimen(900, seed=53, eps_range=(0.3, 1.7), spacing=2.1e-3, wall_gap=0.0))
    _, b = together(ss, 6)
    for i, spec in enumerate(ss):
        _, e = alone(spec, 6)
        assert np.array_equal(b.scenes[i].interactions(True), e.interactions(True)), i
        assert np.array_equal(b.scenes[i].body_state(), e.body_state()), i
    b.close()
