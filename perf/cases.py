"""Performance cases: the calls a user of this framework makes, over the range of its scenes.

Every case is one pass of a running simulation through the public entry points: a scene that has
been loaded and has run its first steps advances by ``steps`` timesteps, and its bodies' kinematic
state and mean stress are read back (``adjoint`` cases: one loss and its gradients).  A pass
continues where the last one ended, as a simulation does.
"""
import math
import os

import numpy as np
import torch

from sudodem_gb300 import Batch, Engine, assemblies
from sudodem_gb300.adjoint import AdjointWindow, wall_force_weights, window_loss
from sudodem_gb300.servo import servo_config

TILE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tests", "golden", "config1_tile.npz")
TILE_PARTICLES = 1600

#: table entries and touching contacts per particle of each kind of scene (for work()): counted on
#: settled or compressed states of these scenes, neither depends on the code
ENTRIES = {"walled": 5.0, "specimen": 10.0, "cell": 14.3, "polydisperse": 14.9, "hertz": 12.0}
TOUCHING = {"walled": 0.2, "specimen": 1.5, "cell": 2.1, "polydisperse": 1.5, "hertz": 1.5}
EVAL_FLOPS = 2735       # one evaluation of a pair's two support points in FP64
BODY_BYTES, ENTRY_BYTES = 216, 256


def listed():
    return [
        # the smallest simulation anyone steps: a few particles in a box, read after every step
        # (a script with a per-step callback); launches and latency are all there is
        {"name": "walled_27_fp64", "kind": "walled", "n": 27, "precision": "fp64", "steps": 1, "warm": 20},
        # gravity deposition of 1,000 particles, the small standard scene (loose, few contacts)
        {"name": "deposition_1000_fp64", "kind": "walled", "n": 1000, "precision": "fp64", "steps": 20, "warm": 40},
        # one servo-controlled cubic specimen between six walls, read every few steps
        {"name": "specimen_2197_mixed", "kind": "specimen", "n": 2197, "precision": "mixed", "steps": 10, "warm": 20},
        # a representative periodic cell, jammed at 120 kPa, an odd number of particles, read after
        # every step
        {"name": "cell_1583_fp64", "kind": "cell", "n": 1583, "precision": "fp64", "steps": 1, "warm": 20},
        # periodic cells of the sizes that element tests are usually run with
        {"name": "cell_12800_mixed", "kind": "cell", "n": 12800, "precision": "mixed", "steps": 5, "warm": 10},
        {"name": "cell_43011_fp64", "kind": "cell", "n": 43011, "precision": "fp64", "steps": 3, "warm": 10},
        # the dense 200,000-particle cell that the benchmark reports, in both precision forms
        {"name": "cell_200000_fp64", "kind": "cell", "n": 200000, "precision": "fp64", "steps": 2, "warm": 6},
        {"name": "cell_200000_mixed", "kind": "cell", "n": 200000, "precision": "mixed", "steps": 3, "warm": 6},
        # near-cubic particles with a 4x size ratio under gravity: ill-conditioned searches
        {"name": "polydisperse_20000_mixed", "kind": "polydisperse", "n": 20000, "precision": "mixed", "steps": 3,
         "warm": 10},
        # the Hertz-Mindlin contact model (Nelder-Mead searches) on a compressed lattice
        {"name": "hertz_20000", "kind": "hertz", "n": 20000, "precision": "fp64", "steps": 5, "warm": 10},
        # a batch of uneven servo-controlled specimens stepped together (parameter studies)
        {"name": "batch_32_fp64", "kind": "batch", "scenes": 32, "lo": 300, "hi": 4000, "precision": "fp64", "steps": 2,
         "warm": 6},
        # gradients of a wall force over a short window: forward and backward through autograd
        {"name": "adjoint_1500", "kind": "adjoint", "n": 1500, "steps": 20, "every": 10, "warm": 50},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["walled", "specimen", "cell", "cell", "polydisperse", "hertz", "batch", "adjoint"])
    precision = rng.choice(["fp64", "mixed"])
    if kind == "batch":
        return {"kind": kind, "scenes": rng.randint(3, 32), "lo": rng.randint(40, 300), "hi": rng.randint(600, 4000),
                "precision": precision, "steps": rng.randint(1, 3), "warm": 6}
    if kind == "adjoint":
        return {"kind": kind, "n": _log(rng, 27, 1500), "steps": rng.randint(5, 20), "every": rng.randint(3, 20),
                "warm": rng.randint(30, 60)}
    hi = {"walled": 20000, "specimen": 12000, "cell": 150000, "polydisperse": 20000, "hertz": 20000}[kind]
    n = _log(rng, 30 if kind != "cell" else 800, hi)
    return {"kind": kind, "n": n, "precision": "fp64" if kind == "hertz" else precision,
            "steps": rng.choice([1, 1, 2, 3, 5, 10]) if n < 20000 else rng.randint(1, 2), "warm": rng.randint(8, 20)}


# ---------------------------------------------------------------------------------------------
# scenes


def _walled(n, seed):
    """Jittered lattice above the floor of a walled box under gravity.  Larger scenes are
    depositions (2.6 mm lattice, 7 x 7 per layer or more); a few particles sit in contact (2.1 mm)."""
    per = 3 if n <= 64 else max(7, int(round(n ** (1.0 / 3.0) * 0.7)))
    spacing = 2.1e-3 if n <= 64 else 2.6e-3
    return assemblies.walled_lattice(n, seed=seed, spacing=spacing, per_side=per, box=(per + 0.7) * spacing)


def _specimen(n, seed, friction=0.5):
    return assemblies.cubic_specimen(n, seed=seed, friction=friction, eps_range=(0.4, 1.6), spacing=2.1e-3,
                                     wall_gap=0.0)


def _servo():
    """100 kPa on the lateral walls, axial strain at the top and bottom ones."""
    return servo_config(z_servo=0, shearMode=1, goalx=1e5, goaly=1e5, goalz=0.05, max_vel=1.0, gain_alpha=0.5,
                        ramp_interval=200, ramp_chunks=20, echo_interval=1000, savedata_interval=1000,
                        target_strain=10.0)


def _cell(n, seed):
    """A jammed periodic cell of n particles: copies of the 1,600-particle tile in a box of whole
    tiles, shifted as a whole by a seeded offset, with seeded velocity fluctuations, and thinned to
    n particles (at most a few per cent are left out)."""
    rng = np.random.default_rng(seed)
    need = max(1, math.ceil(n / TILE_PARTICLES))
    m = max(1, int(round(need ** (1.0 / 3.0))))
    dims = min(((a, b, c) for a in range(1, m + 3) for b in range(a, m + 3) for c in range(b, m + 6)
                if a * b * c >= need), key=lambda d: (d[0] * d[1] * d[2], d[2] - d[0]))
    one = assemblies.config1_dense(TILE, tiles=1, strain_rate=0.1)
    side = one.info["cell_side"]
    vg = np.asarray(one.info["velGrad"]).reshape(3, 3)
    base = rng.uniform(0, side, 3)
    grid = np.stack(np.meshgrid(*[np.arange(d) for d in dims], indexing="ij"), -1).reshape(-1, 3) * side + base
    state = np.tile(one.state, (len(grid), 1))
    shift = np.repeat(grid, TILE_PARTICLES, axis=0)
    state[:, 0:3] += shift
    state[:, 7:10] += shift @ vg.T + rng.normal(0, 1e-3, (len(state), 3))
    keep = np.sort(rng.permutation(len(state))[:n])
    state = state[keep]
    shape5 = np.tile(one.shape5, (len(grid), 1))[keep]
    z = np.zeros(n, np.int32)
    return assemblies.SceneSpec(kind=z, shape5=shape5, wall_axis_sense=np.zeros((n, 2), np.int32), mat=z.copy(),
                                isSphere=z.copy(), state=state, materials=one.materials, params=dict(one.params),
                                info={"periodic": True, "hSize": np.diag(np.array(dims) * side).reshape(9),
                                      "velGrad": vg.reshape(9)})


def _hertz(n, seed):
    per = max(3, int(round(n ** (1.0 / 3.0) * 1.62)))
    lattice = assemblies.walled_lattice(n, seed=seed, box=(per + 1.24) * 2.1e-3, per_side=per, spacing=2.1e-3,
                                        eps_range=(0.5, 1.5))
    return assemblies.hertz_mindlin(lattice, G=1e6, nu=0.3)


def _polydisperse(n, seed):
    return assemblies.config4(seed=seed, n=n, box=0.2 if n > 5000 else 0.05)


SCENES = {"walled": _walled, "specimen": _specimen, "cell": _cell, "polydisperse": _polydisperse, "hertz": _hertz}


def _engine(case, seed, spec):
    eng = Engine(precision=case["precision"])
    eng.load(spec)
    if case["kind"] == "specimen":
        eng.set_servo(_servo())
    if case["kind"] == "cell":
        # the boundary terms that keep a compressed periodic cell's rotations bounded
        eng.set_periodic_fix(True)
    eng.step(case["warm"])
    eng.sync()
    return eng


def _adjoint(case, seed):
    n = case["n"]
    per = max(3, int(round(n ** (1.0 / 3.0))))
    spec = assemblies.walled_lattice(n, seed=seed, spacing=2.1e-3, per_side=per, box=(per + 0.8) * 2.1e-3,
                                     lid_height=(math.ceil(n / per ** 2) + 0.6) * 2.1e-3)
    rng = np.random.default_rng(seed + 100)
    assemblies.per_body_materials(spec, friction=rng.uniform(0.3, 0.7, spec.n_bodies))
    eng = Engine()
    eng.load(spec)
    eng.step(case["warm"])
    window = AdjointWindow.from_engine(eng, spec)
    eng.close()
    m = spec.materials
    leaves = [torch.tensor(np.asarray(v), dtype=torch.float64, requires_grad=True)
              for v in (spec.shape5[:, 3:5], np.tan(m["frictionAngle"]), m["Kn"], m["Ks"])]
    return {"case": case, "window": window, "leaves": leaves, "wF": wall_force_weights(spec.n_bodies, 4, 2)}


def prepare(case, seed):
    if case["kind"] == "adjoint":
        return _adjoint(case, seed)
    if case["kind"] == "batch":
        rng = np.random.default_rng(seed)
        # log-uniform sizes, spread evenly, in a seeded order
        sizes = rng.permutation(np.geomspace(case["lo"], case["hi"], case["scenes"]).astype(int))
        mus = rng.uniform(0.2, 0.8, case["scenes"])
        specs = [_specimen(int(n), seed * 1009 + i, float(mu)) for i, (n, mu) in enumerate(zip(sizes, mus))]
        batch = Batch(len(specs), precision=case["precision"])
        batch.load(specs, servo=_servo())
        batch.step(case["warm"])
        batch.sync()
        return {"case": case, "batch": batch, "out": [_buffer(s.n_bodies) for s in specs]}
    spec = SCENES[case["kind"]](case["n"], seed)
    return {"case": case, "engine": _engine(case, seed, spec), "out": _buffer(spec.n_bodies), "spec": spec}


def _buffer(n):
    """The pinned host buffer a program reads the bodies into."""
    return torch.empty((n, 16), dtype=torch.float64, pin_memory=True).numpy()


def run(state):
    case = state["case"]
    if case["kind"] == "adjoint":
        for t in state["leaves"]:
            t.grad = None
        loss = window_loss(state["window"], *state["leaves"], nsteps=case["steps"], checkpoint_every=case["every"],
                           wF=state["wF"])
        loss.backward()
        return {"loss": loss.detach(), "eps": state["leaves"][0].grad, "mu": state["leaves"][1].grad,
                "Kn": state["leaves"][2].grad, "Ks": state["leaves"][3].grad}
    if case["kind"] == "batch":
        batch = state["batch"]
        batch.step(case["steps"])
        batch.sync()
        servo = np.stack([e.servo_state() for e in batch.scenes])
        rows = np.concatenate([e.kinematics(o) for e, o in zip(batch.scenes, state["out"])])
        return dict(_columns(rows), walls=servo[:, 6:15], box=servo[:, 0:3])
    eng = state["engine"]
    eng.step(case["steps"])
    out = _columns(eng.kinematics(state["out"]))
    out["stress"] = eng.get_stress(1.0)
    return out


def _columns(k):
    return {"pos": k[:, 0:3], "ori": k[:, 3:7], "vel": k[:, 7:10], "angVel": k[:, 10:13], "angMom": k[:, 13:16]}


def work(case):
    """Bytes: the body state and the contact history read, and the contact fields and body state
    written, once per step.  Operations: one evaluation of each touching contact per step (adjoint:
    one per pair and step forward, and its tangents, 17 of them, in the reverse pass)."""
    s = case["steps"]
    if case["kind"] == "adjoint":
        pairs = 7.0 * case["n"]
        flops = s * pairs * (2 * EVAL_FLOPS + 17 * EVAL_FLOPS / 10)
        return {"bytes": s * (2 * 160.0 * case["n"] + 2 * 160.0 * pairs), "flops": flops}
    if case["kind"] == "batch":
        lo, hi = case["lo"], case["hi"]
        n, kind = case["scenes"] * ((hi - lo) / math.log(hi / lo) if hi > lo else lo), "specimen"
    else:
        n, kind = case["n"], case["kind"]
    return {"bytes": s * n * (BODY_BYTES + 200.0 + ENTRY_BYTES * ENTRIES[kind]),
            "flops": s * n * TOUCHING[kind] * EVAL_FLOPS}


# ---------------------------------------------------------------------------------------------
# the timestep in plain numpy, 64 bits (linear contact model, walls or periodic cell): what a pass
# of one step gives from the same starting bodies and interactions (over several steps the
# trajectories of a granular packing part, from the last bit on)

EXACT_BODIES = 15000


def exact(case, seed):
    if case["kind"] not in ("walled", "cell") or case["n"] > EXACT_BODIES or case["steps"] > 1:
        return None
    state = prepare(case, seed)
    eng, spec = state["engine"], state["spec"]
    sim = _Plain(spec, eng.body_state(), eng.interactions(include_potential=True), eng.cell())
    sim.step()
    out = _columns(np.concatenate([sim.pos, sim.ori, sim.vel, sim.ang, sim.mom], axis=1))
    out["stress"] = None   # a reduction over whole contact forces whose sum nearly cancels
    return out


def _dot(a, b):
    return np.einsum("...i,...i->...", a, b)


def _matrices(q):
    w, x, y, z = q.T
    return np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y), 2 * (x * y + w * z),
                     1 - 2 * (x * x + z * z), 2 * (y * z - w * x), 2 * (x * z - w * y), 2 * (y * z + w * x),
                     1 - 2 * (x * x + y * y)], -1).reshape(-1, 3, 3)


def _support(sh, n):
    """Point of the surface of shapes sh (rx, ry, rz, eps1, eps2) whose outward normal is n."""
    rx, ry, rz, e1, e2 = sh.T
    ax, ay, az = np.abs(rx * n[:, 0]), np.abs(ry * n[:, 1]), np.abs(rz * n[:, 2])
    f0 = np.arctan2(np.sign(n[:, 1]) * ay ** (1 / (2 - e1)), np.sign(n[:, 0]) * ax ** (1 / (2 - e1)))
    c0, s0 = np.cos(f0), np.sin(f0)
    f1 = np.arctan2(np.sign(n[:, 2]) * (az * np.abs(c0) ** (2 - e1)) ** (1 / (2 - e2)), ax ** (1 / (2 - e2)))
    c1, s1 = np.cos(f1), np.sin(f1)
    k = np.abs(c1) ** e2
    return np.stack([np.sign(c0) * rx * np.abs(c0) ** e1 * k, np.sign(s0) * ry * np.abs(s0) ** e1 * k,
                     np.sign(s1) * rz * np.abs(s1) ** e2], -1)


def _direction(p):
    return np.stack([np.cos(p[:, 0]) * np.cos(p[:, 1]), np.sin(p[:, 0]) * np.cos(p[:, 1]), np.sin(p[:, 1])], -1)


class _Pairs:
    """Closest points of pairs of superellipsoids: the damped Gauss-Newton search over the two
    angles of the contact direction, all pairs at once, each with its own step control."""

    def __init__(self, shA, RA, xA, rA, shB, RB, xB):
        self.args = shA, RA, xA, shB, RB, xB
        self.rA = rA

    def points(self, i, q):
        shA, RA, xA, shB, RB, xB = (a[i] for a in self.args)
        c = _direction(q)
        p1 = np.einsum("nij,nj->ni", RA, _support(shA, np.einsum("nji,nj->ni", RA, c))) + xA
        p2 = np.einsum("nij,nj->ni", RB, _support(shB, -np.einsum("nji,nj->ni", RB, c))) + xB
        return p1, p2, _dot(c, p2 - p1) > 0

    def search(self, idx, p):
        """From angles p of the pairs idx: (angles, direction, p1, p2, touching)."""
        m = len(idx)
        P1, P2, apart = self.points(idx, p)
        f, con, touch = P2 - P1, np.zeros((m, 3)), np.ones(m, bool)
        p, mu, nu, k = p.copy(), np.zeros(m), np.full(m, 2.0), np.zeros(m, int)
        D = np.full((m, 2), 1e-7)
        out, live = np.ones(m, bool), np.arange(m)
        while len(live):
            # tests before the Jacobian
            a = live
            live = a[(k[a] < 50) & out[a]]
            live = live[np.linalg.norm(f[live], axis=1) > 1e-20]
            touch[live[apart[live]]] = False
            live = live[~apart[live]]
            con[live] = _direction(p[live])
            live = live[np.abs(_dot(f[live], con[live])) / np.linalg.norm(f[live], axis=1) <= 0.95]
            if not len(live):
                break
            J = []
            for j in range(2):
                q = p[live].copy()
                q[:, j] += D[live, j]
                P1[live], P2[live], s = self.points(idx[live], q)
                apart[live] |= s
                J.append((P2[live] - P1[live] - f[live]) / D[live, j][:, None])
            j00, j01, j11 = _dot(J[0], J[0]), _dot(J[0], J[1]), _dot(J[1], J[1])
            t0, t1 = -_dot(J[0], f[live]), -_dot(J[1], f[live])
            go = np.maximum(np.abs(t0), np.abs(t1)) > 1e-15
            live, j00, j01, j11, t0, t1 = (v[go] for v in (live, j00, j01, j11, t0, t1))
            mu[live] = np.where(k[live] == 0, np.maximum(j00, j11), mu[live])
            todo = np.arange(len(live))
            while len(todo):
                a = live[todo]
                b00, b11 = j00[todo] + mu[a], j11[todo] + mu[a]
                det = b00 * b11 - j01[todo] ** 2
                D[a, 0] = (t0[todo] * b11 - t1[todo] * j01[todo]) / det
                D[a, 1] = (t1[todo] * b00 - t0[todo] * j01[todo]) / det
                small = np.linalg.norm(D[a], axis=1) < 1e-5
                out[a[small]] = False
                k[a[small]] += 1
                todo, a = todo[~small], a[~small]
                q = p[a] + D[a]
                P1[a], P2[a], s = self.points(idx[a], q)
                apart[a] |= s
                g = P2[a] - P1[a]
                dF = np.linalg.norm(f[a], axis=1) - np.linalg.norm(g, axis=1)
                dL = D[a, 0] * (mu[a] * D[a, 0] + t0[todo]) + D[a, 1] * (mu[a] * D[a, 1] + t1[todo])
                rho = dF / dL
                ok = rho > 0
                b = a[ok]
                mu[b] *= np.maximum(1 - (2 * rho[ok] - 1) ** 3, 0.3333333333333334)
                nu[b], p[b], f[b] = 2, q[ok], g[ok]
                k[b] += 1
                b = a[~ok]
                mu[b] *= nu[b]
                nu[b] *= 2
                over = nu >= 2.0 ** 31
                out[b[over[b]]] = False
                todo = todo[~ok & ~over[a]]
        return p, con, P1, P2, touch

    def inside(self, i, p, second):
        sh, R, x = (a[i] for a in (self.args[3:] if second else self.args[:3]))
        p = np.abs(np.einsum("nji,nj->ni", R, p - x)) / sh[:, :3]
        e1, e2 = sh[:, 3], sh[:, 4]
        return (p[:, 0] ** (2 / e1) + p[:, 1] ** (2 / e1)) ** (e1 / e2) + p[:, 2] ** (2 / e2) < 1

    def solve(self, p, new):
        every = np.arange(len(p))
        line = self.args[5] - self.args[2]
        centre = np.stack([np.arctan2(line[:, 1], line[:, 0]),
                           np.arctan(line[:, 2] / np.hypot(line[:, 0], line[:, 1]))], -1) + 1e-5
        p = np.where(new[:, None], centre, p)
        res = [np.array(v) for v in self.search(every, p)]
        far = res[4] & (10 * np.linalg.norm(res[3] - res[2], axis=1) > self.rA)
        again = every[far & ~(self.inside(every, res[3], False) & self.inside(every, res[2], True)) & ~new]
        if len(again):
            for r, v in zip(res, self.search(again, centre[again])):
                r[again] = v
        return res


class _Plain:
    """Bodies and interactions advanced by one timestep of the linear contact model."""

    def __init__(self, spec, bodies, recs, cell):
        self.spec, self.par = spec, spec.params
        self.pos, self.ori, self.vel = bodies[:, 0:3].copy(), bodies[:, 3:7].copy(), bodies[:, 7:10].copy()
        self.ang, self.mom = bodies[:, 10:13].copy(), bodies[:, 13:16].copy()
        self.lo, self.hi, self.mass, self.I = bodies[:, 22:25], bodies[:, 25:28], bodies[:, 33], bodies[:, 34:37]
        self.sq = np.asarray(spec.kind) == 0
        sh = np.asarray(spec.shape5)
        self.rb = sh[:, :3].max(1) * np.where((sh[:, 3:] < 1).any(1), math.sqrt(2.0), 1.0)
        self.peri = bool(spec.info.get("periodic"))
        self.h, self.vg, self.pvg = (cell[k:k + 9].reshape(3, 3).copy() for k in (0, 9, 18))
        recs = recs[self.sq[recs[:, 1].astype(int)]]   # no wall-wall pairs
        self.a, self.b = recs[:, 0].astype(int), recs[:, 1].astype(int)
        self.new, self.depth, self.angle = recs[:, 3] == 0, recs[:, 4].copy(), recs[:, 5:7].copy()
        self.normal, self.shear, self.cd = recs[:, 10:13].copy(), recs[:, 29:32].copy(), recs[:, 44:47]

    def step(self):
        dt = self.par["dt"]
        if self.peri:
            self.h += dt * self.vg @ self.h
        a, b = self.a, self.b
        shift = self.cd @ self.h.T if self.peri else np.zeros((len(a), 3))
        apart = ((self.lo[a] >= self.hi[b] + shift) | (self.lo[b] + shift >= self.hi[a])).any(1)
        self.new[apart] = True
        self.shear[apart] = 0
        f, t = self.contacts(np.flatnonzero(~apart), shift)
        self.newton(f, t)

    def contacts(self, e, shift):
        spec, m = self.spec, self.spec.materials
        sh, R = np.asarray(spec.shape5), _matrices(self.ori)
        dt = self.par["dt"]
        a, b, new = self.a[e], self.b[e], self.new[e]
        xb = self.pos[b] + shift[e]
        fresh_shear = new | (self.depth[e] <= 0)
        depth, cp, nrm = np.zeros(len(e)), np.zeros((len(e), 3)), np.zeros((len(e), 3))
        wall = ~self.sq[a]
        near = np.flatnonzero(~wall & ~(np.linalg.norm(self.pos[a] - xb, axis=1) > self.rb[a] + self.rb[b]))
        ia, ib = a[near], b[near]
        pairs = _Pairs(sh[ia], R[ia], self.pos[ia], self.rb[ia], sh[ib], R[ib], xb[near])
        ang, con, p1, p2, touch = pairs.solve(self.angle[e[near]], new[near])
        self.angle[e] = np.where(new[:, None], 0, self.angle[e])
        self.angle[e[near]] = ang
        depth[near] = np.where(touch, _dot(p1 - p2, con), 0)
        cp[near], nrm[near] = 0.5 * (p1 + p2), con / np.maximum(np.linalg.norm(con, axis=1), 1e-300)[:, None]
        hit = np.zeros(len(e), bool)
        hit[near] = touch
        for axis in range(3):
            w = np.flatnonzero(wall & (spec.wall_axis_sense[a, 0] == axis))
            n = np.zeros((len(w), 3))
            n[:, axis] = spec.wall_axis_sense[a[w], 1]
            p = np.einsum("nij,nj->ni", R[b[w]], _support(sh[b[w]], -np.einsum("nji,nj->ni", R[b[w]], n))) + self.pos[b[w]]
            gap = p[:, axis] - self.pos[a[w], axis]
            on = n[:, axis] * gap < 0
            q = p.copy()
            q[:, axis] = self.pos[a[w], axis]
            hit[w], depth[w], cp[w], nrm[w] = on, np.where(on, np.abs(gap), 0), 0.5 * (p + q), n
        # contact law: linear springs, Coulomb cap
        ma, mb = np.asarray(spec.mat)[a], np.asarray(spec.mat)[b]
        kn = np.where(a > 5, 2 * m["Kn"][ma] * m["Kn"][mb] / (m["Kn"][ma] + m["Kn"][mb]), m["Kn"][ma])
        ks = np.where(a > 5, 2 * m["Ks"][ma] * m["Ks"][mb] / (m["Ks"][ma] + m["Ks"][mb]), m["Ks"][ma])
        tan = np.tan(np.where(a > 5, np.minimum(m["frictionAngle"][ma], m["frictionAngle"][mb]), m["frictionAngle"][ma]))
        spin = 0.5 * dt * _dot(nrm, self.ang[a] + self.ang[b])
        field = shift[e] @ self.vg.T
        vrel = self.vel[b] + field + np.cross(self.ang[b], cp - xb) - self.vel[a] - np.cross(self.ang[a], cp - self.pos[a])
        inc = (vrel - _dot(nrm, vrel)[:, None] * nrm) * dt
        s = self.shear[e]
        s = s - np.cross(s, np.cross(self.normal[e], nrm))
        s = s - np.cross(s, spin[:, None] * nrm)
        s = s - _dot(nrm, s)[:, None] * nrm
        s = np.where(fresh_shear[:, None], 0, s) - ks[:, None] * inc
        on = hit & (depth > 1e-18)
        fn = nrm * (depth * kn)[:, None]
        cap = np.linalg.norm(fn, axis=1) * tan
        size = np.linalg.norm(s, axis=1)
        s = s * np.where(size > cap, cap / np.maximum(size, 1e-300), 1)[:, None]
        self.depth[e] = np.where(hit, depth, 0)
        self.normal[e] = np.where(hit[:, None], nrm, self.normal[e])
        self.shear[e] = np.where(on[:, None], s, 0)
        self.new[e] = False
        F = np.where(on[:, None], -fn - s, 0)
        f, t = np.zeros_like(self.pos), np.zeros_like(self.pos)
        np.add.at(f, a, F)
        np.add.at(f, b, -F)
        np.add.at(t, a, np.cross(cp - self.pos[a], F))
        np.add.at(t, b, np.cross(xb - cp, F))
        return f, t

    def newton(self, f, t):
        """Leapfrog with local damping, body by body; walls keep their place."""
        dt, d, sq = self.par["dt"], self.par["damping"], self.sq
        f, t, m, I = f[sq], t[sq], self.mass[sq, None], self.I[sq]
        x, v, w, L, o = self.pos[sq], self.vel[sq], self.ang[sq], self.mom[sq], self.ori[sq]
        acc = f / m + np.asarray(self.par["gravity"])
        fluct = v - x @ self.pvg.T if self.peri else v
        acc = acc * (1 - d * np.sign(acc * (fluct + 0.5 * dt * acc)))
        if self.peri:
            acc = acc + v @ self.pvg.T
        v = v + dt * acc
        t = t * (1 - d * np.sign(t * w))
        R = _matrices(o)

        def rate(mom, q):
            b = np.einsum("nji,nj->ni", R, mom) / I
            qw, qx, qy, qz = q.T
            wx, wy, wz = b.T
            return b, 0.5 * np.stack([-wx * qx - wy * qy - wz * qz, wx * qw - wy * qz + wz * qy,
                                      wx * qz + wy * qw - wz * qx, -wx * qy + wy * qx + wz * qw], -1)

        half = o + rate(L + 0.5 * dt * t, o)[1] * (0.5 * dt)
        L = L + dt * t
        body, dq = rate(L, half)
        o = o + dq * dt
        qv = o[:, 1:]
        c = 2 * np.cross(qv, body)
        w = body + o[:, :1] * c + np.cross(qv, c)
        o = o / np.linalg.norm(o, axis=1)[:, None]
        if self.peri:
            v = v + x @ (self.vg - self.pvg).T
            self.pvg = self.vg.copy()
        x = x + v * dt
        self.pos[sq], self.vel[sq], self.ang[sq], self.mom[sq], self.ori[sq] = x, v, w, L, o
