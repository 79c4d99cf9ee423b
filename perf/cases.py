"""The work a user of this framework has it do, as timed cases.

Every case but the differentiable one is a rollout: body state from page-locked host arrays
(``World.write_bodies``), a few steps (``World.step``), body state back into page-locked host
arrays (``World.bodies``). That is what a control loop, a viewer's frame or a planner's
what-if asks for, and it returns to the same bodies each time, so a pass has the same work
however often it is made. Contacts, joints and their multipliers stay on the GPU between
passes, as they do in a simulation. The differentiable case is a forward over several steps
and its backward.

A case holds: ``kind`` (the scene), the scene's sizes, ``steps`` per pass, ``iterations`` per
step, ``settle`` (steps made before the first pass, so that a pass meets the contacts of a
running simulation) and, where it is not the uniform grid, ``broadphase``. Scenes come from
this package's own generators; the seed moves their random draws, and gives the scenes of
fixed layout (pyramid, rope, batches of worlds) a small random velocity per body.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from avbd_demo3d_b200 import World, scenes

F32 = np.float32
SAP, GRID = scenes.BROADPHASE_SAP, scenes.BROADPHASE_GRID


def listed():
    return [
        # the smallest calls, one step a frame: latency and launches
        # a hanging rope of ball joints
        dict(name="rope20", kind="rope", links=20, steps=1, iterations=10, settle=0),
        # the 210-box benchmark pyramid at a viewer's frame
        dict(name="pyramid20", kind="pyramid", rows=20, steps=1, iterations=10, settle=10),
        # ordinary scenes of hundreds to thousands of bodies
        # mixed primitives (spheres, capsules, cylinders, boxes) falling onto each other
        dict(name="round600", kind="round", bodies=600, steps=2, iterations=10, settle=40),
        # boxes, jointed chains and springs in one scene
        dict(name="mixed6000", kind="mixed", bodies=6000, chains=40, links=16, steps=2, iterations=10, settle=40),
        # a field of box stacks, several steps a frame
        dict(name="stacks4096", kind="stacks", nx=16, ny=16, height=16, steps=4, iterations=10, settle=10),
        # the same with the sweep-and-prune broadphase option, ragged sizes
        dict(name="sap1859", kind="stacks", nx=13, ny=13, height=11, steps=2, iterations=10, settle=10,
             broadphase=SAP),
        # large scenes
        # 20,000 spheres poured onto cylinders
        dict(name="pour20000", kind="pour", bodies=20000, steps=2, iterations=10, settle=40),
        # the 65,536-box stack field, the headline workload
        dict(name="stacks65536", kind="stacks", nx=64, ny=64, height=16, steps=4, iterations=10, settle=10),
        # four times that: data beyond the L2 cache
        dict(name="stacks262144", kind="stacks", nx=128, ny=128, height=16, steps=2, iterations=10, settle=10),
        # many uneven independent worlds in one context (stacks, jointed chains, drop piles of
        # 8 to 2,048 boxes), as a training farm steps them
        dict(name="worlds64", kind="worlds", worlds=64, steps=2, iterations=10, settle=20),
        dict(name="worlds512", kind="worlds", worlds=512, steps=2, iterations=10, settle=20),
        # the differentiable step on the 1,000-box tower: forward with its tape, then backward
        dict(name="adjoint1000", kind="adjoint", nx=10, ny=10, height=10, steps=20, every=10, iterations=10,
             settle=0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rope", "pyramid", "round", "mixed", "stacks", "stacks", "stacks", "sap", "pour", "worlds",
                       "adjoint"])
    c = dict(kind=kind, steps=rng.choice([1, 2, 4]), iterations=rng.choice([5, 8, 10, 10, 15]),
             settle=rng.randint(5, 40))
    if kind == "rope":
        c.update(links=_log(rng, 4, 120), settle=0)
    elif kind == "pyramid":
        c.update(rows=_log(rng, 4, 50))
    elif kind == "round":
        c.update(bodies=_log(rng, 40, 3000))
    elif kind == "mixed":
        n = _log(rng, 300, 6000)
        c.update(bodies=n, chains=max(1, n // 150), links=rng.randint(6, 16))
    elif kind in ("stacks", "sap"):
        height = rng.randint(3, 20)
        columns = _log(rng, 4, (3000 if kind == "sap" else 200000) // height)
        nx = max(1, int(round(math.sqrt(columns) * rng.uniform(0.7, 1.4))))
        c.update(kind="stacks", nx=nx, ny=max(1, columns // nx), height=height)
        if kind == "sap":
            c.update(broadphase=SAP)
        if nx * c["ny"] * height > 60000:
            c.update(steps=min(c["steps"], 2), iterations=min(c["iterations"], 10))
    elif kind == "pour":
        c.update(bodies=_log(rng, 100, 20000))
    elif kind == "worlds":
        c.update(worlds=_log(rng, 4, 400))
    else:
        c.update(nx=rng.randint(1, 10), ny=rng.randint(1, 10), height=rng.randint(2, 10), steps=rng.randint(4, 20),
                 iterations=rng.choice([5, 8, 10]), settle=0)
        c.update(every=rng.choice([4, 5, 10]))
    return c


# ---------------------------------------------------------------------------
# Scenes and states
# ---------------------------------------------------------------------------


def _scene(case, seed):
    """The case's scene, or list of scenes for a batch."""
    kind = case["kind"]
    p = scenes.baseline_params(iterations=case["iterations"], broadphase=case.get("broadphase", GRID))
    s = 1000 + int(seed)
    if kind in ("rope", "pyramid"):
        sc = scenes.rope(case["links"], params=p) if kind == "rope" else scenes.pyramid(case["rows"], params=p)
        noise = np.random.default_rng(s).uniform(-0.05, 0.05, sc.vel.shape).astype(F32)
        sc.vel[:] = np.where(sc.density[:, None] > 0, noise, F32(0.0))
        return sc
    if kind == "round":
        return scenes.round_mix(case["bodies"], seed=s, cols=max(3, round(case["bodies"] ** (1 / 3))), params=p)
    if kind == "mixed":
        side = 40.0 * (case["bodies"] / 6000.0) ** (1 / 3)
        return scenes.mixed_drop(case["bodies"], case["chains"], case["links"], 0.1,
                                 extent=(max(side, 20.0), max(side, 20.0), max(0.75 * side, 12.0)), seed=s, params=p)
    if kind == "pour":
        return scenes.sphere_pour(case["bodies"], seed=s, params=p)
    if kind == "worlds":
        # the farm's worlds are the same for every seed (their counts are array sizes a program
        # keeps); the seed moves the bodies
        batch = scenes.batched_worlds(case["worlds"], seed=3, params=p)
        draws = np.random.default_rng(s)
        for sc in batch:
            noise = draws.uniform(-0.05, 0.05, sc.vel.shape).astype(F32)
            sc.vel[:] = np.where(sc.density[:, None] > 0, noise, F32(0.0))
        return batch
    return scenes.stack_grid(case["nx"], case["ny"], case["height"], seed=s, params=p)


_FIELDS = (("pos", 3), ("quat", 4), ("vel", 3), ("angvel", 3), ("prevvel", 3))


def _pinned(n):
    """Page-locked body state arrays, as a program that reads or writes every frame keeps."""
    return {k: torch.zeros((n, w), dtype=torch.float32, pin_memory=True).numpy() for k, w in _FIELDS}


def prepare(case, seed):
    w = World(_scene(case, seed))
    if case["settle"]:
        w.step(case["settle"])
    start = w.bodies(out=_pinned(w.n))
    state = dict(case=case, world=w, start=start, out=_pinned(w.n))
    if case["kind"] == "adjoint":
        g = np.random.default_rng(seed)
        dyn = w.props["mass"] > 0
        state["d_pos"] = np.where(dyn[:, None], g.standard_normal((w.n, 3)), 0.0)
        state["d_vel"] = np.where(dyn[:, None], 0.1 * g.standard_normal((w.n, 3)), 0.0)
    return state


def run(state):
    case, w = state["case"], state["world"]
    w.write_bodies(**state["start"])
    if case["kind"] == "adjoint":
        w.adjoint_forward(case["steps"], case["every"])
        grad = w.adjoint_backward(d_pos=state["d_pos"], d_vel=state["d_vel"])
        return dict(state=w.bodies(out=state["out"]), grad=grad)
    w.step(case["steps"], sync=False)
    return w.bodies(out=state["out"])


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------


def _sizes(case):
    """(bodies, contacts, joints) of a pass, about: counts a settled scene of the kind has."""
    kind = case["kind"]
    if kind == "rope":
        return case["links"] + 1, 0, case["links"] - 1
    if kind == "pyramid":
        n = case["rows"] * (case["rows"] + 1) // 2
        return n + 1, 8 * n, 0
    if kind == "worlds":
        n = 355 * case["worlds"]  # mean of the log-uniform box counts
        return n, int(1.4 * n), int(0.69 * n)
    if kind in ("round", "pour"):
        return case["bodies"] + 6, case["bodies"], 0
    if kind == "mixed":
        return case["bodies"] + 1, case["bodies"] // 2, case["chains"] * (case["links"] - 1)
    n = case["nx"] * case["ny"] * case["height"]
    return n + 1, 4 * n, 0


def work(case):
    """Body state in and out once (64 B each way) with the static properties (44 B); each
    contact's record (64 B, its share of the manifold's basis and bodies 18 B) and each joint's
    (128 B) in and out once; for the differentiable case the forward's and the backward's state
    in double precision besides. Operations: per iteration and contact or joint, both bodies'
    rows (about 350 each) and the dual update (100); per body the 6x6 solve and the pose update
    (about 300); per step and contact the narrowphase and the warm start (about 1,000). The
    backward replays and reverses: about four times the forward's operations."""
    n, contacts, joints = _sizes(case)
    nbytes = n * (64 + 64 + 44) + 2 * contacts * 82 + 2 * joints * 128
    per_step = case["iterations"] * ((contacts + joints) * 800 + n * 300) + 1000 * contacts
    flops = case["steps"] * per_step
    if case["kind"] == "adjoint":
        nbytes += 2 * n * 13 * 8 + n * 21 * 8
        flops *= 5
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------
# Values in 64 bits
# ---------------------------------------------------------------------------


def _qmul(a, b):
    ax, ay, az, aw = a.T
    bx, by, bz, bw = b.T
    return np.stack([aw * bx + ax * bw + ay * bz - az * by, aw * by - ax * bz + ay * bw + az * bx,
                     aw * bz + ax * by - ay * bx + az * bw, aw * bw - ax * bx - ay * by - az * bz], axis=1)


def _qdiff(a, b):
    """Rotation from b to a: twice the vector part of a b^-1."""
    conj = b * np.array([-1.0, -1.0, -1.0, 1.0])
    return 2.0 * _qmul(a, conj / (b * b).sum(1, keepdims=True))[:, :3]


def _qstep(q, w):
    r = q + 0.5 * _qmul(np.concatenate([w, np.zeros((len(w), 1))], axis=1), q)
    return r / np.linalg.norm(r, axis=1, keepdims=True)


def _rotate(q, v):
    t = 2.0 * np.cross(q[:, :3], v)
    return v + q[:, 3:] * t + np.cross(q[:, :3], t)


def _skew(r):
    z = np.zeros(len(r))
    return np.stack([np.stack([z, -r[:, 2], r[:, 1]], 1), np.stack([r[:, 2], z, -r[:, 0]], 1),
                     np.stack([-r[:, 1], r[:, 0], z], 1)], 1)


def exact(case, seed):
    """A rope's steps in double precision: no body touches another, so the step is the joints'
    alone. A scene with contacts has no such value: its contact features, clamps and friction
    branches are decided by single-precision comparisons, and within a few steps its motion
    depends on every one of them."""
    if case["kind"] != "rope":
        return None
    sc = _scene(case, seed)
    f = lambda a: np.asarray(a, F32)[::-1].astype(np.float64)  # list order: the newest body first
    pos, vel, quat, size, density = f(sc.pos), f(sc.vel), f(sc.quat), f(sc.size), f(sc.density)
    ang, prev = np.zeros_like(vel), vel.copy()
    mass = size.prod(1) * density
    sq = size * size
    moment = (sq.sum(1, keepdims=True) - sq) / 12.0 * mass[:, None]
    p = sc.params
    dt, g, alpha, gamma, beta = (float(F32(x)) for x in (p.dt, p.gravity, p.alpha, p.gamma, p.betaLin))
    n, J = len(pos), sc.n_forces
    a, b = n - 1 - sc.fa, n - 1 - sc.fb
    rA, rB = sc.frA.astype(np.float64), sc.frB.astype(np.float64)
    lam, pen = np.zeros((J, 3)), np.zeros((J, 3))
    dyn = mass > 0
    linked = np.isin(np.arange(n), np.concatenate([a, b]))
    # the rope's links alternate between the two colours of a path, newest link first
    chain = np.flatnonzero(dyn & linked)
    for _ in range(case["steps"]):
        arm = lambda: (_rotate(quat[a], rA), _rotate(quat[b], rB))
        ra, rb = arm()
        C0 = (pos[a] + ra) - (pos[b] + rb)
        lam, pen = lam * alpha * gamma, np.clip(pen * gamma, 1.0, 1e10)
        weight = np.clip((vel[:, 2] - prev[:, 2]) / dt * np.sign(g) / abs(g), 0.0, 1.0)
        pos0, quat0, down = pos.copy(), quat.copy(), np.array([0.0, 0.0, g]) * dt * dt
        inert, inert_q = pos + vel * dt + np.where(dyn[:, None], down, 0.0), _qstep(quat, ang * dt)
        pos = np.where(dyn[:, None], pos + vel * dt + down * weight[:, None], pos)
        quat = np.where(dyn[:, None], inert_q, quat)
        free = dyn & ~linked
        pos[free] = inert[free]
        for _ in range(case["iterations"]):
            for colour in (chain[0::2], chain[1::2]):
                L, A, X = (np.zeros((n, 3, 3)) for _ in range(3))
                L[colour] = (mass[colour] / dt**2)[:, None, None] * np.eye(3)
                A[colour] = (moment[colour] / dt**2)[:, :, None] * np.eye(3)
                RL = mass[:, None] / dt**2 * (pos - inert)
                RA = moment / dt**2 * _qdiff(quat, inert_q)
                ra, rb = arm()
                F = pen * ((pos[a] + ra) - (pos[b] + rb) - alpha * C0) + lam
                for body, sign, r in ((a, 1.0, ra), (b, -1.0, rb)):
                    jang = _skew(-sign * r)
                    kj = pen[:, :, None] * jang
                    v = sign * r
                    H = np.zeros((J, 3, 3))
                    for k in range(3):
                        S = -v[:, k, None, None] * np.eye(3)
                        S[:, :, k] += v
                        H += F[:, k, None, None] * S
                    np.add.at(L, body, pen[:, :, None] * np.eye(3))
                    np.add.at(A, body, jang.transpose(0, 2, 1) @ kj
                              + np.linalg.norm(H, axis=1)[:, :, None] * np.eye(3))
                    np.add.at(X, body, jang.transpose(0, 2, 1) @ (sign * pen[:, :, None] * np.eye(3)))
                    np.add.at(RL, body, sign * F)
                    np.add.at(RA, body, np.einsum("jki,jk->ji", jang, F))
                S = np.concatenate([np.concatenate([L, X.transpose(0, 2, 1)], 2), np.concatenate([X, A], 2)], 1)
                d = np.linalg.solve(S[colour], -np.concatenate([RL, RA], 1)[colour][:, :, None])[:, :, 0]
                pos[colour] += d[:, :3]
                quat[colour] = _qstep(quat[colour], d[:, 3:])
            ra, rb = arm()
            C = (pos[a] + ra) - (pos[b] + rb) - alpha * C0
            lam = pen * C + lam
            pen = np.minimum(pen + np.abs(C) * beta, 1e10)
        prev = vel.copy()
        vel = np.where(dyn[:, None], (pos - pos0) / dt, vel)
        ang = np.where(dyn[:, None], _qdiff(quat, quat0) / dt, ang)
    return dict(pos=pos, quat=quat, vel=vel, angvel=ang, prevvel=prev)
