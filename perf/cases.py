"""Cases of real use for timing the stepping paths through the package's public calls.

Every case is one rollout segment as a host program runs it: the worlds' state goes in from
page-locked host arrays, the worlds advance a control interval or a short horizon in the batched
form, and the state comes back.  Sizes follow the five workloads of `bench.py` and
`tooling_gb300/scenes.py` (chains, free-body piles, quadrupeds, the uneven mix, served rollouts)
and the scenes of the tests (one double pendulum, floating arms, RK4, Newton piles, capsules).

The states are those met in the middle of a run: chains swing from random angles, piles lie on
the ground with stacked, tilted and still falling bodies, quadrupeds stand, walk and lie.  They
are built here from the seed alone (nothing is stepped to make them).  Horizons are short where
contacts or long chains amplify rounding, so that outputs can be compared.
"""
import math

import numpy as np
import torch

from tooling_gb300 import Engine
from tooling_gb300 import model as M

SOLREF, SOLIMP = (0.02, 1.0), (0.9, 0.95, 0.001, 0.5, 2.0)
GRAVITY = (0.0, 0.0, -9.81)
F64 = torch.float64


def listed():
    return [
        # one pendulum stepped once: the smallest call a program makes, host latency and launches
        dict(name="pendulum", kind="tree", worlds=1, hinges=2, base="fixed", rk4=False, dt=1e-3, steps=1),
        # the chain workload: 4096 seven-hinge pendulums over a tenth of its 1000-step horizon
        dict(name="chains_4096x7", kind="tree", worlds=4096, hinges=7, base="fixed", rk4=False, dt=1e-3, steps=100),
        # floating trees with joints about different axes under RK4, newt's default integrator
        dict(name="floating_rk4_1000x11", kind="tree", worlds=1000, hinges=11, base="free", rk4=True, dt=2e-3, steps=20),
        # the long chains of the uneven workload, few worlds: a serial path per world
        dict(name="long_chains_300x61", kind="tree", worlds=300, hinges=61, base="fixed", rk4=False, dt=2e-3, steps=5),
        # a handful of pile worlds, as a planner or a test steps them
        dict(name="piles_10x16", kind="pile", worlds=10, bodies=16, shapes="boxes", solver="pgs", rk4=False, steps=5),
        # the headline workload: 8192 piles of 16 spheres and boxes, one control interval
        dict(name="piles_8192x16", kind="pile", worlds=8192, bodies=16, shapes="boxes", solver="pgs", rk4=False, steps=2),
        # large piles, a ragged count: many contacts per world, few worlds in flight
        dict(name="piles_700x53", kind="pile", worlds=700, bodies=53, shapes="boxes", solver="pgs", rk4=False, steps=2),
        # capsule and sphere piles under RK4 (the other free-body shapes and integrator)
        dict(name="capsules_rk4_1500x12", kind="pile", worlds=1500, bodies=12, shapes="capsules", solver="pgs", rk4=True, steps=2),
        # free bodies under the Newton solver
        dict(name="newton_piles_250x10", kind="pile", worlds=250, bodies=10, shapes="boxes", solver="newton", rk4=False, steps=2),
        # the quadruped workload: 16384 worlds, Newton, new torques, one control interval
        dict(name="quadrupeds_16384", kind="quad", worlds=16384, solver="newton", steps=2),
        # the uneven workload: chains and piles of 2 to 64 bodies in one call
        dict(name="uneven_6000", kind="uneven", worlds=6000, most=64, steps=2),
        # served rollouts: requests with their own control sequences and horizons, continuous batching
        dict(name="served_400", kind="serve", requests=400, most=24, horizon=48, active=256),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same kinds, sizes spread over their logarithm."""
    most = max(_cost(c) for c in listed())
    while True:
        kind = rng.choice(["tree", "tree", "tree", "pile", "pile", "pile", "pile", "quad", "quad", "uneven", "serve"])
        if kind == "tree":
            base = rng.choice(["fixed", "fixed", "free"])
            n = _log(rng, 2, 64 if base == "fixed" else 24)
            # long chains, and floating ones with mixed axes, amplify rounding within tens of steps at this dt
            top = 100 if n <= 8 else 50 if n <= 16 else 25 if n <= 32 else 5
            if base == "free":
                top = 20 if n <= 11 else 4
            c = dict(kind=kind, worlds=_log(rng, 1, 12000), hinges=n, base=base,
                     rk4=rng.random() < 0.3, dt=rng.choice([1e-3, 2e-3]), steps=_log(rng, 1, top))
        elif kind == "pile":
            solver = rng.choice(["pgs", "pgs", "pgs", "newton"])
            shapes = rng.choice(["boxes", "boxes", "capsules"])
            n = _log(rng, 2, 16 if solver == "newton" else 24 if shapes == "capsules" else 64)
            W = _log(rng, 1, 500 if solver == "newton" else 8192)
            top = 2 if solver == "newton" or n > 24 or W * n > 4000 else 5
            c = dict(kind=kind, worlds=W, bodies=n, shapes=shapes, solver=solver, rk4=rng.random() < 0.25,
                     steps=rng.randint(1, top))
        elif kind == "quad":
            W = _log(rng, 1, 16384)
            c = dict(kind=kind, worlds=W, solver=rng.choice(["newton", "newton", "pgs"]),
                     steps=rng.randint(1, 2 if W > 500 else 5))
        elif kind == "uneven":
            c = dict(kind=kind, worlds=_log(rng, 50, 8000), most=_log(rng, 8, 64), steps=rng.randint(1, 2))
        else:
            n = _log(rng, 20, 500)
            c = dict(kind=kind, requests=n, most=_log(rng, 4, 24), horizon=_log(rng, 8, 48),
                     active=max(8, min(256, int(n * rng.uniform(0.3, 1.2)))))
        if _cost(c) <= most:
            return c


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
LINK_FLOPS = 900     # one articulated-body recursion per link and step
ROW_FLOPS = 235      # one PGS row update of newt
PILE_CONTACTS = 1.8  # active contacts per body of a settled pile


def _parts(c):
    """(links x worlds, free bodies x worlds, geoms x worlds, flops) of a pass."""
    k = c["kind"]
    if k == "tree":
        links = c["worlds"] * (c["hinges"] + 1)
        return links, 0, 0, links * c["steps"] * LINK_FLOPS * (4 if c["rk4"] else 1)
    if k == "pile":
        bodies = c["worlds"] * c["bodies"]
        contacts = bodies * PILE_CONTACTS * (1 if c["shapes"] == "boxes" else 0.8)
        if c["solver"] == "pgs":
            f = contacts * 5 * ROW_FLOPS * 50
        else:  # the dense factor and a few Newton iterations over 4 rows per contact
            rows = 4 * contacts / c["worlds"]
            f = c["worlds"] * (rows ** 3 / 3 + 5 * 4 * rows ** 2)
        return 0, bodies, bodies + c["worlds"], f * c["steps"]
    if k == "quad":
        # recursion, 18x18 matrix and factor, about 16 rows through a dense solve
        f = 13 * LINK_FLOPS + 13 * 171 * 20 + 18 ** 3 / 3 + 16 * 18 * 18 + 16 * 16 * 18 * 2 + 16 ** 3 / 3 + 6 * 4 * 16 * 16
        return 13 * c["worlds"], 0, 14 * c["worlds"], c["worlds"] * c["steps"] * f
    if k == "uneven":
        mean = (c["most"] - 1) / math.log((c["most"] + 1) / 2)  # of a log-uniform size
        half = c["worlds"] / 2 * mean
        return half, half, half, c["steps"] * half * (LINK_FLOPS + PILE_CONTACTS * 5 * ROW_FLOPS * 50)
    mean, steps = (c["most"] - 1) / math.log((c["most"] + 1) / 2), (c["horizon"] - 3) / math.log((c["horizon"] + 1) / 4)
    links = c["requests"] * (mean + 1)
    return links, 0, 0, links * steps * LINK_FLOPS


def _cost(c):
    return _parts(c)[3]


def work(case):
    links, bodies, geoms, flops = _parts(case)
    # model (18 floats a link, 20 a body, 10 a geom), then the state read and written
    b = 4 * (links * 18 + bodies * 20 + geoms * 10) + 2 * 4 * (links * 2 + bodies * 13)
    if case["kind"] == "quad":
        b += 4 * 18 * case["worlds"]  # the torques
    if case["kind"] == "serve":
        b += 4 * flops / LINK_FLOPS   # the control sequences
    return {"bytes": b, "flops": flops}


# ---------------------------------------------------------------------------
# models and states
# ---------------------------------------------------------------------------
def _geoms(shape):
    g = np.zeros(shape, M.GEOM_DT)
    g["body"], g["link"] = -1, -1
    g["local_quat"] = (0, 0, 0, 1)
    g["friction"] = 1.0
    g["solref"], g["solimp"], g["condim"] = SOLREF, SOLIMP, 3
    g["group"] = g["mask"] = 0xFFFFFFFF
    return g


def _diag(out, d):
    """Diagonal inertias d (..., 3) into 9-float column-major matrices."""
    out[..., 0], out[..., 4], out[..., 8] = d[..., 0], d[..., 1], d[..., 2]


def _capsule_inertia(m, r, h):
    vc, vs = math.pi * r * r * 2 * h, 4 / 3 * math.pi * r ** 3
    mc = m * vc / (vc + vs)
    ms = m - mc
    zz = 0.5 * mc * r * r + 0.4 * ms * r * r
    xx = mc * (3 * r * r + 4 * h * h) / 12 + 83 / 320 * ms * r * r + ms * (h + 0.375 * r) ** 2
    return np.stack([xx, xx, zz], -1)


def _chains(rng, W, n, base, dt):
    """W chains of n hinges: links (W, n + 1), qpos, qvel, joint torques (the chain workload's
    masses, lengths, damping, angles and torques; a floating base adds a box torso and joints
    about mixed axes)."""
    free = base == "free"
    lk = np.zeros((W, n + 1), M.LINK_DT)
    lk["jp_quat"] = lk["jc_quat"] = (0, 0, 0, 1)
    lk["parent"] = np.arange(-1, n)
    lk["joint"][:, 0], lk["joint"][:, 1:] = (M.JOINT_FREE if free else M.JOINT_FIXED), M.JOINT_HINGE
    lk["axis"][:, 0] = (0, 0, 1)
    ax = rng.integers(0, 3, (W, n)) if free else np.zeros((W, n), np.int64)
    lk["axis"][:, 1:] = np.eye(3, dtype=np.float32)[ax]
    m, length = rng.uniform(0.5, 2.0, (W, n)), rng.uniform(0.2, 0.5, (W, n))
    lk["mass"][:, 0], lk["mass"][:, 1:] = (3.0 if free else 1.0), m
    _diag(lk["inertia"][:, 0], np.broadcast_to([0.05, 0.06, 0.08] if free else [1.0, 1.0, 1.0], (W, 3)))
    _diag(lk["inertia"][:, 1:], _capsule_inertia(m, 0.03, length / 2))
    lk["damping"][:, 1:] = rng.uniform(0.0, 0.1, (W, n))
    lk["jc_pos"][:, 1:, 2] = length / 2
    lk["jp_pos"][:, 2:, 2] = -length[:, :-1] / 2
    q, qd, tau = rng.uniform(-math.pi, math.pi, (W, n)), rng.normal(0, 1, (W, n)), rng.normal(0, 0.5, (W, n))
    if free:
        root = np.concatenate([rng.normal(0, 1, (W, 3)), _unit(rng.normal(0, 1, (W, 4)))], 1)
        q = np.concatenate([root, q], 1)
        qd = np.concatenate([rng.normal(0, 0.5, (W, 6)), qd], 1)
        tau = np.concatenate([np.zeros((W, 6)), tau], 1)
    return lk, q.astype(np.float32), qd.astype(np.float32), tau.astype(np.float32)


def _unit(v):
    return v / np.linalg.norm(v, axis=-1, keepdims=True)


def _qmul(a, b):  # w, x, y, z
    aw, ax, ay, az = np.moveaxis(a, -1, 0)
    bw, bx, by, bz = np.moveaxis(b, -1, 0)
    return np.stack([aw * bw - ax * bx - ay * by - az * bz, aw * bx + ax * bw + ay * bz - az * by,
                     aw * by - ax * bz + ay * bw + az * bx, aw * bz + ax * by - ay * bx + az * bw], -1)


def _rect_gap(px, py, rx, ry, yaw, hx, hy):
    """Distance in the plane from points to yawed rectangles (0 inside)."""
    c, s = np.cos(yaw), np.sin(yaw)
    u, v = c * (px - rx) + s * (py - ry), -s * (px - rx) + c * (py - ry)
    return np.hypot(np.maximum(np.abs(u) - hx, 0), np.maximum(np.abs(v) - hy, 0))


def _rects_meet(ax, ay, aw, ahx, ahy, bx, by, bw, bhx, bhy):
    dx, dy = bx - ax, by - ay
    meet = np.ones(dx.shape, bool)
    for ang in (aw, aw + math.pi / 2, bw, bw + math.pi / 2):
        c, s = np.cos(ang), np.sin(ang)
        ra = ahx * np.abs(np.cos(aw - ang)) + ahy * np.abs(np.sin(aw - ang))
        rb = bhx * np.abs(np.cos(bw - ang)) + bhy * np.abs(np.sin(bw - ang))
        meet &= np.abs(c * dx + s * dy) < ra + rb
    return meet


def _piles(rng, W, n, shapes, count=None):
    """W settled piles of n bodies (`count`: spread as piles of so many, for cutting) dropped one after the other onto what lies below: bodies
    (W, n), geoms (W, n + 1) with the ground plane first, qpos, qvel.  Half spheres, half boxes
    (or capsules, lying); resting bodies penetrate a little and creep, one uncovered body in
    five is still in the air and falls."""
    side = 2.0 * np.sqrt((np.full((W, 1), n) if count is None else count[:, None]) / 16.0)
    sphere = rng.random((W, n)) < 0.5
    r = rng.uniform(0.05, 0.2, (W, n))
    he = rng.uniform(0.05, 0.2, (W, n, 3))
    cr, ch = rng.uniform(0.04, 0.12, (W, n)), rng.uniform(0.05, 0.2, (W, n))
    x, y = side * rng.uniform(-0.5, 0.5, (W, n)), side * rng.uniform(-0.5, 0.5, (W, n))
    yaw = rng.uniform(-math.pi, math.pi, (W, n))
    boxes = shapes == "boxes"
    low = np.where(sphere, r, he[..., 2] if boxes else cr)  # height of the centre on flat ground
    z = np.zeros((W, n))
    covered = np.zeros((W, n), bool)
    bead = np.linspace(-1, 1, 9)
    for k in range(n):  # onto the k bodies already there
        best = low[:, k].copy()
        if k:
            i, j = slice(k, k + 1), slice(0, k)
            if boxes:
                # sphere on sphere, sphere on box top, box bottom on sphere, box on box
                d2, rr = (x[:, i] - x[:, j]) ** 2 + (y[:, i] - y[:, j]) ** 2, r[:, i] + r[:, j]
                ss = np.where(d2 < rr * rr, z[:, j] + np.sqrt(np.maximum(rr * rr - d2, 0)), -1.0)
                g = _rect_gap(x[:, i], y[:, i], x[:, j], y[:, j], yaw[:, j], he[:, j, 0], he[:, j, 1])
                sb = np.where(g < r[:, i], z[:, j] + he[:, j, 2] + np.sqrt(np.maximum(r[:, i] ** 2 - g * g, 0)), -1.0)
                g = _rect_gap(x[:, j], y[:, j], x[:, i], y[:, i], yaw[:, i], he[:, i, 0], he[:, i, 1])
                bs = np.where(g < r[:, j], z[:, j] + he[:, i, 2] + np.sqrt(np.maximum(r[:, j] ** 2 - g * g, 0)), -1.0)
                meet = _rects_meet(x[:, i], y[:, i], yaw[:, i], he[:, i, 0], he[:, i, 1], x[:, j], y[:, j], yaw[:, j],
                                   he[:, j, 0], he[:, j, 1])
                bb = np.where(meet, z[:, j] + he[:, j, 2] + he[:, i, 2], -1.0)
                h = np.where(sphere[:, i], np.where(sphere[:, j], ss, sb), np.where(sphere[:, j], bs, bb))
            else:  # capsules as strings of nine balls
                (px, py, pr), (qx, qy, qr) = (
                    [p[:, e, None] + np.where(sphere[:, e], 0.0, ch[:, e])[..., None] * f(yaw[:, e, None]) * bead
                     for p, f in ((x, np.cos), (y, np.sin))] + [np.where(sphere[:, e], r[:, e], cr[:, e])] for e in (i, j))
                d2 = ((px[..., :, None] - qx[..., None, :]) ** 2 + (py[..., :, None] - qy[..., None, :]) ** 2).min((2, 3))
                rr = pr + qr
                h = np.where(d2 < rr * rr, z[:, j] + np.sqrt(np.maximum(rr * rr - d2, 0)), -1.0)
            covered[:, j] |= h > 0
            best = np.maximum(best, h.max(1))
        z[:, k] = best - rng.uniform(1e-4, 8e-4, W)
    air = ~covered & (rng.random((W, n)) < 0.2)
    z += np.where(air, rng.uniform(0.005, 0.5, (W, n)), 0.0)
    vel = rng.normal(0, 0.03, (W, n, 3))
    vel[..., 2] -= np.where(air, rng.uniform(0, 2.0, (W, n)), 0.0)
    omg = rng.normal(0, 0.1, (W, n, 3))
    tilt = rng.normal(0, 2e-3, (W, n, 3))
    q = np.stack([np.cos(yaw / 2), 0 * yaw, 0 * yaw, np.sin(yaw / 2)], -1)
    q = _qmul(_unit(np.concatenate([np.ones((W, n, 1)), tilt], -1)), q)
    if not boxes:  # a capsule's axis is its local z: turn it down onto local x
        q = np.where(sphere[..., None], q, _qmul(q, np.broadcast_to([math.sqrt(0.5), 0, math.sqrt(0.5), 0], q.shape)))
    qpos = np.concatenate([np.stack([x, y, z], -1), q], -1).astype(np.float32)
    qvel = np.concatenate([vel, omg], -1).astype(np.float32)
    bd = np.zeros((W, n), M.BODY_DT)
    g = _geoms((W, n + 1))
    g["shape"][:, 0] = M.SHAPE_PLANE
    g["body"][:, 1:] = np.arange(n)
    g["friction"][:, 1:] = rng.uniform(0.3, 1.0, (W, n))
    ms = 1000 * 4 / 3 * math.pi * r ** 3
    if boxes:
        mo = 8000 * he.prod(-1)
        s2 = he ** 2
        io = mo[..., None] / 3 * (s2.sum(-1, keepdims=True) - s2)
        size = he
    else:
        mo = 1000 * (math.pi * cr * cr * 2 * ch + 4 / 3 * math.pi * cr ** 3)
        io = _capsule_inertia(mo, cr, ch)
        size = np.stack([cr, ch, 0 * cr], -1)
    bd["mass"] = np.where(sphere, ms, mo)
    _diag(bd["inertia"], np.where(sphere[..., None], (0.4 * ms * r * r)[..., None], io))
    g["shape"][:, 1:] = np.where(sphere, M.SHAPE_SPHERE, M.SHAPE_BOX if boxes else M.SHAPE_CAPSULE)
    g["size"][:, 1:] = np.where(sphere[..., None], np.stack([r, 0 * r, 0 * r], -1), size)
    return bd, g, qpos.reshape(W, -1), qvel.reshape(W, -1)


def _piles_of(rng, sizes):
    """Piles of boxes and spheres in (size, count) blocks: an octave of sizes is made at its largest, then cut."""
    out = {}
    for octave in sorted({s.bit_length() for s, _ in sizes}):
        block = [(s, W) for s, W in sizes if s.bit_length() == octave]
        count = np.concatenate([np.full(W, s) for s, W in block])
        bd, g, q, v = _piles(rng, len(count), block[0][0], "boxes", count)
        a = 0
        for s, W in block:
            out[s] = bd[a:a + W, :s], g[a:a + W, :s + 1], q[a:a + W, :7 * s], v[a:a + W, :6 * s]
            a += W
    return [out[s] for s, _ in sizes]


QUAD_PARENT = [-1] + [p for leg in range(4) for p in (0, 1 + 3 * leg, 2 + 3 * leg)]
QUAD_HIPS = np.array([[0.15, 1.0], [0.15, -1.0], [-0.15, 1.0], [-0.15, -1.0]])


def _quads(rng, W):
    """W quadrupeds of the quadruped workload: three in four stand or walk (each foot on the
    ground or in the air), the rest lie on their bellies; links (W, 13), geoms (W, 14), state and
    joint torques N(0, 2)."""
    lk = np.zeros((W, 13), M.LINK_DT)
    lk["jp_quat"] = lk["jc_quat"] = (0, 0, 0, 1)
    lk["parent"] = QUAD_PARENT
    lk["joint"][:, 0], lk["joint"][:, 1:] = M.JOINT_FREE, M.JOINT_HINGE
    lk["axis"][:, 0] = (0, 0, 1)
    lk["mass"][:, 0], lk["mass"][:, 1:] = 5.0, 0.5
    half = np.array([0.2, 0.1, 0.05])
    _diag(lk["inertia"][:, 0], np.broadcast_to(5.0 / 3 * ((half ** 2).sum() - half ** 2), (W, 3)))
    _diag(lk["inertia"][:, 1:], np.broadcast_to(_capsule_inertia(0.5, 0.02, 0.1), (W, 12, 3)))
    g = _geoms((W, 14))
    g["friction"] = 0.8
    g["shape"][:, 0], g["shape"][:, 1], g["shape"][:, 2:] = M.SHAPE_PLANE, M.SHAPE_BOX, M.SHAPE_CAPSULE
    g["link"][:, 1:] = np.arange(13)
    g["size"][:, 1], g["size"][:, 2:] = half, (0.02, 0.1, 0.0)
    lie = rng.random(W) < 0.25
    h = np.where(lie, 0.05 - rng.uniform(0, 5e-4, W), rng.uniform(0.2, 0.3, W))
    q = np.zeros((W, 12))
    for leg, (hx, sd) in enumerate(QUAD_HIPS):
        a, b, c = 1 + 3 * leg, 2 + 3 * leg, 3 + 3 * leg
        lk["axis"][:, a], lk["axis"][:, b], lk["axis"][:, c] = (1, 0, 0), (0, 1, 0), (0, 1, 0)
        lk["jp_pos"][:, a], lk["jc_pos"][:, a] = (hx, sd * 0.1, 0), (0, -sd * 0.1, 0)
        lk["jp_pos"][:, b], lk["jc_pos"][:, b] = (0, sd * 0.1, 0), (0, 0, 0.1)
        lk["jp_pos"][:, c], lk["jc_pos"][:, c] = (0, 0, -0.1), (0, 0, 0.1)
        s = math.sqrt(0.5)
        g["local_quat"][:, 1 + a] = (-s, 0, 0, s)  # the first link's capsule lies along y
        ab = np.where(lie, rng.normal(0, 0.02, W), rng.normal(0, 0.15, W))
        flex = np.where(lie, 1.50 + rng.normal(0, 0.01, W), 0.9 + rng.normal(0, 0.12, W))
        foot = np.where(rng.random(W) < 0.7, -rng.uniform(1e-4, 8e-4, W), rng.uniform(0.005, 0.05, W))
        reach = (h + sd * 0.2 * np.sin(ab) - 0.02 - foot) / (0.2 * np.cos(ab)) - np.cos(flex)
        knee = np.where(lie, rng.normal(0.05, 0.02, W), -np.arccos(np.clip(reach, -0.99, 0.99)) - flex)
        q[:, 3 * leg:3 * leg + 3] = np.stack([ab, flex, knee], -1)
    yaw = rng.uniform(-math.pi, math.pi, W)
    turn = _qmul(_unit(np.concatenate([np.ones((W, 1)), rng.normal(0, 3e-4, (W, 2)), np.zeros((W, 1))], 1)),
                 np.stack([np.cos(yaw / 2), 0 * yaw, 0 * yaw, np.sin(yaw / 2)], -1))
    root = np.concatenate([rng.normal(0, 1, (W, 2)), h[:, None], turn], 1)
    qpos = np.concatenate([root, q], 1).astype(np.float32)
    qvel = np.concatenate([rng.normal(0, 0.1, (W, 6)), rng.normal(0, 0.5, (W, 12))], 1).astype(np.float32)
    tau = np.concatenate([np.zeros((W, 6)), rng.normal(0, 2.0, (W, 12))], 1).astype(np.float32)
    return lk, g, qpos, qvel, tau


def _batch(links, bodies, geoms, dt, solver=M.SOLVER_PGS, iterations=50, rk4=False):
    """Worlds of blocks of equal size ((W, n) record arrays) as one model batch."""
    def flat(blocks, dt_):
        counts = np.concatenate([np.full(len(b), b.shape[1]) for b in blocks])
        return np.concatenate([b.reshape(-1) for b in blocks]) if counts.sum() else np.zeros(0, dt_), counts
    lk, nl = flat(links, M.LINK_DT)
    bd, nb = flat(bodies, M.BODY_DT)
    gm, ng = flat(geoms, M.GEOM_DT)
    return M.Batch(lk, nl, bd, nb, gm, ng, dt, GRAVITY, solver, iterations,
                   integrator=M.INTEGRATOR_RK4 if rk4 else M.INTEGRATOR_EULER)


def _none(W, dt_):
    return np.zeros((W, 0), dt_)


def _sizes(W, most):
    """Log-uniform sizes 2..most as (size, count) blocks, largest first: the case's, whatever the seed."""
    rng = np.random.default_rng([986, W, most])
    n = np.floor(np.exp(rng.uniform(math.log(2), math.log(most + 1), W))).astype(int).clip(2, most)
    return [(int(s), int((n == s).sum())) for s in np.unique(n)[::-1]]


def _inputs(case, seed):
    """The case's blocks and host arrays, from the seed alone."""
    rng = np.random.default_rng([987, int(seed)])
    k = case["kind"]
    if k == "tree":
        W = case["worlds"]
        lk, q, v, tau = _chains(rng, W, case["hinges"], case["base"], case["dt"])
        b = _batch([lk], [_none(W, M.BODY_DT)], [_none(W, M.GEOM_DT)], case["dt"], rk4=case["rk4"])
        return b, [lk], q.reshape(-1), v.reshape(-1), tau.reshape(-1)
    if k == "pile":
        W = case["worlds"]
        bd, g, q, v = _piles(rng, W, case["bodies"], case["shapes"])
        newton = case["solver"] == "newton"
        b = _batch([_none(W, M.LINK_DT)], [bd], [g], 2e-3, M.SOLVER_NEWTON if newton else M.SOLVER_PGS,
                   20 if newton else 50, case["rk4"])
        return b, [], q.reshape(-1), v.reshape(-1), None
    if k == "quad":
        W = case["worlds"]
        lk, g, q, v, tau = _quads(rng, W)
        newton = case["solver"] == "newton"
        b = _batch([lk], [_none(W, M.BODY_DT)], [g], 2e-3, M.SOLVER_NEWTON if newton else M.SOLVER_PGS,
                   20 if newton else 50)
        return b, [lk], q.reshape(-1), v.reshape(-1), tau.reshape(-1)
    if k == "uneven":
        half = case["worlds"] // 2
        lks, bds, gs, qs, vs, taus = [], [], [], [], [], []
        for n, W in _sizes(half, case["most"]):
            lk, q, v, tau = _chains(rng, W, n, "fixed", 2e-3)
            lks.append(lk), bds.append(_none(W, M.BODY_DT)), gs.append(_none(W, M.GEOM_DT))
            qs.append(q.reshape(-1)), vs.append(v.reshape(-1)), taus.append(tau.reshape(-1))
        chains = len(lks)
        for bd, g, q, v in _piles_of(rng, _sizes(case["worlds"] - half, case["most"])):
            lks.append(_none(len(bd), M.LINK_DT)), bds.append(bd), gs.append(g)
            qs.append(q.reshape(-1)), vs.append(v.reshape(-1)), taus.append(0 * v.reshape(-1))
        b = _batch(lks, bds, gs, 2e-3)
        return b, lks[:chains], np.concatenate(qs), np.concatenate(vs), np.concatenate(taus)
    lks, qs, vs, hs, us = [], [], [], [], []
    for n, W in _sizes(case["requests"], case["most"]):
        lk, q, v, _ = _chains(rng, W, n, "fixed", 2e-3)
        h = np.floor(np.exp(np.random.default_rng([985, n, W]).uniform(math.log(4), math.log(case["horizon"] + 1), W))).astype(np.int32)
        u = rng.normal(0, 1, (W, case["horizon"], n)).astype(np.float32)
        lks.append(lk), qs.append(q.reshape(-1)), vs.append(v.reshape(-1)), hs.append(h), us.append(u)
    W = case["requests"]
    b = _batch(lks, [_none(W, M.BODY_DT)], [_none(W, M.GEOM_DT)], 2e-3)
    return b, lks, np.concatenate(qs), np.concatenate(vs), (hs, us)


def _pinned(a):
    t = torch.empty(a.size, dtype=torch.float32, pin_memory=True).numpy()
    t[:] = a
    return t


def prepare(case, seed):
    """The engine with the worlds allocated, the state in page-locked host arrays."""
    b, _, q, v, tau = _inputs(case, seed)
    eng = Engine()
    ids = eng.upload(b)
    s = dict(kind=case["kind"], eng=eng, ids=ids, batch=b)
    if case["kind"] == "serve":
        hs, us = tau
        u = np.concatenate([x[i, :hs[k][i]].reshape(-1) for k, x in enumerate(us) for i in range(len(x))])
        h = np.concatenate(hs)
        off = np.concatenate([[0], np.cumsum(h * b.nv)[:-1]])
        order = np.random.default_rng([988, len(h)]).permutation(len(h))  # requests of all sizes mixed in time
        qo = [q[b.q_off[i]:b.q_off[i] + b.nq[i]] for i in order]
        vo = [v[b.v_off[i]:b.v_off[i] + b.nv[i]] for i in order]
        s.update(order=order, ids=ids[order], horizons=h[order], arrivals=np.arange(len(h)) * 1e-6,
                 q=np.concatenate(qo), v=np.concatenate(vo), u=u, off=off[order], active=case["active"])
        return s
    s["slots"] = eng.alloc(ids)
    s["q"], s["v"] = _pinned(q), _pinned(v)
    s["out"] = (_pinned(0 * q), _pinned(0 * v))
    s["steps"] = case["steps"]
    s["tau"] = tau if case["kind"] == "quad" else None
    if case["kind"] in ("tree", "uneven"):  # constant torques, set once
        eng.set_qfrc(s["slots"], tau)
    s["split"] = int(b.q_off[np.argmax(b.n_bodies > 0)]), int(b.v_off[np.argmax(b.n_bodies > 0)])
    return s


def run(s):
    """One rollout segment: state in, (new torques,) the steps, state out."""
    eng = s["eng"]
    if s["kind"] == "serve":
        q, v, _, _, _ = eng.serve(s["ids"], s["horizons"], s["arrivals"], s["q"], s["v"], s["u"], s["off"],
                                  max_active=s["active"], real_time=False, steps_per_tick=8)
        return {"qpos": q, "qvel": v}
    eng.set_state(s["slots"], s["q"], s["v"])
    if s["tau"] is not None:
        eng.set_qfrc(s["slots"], s["tau"])
    eng.step(s["steps"])
    q, v = eng.get_state(s["slots"], s["q"].size, s["v"].size, out=s["out"])
    if s["kind"] == "uneven":
        a, b = s["split"]
        return {"chains": [q[:a], v[:b]], "piles": [q[a:], v[b:]]}
    return {"qpos": q, "qvel": v}


# ---------------------------------------------------------------------------
# the same in 64 bits, by plain linear algebra on world matrices
# ---------------------------------------------------------------------------
def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=F64, device=_dev())


def _cross(a, b):
    return torch.linalg.cross(a, b, dim=-1)


def _qrot(q, v, inv=False):  # x, y, z, w
    u, w = (-q[:, :3] if inv else q[:, :3]), q[:, 3:]
    t = 2 * _cross(u, v)
    return v + w * t + _cross(u, t)


class _Tree:
    """Trees of one layout: the equations of motion M qdd + bias = tau in the root link's frame."""

    def __init__(self, lk, dt):
        self.parent, self.n = [int(p) for p in lk["parent"][0]], lk.shape[1]
        self.free = int(lk["joint"][0, 0]) == M.JOINT_FREE
        self.axis, self.jp, self.jc = _t(lk["axis"]), _t(lk["jp_pos"]), _t(lk["jc_pos"])
        self.m, self.damp = _t(lk["mass"]), _t(lk["damping"][:, 1:])
        self.I = _t(lk["inertia"][:, :, [0, 4, 8]])
        self.r = 6 if self.free else 0
        self.nv, self.dt = self.r + self.n - 1, float(np.float32(dt))
        self.damp = torch.cat([torch.zeros(len(self.m), self.r, dtype=F64, device=self.m.device), self.damp], 1)
        self.g = _t(np.float32(GRAVITY)).expand(len(self.m), 3)

    def read(self, q, v):
        """MuJoCo layout -> (root position, quaternion xyzw, hinge angles), rates (omega, v in the body, hinges)."""
        if not self.free:
            return (None, None, q), v
        Q = q[:, [4, 5, 6, 3]]
        Q = Q / Q.norm(dim=1, keepdim=True)
        return (q[:, :3], Q, q[:, 7:]), torch.cat([v[:, 3:6], _qrot(Q, v[:, :3], True), v[:, 6:]], 1)

    def write(self, s, v):
        p, Q, a = s
        if not self.free:
            return a, v
        return (torch.cat([p, Q[:, [3, 0, 1, 2]], a], 1),
                torch.cat([_qrot(Q, v[:, 3:6]), v[:, :3], v[:, 6:]], 1))

    def motion(self, s, v):
        W, nv, z = len(self.m), self.nv, v.new_zeros
        g = _qrot(s[1], self.g, True) if self.free else self.g
        eye = torch.eye(3, dtype=F64, device=v.device).expand(W, 3, 3)
        R, x, Jw, Jv = [eye], [z(W, 3)], [z(W, nv, 3)], [z(W, nv, 3)]
        w, al, ac = [z(W, 3)], [z(W, 3)], [-g]
        if self.free:
            Jw[0][:, 0:3], Jv[0][:, 3:6] = eye, eye
            w[0], ac[0] = v[:, :3], _cross(v[:, :3], v[:, 3:6]) - g
        for i in range(1, self.n):
            p = self.parent[i]
            a = self.axis[:, i]
            th, k = s[2][:, i - 1, None, None], z(W, 3, 3)
            k[:, 0, 1], k[:, 0, 2], k[:, 1, 2] = -a[:, 2], a[:, 1], -a[:, 0]
            k = k - k.transpose(1, 2)
            aw = (R[p] @ a[:, :, None])[:, :, 0]
            R.append(R[p] @ (eye + torch.sin(th) * k + (1 - torch.cos(th)) * (k @ k)))
            d, c = (R[p] @ self.jp[:, i, :, None])[:, :, 0], (R[i] @ self.jc[:, i, :, None])[:, :, 0]
            x.append(x[p] + d - c)
            jw = Jw[p].clone()
            jw[:, self.r + i - 1] += aw
            Jv.append(Jv[p] + _cross(Jw[p], d[:, None].expand_as(jw)) - _cross(jw, c[:, None].expand_as(jw)))
            Jw.append(jw)
            u = aw * v[:, self.r + i - 1, None]
            w.append(w[p] + u)
            al.append(al[p] + _cross(w[p], u))
            ac.append(ac[p] + _cross(al[p], d) + _cross(w[p], _cross(w[p], d)) - _cross(al[i], c)
                      - _cross(w[i], _cross(w[i], c)))
        Rs, Js, Vs = torch.stack(R, 1), torch.stack(Jw, 1), torch.stack(Jv, 1)
        I = (Rs * self.I[:, :, None, :]) @ Rs.transpose(2, 3)
        w, al, ac = torch.stack(w, 1), torch.stack(al, 1), torch.stack(ac, 1)
        IJ = Js @ I
        Mm = torch.einsum("wlac,wlbc->wab", Vs * self.m[:, :, None, None], Vs) + torch.einsum("wlac,wlbc->wab", IJ, Js)
        f, t = self.m[:, :, None] * ac, (I @ al[..., None])[..., 0] + _cross(w, (I @ w[..., None])[..., 0])
        bias = torch.einsum("wlac,wlc->wa", Vs, f) + torch.einsum("wlac,wlc->wa", Js, t)
        return Mm, bias, torch.stack(x, 1), Rs, Vs, Js

    def qdd(self, s, v, tau, fold):
        Mm, bias = self.motion(s, v)[:2]
        return torch.linalg.solve(Mm + torch.diag_embed(self.damp * fold), tau - self.damp * v - bias)

    def advance(self, s, v, dt):
        """Positions by the new rates: the root by its rotation's exponential."""
        p, Q, a = s
        if not self.free:
            return None, None, a + dt * v
        return p + dt * _qrot(Q, v[:, 3:6]), _qexp(Q, v[:, :3], dt), a + dt * v[:, 6:]

    def euler(self, s, v, tau):
        v = v + self.dt * self.qdd(s, v, tau, self.dt)
        return self.advance(s, v, self.dt), v

    def rk4(self, s, v, tau):
        def rate(s, v):
            if not self.free:
                return (None, None, v)
            return _qrot(s[1], v[:, 3:6]), 0.5 * _qmul_t(s[1], v[:, :3]), v[:, 6:]

        def shift(s, d, h):
            return tuple(None if a is None else a + h * b for a, b in zip(s, d))
        dt, ks, st, vt = self.dt, [], s, v
        for h in (dt / 2, dt / 2, dt, None):
            ks.append((rate(st, vt), self.qdd(st, vt, tau, 0.0)))
            if h is not None:
                st, vt = shift(s, ks[-1][0], h), v + h * ks[-1][1]
        for c, (d, a) in zip((1, 2, 2, 1), ks):
            s, v = shift(s, d, c * dt / 6), v + c * dt / 6 * a
        if self.free:
            s = (s[0], s[1] / s[1].norm(dim=1, keepdim=True), s[2])
        return s, v


def _qmul_t(q, w):
    """q (x, y, z, w) times the pure quaternion of w."""
    u, s = q[:, :3], q[:, 3:]
    return torch.cat([s * w + _cross(u, w), -(u * w).sum(1, keepdim=True)], 1)


def _qexp(q, w, dt):
    l = w.norm(dim=1, keepdim=True)
    k = torch.where(l > 0, torch.sin(0.5 * dt * l) / l.clamp_min(1e-300), torch.zeros_like(l))
    n = torch.cos(0.5 * dt * l) * q + _qmul_t(q, k * w)
    return n / n.norm(dim=1, keepdim=True)


def _exact_trees(lk, q, v, tau, dt, steps, rk4):
    T = _Tree(lk, dt)
    s, v = T.read(_t(q), _t(v))
    for _ in range(steps):
        s, v = (T.rk4 if rk4 else T.euler)(s, v, _t(tau))
    q, v = T.write(s, v)
    return q.reshape(-1), v.reshape(-1)


QUAD_HALF = (0.2, 0.1, 0.05)


def _exact_quads(lk, q, v, tau, steps, newton):
    """Euler steps with the soft pyramidal contacts of capsules and torso on the plane z = 0."""
    T = _Tree(lk, 2e-3)
    W, dt, mu, dev = len(T.m), T.dt, float(np.float32(0.8)), T.m.device
    s, v = T.read(_t(q), _t(v))
    tau = _t(tau)
    r, hh = float(np.float32(0.02)), float(np.float32(0.1))
    corner = _t([[a * float(np.float32(QUAD_HALF[0])), b * float(np.float32(QUAD_HALF[1])), c * float(np.float32(QUAD_HALF[2]))]
                 for c in (-1, 1) for b in (-1, 1) for a in (-1, 1)])
    first = torch.tensor([i % 3 == 0 for i in range(12)], device=dev)
    f32 = lambda a: float(np.float32(a))  # noqa: E731
    tc, dmin, dmax, width = max(f32(0.02), 2 * dt), f32(0.9), f32(0.95), f32(0.001)
    for _ in range(steps):
        Mm, bias, x, R, Jv, Jw = T.motion(s, v)
        free = torch.linalg.solve(Mm, tau - bias)
        up = _qrot(s[1], _t([[0, 0, 1.0]]).expand(W, 3), True)  # the plane's normal in the root frame
        e1, e2 = (_qrot(s[1], _t([a]).expand(W, 3), True) for a in ([0, 1.0, 0], [1.0, 0, 0]))
        # candidates in pair order: the torso's corners, then each capsule's two ends
        ax = torch.where(first[None, :, None], R[:, 1:, :, 1], R[:, 1:, :, 2])
        ends = torch.stack([x[:, 1:] + hh * ax, x[:, 1:] - hh * ax], 2).reshape(W, 24, 3)
        pts = torch.cat([corner.expand(W, 8, 3), ends], 1)
        height = s[0][:, 2:3] + (pts * up[:, None]).sum(-1)
        raw = torch.cat([height[:, :8], height[:, 8:] - r], 1)
        below = torch.cat([(corner * up[:, None]).sum(-1) <= 0, torch.ones(W, 24, dtype=torch.bool, device=dev)], 1)
        on = (raw < 0) & below
        pos = pts - up[:, None] * torch.cat([raw[:, :8] / 2, r + raw[:, 8:] / 2], 1)[..., None]
        K = int(on.sum(1).max())
        if K == 0:
            acc = free
        else:
            pick = torch.argsort((~on).to(torch.int8), dim=1, stable=True)[:, :K]
            on, pen = on.gather(1, pick), -raw.gather(1, pick)
            pos = pos.gather(1, pick[..., None].expand(W, K, 3))
            link = torch.tensor([0] * 8 + [1 + i // 2 for i in range(24)], device=dev)[pick]
            at = link[:, :, None, None].expand(W, K, T.nv, 3)
            arm = pos - x.gather(1, link[..., None].expand(W, K, 3))
            Jp = Jv.gather(1, at) + _cross(Jw.gather(1, at), arm[:, :, None].expand(W, K, T.nv, 3))
            dirs = torch.stack([up - mu * e1, up + mu * e1, up - mu * e2, up + mu * e2], 1)
            J = torch.einsum("wkac,wfc->wkfa", Jp, dirs).reshape(W, 4 * K, T.nv) * on.repeat_interleave(4, 1)[..., None]
            wt = torch.einsum("wlac,wab,wlbc->wl", Jv, torch.linalg.inv(Mm), Jv) / 3
            y = (pen.clamp_min(0) / width).clamp(max=1)
            d = dmin + (dmax - dmin) * torch.where(y < 0.5, 2 * y * y, 1 - 2 * (1 - y) ** 2)
            reg = 2 * mu * mu * (1 - d) / d * wt.gather(1, link) * (1 + mu * mu)
            ref = (-2 / (dmax * tc) * (J @ v[..., None])[..., 0]
                   + (d / (dmax * dmax * tc * tc) * pen).repeat_interleave(4, 1))
            b = (J @ free[..., None])[..., 0] * dt - ref * dt
            mask = on.repeat_interleave(4, 1)
            H = J @ torch.linalg.solve(Mm, J.transpose(1, 2)) + torch.diag_embed(reg.repeat_interleave(4, 1))
            H = H + torch.diag_embed((~mask).to(F64))
            b = torch.where(mask, b, torch.zeros_like(b))
            f = torch.zeros_like(b)
            hd = torch.diagonal(H, dim1=1, dim2=2)
            if newton:
                f = _newton64(H, b, 20)
            else:
                hd = torch.diagonal(H, dim1=1, dim2=2)
                for _ in range(50):
                    for k in range(4 * K):
                        f[:, k] = (f[:, k] - ((H[:, k] * f).sum(1) + b[:, k]) / hd[:, k]).clamp_min(0)
            acc = free + torch.linalg.solve(Mm, (J.transpose(1, 2) @ f[..., None])[..., 0]) / dt
        v = v + dt * acc
        s = T.advance(s, v, dt)
    q, v = T.write(s, v)
    return q.reshape(-1), v.reshape(-1)


def _newton64(H, b, iters):
    """newt's contact Newton (newt/src/newton.rs:275-556) on 1/2 x.Hx + b.x, x >= 0, a batch of systems at once:
    full Newton directions, the exact search over each projected ray, its stopping rule."""
    x, n = torch.zeros_like(b), b.shape[1]
    live = torch.ones_like(b[:, 0], dtype=torch.bool)
    mul = lambda v: (H @ v[..., None])[..., 0]  # noqa: E731
    factor = torch.linalg.cholesky(H)
    for _ in range(iters):
        hx = mul(x)
        cur, g = 0.5 * (x * hx).sum(1) + (x * b).sum(1), hx + b
        d = -torch.cholesky_solve(g[..., None], factor)[..., 0]
        live = live & ((g * d).sum(1) < 0)
        free = (x > 0) | ((x == 0) & (d > 0))
        p, s = torch.where(free, x, 0 * x), torch.where(free, d, 0 * d)
        at = torch.where((x > 0) & (d < 0), -x / d, torch.full_like(x, 2.0))
        at = torch.where((at > 0) & (at < 1), at, torch.full_like(x, 2.0))
        u, v = mul(p), mul(s)
        best, best_a, lo = cur, torch.zeros_like(cur), torch.zeros_like(cur)
        for _ in range(n + 1):
            to, j = at.min(1)
            hi = to.clamp_max(1)
            c0, c1, c2 = (p * (0.5 * u + b)).sum(1), (p * v).sum(1) + (b * s).sum(1), (s * v).sum(1)
            opt = torch.where(c2 > 0, torch.minimum(torch.maximum(-c1 / c2, lo), hi), 0.5 * (lo + hi))
            for a in (lo, hi, opt):
                c = c0 + c1 * a + 0.5 * c2 * a * a
                better = (hi - lo > 1e-7) & (c < best)
                best, best_a = torch.where(better, c, best), torch.where(better, a, best_a)
            if bool((to >= 2).all()):
                break
            on = (to < 2).to(F64)
            col = H.gather(1, j[:, None, None].expand(-1, 1, n))[:, 0] * on[:, None]
            j = j[:, None]
            u, v = u - p.gather(1, j) * col, v - s.gather(1, j) * col
            gone = torch.zeros_like(p).scatter(1, j, on[:, None]) > 0
            p, s = torch.where(gone, 0 * p, p), torch.where(gone, 0 * s, s)
            at, lo = torch.where(gone, torch.full_like(at, 2.0), at), torch.where(on > 0, hi, lo)
            # a system past its last window has lo = hi = 1 and takes no candidate
            lo = torch.where(on > 0, lo, torch.ones_like(lo))
        live = live & (best_a > 0) & (cur - best > 1e-7 * (1 + cur.abs()))
        x = torch.where(live[:, None], (x + best_a[:, None] * d).clamp_min(0), x)
        if not bool(live.any()):
            break
    return x


def exact(case, seed):
    """The outputs in 64 bits.  Free-body piles have none: fifty ordered Gauss-Seidel sweeps over
    every contact of every world, with box clipping, take minutes in plain numpy."""
    k = case["kind"]
    if k == "pile":
        return None
    _, lks, q, v, tau = _inputs(case, seed)

    def blocks():
        a = c = 0
        for lk in lks:
            W, free = len(lk), int(lk["joint"][0, 0]) == M.JOINT_FREE
            nq, nv = lk.shape[1] - 1 + 7 * free, lk.shape[1] - 1 + 6 * free
            yield lk, slice(a, a + W * nq), slice(c, c + W * nv), W
            a, c = a + W * nq, c + W * nv
    outs = []
    if k == "quad":
        for lk, a, c, W in blocks():
            outs.append(_exact_quads(lk, q[a].reshape(W, -1), v[c].reshape(W, -1), tau[c].reshape(W, -1), case["steps"],
                                     case["solver"] == "newton"))
    elif k == "serve":
        hs, us = tau
        for (lk, a, c, W), h, u in zip(blocks(), hs, us):
            T = _Tree(lk, 2e-3)
            s, w = T.read(_t(q[a].reshape(W, -1)), _t(v[c].reshape(W, -1)))
            u, h = _t(u), torch.as_tensor(h, device=_dev())
            for t in range(int(h.max())):
                s2, w2 = T.euler(s, w, u[:, t])
                go = (t < h)[:, None]
                s, w = (None, None, torch.where(go, s2[2], s[2])), torch.where(go, w2, w)
            outs.append(T.write(s, w))
        b = _inputs(case, seed)[0]
        order = np.random.default_rng([988, len(b)]).permutation(len(b))
        Q = np.concatenate([o[0].reshape(-1).cpu().numpy() for o in outs])
        V = np.concatenate([o[1].reshape(-1).cpu().numpy() for o in outs])
        return {"qpos": np.concatenate([Q[b.q_off[i]:b.q_off[i] + b.nq[i]] for i in order]),
                "qvel": np.concatenate([V[b.v_off[i]:b.v_off[i] + b.nv[i]] for i in order])}
    else:
        dt, rk4 = case.get("dt", 2e-3), case.get("rk4", False)
        for lk, a, c, W in blocks():
            outs.append(_exact_trees(lk, q[a].reshape(W, -1), v[c].reshape(W, -1), tau[c].reshape(W, -1), dt,
                                     case["steps"], rk4))
    Q, V = (np.concatenate([o[i].cpu().numpy() for o in outs]) for i in (0, 1))
    if k == "uneven":
        return {"chains": [Q, V], "piles": [None, None]}
    return {"qpos": Q, "qvel": V}
