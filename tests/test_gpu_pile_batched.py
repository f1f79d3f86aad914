"""The batched pile step (pile_batched.cu) against the FP64 oracle where its
launches can go wrong: worlds at the edges of the size classes, stacks with
more rounds than the sweeps' schedule holds and with rows past their shared
memory, worlds without contacts, bodies whose inverse inertia is not diagonal,
different iteration counts in one block, and every number of lanes per world.

Tolerance: a world's step may be no further from FP64 than twice newt's own
f32 step (the oracle's float build), or 4e-6 of the world's largest value (32
roundings of 2^-23), whichever is larger.  Depths are at least 1e-4 m, so that
no contact is at the edge of being active."""
import numpy as np
import pytest

import oracle_py
from tooling_gb300 import api as A
from tooling_gb300 import model as M

pytestmark = pytest.mark.gpu


def _inertia(rng, mass, general):
    d = mass * rng.uniform(0.002, 0.01, 3)
    if not general:
        return M._diag9(*[float(x) for x in d])
    Q, _ = np.linalg.qr(rng.normal(size=(3, 3)))
    return [float(x) for x in (Q * d @ Q.T).T.reshape(-1)]


def stack(rng, n, general=False):
    """n boxes one on another, each pair a little apart sideways."""
    w = M.WorldModel(dt=2e-3, iterations=int(rng.integers(20, 60)))
    w.add_geom(M.static_plane())
    q, z = [], 0.0
    for i in range(n):
        h = rng.uniform(0.06, 0.12, 3)
        mass = float(rng.uniform(0.5, 3.0))
        b = w.add_body(mass, _inertia(rng, mass, general))
        w.add_geom(M.Geom(shape=M.SHAPE_BOX, body=b, size=tuple(float(x) for x in h), friction=float(rng.uniform(0.3, 1.0))))
        z += float(h[2]) - rng.uniform(2e-4, 6e-4)
        yaw = rng.uniform(-0.3, 0.3)
        q += [*rng.uniform(-0.01, 0.01, 2), z, np.cos(yaw / 2), *rng.normal(0, 3e-4, 2), np.sin(yaw / 2)]
        z += float(h[2])
    return w, q


def spread(rng, n, general=False, high=False):
    """n spheres on a grid, touching the ground (or none of them: high)."""
    w = M.WorldModel(dt=2e-3, iterations=int(rng.integers(20, 60)))
    w.add_geom(M.static_plane())
    q = []
    for i in range(n):
        r = float(rng.uniform(0.1, 0.14))
        mass = float(rng.uniform(0.5, 3.0))
        b = w.add_body(mass, _inertia(rng, mass, general))
        w.add_geom(M.Geom(shape=M.SHAPE_SPHERE, body=b, size=(r, 0, 0), friction=float(rng.uniform(0.3, 1.0))))
        u = rng.normal(size=4)
        q += [0.2 * (i % 8) + rng.uniform(-0.01, 0.01), 0.2 * (i // 8) + rng.uniform(-0.01, 0.01),
              r + (1.0 if high else -rng.uniform(2e-4, 1e-3)), *(u / np.linalg.norm(u))]
    return w, q


SHAPES = {32: 0, 16: 1, 8: 2}


@pytest.mark.parametrize("lanes", [32, 16, 8])
@pytest.mark.parametrize("n", [1, 8, 9, 20, 21, 63, pytest.param(64, marks=pytest.mark.xfail(strict=True, reason=(
    "the broadphase sorts 64 geoms: beside a plane, the last body of a 64-body world meets no other body in any form")))])
def test_spread_worlds_match_fp64(n, lanes):
    rng = np.random.default_rng([5, n])
    _check([spread(rng, n, general=w % 2 == 1, high=w == 3) for w in range(7)], lanes)


@pytest.mark.parametrize("lanes", [32, 16, 8])
@pytest.mark.parametrize("n", [3, 12, 20])
def test_stacks_match_fp64(n, lanes):
    rng = np.random.default_rng([6, n])
    _check([stack(rng, n, general=w % 2 == 1) for w in range(5)], lanes)


def _check(worlds, lanes):
    P = M.PackedModels([w for w, _ in worlds])
    nb = len(worlds[0][0].bodies)
    rng = np.random.default_rng(9)
    q = np.array([x for _, x in worlds], np.float32).reshape(len(worlds), 7 * nb)
    for k in range(nb):
        q[:, 7 * k + 3:7 * k + 7] /= np.linalg.norm(q[:, 7 * k + 3:7 * k + 7], axis=1, keepdims=True)
    v = rng.normal(0, 0.1, (len(worlds), 6 * nb)).astype(np.float32)
    eng = A.Engine()
    eng.set_launch_choice(persistent=True, persistent_shape=SHAPES[lanes])
    slots = eng.alloc(eng.upload(P))
    eng.set_state(slots, q.reshape(-1), v.reshape(-1))
    eng.step(1)
    gq, gv = eng.get_state(slots, q.size, v.size)
    assert not eng.status(slots).any()
    imps = [eng.impulses(int(s)) for s in slots]
    eng.close()
    gq, gv = gq.reshape(q.shape), gv.reshape(v.shape)
    for w in range(len(worlds)):
        run = lambda p: oracle_py.run(P, np.array([w]), q[w], v[w], None, 1, precision=p)
        (q32, v32), (q64, v64) = run(0), run(1)
        i32, i64 = (oracle_py.impulses(P, w, q[w], v[w], precision=p) for p in (0, 1))
        _, d = oracle_py.contacts(P, w, q[w], v[w])
        assert len(d) == 0 or np.abs(d[:, 6]).min() > 1e-5
        got = imps[w].reshape(-1, 4)[d[:, 6] > 0].reshape(-1) if len(d) else imps[w][:0]
        assert len(got) == len(i64)
        for x, f32, f64 in ((gq[w], q32, q64), (gv[w], v32, v64), (got, i32, i64)):
            if len(f64):
                tol = max(2 * np.abs(f32 - f64).max(), 4e-6 * max(1.0, np.abs(f64).max()))
                assert np.abs(x - f64).max() <= tol
