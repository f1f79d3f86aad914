"""Tree-contact worlds of more than 32 rows beside smaller ones (tc_k_small's
own general solve where a world has a block to itself, tc_k_listed where
worlds share blocks): the FP64 oracle's step within the bars of
test_gpu_tc_small.py from both, and the same digits whatever the neighbours."""
import time

import numpy as np
import pytest

import oracle_py
from test_gpu_tc_small import crawler
from tooling_gb300 import api as A
from tooling_gb300 import model as M

pytestmark = pytest.mark.gpu
JOINTS, WORLDS = 14, 24


def _worlds(solver):
    """`WORLDS` worlds of 4, 28, 32, 36 and 56 rows and without contact, one layout."""
    out = []
    for w in range(WORLDS):
        rng = np.random.default_rng([41, w])
        m = crawler(rng, JOINTS, 14, solver, False, 3, 0.8)
        feet = [1, 7, 8, 9, 14, 0][w % 6]
        for g in m.geoms:  # spheres of the links past the feet shrink off the plane
            if g.link >= feet:
                g.size = (1e-3, 0.0, 0.0)
        out.append(m)
    nq, nv = out[0].nq, out[0].nv
    q = np.zeros((WORLDS, nq), np.float32)
    rng = np.random.default_rng(42)
    q[:, 2], q[:, 3] = 0.0295, 1.0
    q[:, 7:] = rng.normal(0, 1e-3, (WORLDS, nq - 7))
    return M.PackedModels(out), q, rng.normal(0, 0.1, (WORLDS, nv)).astype(np.float32)


def _step(P, q, v, copies):
    eng = A.Engine()
    n, nq, nv = len(q), q.shape[1], v.shape[1]
    slots = eng.alloc(np.tile(eng.upload(P), copies))
    eng.set_state(slots, np.tile(q, (copies, 1)).reshape(-1), np.tile(v, (copies, 1)).reshape(-1))
    eng.step(1)
    gq, gv = eng.get_state(slots, copies * q.size, copies * v.size)
    rows = [4 * int((eng.contacts(int(s))[1][:, 6] > 0).sum()) for s in slots[:n]]
    assert not (eng.status(slots) & 0x3).any()
    eng.close()
    return gq.reshape(copies, n, nq), gv.reshape(copies, n, nv), rows


@pytest.mark.parametrize("solver", [M.SOLVER_NEWTON, M.SOLVER_PGS])
def test_large_worlds_beside_small_ones(solver):
    P, q, v = _worlds(solver)
    gq, gv, rows = _step(P, q, v, 1)
    assert {0, 32} <= set(rows) and 36 in rows and max(rows) == 56
    for w in range(WORLDS):
        run = lambda p: oracle_py.run(P, np.array([w]), q[w], v[w], None, 1, precision=p)
        (q32, v32), (q64, v64) = run(0), run(1)
        tol = max(2 * np.abs(v32 - v64).max(), 1e-4 * np.abs(v64 - v[w]).max())
        assert np.abs(gv[0, w] - v64).max() <= tol, w
        assert np.abs(gq[0, w] - q64).max() <= max(2 * np.abs(q32 - q64).max(), 2e-3 * tol, 2e-7), w
    # more than eight worlds an SM: blocks of four and the list; more than 64: a part of them in the blocks
    for per_sm in (8, 64):
        hq, hv, _ = _step(P, q, v, per_sm * 192 // WORLDS + 1)
        assert (hq == gq[0]).all() and (hv == gv[0]).all()


def test_a_large_world_does_not_hold_up_its_neighbours():
    """6000 worlds, a quarter of them with 56 rows, take less than 0.55 of the time that 56 rows everywhere take
    (a quarter of it and the small worlds'; all of it where a block's small worlds wait for its large one)."""
    P, q, v = _worlds(M.SOLVER_NEWTON)
    took = []
    for pick in ([4] * 4, [4, 0, 5, 0]):
        eng = A.Engine()
        slots = eng.alloc(np.tile(eng.upload(P)[pick], 1500))
        Q, V = np.tile(q[pick], (1500, 1)).reshape(-1), np.tile(v[pick], (1500, 1)).reshape(-1)
        ts = []
        for _ in range(5):
            eng.set_state(slots, Q, V)
            eng.sync()
            t = time.perf_counter()
            eng.step(1)
            eng.sync()
            ts.append(time.perf_counter() - t)
        took.append(min(ts))
        eng.close()
    assert took[1] < 0.55 * took[0]
