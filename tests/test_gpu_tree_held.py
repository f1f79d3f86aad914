"""Trees that are held or freed cost the batched step next to nothing, and
their neighbours step as without them."""
import time

import numpy as np
import pytest

from test_gpu_tree_lanes import tree
from tooling_gb300 import api as A
from tooling_gb300 import model as M

pytestmark = pytest.mark.gpu


def _took(eng, steps):
    ts = []
    for _ in range(5):
        eng.sync()
        t = time.perf_counter()
        eng.step(steps)
        eng.sync()
        ts.append(time.perf_counter() - t)
    return min(ts)


def test_worlds_that_are_not_stepped_cost_nothing():
    """12000 chains of 25 links, 20 env-steps: with none of them to step under a quarter of the time of all."""
    m = tree(np.random.default_rng(3), 25, False, False, False, jointmix=False)
    eng = A.Engine()
    slots = eng.alloc(np.repeat(eng.upload(M.PackedModels([m])), 12000))
    live = _took(eng, 20)
    eng.hold(slots[:6000])
    eng.free(slots[6000:])
    assert _took(eng, 20) < 0.25 * live
    eng.close()


def test_worlds_beside_held_ones_step_the_same():
    rng = np.random.default_rng(4)
    m, n = tree(rng, 12, True, False, True, jointmix=False), 23
    q, v = rng.uniform(-1, 1, (n, m.nq)).astype(np.float32), rng.normal(0, 1, (n, m.nv)).astype(np.float32)
    q[:, 3:7] /= np.linalg.norm(q[:, 3:7], axis=1, keepdims=True)
    held = np.array([1, 4, 5, 6, 7, 10, 16, 17, 18, 19, 22])  # parts of blocks of four, and two whole ones
    out = []
    for hold in (False, True):
        eng = A.Engine()
        slots = eng.alloc(np.repeat(eng.upload(M.PackedModels([m])), n))
        eng.set_state(slots, q.reshape(-1), v.reshape(-1))
        was = eng.get_state(slots, q.size, v.size)
        if hold:
            eng.hold(slots[held])
        eng.step(3)
        out.append([x.reshape(n, -1) for x in eng.get_state(slots, q.size, v.size)])
        eng.close()
    rest = np.setdiff1d(np.arange(n), held)
    for a, b, w in zip(out[0], out[1], was):
        assert np.array_equal(a[rest], b[rest]) and np.array_equal(b[held], w.reshape(n, -1)[held])
