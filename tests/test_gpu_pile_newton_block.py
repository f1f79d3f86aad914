"""The free-body Newton solve by a block per world (pile_newton.cu) against
the FP64 oracle where it can go wrong: one contact's rows, worlds of every
size of block (up to 32, 128 and 224 rows) and past the largest in one call, worlds without contact beside others, and RK4.

Bars (those of the free-body Newton tests): no further from FP64 than twice
newt's own f32 step (the oracle's float build), or 1e-4 m/s and 2e-6 m where
newt's is closer."""
import numpy as np
import pytest

import oracle_py
from test_gpu_pile_batched import spread, stack
from tooling_gb300 import api as A
from tooling_gb300 import model as M

pytestmark = pytest.mark.gpu


def _check(worlds, iterations=20, rk4=False):
    for m, _ in worlds:
        m.solver, m.iterations = M.SOLVER_NEWTON, iterations
        m.integrator = M.INTEGRATOR_RK4 if rk4 else M.INTEGRATOR_EULER
    P = M.PackedModels([m for m, _ in worlds])
    q = [np.array(x, np.float32) for _, x in worlds]
    rng = np.random.default_rng(11)
    v = [rng.normal(0, 0.05, 6 * len(m.bodies)).astype(np.float32) for m, _ in worlds]
    eng = A.Engine()
    slots = eng.alloc(eng.upload(P))
    eng.set_state(slots, np.concatenate(q), np.concatenate(v))
    eng.step(1)
    gq, gv = eng.get_state(slots, sum(map(len, q)), sum(map(len, v)))
    assert not (eng.status(slots) & 0x3).any()
    a = b = contacts = 0
    for w in range(len(worlds)):
        pairs, data = oracle_py.contacts(P, w, q[w], v[w])
        got, _ = eng.contacts(int(slots[w]))
        assert np.array_equal(got, pairs)
        contacts += len(pairs)
        run = lambda p: oracle_py.run(P, np.array([w]), q[w], v[w], None, 1, precision=p, integrator=0 if rk4 else 1)
        (q32, v32), (q64, v64) = run(0), run(1)
        wq, wv = gq[a:a + len(q[w])], gv[b:b + len(v[w])]
        a, b = a + len(q[w]), b + len(v[w])
        assert np.abs(wv - v64).max() <= max(2 * np.abs(v32 - v64).max(), 1e-4), w
        assert np.abs(wq - q64).max() <= max(2 * np.abs(q32 - q64).max(), 2e-6), w
    assert contacts
    eng.close()


@pytest.mark.parametrize("n", [1, 8, 9, 20, 32, 33])  # four rows a sphere
def test_spread_worlds_match_fp64(n):
    rng = np.random.default_rng([6, n])
    _check([spread(rng, n, general=w % 2 == 1, high=w == 3) for w in range(5)])


@pytest.mark.parametrize("n,rk4", [(2, False), (3, True), (8, False), (9, False)])  # sixteen rows a box
def test_stacks_match_fp64(n, rk4):
    rng = np.random.default_rng([7, n])
    _check([stack(rng, n, general=w % 2 == 1) for w in range(4)], rk4=rk4)


def test_more_worlds_than_one_wave_match_fp64():
    """Past three worlds an SM the smallest take their own launch."""
    rng = np.random.default_rng(9)
    _check([spread(rng, (1, 2, 6, 9)[w % 4], general=w % 2 == 1, high=w % 16 == 15) for w in range(480)])
