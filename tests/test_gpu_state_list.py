"""Worlds named in no order (world_io.cu, state_move_list): more runs than a
call moves as runs, the same values one world at a time, one launch however
often a slot is named, and none where no named world carries a force."""
import numpy as np
import pytest

from test_gpu_pile_batched import spread
from test_gpu_state_runs import _host, _state
from test_gpu_tree_lanes import tree
from tooling_gb300 import Engine
from tooling_gb300 import model as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pinned", [True, False])
@pytest.mark.parametrize("run", [1, 7, 8, 9])  # lists below eight worlds a run on average
def test_listed_worlds_keep_their_values(run, pinned):
    rng = np.random.default_rng([11, run])
    n = 130 * run + 3
    kinds = [tree(rng, 9, False, False, False, jointmix=False), spread(rng, 33)[0]]
    eng = Engine()
    ids = eng.upload(M.PackedModels(kinds))
    k = np.arange(n) // run % 2
    slots = eng.alloc(ids[k])
    order = np.concatenate([np.arange(a, min(a + run, n)) for a in rng.permutation(np.arange(0, n, run))])
    x = [_state(rng, kinds[k[i]]) for i in order]
    q, v = (_host(np.concatenate([s[j] for s in x]).astype(np.float32), pinned) for j in (0, 1))
    before = eng.launch_count()
    eng.set_state(slots[order], q, v)
    assert eng.launch_count() == before + 1
    gq, gv = eng.get_state(slots[order], q.size, v.size, out=(_host(0 * q, pinned), _host(0 * v, pinned)))
    assert np.abs(gq - q).max() <= 4e-7 * np.abs(q).max() and np.array_equal(gv, v)
    a = b = 0
    for i in order[:60]:
        m = kinds[k[i]]
        oq, ov = eng.get_state(slots[i:i + 1], m.nq, m.nv)
        assert np.array_equal(oq, gq[a:a + m.nq]) and np.array_equal(ov, gv[b:b + m.nv])
        a, b = a + m.nq, b + m.nv
    eng.close()


def test_a_slot_named_again_costs_no_launch_and_keeps_the_last_forces():
    rng = np.random.default_rng(12)
    m, n = tree(rng, 6, False, False, False, jointmix=False), 300
    eng = Engine()
    slots = eng.alloc(np.repeat(eng.upload(M.PackedModels([m])), n))
    st = [_state(rng, m) for _ in range(n)]
    q, v = (np.concatenate([s[j] for s in st]).astype(np.float32) for j in (0, 1))
    tau = rng.normal(size=(n, m.nv)).astype(np.float32)

    def step(order, values):
        eng.set_state(slots, q, v)
        before = eng.launch_count()
        eng.set_qfrc(slots[order], values.reshape(-1))
        assert eng.launch_count() == before + 1
        eng.step(1)
        return eng.get_state(slots, q.size, v.size)

    ref = step(np.arange(n), tau)
    a, b = rng.permutation(n), rng.permutation(n)
    got = step(np.concatenate([a, b]), np.concatenate([tau[a] + 9, tau[b]]))
    assert np.array_equal(ref[0], got[0]) and np.array_equal(ref[1], got[1])
    eng.close()


def test_forces_of_free_bodies_move_nothing():
    rng = np.random.default_rng(13)
    pile, chain = spread(rng, 4)[0], tree(rng, 4, False, False, False, jointmix=False)
    eng = Engine()
    ids = eng.upload(M.PackedModels([pile, chain]))
    slots = eng.alloc(ids[[0, 0, 1, 0]])
    before = eng.launch_count()
    eng.set_qfrc(slots[[0, 1, 3]], np.ones(3 * pile.nv, np.float32))
    assert eng.launch_count() == before
    eng.set_qfrc(slots, np.ones(3 * pile.nv + chain.nv, np.float32))
    assert eng.launch_count() == before + 1
    eng.close()
