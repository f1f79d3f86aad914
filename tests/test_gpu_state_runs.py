"""State and forces in and out by runs of worlds (world_io.cu): one run and
many, tiles that are not full, more runs than a launch's parameters hold,
interleaved groups of trees and piles, page-locked and ordinary arrays, and
slots named twice.  What goes in comes out: coordinates and rates of fixed
bases bit for bit, quaternions and the free roots' rotated velocities to 4e-7
of their largest value (four roundings of 2^-23)."""
import numpy as np
import pytest
import torch

from tooling_gb300 import Engine, NewtError
from tooling_gb300 import model as M
from test_gpu_pile_batched import spread
from test_gpu_tree_lanes import tree

pytestmark = pytest.mark.gpu


def _state(rng, m):
    q, v = rng.normal(size=m.nq), rng.normal(size=m.nv)
    free = [7 * i for i in range(len(m.bodies))] if m.bodies else [0] if m.links[0].joint == M.JOINT_FREE else []
    for o in free:
        q[o + 3:o + 7] /= np.linalg.norm(q[o + 3:o + 7])
    return q, v


def _host(a, pinned):
    return torch.from_numpy(a.copy()).pin_memory().numpy() if pinned else a.copy()


@pytest.mark.parametrize("pinned", [True, False])
@pytest.mark.parametrize("worlds,order", [(1, "as is"), (32, "as is"), (33, "as is"), (70, "by two"), (400, "shuffled")])
def test_what_goes_in_comes_out(worlds, order, pinned):
    rng = np.random.default_rng([9, worlds])
    kinds = [tree(rng, 5, False, False, False, jointmix=False), tree(rng, 12, True, False, False, jointmix=False),
             spread(rng, 3)[0], spread(rng, 40)[0], tree(rng, 65, False, False, False, jointmix=False)]
    models = [kinds[w % len(kinds)] for w in range(worlds)]
    P = M.PackedModels(kinds)
    eng = Engine()
    ids = eng.upload(P)
    slots = eng.alloc([ids[w % len(kinds)] for w in range(worlds)])
    perm = {"as is": np.arange(worlds), "by two": np.concatenate([np.arange(0, worlds, 2), np.arange(1, worlds, 2)]),
            "shuffled": rng.permutation(worlds)}[order]
    x = [_state(rng, m) for m in models]
    q = _host(np.concatenate([x[i][0] for i in perm]).astype(np.float32), pinned)
    v = _host(np.concatenate([x[i][1] for i in perm]).astype(np.float32), pinned)
    eng.set_state(slots[perm], q, v)
    out = _host(np.zeros_like(q), pinned), _host(np.zeros_like(v), pinned)
    gq, gv = eng.get_state(slots[perm], q.size, v.size, out=out)
    a = b = 0
    for i in perm:
        m = models[i]
        for got, ref in ((gq[a:a + m.nq], q[a:a + m.nq]), (gv[b:b + m.nv], v[b:b + m.nv])):
            if m.bodies or m.links[0].joint == M.JOINT_FREE:
                assert np.abs(got - ref).max() <= 4e-7 * np.abs(ref).max()
            else:
                assert np.array_equal(got, ref)
        a, b = a + m.nq, b + m.nv
    # one world at a time, in the slots' order: the same values
    a = b = 0
    for i in perm[:40]:
        m = models[i]
        oq, ov = eng.get_state(slots[i:i + 1], m.nq, m.nv)
        assert np.array_equal(oq, gq[a:a + m.nq]) and np.array_equal(ov, gv[b:b + m.nv])
        a, b = a + m.nq, b + m.nv
    eng.close()


def test_forces_reach_their_worlds_and_the_last_of_two_stays():
    rng = np.random.default_rng(10)
    m, n = tree(rng, 6, False, False, False, jointmix=False), 150
    pile = spread(rng, 2)[0]
    eng = Engine()
    ids = eng.upload(M.PackedModels([m, pile]))
    kinds = np.arange(n) % 3 == 2  # a pile after every two trees
    slots = eng.alloc([ids[int(k)] for k in kinds])
    nv = np.where(kinds, pile.nv, m.nv)
    tau = [rng.normal(size=k).astype(np.float32) for k in nv]
    st = [_state(rng, pile if k else m) for k in kinds]
    q, v = (np.concatenate([s[j] for s in st]).astype(np.float32) for j in (0, 1))

    def step(order):
        eng.set_state(slots, q, v)
        eng.set_qfrc(slots, np.zeros(nv.sum(), np.float32))
        eng.set_qfrc(slots[order], np.concatenate([tau[i] if k >= len(order) - n else 9 + tau[i] for k, i in enumerate(order)]))
        eng.step(1)
        return eng.get_state(slots, q.size, v.size)

    ref = step(np.arange(n))
    for order in (rng.permutation(n), np.concatenate([rng.permutation(n)[:40], rng.permutation(n)])):
        got = step(order)
        assert np.array_equal(ref[0], got[0]) and np.array_equal(ref[1], got[1])
    with pytest.raises(NewtError):
        eng.set_state(np.array([slots[0], slots[0]]), np.zeros(2 * m.nq, np.float32), np.zeros(2 * m.nv, np.float32))
    eng.free(slots[:1])
    for call in (lambda: eng.set_state(slots[:1], q[:m.nq], v[:m.nv]), lambda: eng.get_state(slots[:1], m.nq, m.nv),
                 lambda: eng.set_qfrc(slots[:1], tau[0])):
        with pytest.raises(NewtError):
            call()
    eng.close()
