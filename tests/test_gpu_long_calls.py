"""Calls of more env-steps than one graph holds: the same digits as the call in
parts, the work counters and the contacts of the whole call, lengths around
the graph's, and memory that does not grow with the length."""
import numpy as np
import pytest
import torch

from test_gpu_pile_batched import stack
from test_gpu_tc_small import crawler
from test_gpu_tree_lanes import tree
from tooling_gb300 import api as A
from tooling_gb300 import model as M

pytestmark = pytest.mark.gpu


def _load(eng):
    """Piles of two size classes, Newton piles, trees and trees in contact; (slots, nq, nv, the piles' slots)."""
    rng = np.random.default_rng(21)
    piles = [stack(rng, n) for n in (3, 3, 9, 2, 2, 12)]
    newton = [stack(rng, 2) for _ in range(3)]
    for m, _ in newton:
        m.solver, m.iterations = M.SOLVER_NEWTON, 20
    trees = [tree(rng, 6, free, False, rk4, jointmix=False) for free in (False, True) for rk4 in (False, True)]
    walkers = [crawler(rng, 12, 9, M.SOLVER_NEWTON, False, 3, 0.8) for _ in range(3)]
    models = [m for m, _ in piles + newton] + trees + walkers
    q = [np.array(x) for _, x in piles + newton]
    for m in trees:
        x = rng.uniform(-1, 1, m.nq)
        if m.links[0].joint == M.JOINT_FREE:
            x[3:7] /= np.linalg.norm(x[3:7])
        q.append(x)
    for m in walkers:
        x = rng.normal(0, 1e-3, m.nq)
        x[:7] = 0.0, 0.0, 0.0295, 1.0, 0.0, 0.0, 0.0
        q.append(x)
    slots = eng.alloc(eng.upload(M.PackedModels(models)))
    q = np.concatenate(q).astype(np.float32)
    v = np.concatenate([rng.normal(0, 0.05, m.nv) for m in models]).astype(np.float32)
    eng.set_state(slots, q, v)
    return slots, q.size, v.size, slots[:len(piles)]


def _read(eng, slots, nq, nv):
    q, v = eng.get_state(slots, nq, nv)
    found = [np.concatenate([x.reshape(-1).astype(np.float64) for x in eng.contacts(int(s))]) for s in slots]
    return [q, v, eng.get_qacc(slots, nv), eng.status(slots)] + found


@pytest.mark.parametrize("n", [127, 128, 129, 256, 257, 300])  # a graph holds 128 env-steps
def test_a_long_call_is_its_parts(n):
    parts = [100] * (n // 100) + [n % 100] * (n % 100 > 0)
    got, work = [], []
    for calls in ([n], parts):
        eng = A.Engine()
        slots, nq, nv, piles = _load(eng)
        counted = np.zeros(3)
        for k in calls:
            eng.step(k)
            w = eng.fused_profile()[1]
            counted += [w["contacts"], w["rounds"], w["levels"]]
            assert w["worlds"] == len(piles)
        got.append(_read(eng, slots, nq, nv))
        work.append(counted)
        eng.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b)
    assert np.array_equal(*work) and (work[0] > 0).all()


def test_alternating_lengths_keep_their_own_graphs():
    ref, eng = A.Engine(), A.Engine()
    slots, nq, nv, _ = _load(ref)
    other, _, _, _ = _load(eng)
    for k in (130, 2, 130, 258, 2, 1):  # pieces stay while ends change
        eng.step(k)
    for _ in range(523):
        ref.step(1)
    for a, b in zip(_read(ref, slots, nq, nv), _read(eng, other, nq, nv)):
        assert np.array_equal(a, b)
    # a model added in between: both graphs are captured again
    extra = [(e, e.alloc(e.upload(M.PackedModels([stack(np.random.default_rng(5), 4)[0]])))) for e in (ref, eng)]
    state = np.array(stack(np.random.default_rng(5), 4)[1], np.float32)
    for e, s in extra:
        e.set_state(s, state, np.zeros(24, np.float32))
    eng.step(140)
    for _ in range(140):
        ref.step(1)
    for (e, s), (f, t) in zip(extra[:1], extra[1:]):
        assert all(np.array_equal(a, b) for a, b in zip(e.get_state(s, 28, 24), f.get_state(t, 28, 24)))
    for a, b in zip(_read(ref, slots, nq, nv), _read(eng, other, nq, nv)):
        assert np.array_equal(a, b)
    ref.close()
    eng.close()


def test_a_call_takes_no_memory_for_its_length():
    """10000 env-steps of one pile in under 16 MB of the device (in one graph they took 50)."""
    m, q = stack(np.random.default_rng(2), 1)
    eng = A.Engine()
    slots = eng.alloc(eng.upload(M.PackedModels([m])))
    eng.set_state(slots, np.array(q, np.float32), np.zeros(6, np.float32))
    eng.step(200)
    eng.sync()
    free = torch.cuda.mem_get_info()[0]
    eng.step(10000)
    eng.sync()
    assert free - torch.cuda.mem_get_info()[0] < 16 << 20
    eng.close()
