"""Many of the smallest trees in the batched form (tree_lanes.cu): the digits
of the same worlds alone, the FP64 oracle's step within the bars of
test_gpu_tree_lanes.py, blocks that are not full, held worlds, both
integrators and both roots in one call, and larger trees beside them."""
import numpy as np
import pytest
import torch

import oracle_py
from test_gpu_tree_lanes import tree
from tooling_gb300 import api as A
from tooling_gb300 import model as M

pytestmark = pytest.mark.gpu


def _states(rng, m, n):
    q, v = rng.uniform(-1.5, 1.5, (n, m.nq)), rng.normal(0, 1, (n, m.nv))
    if m.links[0].joint == M.JOINT_FREE:
        q[:, 3:7] /= np.linalg.norm(q[:, 3:7], axis=1, keepdims=True)
    return q.astype(np.float32), v.astype(np.float32), rng.normal(0, 0.5, (n, m.nv)).astype(np.float32)


@pytest.mark.parametrize("links", [2, 3, 4])
def test_many_small_trees_match_fp64(links):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng([51, links])
    # four kinds: both roots, both integrators; a third with a slide
    kinds = [tree(rng, links, free, links == 4, rk4, jointmix=False) for free in (False, True) for rk4 in (False, True)]
    for m in kinds[1:3]:
        m.links[1].joint = M.JOINT_SLIDE
    large = tree(rng, 9, False, False, False, jointmix=False)
    W = 120 * sms + 45  # more than a wave
    eng = A.Engine()
    P = M.PackedModels(kinds + [large])
    ids = eng.upload(P)
    k = np.arange(W) % 4
    slots = eng.alloc(ids[k])
    beside = eng.alloc(ids[4:])
    st = [_states(rng, m, 3) for m in kinds]  # three states a kind, repeated over its worlds
    pick = lambda j: np.concatenate([st[a][j][b] for a, b in zip(k, np.arange(W) // 4 % 3)])
    eng.set_state(slots, pick(0), pick(1))
    eng.set_qfrc(slots, pick(2))
    lq, lv, _ = _states(rng, large, 1)
    eng.set_state(beside, lq.reshape(-1), lv.reshape(-1))
    held = slots[5::97]
    eng.hold(held)
    nq, nv = sum(kinds[a].nq for a in k), sum(kinds[a].nv for a in k)
    before = eng.get_state(slots, nq, nv)
    eng.step(2)
    q, v = eng.get_state(slots, nq, nv)
    assert not eng.status(slots).any()
    oq, ov = eng.get_state(beside, large.nq, large.nv)
    acc = eng.get_qacc(slots[:12], 3 * sum(m.nv for m in kinds))
    eng.close()
    # the first of them alone
    eng = A.Engine()
    few = eng.alloc(eng.upload(P)[k[:12]])
    n, m = 3 * sum(x.nq for x in kinds), 3 * sum(x.nv for x in kinds)
    eng.set_state(few, pick(0)[:n], pick(1)[:m])
    eng.set_qfrc(few, pick(2)[:m])
    eng.hold(few[5:6])  # as among the many
    eng.step(2)
    alone = eng.get_state(few, n, m) + (eng.get_qacc(few, m),)
    eng.close()
    assert np.array_equal(alone[0], q[:n]) and np.array_equal(alone[1], v[:m]) and np.array_equal(alone[2], acc)
    ref = {}
    for a, m in enumerate(kinds):
        for b in range(3):
            x, y, tau = (st[a][j][b] for j in range(3))
            run = lambda p: oracle_py.run(P, np.array([a]), x, y, tau, 2, precision=p, integrator=0 if m.integrator == M.INTEGRATOR_RK4 else 1)
            ref[a, b] = run(0) + run(1)
    seen = set()
    i = j = 0
    still = set(held.tolist())
    for w in range(W):
        a, b = k[w], w // 4 % 3
        m = kinds[a]
        got, was = ((x[i:i + m.nq], y[j:j + m.nv]) for x, y in ((q, v), before))
        i, j = i + m.nq, j + m.nv
        q32, v32, q64, v64 = ref[a, b]
        if int(slots[w]) in still:
            assert np.array_equal(got[0], was[0]) and np.array_equal(got[1], was[1])
            continue
        key = (a, b) + tuple(g.tobytes() for g in got)
        if key in seen:  # the same digits as a world that was compared
            continue
        seen.add(key)
        for g, f32, f64 in ((got[0], q32, q64), (got[1], v32, v64)):
            assert np.abs(g - f64).max() <= max(2 * np.abs(f32 - f64).max(), 2e-6 * max(1.0, np.abs(f64).max()))
    assert len(seen) == 12
    r32, r64 = (oracle_py.run(P, np.array([4]), lq[0], lv[0], None, 2, precision=p) for p in (0, 1))
    for g, f32, f64 in ((oq, r32[0], r64[0]), (ov, r32[1], r64[1])):
        assert np.abs(g - f64).max() <= max(2 * np.abs(f32 - f64).max(), 2e-6 * max(1.0, np.abs(f64).max()))
    assert np.isfinite(acc).all() and np.abs(acc).max() > 0
