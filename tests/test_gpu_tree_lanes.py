"""Trees without contact in the batched form (eight lanes per world, four
worlds per block; tree_lanes.cu) against the FP64 oracle, where its passes can
go wrong: the smallest and the largest trees and the sizes around its buckets,
world counts that leave a block part empty, branching trees, every joint type,
armature and damping, both roots, and both integrators in one block.

Tolerance: each world's step may be no further from FP64 than twice newt's own
f32 step (the oracle's float build), or 2e-6 of the world's largest value (16
roundings of 2^-23), whichever is larger."""
import numpy as np
import pytest

import oracle_py
from tooling_gb300 import api as A
from tooling_gb300 import model as M

pytestmark = pytest.mark.gpu


def tree(rng, n_links, free, branching, rk4, jointmix=True):
    w = M.WorldModel(dt=2e-3, integrator=M.INTEGRATOR_RK4 if rk4 else M.INTEGRATOR_EULER)
    for i in range(n_links):
        if i == 0:
            joint, parent = (M.JOINT_FREE if free else M.JOINT_FIXED), -1
        else:
            joint = int(rng.choice([M.JOINT_HINGE, M.JOINT_HINGE, M.JOINT_SLIDE, M.JOINT_FIXED])) if jointmix else M.JOINT_HINGE
            parent = int(rng.integers(max(0, i - 4), i)) if branching else i - 1
        ax = rng.normal(size=3)
        d = rng.uniform(0.02, 0.1, 3)
        w.push_link(M.Link(parent=parent, joint=joint, axis=ax / np.linalg.norm(ax) * rng.uniform(0.5, 2.0),
                           damping=rng.uniform(0, 0.2) if i else 0.0, armature=rng.uniform(0, 0.05) if i else 0.0,
                           free_damping=rng.uniform(0, 0.3) if free and i == 0 else 0.0,
                           jp_pos=rng.normal(0, 0.15, 3), jc_pos=rng.normal(0, 0.15, 3) if i else (0, 0, 0),
                           mass=rng.uniform(0.5, 2.0), inertia=M._diag9(*d)))
    return w


CASES = [(n, free, branching, worlds) for n, free, branching, worlds in
         [(1, True, False, 3), (2, False, False, 1), (2, True, False, 5), (7, False, True, 4), (8, True, True, 6),
          (9, False, False, 7), (16, True, False, 2), (17, True, True, 5), (32, False, True, 3), (33, True, False, 3),
          (64, False, False, 2), (64, True, True, 5), (65, False, False, 1)]]


@pytest.mark.parametrize("n,free,branching,worlds", CASES)
def test_tree_step_matches_fp64(n, free, branching, worlds):
    rng = np.random.default_rng([77, n, free, branching, worlds])
    # hinges only in the serial trees: there the links' own order is the path
    models = [tree(rng, n, free, False, w % 2 == 1, jointmix=False) for w in range(worlds)]
    if branching:  # one layout for the group, other parameters and integrators
        first = tree(rng, n, free, True, False)
        models = []
        for w in range(worlds):
            m = tree(rng, n, free, True, w % 3 == 2)
            for a, b in zip(m.links, first.links):
                a.parent, a.joint = b.parent, b.joint
            models.append(m)
    P = M.PackedModels(models)
    nq, nv = models[0].nq, models[0].nv
    if nv == 0:
        pytest.skip("no degrees of freedom")
    q = rng.uniform(-1.5, 1.5, (worlds, nq)).astype(np.float32)
    if free:
        quat = rng.normal(size=(worlds, 4))
        q[:, 3:7] = quat / np.linalg.norm(quat, axis=1, keepdims=True)
    v = rng.normal(0, 1, (worlds, nv)).astype(np.float32)
    tau = rng.normal(0, 0.5, (worlds, nv)).astype(np.float32)
    eng = A.Engine()
    slots = eng.alloc(eng.upload(P))
    eng.set_state(slots, q.reshape(-1), v.reshape(-1))
    eng.set_qfrc(slots, tau.reshape(-1))
    eng.step(2)
    gq, gv = eng.get_state(slots, nq * worlds, nv * worlds)
    assert not eng.status(slots).any()
    eng.close()
    gq, gv = gq.reshape(worlds, nq), gv.reshape(worlds, nv)
    for w in range(worlds):
        integ = 0 if models[w].integrator == M.INTEGRATOR_RK4 else 1
        run = lambda p: oracle_py.run(P, np.array([w]), q[w], v[w], tau[w], 2, precision=p, integrator=integ)
        (q32, v32), (q64, v64) = run(0), run(1)
        for got, f32, f64 in ((gq[w], q32, q64), (gv[w], v32, v64)):
            tol = max(2 * np.abs(f32 - f64).max(), 2e-6 * max(1.0, np.abs(f64).max()))
            assert np.abs(got - f64).max() <= tol
