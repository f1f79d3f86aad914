"""The batched pile launches' work counters (newt_gpu_pile_fused_profile):
contacts, dependency levels and their groups of eight contacts as counted here
from the contact lists, whatever lanes a world has."""
import numpy as np
import pytest

from test_gpu_pile_batched import SHAPES, spread, stack
from tooling_gb300 import api as A
from tooling_gb300 import model as M

pytestmark = pytest.mark.gpu


def _levels(pairs, depth):
    """Sizes of the levels: a contact's is one past the highest of the earlier active ones on its bodies."""
    last, sizes = {}, []
    for (a, b), d in zip(pairs.tolist(), depth):
        if d <= 0:
            continue
        v = max([last.get(g, 0) for g in (a, b) if g > 0] + [0])  # geom 0: the plane
        for g in (a, b):
            last[g] = v + 1
        if v == len(sizes):
            sizes.append(0)
        sizes[v] += 1
    return sizes


@pytest.mark.parametrize("lanes", [32, 16, 8])
def test_counters_are_those_of_the_contacts(lanes):
    rng = np.random.default_rng(31)
    worlds = [stack(rng, 3), stack(rng, 9), spread(rng, 17), spread(rng, 8), spread(rng, 40), spread(rng, 5, high=True)]
    eng = A.Engine()
    eng.set_launch_choice(persistent=True, persistent_shape=SHAPES[lanes])
    slots = eng.alloc(eng.upload(M.PackedModels([w for w, _ in worlds])))
    q = [np.array(x, np.float32) for _, x in worlds]
    v = [np.zeros(6 * len(w.bodies), np.float32) for w, _ in worlds]
    eng.set_state(slots, np.concatenate(q), np.concatenate(v))
    want = np.zeros(3, int)
    eng.step(1)
    for (w, _), s in zip(worlds, slots):
        pairs, data = eng.contacts(int(s))
        sizes = _levels(pairs, data[:, 6]) if len(pairs) else []
        want += [sum(sizes), w.iterations * sum((n + 7) // 8 for n in sizes), len(sizes)]
    got = eng.fused_profile()[1]
    eng.close()
    assert want.min() > 0
    assert [got["contacts"], got["rounds"], got["levels"]] == want.tolist() and got["worlds"] == len(worlds)
