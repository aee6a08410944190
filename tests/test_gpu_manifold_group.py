"""Box pairs by eight lanes and by one thread: the oracle's slots for cubes and
boxes at every kind of axis, face and edge contacts, aligned and coincident
ones, 4 and 8 contacts a pair, and counts on both sides of the line."""
import numpy as np
import pytest

import oracle_lib as O
from diomedes_gb300 import abi, compute, physics as ph

pytestmark = pytest.mark.gpu


def _boxes(n, seed):
    rng = np.random.default_rng(seed)
    items = []
    for k in range(n):
        p = rng.uniform(-1.2, 1.2, 3)
        if k % 5 == 0:
            p = np.round(p)  # aligned: equal overlaps, shared faces
        q = rng.normal(size=4) if k % 5 else np.array([0.0, 0.0, 0.0, 1.0])
        if k % 7 == 0:
            q = np.array([0.0, 0.70710677, 0.0, 0.70710677])
        q = tuple(q / np.linalg.norm(q))
        if k % 2:
            items.append(ph.cube(tuple(p), 0.5, 1.0, orientation=q))
        else:
            items.append(ph.box(tuple(p), tuple(rng.uniform(0.2, 0.9, 3)), 1.0, orientation=q))
    items.append(ph.cube((0.0, 0.0, 0.0), 0.5, 1.0))
    items.append(ph.cube((0.0, 0.0, 0.0), 0.5, 1.0))  # coincident with the last
    items.append(ph.sphere((0.0, 0.0, 0.0), 0.4, 1.0))
    items.append(ph.sphere((0.3, 0.0, 0.0), 0.4, 1.0))
    return ph.pack_bodies(items)[0]


@pytest.mark.parametrize("per_pair", [4, 8])
@pytest.mark.parametrize("count", [1, 3, 16, 17, 1900, 65535, 65536, 65537])
def test_slots_match_oracle(count, per_pair):
    b = _boxes(60, per_pair)
    pairs, _ = O.broad(b)
    want = O.narrow(b, pairs, per_pair=per_pair)
    valid = (want["valid"] != 0).reshape(-1, per_pair).sum(1)
    assert len(pairs) > 500 and (valid == 0).any() and (valid == 1).any() and (valid >= 4).any()
    pick = (np.arange(count) * 7919) % len(pairs)
    with compute.NarrowPhaseCompute(len(b), count) as npc:
        npc.configure(contacts_per_pair=per_pair)
        npc.submit(b, pairs[pick])
        got = npc.read(per_pair)
    want = want.reshape(len(pairs), per_pair)[pick].reshape(-1)
    assert np.array_equal(got.view(np.uint8), want.view(np.uint8))
