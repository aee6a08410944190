"""GJK with eight lanes a pair and with one (as many pairs as fill the grid),
EPA with pairs taken as warps become free: the oracle's slots at the line
between the two, and the same slots for every copy of a pair."""
import numpy as np
import pytest

import oracle_lib as O
from diomedes_gb300 import abi, compute, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 7, 8, 33, 9727, 9728, 9729, 20000])
def test_copies_of_pairs_match_oracle(count):
    sc = scenes.mixed_pile(n=300, extent=5.0)
    pairs, _ = O.broad(sc.bodies, hull=sc.hull_vertices)
    tags = sc.bodies["shape"]["tag"]
    both = tags[pairs["a"]], tags[pairs["b"]]
    pairs = pairs[(both[0] != both[1]) | (both[0] == abi.HULL)]  # neither both spheres nor both cubes
    want = O.narrow(sc.bodies, pairs, hull=sc.hull_vertices)
    assert len(pairs) > 50 and want["valid"].any()
    pick = np.arange(count) % len(pairs)
    with compute.NarrowPhaseCompute(sc.n, count, max_hull_vertices=len(sc.hull_vertices)) as npc:
        npc.set_hull_vertices(sc.hull_vertices)
        got = npc.run(sc.bodies, pairs[pick])
    want = np.asarray(want).reshape(len(pairs), -1)[pick].reshape(-1)
    assert np.array_equal(got.view(np.uint8), want.view(np.uint8))
