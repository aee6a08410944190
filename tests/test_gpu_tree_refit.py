"""The global trees' refit, which unites a CTA's 256 leaves in shared memory
and the levels above through L2, and the walk over nodes that name their two
children in one word: scenes whose ranges start and end off the CTAs' edges,
equal Morton codes (deep trees), and counts on both sides of the line between
split and whole walks."""
import numpy as np
import pytest

import oracle_lib as O
from diomedes_gb300 import abi, compute, physics as ph, scenes

pytestmark = pytest.mark.gpu


def _field(n, seed, coincident=0):
    """n bodies on a loose grid, the first `coincident` of them at one centre."""
    rng = np.random.default_rng(seed)
    side = int(np.ceil(n ** (1.0 / 3.0)))
    items = []
    for k in range(n):
        p = np.array([k % side, (k // side) % side, k // (side * side)]) * 1.3 + rng.uniform(-0.2, 0.2, 3)
        if k < coincident:
            p = np.zeros(3)
        r = 0.02 if k < coincident else 0.5
        items.append(ph.sphere(tuple(p), r, 1.0) if k % 2 else ph.cube(tuple(p), r, 1.0))
    b, s = ph.pack_bodies(items)
    return scenes.Scene(f"field{n}", b, s, containers=[scenes.ground()], options=ph.avbd_options(iterations=2))


@pytest.mark.parametrize("precision,sizes", [(abi.PREC_F32, (3, 2049, 255, 2304, 1)),
                                             (abi.PREC_F32, (2303, 2561)),
                                             (abi.PREC_F64, (7, 1025, 1279, 1024, 1281)),
                                             (abi.PREC_SPLIT, (2, 2050, 1))])
def test_scenes_off_the_refit_edges_match_oracle(precision, sizes):
    packed = scenes.pack([_field(n, i, coincident=20 if n > 2000 else 0) for i, n in enumerate(sizes)])
    ow = O.World(packed, precision=precision)
    ow.step(packed.options, 2)
    cap = compute.capacity(packed.n, max_pairs=16 * packed.n, max_contacts=64 * packed.n, max_scenes=len(sizes))
    with compute.World(cap, precision=precision, bvh_rebuild_period=2) as w:
        w.upload(packed.bodies, packed.state, **packed.upload_kwargs())
        w.step(packed.options, 2)
        got, want, st = (*w.download(), w.contacts()), (*ow.download(), ow.contacts()), w.stats()
    assert st["error_flags"] == 0 and st["pairs"] > 190
    for g, r in zip(got, want):
        assert np.array_equal(np.ascontiguousarray(g).view(np.uint8), np.ascontiguousarray(r).view(np.uint8))


@pytest.mark.parametrize("n", [2049, 40001, 152 * 512 + 3])
def test_tree_pairs_equal_the_dense_sweep(n):
    b = _field(n, n).bodies
    got = []
    for broad in (0, 1):
        with compute.NarrowPhaseCompute(n, 16 * n) as npc:
            npc.configure(broad_phase=broad)
            npc.submit_broad(b)
            got.append(npc.read_pairs(npc.read_pair_count()))
    assert len(got[0]) and np.array_equal(got[0], got[1])
