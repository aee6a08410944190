"""The shared-memory trees walked by several CTAs a chunk and the pairs ranked
in shared memory: sizes around a part's four warps, lists on both sides of the
ranked length, scratch that overflows, and chunks of several sizes at once."""
import numpy as np
import pytest

import oracle_lib as O
from diomedes_gb300 import abi, compute, physics as ph, scenes

pytestmark = pytest.mark.gpu


def _cloud(n, spacing, seed, big=0):
    """n spheres and cubes of half size 0.5 on a grid of the spacing; the first
    `big` of them span everything."""
    rng = np.random.default_rng(seed)
    side = max(1, int(np.ceil(n ** (1.0 / 3.0))))
    items = []
    for k in range(n):
        p = np.array([k % side, (k // side) % side, k // (side * side)]) * spacing + rng.uniform(-0.1, 0.1, 3)
        r = 2.0 * side if k < big else 0.5
        items.append(ph.cube(tuple(p), r, 1.0) if k % 3 else ph.sphere(tuple(p), r, 1.0))
    rng.shuffle(items)
    return ph.pack_bodies(items)


@pytest.mark.parametrize("n,spacing,big", [(2, 0.9, 0), (31, 0.9, 0), (127, 0.9, 1), (128, 0.5, 0), (256, 0.3, 0),
                                           (257, 0.9, 2), (1024, 0.7, 3), (1300, 0.4, 0), (2047, 0.9, 1),
                                           (2048, 0.6, 0)])
def test_pairs_equal_the_oracle(n, spacing, big):
    b, _ = _cloud(n, spacing, n, big)
    want, _ = O.broad(b)
    with compute.NarrowPhaseCompute(n, max(64, len(want))) as npc:
        for _ in range(2):
            npc.submit_broad(b)
            got = npc.read_pairs(npc.read_pair_count())
            assert np.array_equal(got, want)
    assert len(want)


@pytest.mark.parametrize("precision", [abi.PREC_F32, abi.PREC_F64])
def test_chunks_of_many_sizes_match_oracle(precision):
    parts = []
    for i, (n, spacing) in enumerate([(900, 0.9), (1, 1.0), (130, 0.35), (1000, 0.8), (20, 0.2), (600, 1.1)]):
        b, s = _cloud(n, spacing, i, big=1 if n == 600 else 0)
        parts.append(scenes.Scene(f"cloud{i}", b, s, options=ph.avbd_options(iterations=1)))
    sc = scenes.pack(parts)
    ow = O.World(sc, precision=precision, threads=8)
    ow.step(sc.options, 1)
    cap = compute.capacity(sc.n, max_pairs=40 * sc.n, max_contacts=160 * sc.n, max_scenes=len(parts))
    with compute.World(cap, precision=precision) as w:
        w.upload(sc.bodies, sc.state, **sc.upload_kwargs())
        w.step(sc.options, 1)
        got, want, st = (*w.download(), w.contacts()), (*ow.download(), ow.contacts()), w.stats()
    assert st["error_flags"] == 0 and st["pairs"] > sc.n
    for g, r in zip(got, want):
        assert np.array_equal(np.ascontiguousarray(g).view(np.uint8), np.ascontiguousarray(r).view(np.uint8))
