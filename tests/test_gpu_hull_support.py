"""Hull supports with four running maxima, the six-way AABB pass and the
container test's bounding radius against the oracle, bit for bit: vertex
counts around the stride, repeated vertices (ties), hulls resting in a
container's corner, and detection over the same bodies."""
import numpy as np
import pytest

import oracle_lib as O
from diomedes_gb300 import compute, physics as ph, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 2, 3, 4, 5, 7, 8, 9, 42])
def test_hulls_in_a_corner_match_oracle(count):
    rng = np.random.default_rng(count)
    items, pool = [], []
    for k in range(40):
        v = rng.normal(size=(count, 3)).astype(np.float32)
        v *= np.float32(0.4) / np.maximum(np.linalg.norm(v, axis=1, keepdims=True), np.float32(1e-3))
        if count > 4:
            v[count // 2] = v[0]  # a tie between vertices
            v[-1] = v[1]
        q = rng.normal(size=4)
        items.append(ph.hull(tuple(rng.uniform(-1.8, 1.8, 3)), len(pool) * count, v, 1.0,
                             orientation=tuple(q / np.linalg.norm(q)), velocity=tuple(rng.uniform(-3, 3, 3))))
        pool.append(v)
    b, s = ph.pack_bodies(items)
    hv = np.zeros((len(pool) * count, 4), np.float32)
    hv[:, :3] = np.concatenate(pool)
    sc = scenes.Scene("hulls", b, s, containers=[ph.container((0, 0, 0), 2.0)], hull_vertices=hv,
                      options=ph.avbd_options(), steps=4)
    ow = O.World(sc)
    ow.step(sc.options, 4)
    cap = compute.capacity(sc.n, max_pairs=2000, max_contacts=8000, max_hull_vertices=len(hv))
    with compute.World(cap) as w:
        w.upload(b, s, **sc.upload_kwargs())
        w.step(sc.options, 4)
        got, want = (*w.download(), w.contacts()), (*ow.download(), ow.contacts())
    for g, r in zip(got, want):
        assert np.array_equal(np.ascontiguousarray(g).view(np.uint8), np.ascontiguousarray(r).view(np.uint8))
    assert count < 4 or len(want[2])
