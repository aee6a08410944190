"""Pairs and rows put in order by rank, and the warm start found from where a
row stands: lists on both sides of the counted lengths, bodies of many rows, and
contacts that come, go and shift the sections between steps."""
import numpy as np
import pytest

import oracle_lib as O
from diomedes_gb300 import abi, compute, physics as ph, scenes

pytestmark = pytest.mark.gpu


def _plates(n, seed):
    """n small bodies in motion around three plates of 20, 300 and 500
    neighbours, at the first, a middle and the last index."""
    rng = np.random.default_rng(seed)
    plates = {0: (0.0, 11.0), n // 2: (40.0, 8.0), n - 1: (80.0, 2.0)}
    items = []
    for k in range(n):
        if k in plates:
            x, half = plates[k]
            items.append(ph.box((x, 0.0, 0.0), (half, 0.5, half), 50.0) if hasattr(ph, "box")
                         else ph.cube((x, -half, 0.0), half, 50.0))
            continue
        x = (0.0, 40.0, 80.0)[k % 3] + rng.uniform(-12, 12)
        p = (x, rng.uniform(0.6, 3.0), rng.uniform(-12, 12))
        v = tuple(rng.uniform(-6, 6, 3))
        items.append(ph.cube(p, 0.3, 1.0, velocity=v) if k % 2 else ph.sphere(p, 0.3, 1.0, velocity=v))
    return ph.pack_bodies(items)


@pytest.mark.parametrize("n,per_pair,precision,lag", [(900, 4, abi.PREC_F32, 0), (2400, 4, abi.PREC_F32, 0),
                                                      (2400, 8, abi.PREC_F32, 1), (1200, 8, abi.PREC_F64, 0),
                                                      (2300, 4, abi.PREC_SPLIT, 0)])
def test_plates_match_oracle(n, per_pair, precision, lag):
    b, s = _plates(n, n)
    sc = scenes.Scene("plates", b, s, containers=[ph.container((40, 0, 0), 60.0)],
                      options=ph.avbd_options(gravity=(0, -30.0, 0), iterations=3))
    ow = O.World(sc, precision=precision, contacts_per_pair=per_pair, contact_lag=lag, threads=8)
    cap = compute.capacity(n, max_pairs=40 * n, max_contacts=200 * n)
    rows = []
    with compute.World(cap, precision=precision, contacts_per_pair=per_pair, contact_lag=lag) as w:
        w.upload(sc.bodies, sc.state, **sc.upload_kwargs())
        for _ in range(6):
            ow.step(sc.options, 1)
            w.step(sc.options, 1)
            got, want = (*w.download(), w.contacts()), (*ow.download(), ow.contacts())
            for g, r in zip(got, want):
                assert np.array_equal(np.ascontiguousarray(g).view(np.uint8), np.ascontiguousarray(r).view(np.uint8))
            rows.append(len(want[2]))
        assert w.stats()["error_flags"] == 0
    assert rows[-1] > 100 and len(set(rows)) > 1
