"""A dynamic body with thousands of contact rows: its incidence list is written
whole and in order whatever its length, in the chunk solve and per phase, with
both schedules."""
import numpy as np
import pytest

import oracle_lib as O
from diomedes_gb300 import abi, compute, physics as ph, scenes

pytestmark = pytest.mark.gpu


def _loaded_plate(n):
    """n cubes resting on a dynamic plate, four rows each against it."""
    side = int(np.ceil(np.sqrt(n)))
    half = 0.3 * side
    items = [ph.box((0.0, -0.5, 0.0), (half, 0.5, half), 500.0)]
    for k in range(n):
        x, z = ((k % side) - (side - 1) / 2) * 0.55, ((k // side) - (side - 1) / 2) * 0.55
        items.append(ph.cube((x, 0.195, z), 0.2, 1.0, velocity=(0.0, -0.1 * (k % 3), 0.0)))
    b, s = ph.pack_bodies(items)
    return scenes.Scene("loaded_plate", b, s, containers=[ph.container((0, 200.0 - 1.0, 0), 200.0)],
                        options=ph.avbd_options(gravity=(0, -9.81, 0), iterations=2))


# 4,400 and 8,400 rows on the plate (4,095 to 4,097 around a power of two)
@pytest.mark.parametrize("n,per_pair,launch,mode", [
    (1023, 4, abi.SOLVE_AUTO, 0), (1024, 4, abi.SOLVE_PER_PHASE, 0), (1100, 4, abi.SOLVE_AUTO, 0),
    (1100, 4, abi.SOLVE_AUTO, 1), (1100, 8, abi.SOLVE_PER_PHASE, 0), (1100, 8, abi.SOLVE_PER_PHASE, 1),
    (2100, 4, abi.SOLVE_AUTO, 0), (2100, 8, abi.SOLVE_AUTO, 1)])
def test_loaded_plate_matches_oracle(n, per_pair, launch, mode):
    sc = _loaded_plate(n)
    ow = O.World(sc, solver_mode=mode, contacts_per_pair=per_pair, threads=8)
    cap = compute.capacity(sc.n, max_pairs=16 * sc.n, max_contacts=64 * sc.n)
    with compute.World(cap, solver_mode=mode, contacts_per_pair=per_pair, batched_solver=launch) as w:
        w.upload(sc.bodies, sc.state, **sc.upload_kwargs())
        for _ in range(3):
            ow.step(sc.options, 1)
            w.step(sc.options, 1)
            for g, r in zip((*w.download(), w.contacts()), (*ow.download(), ow.contacts())):
                assert np.array_equal(np.ascontiguousarray(g).view(np.uint8), np.ascontiguousarray(r).view(np.uint8))
        rows = w.contacts()
        assert w.stats()["error_flags"] == 0
    assert int(np.count_nonzero((rows["a"] == 0) | (rows["b"] == 0))) >= 4 * n
