"""The grouped primal (incidence-parallel row terms, serial-order sums) against
the oracle, bit for bit, at one, two and four bodies a warp: plates carrying
68 rows beside bodies with four and with none, last groups that are not full,
both solver schedules, in all precisions."""
import numpy as np
import pytest

import oracle_lib as O
from diomedes_gb300 import abi, compute, scenes
from test_gpu_parity import _platform_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("copies,precision,mode", [(1, 0, 0), (223, 0, 0), (223, 1, 0), (461, 0, 0), (461, 2, 0),
                                                   (223, 0, 1)])
def test_grouped_primal_matches_oracle(copies, precision, mode):
    parts = [_platform_scene(), scenes.box_demo(count=11)] + [_platform_scene()] * copies
    for p in parts:
        p.options = parts[0].options
    sc = scenes.pack(parts)
    ow = O.World(sc, precision=precision, solver_mode=mode, threads=8)
    ow.step(sc.options, 3)
    cap = compute.capacity(sc.n, max_pairs=16 * sc.n, max_contacts=64 * sc.n, max_scenes=sc.n_scenes)
    with compute.World(cap, precision=precision, solver_mode=mode, batched_solver=abi.SOLVE_PER_PHASE) as w:
        w.upload(sc.bodies, sc.state, **sc.upload_kwargs())
        w.step(sc.options, 3)
        got, want = w.download(), ow.download()
        rows, ref = w.contacts(), ow.contacts()
    for g, r in zip((*got, rows), (*want, ref)):
        assert np.array_equal(np.ascontiguousarray(g).view(np.uint8), np.ascontiguousarray(r).view(np.uint8))
