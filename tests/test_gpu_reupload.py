"""A world uploaded over another in the same context: larger, smaller, of other
scene sizes and kinds, from an image too; nothing of the former one's scene
table is read for the new bodies."""
import numpy as np
import pytest

import oracle_lib as O
from diomedes_gb300 import abi, compute, scenes

pytestmark = pytest.mark.gpu


def _same(w, ow):
    for g, r in zip((*w.download(), w.contacts()), (*ow.download(), ow.contacts())):
        assert np.array_equal(np.ascontiguousarray(g).view(np.uint8), np.ascontiguousarray(r).view(np.uint8))


@pytest.mark.parametrize("precision,mode", [(abi.PREC_F32, 0), (abi.PREC_F32, 1), (abi.PREC_SPLIT, 0),
                                            (abi.PREC_F64, 0)])
def test_uploads_over_one_another(precision, mode):
    worlds = [scenes.pyramid(levels=3), scenes.batched(n_scenes=40, lo=16, hi=200, seed=1),
              scenes.constraints_demo(), scenes.cube_field(nx=16, nz=16, ny=9), scenes.pyramid(levels=20),
              scenes.batched(n_scenes=3, lo=300, hi=900, seed=2)]
    n = max(sc.n for sc in worlds)
    cap = compute.capacity(n, max_pairs=16 * n, max_contacts=64 * n, max_scenes=max(sc.n_scenes for sc in worlds),
                           max_joints=max(len(sc.constraints) for sc in worlds))
    with compute.World(cap, precision=precision, solver_mode=mode) as w:
        for sc in worlds:
            ow = O.World(sc, precision=precision, solver_mode=mode, threads=8)
            w.upload(sc.bodies, sc.state, **sc.upload_kwargs())
            w.step(sc.options, 2)
            ow.step(sc.options, 2)
            _same(w, ow)
            image = w.checkpoint()
        w.upload(worlds[0].bodies, worlds[0].state, **worlds[0].upload_kwargs())
        w.step(worlds[0].options, 1)
        w.resume(image)  # the last world, larger than the one in force
        w.step(sc.options, 1)
        ow.step(sc.options, 1)
        _same(w, ow)
