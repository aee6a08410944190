"""A step of no iterations: the pose that each schedule leaves, in every
precision and with either solve launch."""
import numpy as np
import pytest

import oracle_lib as O
from diomedes_gb300 import abi, compute, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [abi.PREC_F32, abi.PREC_SPLIT, abi.PREC_F64])
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("launch,block", [(abi.SOLVE_AUTO, 0), (abi.SOLVE_AUTO, 640), (abi.SOLVE_PER_PHASE, 0)])
@pytest.mark.parametrize("iterations", [0, 1])
def test_steps_of_few_iterations(precision, mode, launch, block, iterations):
    sc = scenes.pack([scenes.box_demo(), scenes.constraints_demo(), scenes.pyramid(levels=4, gap=-0.01)])
    sc.options.iterations = iterations
    ow = O.World(sc, precision=precision, solver_mode=mode)
    cap = compute.capacity(sc.n, max_pairs=64 * sc.n, max_contacts=200 * sc.n, max_joints=len(sc.constraints),
                           max_scenes=sc.n_scenes)
    with compute.World(cap, precision=precision, solver_mode=mode, batched_solver=launch, block_size=block) as w:
        w.upload(sc.bodies, sc.state, **sc.upload_kwargs())
        for _ in range(3):
            ow.step(sc.options, 1)
            w.step(sc.options, 1)
            for g, r in zip((*w.download(), w.contacts()), (*ow.download(), ow.contacts())):
                assert np.array_equal(np.ascontiguousarray(g).view(np.uint8), np.ascontiguousarray(r).view(np.uint8))
