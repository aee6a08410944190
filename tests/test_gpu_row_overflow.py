"""More contact rows than max_contacts: a call of several steps reports the
capacity error with the rows that fit kept, and the world is usable after the
next upload."""
import numpy as np
import pytest

import oracle_lib as O
from diomedes_gb300 import abi, compute, scenes

pytestmark = pytest.mark.gpu


# a falling pyramid grows to 374 pair rows and 418 rows: one, the container's
# alone, below and about the pair rows, and between them and all rows
@pytest.mark.parametrize("cap", [1, 44, 300, 374, 400])
@pytest.mark.parametrize("launch,mode", [(abi.SOLVE_AUTO, 0), (abi.SOLVE_PER_PHASE, 0), (abi.SOLVE_AUTO, 1)])
def test_steps_beyond_the_row_capacity(cap, launch, mode):
    sc, small = scenes.pyramid(levels=11), scenes.pyramid(levels=1)
    with compute.World(compute.capacity(sc.n, max_pairs=64 * sc.n, max_contacts=cap), batched_solver=launch,
                       solver_mode=mode) as w:
        w.upload(sc.bodies, sc.state, **sc.upload_kwargs())
        with pytest.raises(abi.DioError) as e:
            w.step(sc.options, 60)
        assert e.value.status == abi.DIO_ERR_CAPACITY
        assert len(w.contacts()) <= cap  # (the last step need not be among those that overflowed)
        if cap < 4:
            return
        ow = O.World(small, solver_mode=mode)
        w.upload(small.bodies, small.state, **small.upload_kwargs())
        w.step(small.options, 30)
        ow.step(small.options, 30)
        for g, r in zip((*w.download(), w.contacts()), (*ow.download(), ow.contacts())):
            assert np.array_equal(np.ascontiguousarray(g).view(np.uint8), np.ascontiguousarray(r).view(np.uint8))
