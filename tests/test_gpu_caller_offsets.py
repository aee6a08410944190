"""A caller's row offsets that step back: a body whose list would end before it
starts has no rows, in every primal variant's way of walking the lists."""
import numpy as np
import pytest

import oracle_lib as O
from diomedes_gb300 import compute, physics as ph, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", [5, 0, 6, 10])
@pytest.mark.parametrize("name", ["pyramid", "box_demo", "cube_field"])
def test_offsets_that_step_back(name, variant):
    sc = {"pyramid": lambda: scenes.pyramid(levels=6, gap=-0.01), "box_demo": scenes.box_demo,
          "cube_field": lambda: scenes.cube_field(nx=8, nz=8, ny=4, spacing=0.45)}[name]()
    cont = sc.containers[0]
    pairs, _ = O.broad(sc.bodies)
    slots = O.narrow(sc.bodies, pairs)
    rows, off, idx = O.prepare_contacts(sc.bodies, sc.state, slots, None, cont, sc.options)
    # body 0: an empty list that starts past the others; body 1: one that
    # steps back to the start; from body 2 on the lists as they were
    lists = idx[off[2]:]
    assert len(lists) > 8
    offsets = (off - off[2]).astype(np.uint32)
    offsets[0] = offsets[1] = len(lists)
    args = (sc.state, sc.bodies["position"][:, :3], sc.bodies["orientation"], rows, sc.constraints, offsets, lists,
            ph.run_options(sc.options))
    ref = O.avbd_run(*args)
    with compute.AvbdCompute(sc.n, len(rows), max_joints=max(1, len(sc.constraints))) as ac:
        ac.configure(primal_variant=variant)
        got = ac.run(*args)
    for k in ref:
        assert np.array_equal(np.ascontiguousarray(got[k]).view(np.uint8),
                              np.ascontiguousarray(ref[k]).view(np.uint8)), k
