"""A caller's rows, lists and indices that reach beyond the call's arrays are
reported, nothing beyond the buffers is read, and the context solves on."""
import numpy as np
import pytest

import oracle_lib as O
from diomedes_gb300 import abi, compute, physics as ph, scenes

pytestmark = pytest.mark.gpu


def _inputs():
    sc = scenes.pyramid(levels=6, gap=-0.01)
    pairs, _ = O.broad(sc.bodies)
    rows, off, idx = O.prepare_contacts(sc.bodies, sc.state, O.narrow(sc.bodies, pairs), None, sc.containers[0],
                                        sc.options)
    return sc, rows, off, idx


@pytest.mark.parametrize("what", ["index", "no rows", "body a", "body b", "list", "last list"])
@pytest.mark.parametrize("value", [0, 7, 1 << 20, 0xFFFFFFF0])
def test_out_of_range_input_is_reported(what, value):
    sc, rows, off, idx = _inputs()
    n, m = sc.n, len(rows)
    r2, o2, i2 = rows.copy(), off.copy(), idx.copy()
    if what == "index":
        i2[3] = min(m + value, 0xFFFFFFFE)
    elif what == "no rows":
        r2 = rows[:0]
    elif what == "body a":
        r2["a"][5] = min(n + value, 0xFFFFFFFE)
    elif what == "body b":
        r2["b"][5] = min(n + value, 0xFFFFFFFE)
    elif what == "list":
        o2[7] = off[n] + 1 + min(value, 0xFFFF0000)
    else:
        o2[n - 1], o2[n] = off[n] + 1 + min(value, 0xFFFF0000), off[n]
        o2[n - 2] = 0  # the list before runs from the start to beyond the end
    pos, quat, ro = sc.bodies["position"][:, :3], sc.bodies["orientation"], ph.run_options(sc.options)
    with compute.AvbdCompute(n, m) as ac:
        with pytest.raises(abi.DioError) as e:
            ac.run(sc.state, pos, quat, r2, sc.constraints, o2, i2, ro)
        assert e.value.status == abi.DIO_ERR_INVALID
        got = ac.run(sc.state, pos, quat, rows, sc.constraints, off, idx, ro)
    ref = O.avbd_run(sc.state, pos, quat, rows, sc.constraints, off, idx, ro)
    for k in ref:
        assert np.array_equal(np.ascontiguousarray(got[k]).view(np.uint8),
                              np.ascontiguousarray(ref[k]).view(np.uint8)), k
