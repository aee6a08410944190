"""Checkpoint rows copied in one piece and in several (more row bytes than the
staging buffer): the image of a resumed world is the image, and it steps on as
the oracle does."""
import numpy as np
import pytest

import oracle_lib as O
from diomedes_gb300 import abi, compute, physics as ph, scenes

pytestmark = pytest.mark.gpu


def _cornered(n):
    """n scenes of one cube in the corner of its box: twelve rows each."""
    b, s = ph.pack_bodies([ph.cube((0.51 + 4 * k, 0.51, 0.51), 0.5, 1.0) for k in range(n)])
    b["position"][:, 0] -= 4 * np.arange(n, dtype=np.float32)
    b["position"][:, :3] -= 0.02 + 0.001 * (np.arange(n) % 7)[:, None].astype(np.float32)
    return scenes.Scene("cornered", b, s, scene_offsets=np.arange(n + 1, dtype=np.uint32),
                        containers=[ph.container((2, 2, 2), 2.0)] * n, options=ph.avbd_options(iterations=3))


@pytest.mark.parametrize("precision", [abi.PREC_F32, abi.PREC_SPLIT, abi.PREC_F64])
@pytest.mark.parametrize("n", [1, 65, 300])
def test_row_images(n, precision):
    sc = _cornered(n)
    ow = O.World(sc, precision=precision)
    cap = compute.capacity(n, max_pairs=1, max_contacts=12 * n, max_scenes=n)
    with compute.World(cap, precision=precision) as w, compute.World(cap, precision=precision) as v:
        w.upload(sc.bodies, sc.state, **sc.upload_kwargs())
        w.step(sc.options, 2)
        ow.step(sc.options, 2)
        image = w.checkpoint()
        assert compute.checkpoint_header(image)["rows"] == len(ow.contacts()) > 8 * n
        v.resume(image)
        assert v.checkpoint() == image
        for x in (w, v):
            x.step(sc.options, 2)
        ow.step(sc.options, 2)
        for x in (w, v):
            for g, r in zip((*x.download(), x.contacts()), (*ow.download(), ow.contacts())):
                assert np.array_equal(np.ascontiguousarray(g).view(np.uint8), np.ascontiguousarray(r).view(np.uint8))
