"""The scene-chunk solve's shapes against the oracle, bit for bit: worlds that
take a cluster of 1, 2, 4 and 8 CTAs (3 to 2,048 bodies, block and slot
remainders, scenes without contacts, joints across CTAs), whole-SM chunks
(more chunks than SMs; block_size 640), all precisions and both schedules,
and a switch of the schedule after the upload."""
import numpy as np
import pytest

import oracle_lib as O
from diomedes_gb300 import compute, scenes

pytestmark = pytest.mark.gpu


def _scene(kind, n):
    if kind == "pyramid":
        return scenes.pyramid(levels=n)
    if kind == "field":
        return scenes.cube_field(nx=n, nz=4, ny=4)
    if kind == "batch":
        return scenes.batched(n_scenes=n, lo=16, hi=300, seed=n)
    return scenes.batched(n_scenes=2, lo=n, hi=n + 1, seed=n)


def _same(w, ow):
    for g, r in zip((*w.download(), w.contacts()), (*ow.download(), ow.contacts())):
        assert np.array_equal(np.ascontiguousarray(g).view(np.uint8), np.ascontiguousarray(r).view(np.uint8))


def _world(sc, **cfg):
    cap = compute.capacity(sc.n, max_pairs=16 * sc.n + 64, max_contacts=64 * sc.n + 64,
                           max_joints=max(1, len(sc.constraints)), max_scenes=sc.n_scenes)
    w = compute.World(cap, **cfg)
    w.upload(sc.bodies, sc.state, **sc.upload_kwargs())
    return w


@pytest.mark.parametrize("kind,n,precision,mode,block", [
    ("pyramid", 2, 0, 0, 0), ("pyramid", 9, 0, 0, 0), ("pyramid", 9, 0, 1, 0), ("field", 17, 0, 0, 0),
    ("field", 128, 0, 0, 0), ("field", 20, 2, 0, 0), ("field", 70, 1, 0, 0), ("single", 2047, 0, 0, 0),
    ("single", 2047, 0, 1, 0), ("single", 1025, 1, 0, 0), ("single", 1300, 2, 1, 0), ("single", 2047, 0, 0, 640),
    ("batch", 400, 0, 0, 0), ("batch", 400, 0, 1, 640), ("batch", 31, 1, 1, 0)])
def test_solve_shapes_match_oracle(kind, n, precision, mode, block):
    sc = _scene(kind, n)
    ow = O.World(sc, precision=precision, solver_mode=mode, threads=8)
    ow.step(sc.options, 3)
    with _world(sc, precision=precision, solver_mode=mode, block_size=block) as w:
        w.step(sc.options, 3)
        _same(w, ow)


def test_schedule_switched_after_the_upload():
    sc = scenes.pyramid(levels=8)
    ow = O.World(sc)
    with _world(sc) as w:
        w.step(sc.options, 2)
        ow.step(sc.options, 2)
        _same(w, ow)
        w.configure(block_size=640)
        w.step(sc.options, 2)
        ow.step(sc.options, 2)
        _same(w, ow)
