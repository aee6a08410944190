"""The FP64 scene-chunk solve, which an FP64 world takes where it is estimated
the faster: whole-SM chunks (block_size 640) and clusters (worlds stepped
together), both schedules; the timed launches show that it ran."""
import numpy as np
import pytest

import oracle_lib as O
from diomedes_gb300 import abi, compute, scenes

pytestmark = pytest.mark.gpu


def _scene(kind, n):
    if kind == "pyramid":
        return scenes.pyramid(levels=n, gap=-0.01)
    if kind == "field":
        return scenes.cube_field(nx=n, nz=4, ny=4, spacing=0.45)
    if kind == "batch":
        return scenes.batched(n_scenes=n, lo=16, hi=300, seed=n)
    return scenes.batched(n_scenes=2, lo=n, hi=n + 1, seed=n)


def _world(sc, **cfg):
    w = compute.World(compute.capacity(sc.n, max_pairs=24 * sc.n + 64, max_contacts=64 * sc.n + 64,
                                       max_joints=max(1, len(sc.constraints)), max_scenes=sc.n_scenes),
                      precision=abi.PREC_F64, profile=1, **cfg)
    w.upload(sc.bodies, sc.state, **sc.upload_kwargs())
    return w


def _same(got, ref):
    for g, r in zip(got, ref):
        assert np.array_equal(np.ascontiguousarray(g).view(np.uint8), np.ascontiguousarray(r).view(np.uint8))


@pytest.mark.parametrize("kind,n,mode", [("pyramid", 2, 0), ("pyramid", 9, 0), ("pyramid", 9, 1), ("field", 17, 0),
                                         ("field", 17, 1), ("single", 400, 0), ("batch", 31, 0)])
def test_whole_sm_chunks(kind, n, mode):
    sc = _scene(kind, n)
    ow = O.World(sc, precision=abi.PREC_F64, solver_mode=mode, threads=8)
    with _world(sc, solver_mode=mode, block_size=640) as w:
        for _ in range(3):
            w.step(sc.options, 1)
            ow.step(sc.options, 1)
            _same((*w.download(), w.contacts()), (*ow.download(), ow.contacts()))
        assert w.stats()["chunk_launches"] == 3


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("kind,n", [("pyramid", 3), ("field", 20), ("field", 70), ("single", 1025), ("single", 2047),
                                    ("batch", 31)])
@pytest.mark.parametrize("block", [0, 640])
def test_worlds_together(kind, n, mode, block):
    """Clusters, or whole-SM chunks where the scenes fit one (1,024 bodies)."""
    sc = _scene(kind, n)
    ow = O.World(sc, precision=abi.PREC_F64, solver_mode=mode, threads=8)
    ow.step(sc.options, 1)
    worlds = [_world(sc, solver_mode=mode, block_size=block) for _ in range(3)]
    phases = _world(sc, solver_mode=mode, batched_solver=abi.SOLVE_PER_PHASE)
    for k in range(3):
        for group in (worlds, [phases]):
            bs = [w.download() for w in group]
            compute.step_host(group, [b for b, _ in bs], [s for _, s in bs], sc.options, 1)
        got = [(*w.download(), w.contacts()) for w in (*worlds, phases)]
        for g in got[1:]:
            _same(g, got[0])
        if k == 0:
            _same(got[0], (*ow.download(), ow.contacts()))
    assert worlds[0].stats()["chunk_launches"] == 3 and phases.stats()["chunk_launches"] == 0
    for w in (*worlds, phases):
        w.close()
