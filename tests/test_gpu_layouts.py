"""One world laid out for several numbers of worlds stepped together, in turn:
each call takes the layout of its own count, a world stepped alone the whole
GPU's, and the bits are those of a world stepped alone throughout."""
import numpy as np
import pytest

import oracle_lib as O
from diomedes_gb300 import abi, compute, scenes

pytestmark = pytest.mark.gpu


def _world(sc, **cfg):
    w = compute.World(compute.capacity(sc.n, max_pairs=24 * sc.n, max_contacts=64 * sc.n, max_scenes=sc.n_scenes,
                                       max_joints=max(1, len(sc.constraints))), **cfg)
    w.upload(sc.bodies, sc.state, **sc.upload_kwargs())
    return w


def _same(got, ref):
    for g, r in zip(got, ref):
        assert np.array_equal(np.ascontiguousarray(g).view(np.uint8), np.ascontiguousarray(r).view(np.uint8))


def _group(worlds, sc, steps):
    bs = [w.download() for w in worlds]
    compute.step_host(worlds, [b for b, _ in bs], [s for _, s in bs], sc.options, steps)


def test_groups_alone_and_schedules_in_turn():
    sc = scenes.pack([scenes.pyramid(levels=9, gap=-0.01), scenes.constraints_demo(), scenes.box_demo()])
    ow = O.World(sc)
    worlds = [_world(sc) for _ in range(9)]
    w = worlds[0]
    # more counts than layouts are kept, each with others in between
    for count in (1, 3, 2, 9, 0, 6, 5, 4, 0, 3, 2):
        if count:
            _group(worlds[:count], sc, 2)
        else:
            w.step(sc.options, 2)
        ow.step(sc.options, 2)
        _same((*w.download(), w.contacts()), (*ow.download(), ow.contacts()))
    alone = _world(sc, batched_solver=abi.SOLVE_PER_PHASE)
    _group([alone], sc, 22)
    for mode, count in ((1, 0), (0, 3), (1, 3), (0, 0), (0, 3)):
        for x in (w, alone):
            x.configure(solver_mode=mode)
        if count:
            _group(worlds[:count], sc, 2)
        else:
            w.step(sc.options, 2)
        alone.step(sc.options, 2)
        _same((*w.download(), w.contacts()), (*alone.download(), alone.contacts()))
    for x in (*worlds, alone):
        x.close()


@pytest.mark.parametrize("precision,mode", [(abi.PREC_F32, 0), (abi.PREC_F32, 1), (abi.PREC_SPLIT, 0)])
def test_bodies_turned_static_between_layouts(precision, mode):
    sc = scenes.batched(n_scenes=24, lo=16, hi=300, seed=3)
    cfg = dict(precision=precision, solver_mode=mode)
    worlds = [_world(sc, **cfg) for _ in range(3)]
    ref = _world(sc, batched_solver=abi.SOLVE_PER_PHASE, **cfg)
    rng = np.random.default_rng(1)
    for k, count in enumerate((3, 1, 3, 2, 1, 3)):
        b, s = ref.download()
        turn = rng.random(sc.n) < 0.2
        fixed = turn & (s["inv_mass"] != 0)
        s["inv_mass"][fixed], s["inv_moment"][fixed] = 0.0, 0.0
        if k % 2:
            s["inv_mass"][turn & ~fixed], s["inv_moment"][turn & ~fixed, :3] = 2.0, 9.0
        for x in (*worlds, ref):
            x.set_state(b, s)
        _group(worlds[:count], sc, 1)
        _group([ref], sc, 1)
        _same((*worlds[0].download(), worlds[0].contacts()), (*ref.download(), ref.contacts()))
    for x in (*worlds, ref):
        x.close()


def test_a_world_stepped_alone_is_laid_out_alone():
    """An FP64 world whose solve goes per phase alone and as one launch where
    the GPU is shared: which one ran is seen from the timed launches."""
    sc = scenes.cube_field(nx=20, nz=4, ny=4)
    worlds = [_world(sc, precision=abi.PREC_F64, profile=1) for _ in range(3)]
    w = worlds[0]
    ran = []
    for count in (0, 3, 0, 3, 0):
        w.reset_timers()
        if count:
            _group(worlds, sc, 2)
        else:
            w.step(sc.options, 2)
        st = w.stats()
        ran.append((st["primal_launches"], st["chunk_launches"]))
    assert ran == [(20, 0), (0, 2)] * 2 + [(20, 0)]
    for x in worlds:
        x.close()


@pytest.mark.parametrize("precision", [abi.PREC_F32, abi.PREC_SPLIT, abi.PREC_F64])
@pytest.mark.parametrize("mode", [0, 1])
def test_solve_launch_switched_after_the_upload(precision, mode):
    """The chunk solve's list is ordered by its CTAs, the per-phase solve's by
    signature alone; a bodies' update between them is ordered for the one in
    force."""
    sc = scenes.pack([scenes.pyramid(levels=9, gap=-0.01), scenes.constraints_demo(), scenes.box_demo(),
                      scenes.pyramid(levels=5, gap=-0.01)])
    ow = O.World(sc, precision=precision, solver_mode=mode)
    with _world(sc, precision=precision, solver_mode=mode, block_size=640) as w:
        for launch in (abi.SOLVE_AUTO, abi.SOLVE_PER_PHASE, abi.SOLVE_AUTO, abi.SOLVE_PER_PHASE):
            w.configure(batched_solver=launch)
            w.step(sc.options, 2)
            ow.step(sc.options, 2)
            _same((*w.download(), w.contacts()), (*ow.download(), ow.contacts()))


def test_tuner_times_the_primal_shapes_where_no_chunk_solve_runs():
    """An FP64 batch whose scenes fit the chunk solve but go per phase either
    way: the tuner goes on to the primal shapes."""
    sc = scenes.batched(n_scenes=12, lo=600, hi=1600, seed=5)
    with _world(sc, precision=abi.PREC_F64, profile=1) as w:
        w.step(sc.options, 1)
        assert w.stats()["chunk_launches"] == 0
        w.configure(profile=0)
        before = w.download_f64()
        assert w.autotune(sc.options, trial_steps=1)["batched_solver"] == abi.SOLVE_PER_PHASE
        _same(w.download_f64(), before)
