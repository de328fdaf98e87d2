"""The cooperative launches (csrc/team.cuh) as several blocks on the CPU: the
refiner's own sources compiled with tests/emu/team_emu.h, whose blocks run one
at a time from barrier to barrier in a chosen order.  Whatever the order, every
block has to take the same way through the barriers and the mesh is the
oracle's byte for byte.  Order 0 lets the first block run ahead of all others
(it runs the small flip steps), order 1 lets it come last."""
import ctypes

import numpy as np
import pytest

from gpu_cdt_refine_b200 import cdtio, inputs, refine, triangulate
from oracle import oracle_py

from test_emulated_kernels import _same, emulated  # noqa: F401  (fixture)

teams = pytest.mark.parametrize("emulated", ["libgqm_emu_teams.so"], indirect=True)


def _schedule(order):
    L = refine.lib()
    L.gqm_emu_schedule.argtypes = [ctypes.c_int]
    L.gqm_emu_schedule(order)
    return L


@teams
@pytest.mark.parametrize("order", [0, 1, 2, 3])
@pytest.mark.parametrize("points", [1500, 3000])  # one launch; the flip loop's own launch
@pytest.mark.parametrize("shape", [dict(), dict(small_limit=-1), dict(small_limit=40), dict(small_cluster=8)],
                         ids=["default", "no small steps", "both", "small team"])
def test_flip_loop_in_any_order_of_blocks(emulated, order, points, shape):  # noqa: F811
    cdt = inputs.plain_small(seed=7100 + points, n=points, nseg=points // 15)
    L = _schedule(order)
    ctx = refine.Context(0)
    try:
        ctx.set_tuning(**shape)
        st = ctx.run_host(cdt, refine.make_options(20.0, 1, 1))
        got = ctx.result()
    finally:
        ctx.close()
    assert L.gqm_emu_stuck_count() == 0
    want, info = oracle_py.refine(cdt, 20.0, 1, 1)
    _same(got, want)
    assert st["rounds"] == info["rounds"] and st["flip_steps"] > 0


@teams
@pytest.mark.parametrize("order", [0, 1, 2])
@pytest.mark.parametrize("limit", [40, 300])
def test_small_team_of_some_of_the_blocks(emulated, order, limit):  # noqa: F811
    cdt = inputs.plain_small(seed=7150, n=1500, nseg=100)
    L = _schedule(order)
    L.gqm_emu_set_blocks(12)
    ctx = refine.Context(0)
    try:
        ctx.set_tuning(small_cluster=8, small_limit=limit)
        ctx.run_host(cdt, refine.make_options(20.0, 1, 1))
        got = ctx.result()
    finally:
        L.gqm_emu_set_blocks(4)
        ctx.close()
    assert L.gqm_emu_stuck_count() == 0
    _same(got, oracle_py.refine(cdt, 20.0, 1, 1)[0])


@teams
@pytest.mark.parametrize("order", [0, 1, 2])
def test_batch_teams_in_any_order_of_blocks(emulated, order):  # noqa: F811
    doms = [inputs.plain_small(seed=7200 + i, n=n, nseg=n // 15) for i, n in enumerate([900, 300])]
    L = _schedule(order)
    got, _ = refine.refine_batch_persistent(doms, 20.0)
    assert L.gqm_emu_stuck_count() == 0
    for d, g in zip(doms, got):
        _same(g, oracle_py.refine(d, 20.0, 1, 1)[0])


@teams
@pytest.mark.parametrize("order", [0, 1, 2, 3])
@pytest.mark.parametrize("points,segments", [(1100, 60), (1100, 0), (4000, 400)])
def test_triangulation_in_any_order_of_blocks(emulated, order, points, segments):  # noqa: F811
    pts = inputs.uniform_points(points, 0.0, 1000.0, 7300 + points)
    seg = inputs.pick_segments(pts, segments, 7301) if segments else np.zeros((0, 2), np.int32)
    L = _schedule(order)
    got = triangulate.build_cdt_gpu(pts, seg)
    assert L.gqm_emu_stuck_count() == 0
    assert cdtio.same_mesh(inputs.build_cdt(pts, seg), got)


@teams
@pytest.mark.parametrize("points", [1500, 3000])  # one launch; the flip loop's own launch
@pytest.mark.parametrize("wait", [200, 1003, 2506])
def test_context_recovers_from_a_wait_that_ran_out(emulated, points, wait):  # noqa: F811
    """The waits of a launch are given up in the middle of a flip loop: that call
    reports it, and the next on the same context gives the oracle's mesh."""
    cdt = inputs.plain_small(seed=7500 + points, n=points, nseg=points // 15)
    want, _ = oracle_py.refine(cdt, 20.0, 1, 1)
    L = _schedule(2)
    L.gqm_emu_break_at.argtypes = [ctypes.c_longlong]
    opt = refine.make_options(20.0, 1, 1)
    opt.max_rounds = 500  # ends a loop that never does
    ctx = refine.Context(0)
    try:
        ctx.set_tuning(small_limit=-1)  # every step by all blocks
        L.gqm_emu_break_at(wait)
        with pytest.raises(refine.RefineError) as e:
            ctx.run_host(cdt, opt)
        assert e.value.status == -5
        for _ in range(2):
            ctx.run_host(cdt, opt)
            _same(ctx.result(), want)
    finally:
        L.gqm_emu_break_at(-1)
        ctx.close()


@teams
def test_autotune_chooses_among_launches_that_differ(emulated):  # noqa: F811
    """Two and one of four blocks are tried beside all four; an input that one
    block refines has nothing to choose there (six runs: no clock's noise does)."""
    _schedule(2)
    opt = refine.make_options(20.0, 1, 1)
    for points, grids in ((1500, (592, 2, 1)), (300, (592,))):
        cdt = inputs.plain_small(seed=7550, n=points, nseg=points // 15)
        for _ in range(6):
            ctx = refine.Context(0)
            try:
                chosen, _ = ctx.autotune(cdt, opt)
                assert chosen["step_grid"] in grids and chosen == ctx.tuning()
                ctx.run_host(cdt, opt)
                _same(ctx.result(), oracle_py.refine(cdt, 20.0, 1, 1)[0])
            finally:
                ctx.close()
