"""A small mesh refined by a context whose buffers have grown with a large one,
on the CPU build of the refiner's sources (tests/emu): the mesh is the oracle's,
also where its own slots grow into what the large one left, and the call does
not do work for the buffers' size."""
import time

import pytest

from gpu_cdt_refine_b200 import inputs, refine
from oracle import oracle_py

from test_emulated_kernels import _same, emulated  # noqa: F401  (fixture)


def _best(ctx, cdt, opt):
    t = []
    for _ in range(7):
        t0 = time.perf_counter()
        ctx.run_host(cdt, opt)
        t.append(time.perf_counter() - t0)
    return min(t)


def test_small_call_keeps_its_time(emulated):  # noqa: F811
    small = inputs.plain_small(seed=7600, n=100, nseg=5)
    large = inputs.plain_small(seed=7601, n=60_000, nseg=50)
    opt = refine.make_options(20.0, 1, 1)
    ctx = refine.Context(0)
    try:
        before = _best(ctx, small, opt)
        ctx.run_host(large, refine.make_options(1.0, 1, 1))  # grows the buffers, refines little
        after = _best(ctx, small, opt)
        _same(ctx.result(), oracle_py.refine(small, 20.0, 1, 1)[0])
    finally:
        ctx.close()
    assert after < 2.0 * before + 2e-4, (before, after)


@pytest.mark.parametrize("theta", [20.0, 24.0])
def test_growth_into_used_slots(emulated, theta):  # noqa: F811
    """60 points in clusters grow past their first capacities."""
    large = inputs.clustered(seed=7602, n=1500, nseg=100)
    ctx = refine.Context(0)
    try:
        for k in range(4):
            ctx.run_host(large, refine.make_options(20.0, 1, 1))
            small = inputs.clustered(seed=7603 + k, n=60, nseg=6)
            ctx.run_host(small, refine.make_options(theta, 1, 1))
            got = ctx.result()
            assert got.numberofpoints > 90  # 60 and a block of 30
            _same(got, oracle_py.refine(small, theta, 1, 1)[0])
    finally:
        ctx.close()
