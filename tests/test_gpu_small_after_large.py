"""A small mesh refined by a context whose buffers have grown with a large one:
the oracle's mesh, in the device time it takes on a fresh context."""
import numpy as np
import pytest

from gpu_cdt_refine_b200 import inputs, refine
from oracle import oracle_py

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("points", [500, 6000])  # one block; a team
def test_small_call_keeps_its_time(gpu, points):
    small = inputs.plain_small(seed=7700, n=points, nseg=points // 20)
    large = inputs.clustered(seed=7701, n=1_000_000, nseg=1000)
    opt = refine.make_options(20.0, 1, 1)
    ctx = refine.Context(0)
    try:
        before = min(ctx.run_host(small, opt)["device_ms"] for _ in range(8))
        ctx.run_host(large, opt)
        after = min(ctx.run_host(small, opt)["device_ms"] for _ in range(8))
        got = ctx.result()
    finally:
        ctx.close()
    want, _ = oracle_py.refine(small, 20.0, 1, 1)
    for f in ("pointlist", "trianglelist", "neighborlist", "segmentlist"):
        assert np.array_equal(getattr(got, f).view(np.uint8), getattr(want, f).view(np.uint8)), f
    assert after < 1.15 * before, (before, after)
