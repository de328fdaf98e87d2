"""Launch shapes (gqm_tuning) on the GPU: the small team of several blocks and
the 255-register form of the flip loop (csrc/flipcl.cu) run where they are asked
for, at sizes that a context with the default shape refines in one launch, and
give the oracle's mesh."""
import numpy as np
import pytest

from gpu_cdt_refine_b200 import inputs, refine
from oracle import oracle_py

pytestmark = pytest.mark.gpu

ONE_LAUNCH = 2  # kernel launches of a one-launch refinement


@pytest.mark.parametrize("points", [60, 1100, 30_001])
@pytest.mark.parametrize("shape,one", [
    (dict(), True), (dict(small_cluster=8), False), (dict(small_cluster=16, small_limit=3000), False),
    (dict(small_cluster=8, small_limit=-1), False), (dict(check_blocks_per_sm=1), False),
    (dict(check_blocks_per_sm=1, small_cluster=16, step_grid=20), False)])
def test_shape_runs_where_it_exists(gpu, points, shape, one):
    cdt = inputs.plain_small(seed=7900 + points, n=points, nseg=points // 20)
    ctx = refine.Context(0)
    try:
        ctx.set_tuning(**shape)
        st = ctx.run_host(cdt, refine.make_options(20.0, 1, 1))
        got = ctx.result()
    finally:
        ctx.close()
    assert (st["kernel_launches"] == ONE_LAUNCH) == one
    want, info = oracle_py.refine(cdt, 20.0, 1, 1)
    assert st["rounds"] == info["rounds"]
    for f in ("pointlist", "trianglelist", "neighborlist", "segmentlist"):
        assert np.array_equal(getattr(got, f).view(np.uint8), getattr(want, f).view(np.uint8)), f


@pytest.mark.parametrize("shape", [dict(small_cluster=8), dict(check_blocks_per_sm=1)])
def test_exact_predicates(gpu, shape):
    cdt = inputs.clustered(seed=7990, n=20_000, nseg=1000)
    outs = []
    for s in (dict(), shape):
        ctx = refine.Context(0)
        try:
            ctx.set_tuning(**s)
            ctx.run_host(cdt, refine.make_options(20.0, 1, 1, refine.PRED_EXACT))
            outs.append(ctx.result())
        finally:
            ctx.close()
    for f in ("pointlist", "trianglelist", "neighborlist", "segmentlist"):
        assert np.array_equal(getattr(outs[0], f).view(np.uint8), getattr(outs[1], f).view(np.uint8)), f
