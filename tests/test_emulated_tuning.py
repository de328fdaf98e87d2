"""Launch shapes (gqm_tuning) on the CPU build of the refiner's sources
(tests/emu): a shape that the one-launch refinement does not have is run by the
form that has it, at every size, and the mesh stays the oracle's."""
import pytest

from gpu_cdt_refine_b200 import inputs, refine
from oracle import oracle_py

from test_emulated_kernels import _same, emulated  # noqa: F401  (fixture)

ONE_LAUNCH = 2  # kernel launches of a one-launch refinement


@pytest.mark.parametrize("points", [40, 900])
@pytest.mark.parametrize("shape,one", [
    (dict(), True), (dict(small_limit=-1), True), (dict(step_grid=8), True),
    (dict(small_cluster=8), False), (dict(small_cluster=16, small_limit=2000), False),
    (dict(check_blocks_per_sm=1), False)])
def test_shape_runs_where_it_exists(emulated, points, shape, one):  # noqa: F811
    cdt = inputs.plain_small(seed=7800 + points, n=points, nseg=points // 20)
    ctx = refine.Context(0)
    try:
        ctx.set_tuning(**shape)
        st = ctx.run_host(cdt, refine.make_options(20.0, 1, 1))
        got = ctx.result()
    finally:
        ctx.close()
    assert (st["kernel_launches"] == ONE_LAUNCH) == one
    _same(got, oracle_py.refine(cdt, 20.0, 1, 1)[0])
