"""The flip-flop loop's launch (csrc/flipcl.cu) at the edges of its teams.

A refinement uses one block per 1,024 input triangles, hands steps of at most
small_limit queued triangles to the small team, keeps the decisions of a step of
at most 1,024 triangles in shared memory, and orders competing subsegment stores
with a scan up to 2,048 queue entries and with a bitmap beyond: each side of each
of these gives the oracle's output byte for byte."""
import numpy as np
import pytest

from gpu_cdt_refine_b200 import inputs, refine
from oracle import oracle_py

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("points,nseg", [(40, 3), (520, 26), (1100, 200), (4096, 900), (30_001, 6000)])
@pytest.mark.parametrize("limit", [0, 1, 33, 1025, 5000])
def test_team_edges(gpu, points, nseg, limit):
    cdt = inputs.plain_small(seed=7000 + points, n=points, nseg=nseg)
    want, info = oracle_py.refine(cdt, 20.0, 1, 1)
    ctx = refine.Context(0)
    try:
        ctx.set_tuning(small_limit=limit)
        st = ctx.run_host(cdt, refine.make_options(20.0, 1, 1))
        got = ctx.result()
    finally:
        ctx.close()
    assert st["rounds"] == info["rounds"]
    for f in ("pointlist", "trianglelist", "neighborlist", "segmentlist"):
        assert np.array_equal(getattr(got, f).view(np.uint8), getattr(want, f).view(np.uint8)), f
