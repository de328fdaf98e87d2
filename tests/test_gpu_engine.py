"""The one-launch refinement and the teams of the persistent batch
(csrc/engine.cuh) at the edges of their rules.

An input of up to 2,048 triangles is refined by one block, a larger one by 16 or
more, beyond 2^20 triangles by the graph; a batch's teams have as many blocks as
its domains leave.  Every side gives the oracle's output byte for byte."""
import numpy as np
import pytest

from gpu_cdt_refine_b200 import inputs, refine
from oracle import oracle_py

pytestmark = pytest.mark.gpu

FIELDS = ("pointlist", "trianglelist", "neighborlist", "segmentlist")


def _same(a, b):
    for f in FIELDS:
        assert np.array_equal(getattr(a, f).view(np.uint8), getattr(b, f).view(np.uint8)), f


@pytest.mark.parametrize("points,mode,policy", [(4, 1, 1), (37, 0, 0), (1020, 1, 1), (1050, 1, 1), (1050, 0, 0),
                                                (9000, 0, 1), (60_000, 1, 0)])
def test_one_launch_matches_oracle(gpu, points, mode, policy):
    cdt = inputs.plain_small(seed=8100 + points, n=points, nseg=max(1, points // 20))
    got, ps, ts, st = refine.refine(cdt, 20.0, policy, mode, with_status=True)
    want, info = oracle_py.refine(cdt, 20.0, policy, mode)
    _same(got, want)
    assert np.array_equal(ps, info["pstatus"]) and np.array_equal(ts, info["tstatus"])
    assert st["rounds"] == info["rounds"] and st["kernel_launches"] == 2


def test_one_launch_round_limit_and_bad_input(gpu):
    cdt = inputs.plain_small(seed=8200, n=3000, nseg=100)
    with pytest.raises(refine.RefineError) as e:
        refine.refine(cdt, 20.0, max_rounds=1)
    assert e.value.status == -2
    want, _ = refine.refine(cdt, 20.0)
    cdt.trianglelist[5, 2] = 10**6
    with pytest.raises(refine.RefineError) as e:
        refine.refine(cdt, 20.0)
    assert e.value.status == -1
    cdt = inputs.plain_small(seed=8200, n=3000, nseg=100)
    _same(refine.refine(cdt, 20.0)[0], want)


@pytest.mark.parametrize("sizes", [[30_000], [300, 20_000], [700, 900, 4000, 12_000, 260], [400] * 40, [250] * 200])
def test_batch_teams_match_oracle(gpu, sizes):
    doms = [inputs.plain_small(seed=8300 + 7 * k, n=n, nseg=max(1, n // 20)) for k, n in enumerate(sizes)]
    got, stats, rep = refine.refine_batch_persistent(doms, 20.0, with_report=True)
    assert rep["fallbacks"] == 0 and rep["grid"] >= min(len(sizes), 148)
    for k, (d, g, st) in enumerate(zip(doms, got, stats)):
        if k % 10 == 0 or len(sizes) < 10:
            want, info = oracle_py.refine(d, 20.0, 1, 1)
            _same(g, want)
            assert st["rounds"] == info["rounds"]


@pytest.mark.parametrize("ring", [30, 52, 53, 120, 700])
def test_large_cavities_match_oracle(gpu, ring):
    """Points on a circle: the first Steiner points' cavities hold nearly every
    triangle, on both sides of the cap of fifty."""
    a = 2 * np.pi * (np.arange(ring) + 0.3 * np.random.default_rng(ring).uniform(-1, 1, ring)) / ring
    pts = np.stack([100 * np.cos(a), 100 * np.sin(a)], 1)
    cdt = inputs.build_cdt(pts, np.zeros((0, 2), np.int32))
    got, st = refine.refine(cdt, 20.0)
    want, info = oracle_py.refine(cdt, 20.0, 1, 1)
    _same(got, want)
    assert st["rounds"] == info["rounds"]
    one, _ = refine.refine_batch_persistent([cdt], 20.0)
    _same(one[0], want)
