"""Contexts and triangulations used by several threads at once share the
multiprocessors (csrc/sm_share.h): the results are those of the same calls one
after another."""
import threading

import numpy as np
import pytest

from gpu_cdt_refine_b200 import inputs, refine, triangulate

pytestmark = pytest.mark.gpu

FIELDS = ("pointlist", "trianglelist", "neighborlist", "segmentlist")


def _same(a, b):
    for f in FIELDS:
        assert np.array_equal(getattr(a, f).view(np.uint8), getattr(b, f).view(np.uint8)), f


def _in_threads(works):
    errors = []

    def run(w):
        try:
            w()
        except BaseException as e:  # noqa: B036  (handed to the test's thread)
            errors.append(e)

    pool = [threading.Thread(target=run, args=(w,)) for w in works]
    for t in pool:
        t.start()
    for t in pool:
        t.join()
    if errors:
        raise errors[0]


@pytest.mark.parametrize("sizes", [(500, 9000, 60_000, 200_000), (60_000,) * 6, (600_000, 700, 700_000)])
def test_contexts_in_threads(gpu, sizes):
    """The last case mixes the one-launch form and the graph (above 2^20 triangles)."""
    opt = refine.make_options(20.0, 1, 1)
    doms = [inputs.plain_small(seed=7800 + k, n=n, nseg=n // 20) for k, n in enumerate(sizes)]
    want = [refine.refine(d, 20.0)[0] for d in doms]

    def work(k):
        def w():
            ctx = refine.Context(0)
            try:
                for _ in range(4):
                    ctx.run_host(doms[k], opt)
                    _same(ctx.result(), want[k])
            finally:
                ctx.close()
        return w

    _in_threads([work(k) for k in range(len(doms))])


def test_triangulations_and_refinements_in_threads(gpu):
    opt = refine.make_options(20.0, 1, 1)
    cases = []
    for k, n in enumerate((2000, 20_011, 150_000)):
        pts = inputs.uniform_points(n, 0.0, 1000.0, 7900 + k)
        seg = inputs.pick_segments(pts, n // 20, 7901 + k)
        cdt = triangulate.build_cdt_gpu(pts, seg)
        cases.append((pts, seg, cdt, refine.refine(cdt, 20.0)[0]))

    def build(c):
        def w():
            for _ in range(5):
                _same(triangulate.build_cdt_gpu(c[0], c[1]), c[2])
        return w

    def mesh(c):
        def w():
            ctx = refine.Context(0)
            try:
                for _ in range(5):
                    ctx.run_host(c[2], opt)
                    _same(ctx.result(), c[3])
            finally:
                ctx.close()
        return w

    _in_threads([f(c) for c in cases for f in (build, mesh)])
