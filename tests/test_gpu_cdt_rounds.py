"""The insertion rounds of the GPU CDT builder (csrc/cdt_gpu.cu) at the edges of
their launch: one block up to 1,024 points and 16 or more beyond, flip rounds of
at most 256 dirty triangles by the first block, chunks of the pending list with
remainders.  The mesh is the exact CPU builder's (general position: unique up to
numbering), and a repeated build gives the same numbering."""
import numpy as np
import pytest

from gpu_cdt_refine_b200 import inputs, triangulate
from gpu_cdt_refine_b200.cdtio import same_mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4, 33, 257, 1024, 1025, 5003, 8193, 75_777])
@pytest.mark.parametrize("clustered", [False, True])
def test_rounds_match_cpu_builder(gpu, n, clustered):
    pts = (inputs.cluster_points(n, 8, 1000.0, 5.0, 100.0, 0.1, n) if clustered
           else inputs.uniform_points(n, 0.0, 1000.0, n))
    seg = inputs.pick_segments(pts, max(1, n // 20), n + 1)
    got, st = triangulate.build_cdt_gpu(pts, seg, with_stats=True)
    want = inputs.build_cdt(pts, seg)
    assert same_mesh(got, want)
    again = triangulate.build_cdt_gpu(pts, seg)
    assert np.array_equal(got.trianglelist, again.trianglelist)
    assert np.array_equal(got.neighborlist, again.neighborlist)
    assert np.array_equal(got.segmentlist, again.segmentlist)
