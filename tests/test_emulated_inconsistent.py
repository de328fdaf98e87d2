"""Meshes whose indices are in range but whose neighbour lists contradict one
another, on the CPU build of the refiner's sources (tests/emu): the refinement
ends with the error that a step recorded, soon after that step, and the context
refines a sound input as the oracle does afterwards.  (The reference trusts its
input.)"""
import ctypes

import numpy as np
import pytest

from gpu_cdt_refine_b200 import inputs, refine
from oracle import oracle_py

from test_emulated_kernels import _same, emulated  # noqa: F401  (fixture)


def _scrambled(seed):
    rng = np.random.default_rng(seed)
    cdt = inputs.plain_small(seed=900 + seed % 5, n=int(rng.integers(60, 700)), nseg=20)
    nb, tr = cdt.neighborlist.copy(), cdt.trianglelist.copy()
    for _ in range(int(rng.integers(1, 6))):
        t, e = rng.integers(0, len(nb)), rng.integers(0, 3)
        if seed % 6 in (0, 1):
            nb[t, e] = rng.integers(0, len(nb))
        elif seed % 6 == 2:
            nb[t, e] = -1
        elif seed % 6 == 4:
            tr[t] = tr[t][::-1]
    cdt.neighborlist, cdt.trianglelist = nb, tr
    return cdt


# 16, 22: a walk does not end; 84: a point to be deleted lies on the boundary
@pytest.mark.parametrize("seed,status", [(16, -3), (22, -3), (84, -5)])
def test_ends_with_the_first_error(emulated, seed, status):  # noqa: F811
    ctx = refine.Context(0)
    try:
        L = refine.lib()
        keep = []
        cin = refine._cdt_in(_scrambled(seed), keep)
        st = refine.Stats()
        opt = refine.make_options(20.0, 1, 1)
        assert L.gqm_context_run(ctx._h, ctypes.byref(cin), 0, ctypes.byref(opt), ctypes.byref(st)) == status
        assert st.flip_steps < 10_000  # not the loops' own limit of 64 million
        sound = inputs.plain_small(seed=901, n=400, nseg=20)
        ctx.run_host(sound, opt)
        _same(ctx.result(), oracle_py.refine(sound, 20.0, 1, 1)[0])
    finally:
        ctx.close()
