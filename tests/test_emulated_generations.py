"""Generations of the flip steps (claims, stamps and edge maps of csrc/
kernels.cuh) over the life of a context, on the CPU build of the refiner's
sources (tests/emu): a context that has used up its 32-bit generations keeps
giving the oracle's mesh."""
import ctypes

import pytest

from gpu_cdt_refine_b200 import inputs, refine
from oracle import oracle_py

from test_emulated_kernels import _same, emulated  # noqa: F401  (fixture)


@pytest.mark.parametrize("points", [600, 3000])  # one launch; the flip loop's own launch
@pytest.mark.parametrize("gen", [2**32 - 20, 2**32 - 1000, 2**31 - 50, 2**30 - 1, 2**30])
def test_generations_near_their_end(emulated, points, gen):  # noqa: F811
    L = refine.lib()
    L.gqm_emu_set_generation.argtypes = [ctypes.c_void_p, ctypes.c_uint]
    cdt = inputs.plain_small(seed=7400 + points, n=points, nseg=points // 15)
    want, _ = oracle_py.refine(cdt, 20.0, 1, 1)
    opt = refine.make_options(20.0, 1, 1)
    opt.max_rounds = 500  # ends a loop that never does
    ctx = refine.Context(0)
    try:
        ctx.run_host(cdt, opt)
        L.gqm_emu_set_generation(ctx._h, gen)
        for _ in range(3):
            ctx.run_host(cdt, opt)
            _same(ctx.result(), want)
    finally:
        ctx.close()
