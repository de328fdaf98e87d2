"""The sharing of the multiprocessors among calls that run side by side
(csrc/sm_share.h): the rule itself (tests/emu/share_check.cpp), and the blocks
that gqm_refine_batch's launches get, on the CPU build of the refiner's sources
with several blocks to a launch."""
import os
import subprocess

from gpu_cdt_refine_b200 import inputs, refine
from oracle import oracle_py

from test_emulated_kernels import EMU, _same, emulated  # noqa: F401  (fixture)
from test_emulated_teams import _schedule, teams


def test_rule(tmp_path):
    exe = str(tmp_path / "share_check")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-pthread", "-o", exe, os.path.join(EMU, "share_check.cpp")])
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.stdout.strip() == "ok" and out.returncode == 0, out.stdout


def _largest_launch(doms, workers, blocks=12):
    L = _schedule(2)
    L.gqm_emu_set_blocks(blocks)
    L.gqm_emu_largest_launch()
    try:
        got, _ = refine.refine_batch(doms, 20.0, workers=workers)
        n = L.gqm_emu_largest_launch()
    finally:
        L.gqm_emu_set_blocks(4)
    for d, g in zip(doms, got):
        _same(g, oracle_py.refine(d, 20.0, 1, 1)[0])
    return n


@teams
def test_batch_gives_a_large_domain_its_part(emulated):  # noqa: F811
    """Beside small domains the large one gets most of the blocks, not one part in
    as many as there are workers."""
    doms = [inputs.plain_small(seed=7560 + n, n=n, nseg=10) for n in (1900, 60, 50, 40)]
    assert _largest_launch(doms, 4) >= 10
    assert _largest_launch(doms[:1], 4) == 12
