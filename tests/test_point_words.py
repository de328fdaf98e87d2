"""Point status bytes are changed by atomics on whole words (csrc/kernels.cuh,
delete_point): none reaches past the status array (tests/emu/point_words.cpp,
the refiner's sources under the address sanitizer)."""
import os
import subprocess

from test_emulated_kernels import EMU, ROOT


def test_last_point_deleted_within_the_array(tmp_path):
    exe = str(tmp_path / "point_words")
    csrc = os.path.join(ROOT, "gpu_cdt_refine_b200", "csrc")
    flags = ["-O1", "-g", "-std=c++17", "-fsanitize=address", "-Wno-unused-result", "-x", "c++",
             "-I" + os.path.join(EMU, "cuda_fake"), "-I" + os.path.join(ROOT, "include")]
    subprocess.check_call(["g++", *flags, "-o", exe, os.path.join(EMU, "point_words.cpp"),
                           os.path.join(csrc, "batch.cu"), os.path.join(csrc, "flipcl.cu")])
    run = subprocess.run([exe], capture_output=True, text=True, env={**os.environ, "ASAN_OPTIONS": "detect_leaks=0"})
    assert run.returncode == 0, run.stderr[:2000]
