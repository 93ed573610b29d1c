"""The convolutions' host plan over every shape that the entry points accept."""
import os
import subprocess

from conftest import PKG, ROOT


def test_weight_gradient_plan_fits_every_shape(tmp_path):
    """Channels 8 to 128 by 8, widths to 140, 1 to 64 splits, 27 taps and 1."""
    exe = str(tmp_path / "conv_plan_check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", os.path.join(ROOT, "include"), "-I", os.path.join(PKG, "csrc"),
                    os.path.join(ROOT, "tests", "cuda", "conv_plan_check.cpp"), "-o", exe], check=True)
    plans, memory, limits = map(int, subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split())
    assert plans > 4_000_000 and memory == 0 and limits == 0
