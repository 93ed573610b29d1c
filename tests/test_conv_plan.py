"""The convolutions' host plans over every shape that the entry points accept."""
import os
import subprocess

import pytest

from conftest import PKG, ROOT


@pytest.fixture(scope="module")
def counts(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("plan") / "conv_plan_check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", os.path.join(ROOT, "include"), "-I", os.path.join(PKG, "csrc"),
                    os.path.join(ROOT, "tests", "cuda", "conv_plan_check.cpp"), "-o", exe], check=True)
    return list(map(int, subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split()))


def test_plans_fit_every_shape(counts):
    """Channels 8 to 128 by 8, widths to 140, 1 to 64 splits, 27 taps and 1."""
    plans, memory, limits = counts[:3]
    assert plans > 12_000_000 and memory == 0 and limits == 0


def test_grids_that_numbered_rows_do_not_suit_are_gathered(counts):
    """Six grids, three calls each: numbered rows beyond 31 bits, and one voxel to a plane."""
    assert counts[3] == 18
