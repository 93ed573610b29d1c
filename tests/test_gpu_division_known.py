"""The streamline pass divides by known divisors through one correctly rounded reciprocal
(div_known, wt_lattice.cuh): builds tests/cuda/div_known_check.cu and checks it against
IEEE division bit for bit, over its whole range of divisors and past both ends."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(os.path.dirname(HERE), "f1-wind-tunnel_gb300"))


def test_div_known_matches_ieee_division(tmp_path):
    import build
    exe = str(tmp_path / "div_known_check")
    subprocess.run([build.nvcc(), *[f for f in build.NVCC_FLAGS if f != "-lineinfo"], "-I", build.CSRC,
                    os.path.join(HERE, "cuda", "div_known_check.cu"), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=600).stdout.split()
    bad, cases = int(out[0]), int(out[1])
    assert cases == 2 << 30 and bad == 0
