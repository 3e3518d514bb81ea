"""The reciprocal of the secular solver, by itself: within one unit of the last
place of the correctly rounded 1/x for |x| from 2^-1000 to 2^1000 (8 million
numbers, every binade's ends among them), and not a number where its comment
says so.

Bound: each step squares the relative error (the approximation has about 20
bits), so only the last rounding is left, half a unit; the correctly rounded
value is at most half a unit from 1/x too, so the two are equal or neighbours."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "nrgljubljana-old_b200", "csrc")


def test_against_the_division(tmp_path):
    exe = str(tmp_path / "rcp_newton_check")
    subprocess.run([os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc"), "-gencode", "arch=compute_100a,code=sm_100a",
                    "-O3", "-std=c++17", "-I" + CSRC, os.path.join(HERE, "cpp", "rcp_newton_check.cu"), "-o", exe],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    worst, *special = (int(v) for v in r.stdout.split())
    assert worst <= 1
    assert special == [1, 1, 1]  # 0, a subnormal number, infinity
