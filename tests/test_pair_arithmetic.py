"""The straight-line quotients and roots of the flat kernels (ez_pair.cuh) and
their division by 12 are the IEEE operations wherever the guard accepts the
operands: tests/cuda/pair_check.cu, compiled here, compares every FP32
mantissa, every FP32 pattern of the division by 12, and random and
near-boundary operands of both precisions, those at the guard's thresholds
among them."""
import os
import subprocess

import pytest

from coffee_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.gpu
def test_straight_line_arithmetic_is_ieee(tmp_path):
    exe = str(tmp_path / "pair_check")
    subprocess.run([build.nvcc_path(), "-O3", "-std=c++17", *build.ARCH, "-I", build.INCLUDE, "-I",
                    build.CSRC, os.path.join(HERE, "cuda", "pair_check.cu"), "-o", exe], check=True,
                   capture_output=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=300).stdout
    print(out)
    lines = [line.split() for line in out.splitlines()]
    assert len(lines) == 9
    for name, n, bad in lines:
        assert int(n) > 1e6 and int(bad) == 0, out
