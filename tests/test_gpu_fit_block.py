"""The chunked spline fits (k_fit_block) against the whole-line sweeps they stand in for, bit for bit:
tests/fit_block_check.cu runs both kernels on the same axes -- FP64 and FP32, orders 4 and 3, 32, 16 and
8 lines per block, x, y and z, even and stretched lines, the plain and the transposed solve -- over
random, constant, partly zero, wide-ranging and NaN lines, with the measured warm-up and with one of a
single element, after which nearly every chunk has to be swept again."""
import concurrent.futures as cf
import os
import subprocess

import pytest

from libcfd2lcs_b200.build import ARCH, CSRC, NVCC

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def programs(tmp_path_factory):
    d = tmp_path_factory.mktemp("fit_block")

    def compile_(real):
        out = str(d / real)
        cmd = [NVCC, "-O3", "-std=c++17", "-DREAL=" + real, "-I", CSRC, os.path.join(HERE, "fit_block_check.cu"),
               os.path.join(CSRC, "spline_host.cpp"), "-o", out] + ARCH
        r = subprocess.run(cmd, capture_output=True, text=True)
        assert r.returncode == 0, r.stderr
        return out

    reals = ("double", "float")
    with cf.ThreadPoolExecutor(2) as ex:
        return dict(zip(reals, ex.map(compile_, reals)))


@pytest.mark.parametrize("real", ["double", "float"])
def test_chunked_fit_has_the_bits_of_the_whole_line_sweeps(programs, real):
    r = subprocess.run([programs[real]], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr
    lines = r.stdout.splitlines()
    assert sum("warm 1" in q for q in lines) >= 100 and sum("transposed" in q for q in lines) >= 100
    assert sum(q.split()[1] == "rule" for q in lines) >= 15
    assert [q for q in lines if not q.startswith("0 ")] == []
