"""Both forms of divByRecip (integer pipe, and Newton corrections on the FP64
pipe) against the IEEE division, bit for bit, on the host and on the GPU."""

import os
import subprocess

import pytest

from geometricvofext_gb300 import build as B

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _check(tmp_path, where, n, seed):
    out = str(tmp_path / "newton_div_check")
    cmd = [B.nvcc(), *B.ARCH, "-O2", "-std=c++17", "-fmad=false", "-Xcompiler", "-ffp-contract=off", "-I",
           os.path.join(ROOT, "geometricvofext_gb300", "csrc"), "-I", os.path.join(ROOT, "include"),
           os.path.join(ROOT, "tests", "cpp", "newton_div_check.cu"), "-o", out]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([out, where, str(n), str(seed)], capture_output=True, text=True, check=True, timeout=300)
    assert r.stdout.split() == ["0", "0", "0"]


def test_both_quotients_are_ieee_on_the_host(tmp_path):
    _check(tmp_path, "host", 20000000, 3)


@pytest.mark.gpu
def test_both_quotients_are_ieee_on_the_gpu(tmp_path):
    _check(tmp_path, "gpu", 1 << 28, 4)
