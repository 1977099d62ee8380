"""The quotient through a reciprocal on the integer pipe (divByRecip) against
the IEEE division, on the host side of the code."""

import os
import subprocess

from geometricvofext_gb300 import build as B

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_integer_quotient_is_ieee(tmp_path):
    out = str(tmp_path / "int_div_check")
    cmd = [B.nvcc(), *B.ARCH, "-O2", "-std=c++17", "-Xcompiler", "-ffp-contract=off", "-I",
           os.path.join(ROOT, "geometricvofext_gb300", "csrc"), "-I", os.path.join(ROOT, "include"),
           os.path.join(ROOT, "tests", "cpp", "int_div_check.cu"), "-o", out]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    for seed in (1, 2):
        r = subprocess.run([out, "20000000", str(seed)], capture_output=True, text=True, check=True)
        assert r.stdout.split() == ["0"]
