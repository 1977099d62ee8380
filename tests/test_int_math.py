"""int_math.cuh (products, quotients and settled differences of doubles on the
integer pipe) against the IEEE operations, on the host side of the code."""

import os
import subprocess

from geometricvofext_gb300 import build as B

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_integer_products_are_ieee(tmp_path):
    out = str(tmp_path / "int_math_check")
    cmd = [B.nvcc(), *B.ARCH, "-O2", "-std=c++17", "-Xcompiler", "-ffp-contract=off", "-I",
           os.path.join(ROOT, "geometricvofext_gb300", "csrc"), "-I", os.path.join(ROOT, "include"),
           os.path.join(ROOT, "tests", "cpp", "int_math_check.cu"), "-o", out]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    for seed in (1, 2):
        r = subprocess.run([out, "3000000", str(seed)], capture_output=True, text=True, check=True)
        for line in r.stdout.split("\n")[:-1]:
            cases, refused, bad = (int(x) for x in line.split())
            assert bad == 0 and refused < 0.6 * cases
