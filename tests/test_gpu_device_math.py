"""Quotients and roots of the trace kernels (csrc/device_math.cuh) against the
compiler's correctly rounded ones, on 2^28 operand pairs.

Bounds, from the forms' error terms: the corrected result before its last
rounding is off by at most 2 ulp x 2^-22 (the quotient's or root's own error
times the reciprocal's), so it rounds to the correct float or, where the exact
value lies that near a rounding boundary, to its neighbour: at most 1 ulp, in
less than one of 2^19 operands.  (rcp_rn's last bit comes from one Newton step:
0.5 ulp + 2^-23 of one before its rounding.)
"""
import os
import subprocess

import pytest

from dvsrender4deepspace_gb300 import build

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


def test_quotients_and_roots_are_the_operators(tmp_path):
    exe = str(tmp_path / "device_math_selftest")
    subprocess.run([build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "-fmad=false", "-prec-div=true", "-prec-sqrt=true",
                    "-I", build.CSRC, os.path.join(HERE, "device_math_selftest.cu"), "-o", exe], check=True)
    n = 1 << 28
    out = subprocess.run([exe, str(n)], check=True, capture_output=True, text=True, timeout=120).stdout
    rows = {line.split()[0]: [int(v) for v in line.split()[1:]] for line in out.splitlines()}
    assert rows["corners"] == [1]
    for f in ("div_rn", "div_by", "rcp_rn", "sqrt_rn"):
        differ, worst = rows[f]
        assert worst <= 1 and differ <= n >> 19, (f, differ, worst)
