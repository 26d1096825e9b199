"""Reciprocals of the trace kernels (csrc/device_math.cuh) over the ranges they
are used in: rcp_rn for every normal float up to 2^126, rcp_small for every one
from 2^-128 to 2^124.  As test_gpu_device_math.py states, a result is the correctly
rounded one or, rarely, its neighbour.  The FP64 quotients by a divisor known
beforehand: their own error before the last rounding is 2^-52 ulp, so none of
2^26 pairs differs from the operator.  And the triangle that needs the latter:
one so small that the watertight test's determinant is denormal is hit.
"""
import os
import subprocess

import numpy as np
import pytest

from dvsrender4deepspace_gb300 import CamRayCaster, DeviceScene, build

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
HAPKE = dict(b=0.3, c=0.4, hS=0.06, hC=1.0, thetap=0.349066, w=0.25, B_S0=1.0, B_C0=0.0, phi=0.3)


def test_reciprocals_over_their_ranges(tmp_path):
    exe = str(tmp_path / "device_math_ranges_selftest")
    subprocess.run([build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "-fmad=false", "-prec-div=true",
                    "-I", build.CSRC, os.path.join(HERE, "device_math_ranges_selftest.cu"), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=120).stdout
    rows = {line.split()[0]: [int(v) for v in line.split()[1:]] for line in out.splitlines()}
    for f, n in (("rcp_rn", 2 * 252 << 23), ("rcp_small", 2 * 250 << 23)):
        differ, worst = rows[f]
        assert worst <= 1 and differ <= n >> 19, (f, differ, worst)
    assert rows["beyond_finite"] == [0]
    assert rows["quotient"] == [0] and rows["product"][0] > 1 << 20


@pytest.mark.parametrize("size", [1e-3, 1e-12, 3e-20])
def test_smallest_triangles_are_hit(size):
    """The clamp of a zero direction component at 1e-20 leaves a box of 3e-20 open for three units of distance."""
    V = np.array([[-size, -size, 0], [size, -size, 0], [0, size, 0]], np.float32)
    N = np.tile(np.float32([0, 0, 1]), (3, 1))
    cam = dict(width=3, height=3, fx=10.0, fy=10.0, cx=1.0, cy=1.0)  # the middle pixel's ray is -z
    scene = DeviceScene(V, N, np.array([[0, 1, 2]], np.uint32), cam, 1, HAPKE, geometry=2)
    pose = dict(position=(0, 0, 2), rotation=(0, 0, 0, 1), light=(0, 0, 1), intensity=1000)
    depth = np.asarray(CamRayCaster(scene).render_state(pose)[1])
    assert abs(depth[4] - 2.0) < 1e-4
    assert (np.delete(depth, 4) == -1.0).all()
