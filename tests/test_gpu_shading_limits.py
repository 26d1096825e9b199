"""Materials and normals at the ends of their ranges: values that the quotients
and roots without range checks cannot take and the shading handles beside them.
Each goes through both samplers -- a frame (packets of sub-rays) and an exposure
of eight equal poses (temporal packets).
"""
import numpy as np
import pytest

from dvsrender4deepspace_gb300 import CamRayCaster, DeviceScene, OpticalError, terrain, trajectory

pytestmark = pytest.mark.gpu

HAPKE = dict(b=0.3, c=0.4, hS=0.06, hC=1.0, thetap=0.349066, w=0.25, B_S0=1.0, B_C0=0.0, phi=0.3)
CAM = dict(width=41, height=31, fx=40.0, fy=40.0, cx=20.5, cy=15.5)
POSE = trajectory.StraightPass((5.0, -8.0, 350.0), (0.0, 0.0, 0.0), trajectory.sun_direction(30, 40), 1000.0, 0.4).state(0)


@pytest.fixture(scope="module")
def ground():
    return terrain.terrain_mesh(48, seed=3)


def renders(scene, pose=POSE):
    """The callables that give a scene's image through each sampler."""
    caster = CamRayCaster(scene)
    return (lambda: np.asarray(caster.render_state(pose)[0]),
            lambda: np.asarray(caster.render_blur([pose] * 8, [1.0] + [0.0] * 7)))


@pytest.mark.parametrize("ss", [1, 2])
def test_short_normals_keep_their_direction(ground, ss):
    """Vertex normals of length 2^-65, whose squares are denormal: the squared
    length keeps 19 bits, an error that the second normalization of a lit sample
    takes out again, so the image is that of the unit normals to float rounding."""
    V, N, I = ground
    want = renders(DeviceScene(V, N, I, CAM, ss, HAPKE))
    got = renders(DeviceScene(V, np.asarray(N) * np.float32(2.0 ** -65), I, CAM, ss, HAPKE))
    for g, w in zip(got, want):
        g, w = g(), w()
        assert (w > 0).mean() > 0.5
        np.testing.assert_allclose(g, w, rtol=1e-5, atol=0)
