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


@pytest.mark.parametrize("width", [1e-33, 1e-36, 1e-39, 1e-44])
def test_opposition_surge_of_no_width(ground, width):
    """The surge 1 / (1 + tan(g/2) / hS) is below 1e-15 for every ray of this view at hS = 1e-20 and below."""
    V, N, I = ground
    base = DeviceScene(V, N, I, CAM, 2, dict(HAPKE, hS=1e-20))
    for g, w in zip(renders(base.view(CAM, 2, dict(HAPKE, hS=width))), renders(base)):
        w = w()
        assert (w > 0).mean() > 0.5
        np.testing.assert_array_equal(g(), w)


def test_infinite_porosity_factor_is_reported(ground):
    """K = -log(1 - p) / p is infinite where p = 1.209 phi^(2/3) rounds to 1:
    lit samples are then infinite, and the call reports them as before."""
    V, N, I = ground
    base = DeviceScene(V, N, I, CAM, 1, HAPKE)
    phi, reported = np.float32((1.0 / 1.209) ** 1.5), 0
    for _ in range(8):
        phi = np.nextafter(phi, np.float32(0))
    for _ in range(17):
        errors = 0
        for render in renders(base.view(CAM, 1, dict(HAPKE, phi=float(phi)))):
            try:
                render()
            except OpticalError:
                errors += 1
        assert errors in (0, 2)
        reported += errors == 2
        phi = np.nextafter(phi, np.float32(1))
    assert reported > 0


def test_lobe_without_width_is_reported():
    """b = 1 - 2^-13: at opposition (sun behind the camera, nadir pixel)
    1 - 2 b + b^2 rounds to 0 in floats, and the forward lobe is infinite."""
    V = np.array([[-100, -100, 0], [100, -100, 0], [100, 100, 0], [-100, 100, 0]], np.float32)
    N = np.tile(np.float32([0, 0, 1]), (4, 1))
    I = np.array([[0, 1, 2], [0, 2, 3]], np.uint32)
    cam = dict(width=3, height=3, fx=10.0, fy=10.0, cx=1.0, cy=1.0)  # one ray a pixel: the middle one looks along -z
    pose = dict(position=(1.0, 2.0, 10.0), rotation=(0, 0, 0, 1), light=(0, 0, 1), intensity=1000)
    b = np.float32(1.0 - 2.0 ** -13)
    assert np.float32(np.float32(1) - np.float32(2) * b) + b * b == 0
    scene = DeviceScene(V, N, I, cam, 1, dict(HAPKE, b=float(b), c=0.5, thetap=0.0))
    for render in renders(scene, pose):
        with pytest.raises(OpticalError):
            render()
