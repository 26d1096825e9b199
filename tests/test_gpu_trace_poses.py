"""Traces of few poses (camera frames; sub-rays of one or more pixels in a
packet) against the temporal packets of eight equal poses, and the depths of
events against a frame's.

The eight-pose exposure with the weights 1, 0, ... is the frame's image through
trace_cells_kernel.  Every ray and every sum is the same arithmetic in the same
order, so the images are equal up to exact ties in hit distance (two triangles
with a common edge: 1e-7 of a sub-ray).
"""
import numpy as np
import pytest

from dvsrender4deepspace_gb300 import CamRayCaster, DeviceScene, EventSensor, terrain, trajectory
from tests.test_gpu_batch import physic
from tests.test_gpu_trace_beam import Tilted

pytestmark = pytest.mark.gpu

HAPKE = dict(b=0.3, c=0.4, hS=0.06, hC=1.0, thetap=0.349066, w=0.25, B_S0=1.0, B_C0=0.0, phi=0.3)


@pytest.fixture(scope="module")
def scenes():
    V, N, I = terrain.terrain_mesh(96, seed=11)
    tiny = dict(width=2, height=2, fx=2.0, fy=2.0, cx=1.0, cy=1.0)
    return {g: DeviceScene(V, N, I, tiny, 1, HAPKE, geometry=g) for g in range(4)}


# one sub-ray: lone pixels, a part of a packet, several items, and enough pixels for full packets; then sub-ray counts
# below, at and above a packet's 32 lanes, odd ones, and images large enough for items of many pixels
@pytest.mark.parametrize("width,height,ss,geometry", [
    (1, 1, 1, 0), (7, 5, 1, 3), (64, 48, 1, 2), (330, 240, 1, 0), (3, 3, 2, 0), (200, 150, 2, 3), (121, 91, 3, 1),
    (200, 150, 4, 0), (65, 33, 5, 2), (31, 7, 6, 0), (160, 121, 6, 3), (40, 31, 9, 1), (5, 3, 17, 0), (320, 200, 8, 3)])
@pytest.mark.parametrize("tilt", [0.0, 0.5])
def test_frames_equal_the_temporal_packets(scenes, width, height, ss, geometry, tilt):
    cam = dict(width=width, height=height, fx=0.9 * width, fy=0.9 * width, cx=width / 2, cy=height / 2)
    caster = CamRayCaster(scenes[geometry].view(cam, ss))
    pose = Tilted(450.0, tilt, 0.6 if tilt else 0.0).state(0.0)
    image, depth = caster.render_state(pose)
    want = caster.render_blur([pose] * 8, [1.0] + [0.0] * 7)
    np.testing.assert_allclose(image, want, rtol=1e-6, atol=0)
    assert np.all((depth > 0) | (depth == -1.0))
    assert (depth > 0).any() or width == 1  # the one wide pixel, tilted, looks past the terrain


@pytest.mark.parametrize("ss,geometry", [(1, 0), (3, 2), (4, 1), (6, 3)])
def test_event_depths_equal_a_frame(scenes, ss, geometry):
    cam = dict(width=37, height=29, fx=40.0, fy=40.0, cx=18.5, cy=14.5)
    view = scenes[geometry].view(cam, ss)
    pose = trajectory.StraightPass((40.0, 25.0, 420.0), (0.0, 0.0, 0.0), trajectory.sun_direction(35, 50), 1000.0, 0.3).state(0)
    sensor = EventSensor(view, physic(photon_shot_noise=0))
    sensor.initialize(pose, 0.0)
    ev = sensor.process((dict(pose, intensity_rate=8e6), dict(pose, intensity_rate=-8e6), 0.0, 2e-3))
    assert len(ev) > 500
    depth = CamRayCaster(view).render_state(pose)[1].reshape(29, 37)
    # the sensor renormalizes the pose's quaternion, whose last bit may move the ray
    np.testing.assert_allclose(ev["depth"], depth[ev["y"], ev["x"]], rtol=2e-6)
