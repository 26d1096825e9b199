"""Traces whose warps share one walk of the tree (beams) against the walk per
packet, through sensors that differ only in their packet shape.

Four cells per warp never use beams; 32 do wherever a warp's item holds enough
packets.  The leaves a ray tests are the same either way, so the circuits are
driven by the same radiance up to exact ties in hit distance, whose two
triangles share the edge (1e-7 of one sub-ray): the receptor's log voltage then
moves by less than 1e-9, while a missing leaf would move it by 1e-4 and more.
"""
import math

import numpy as np
import pytest

from dvsrender4deepspace_gb300 import DeviceScene, EventSensor, terrain, trajectory
from tests.test_gpu_batch import physic

pytestmark = pytest.mark.gpu


class Tilted:
    """A straight pass whose camera looks off nadir."""

    def __init__(self, altitude, tilt, yaw):
        self.p = trajectory.StraightPass((31.0, -17.0, altitude), (60.0, 25.0, 0.0), trajectory.sun_direction(25, 70),
                                         1000.0, yaw)
        self.tilt = tilt

    def state(self, t):
        s = self.p.state(t)
        x, y, z, w = s["rotation"]
        a, b = math.sin(self.tilt / 2), math.cos(self.tilt / 2)
        # yaw, then a tilt about the camera's x axis
        s["rotation"] = (w * a + x * b, y * b + z * a, z * b - y * a, w * b - x * a)
        return s


@pytest.mark.parametrize("width,height,fx,ss,cells,geometry,altitude,tilt,yaw", [
    (346, 260, 300.0, 1, 64, 0, 900.0, 0.0, 0.0),     # one sub-ray: items of several pixels and both cell groups;
                                                      # axis-aligned view: directions that change sign in an item
    (346, 260, 300.0, 1, 97, 3, 900.0, 0.3, 0.7),     # a last cell group of one cell
    (160, 120, 150.0, 3, 33, 2, 600.0, 0.2, 0.4),     # odd sub-ray count
    (96, 64, 90.0, 4, 640, 0, 700.0, 0.0, 1.1),       # many cell groups an item
    (64, 48, 50.0, 4, 40, 1, 2500.0, 0.5, 0.3),       # wide pixels: more leaves than a list holds
    (40, 30, 400.0, 16, 13, 3, 800.0, 0.9, 0.2),      # a view past the terrain: empty lists
    (40, 30, 400.0, 16, 13, 3, 400.0, 0.6, 0.2),      # narrow pixels, oblique view; eight cells a warp
    (31, 17, 30.0, 5, 8, 0, 500.0, 1.2, 0.0),         # rays over the horizon
])
def test_beams_change_no_circuit(width, height, fx, ss, cells, geometry, altitude, tilt, yaw):
    V, N, I = terrain.terrain_mesh(128, seed=4)
    cam = dict(width=width, height=height, fx=fx, fy=fx, cx=width / 2, cy=height / 2)
    hap = dict(b=0.3, c=0.4, hS=0.06, hC=1.0, thetap=0.349066, w=0.25, B_S0=1.0, B_C0=0.0, phi=0.3)
    scene = DeviceScene(V, N, I, cam, ss, hap, geometry=geometry)
    traj = Tilted(altitude, tilt, yaw)
    ivs = trajectory.horizons(traj, 0.0, 1e-6, cells)
    phys = physic(photon_shot_noise=0, threshold_std=0)
    states = {}
    for cw in (4, 32):
        s = EventSensor(scene, phys)
        s.set_tuning(cw, 1)
        s.initialize(traj.state(0.0), 0.0)
        s.process_many(ivs)
        st = s.stats()
        states[cw] = (s.read_state(), st["primary_rays"], st["shadow_rays"])
    (a, pa), prim_a, shad_a = states[4]
    (b, pb), prim_b, shad_b = states[32]
    assert prim_a == prim_b and shad_a == shad_b
    np.testing.assert_allclose(b[:, 0], a[:, 0], rtol=0, atol=1e-9)
    np.testing.assert_array_equal(pb, pa)
    assert np.isfinite(a[:, 0]).all()
    assert shad_a > 0 or altitude * math.tan(tilt) > 900.0
