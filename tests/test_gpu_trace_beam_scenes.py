"""Items that share a walk of the tree against the walk per packet (see
test_gpu_trace_beam.py, whose tolerance this is) on geometry that a terrain
seen from above does not have: the inside of a bowl, a mesh whose triangles
all lie twice in the same place, suns along an axis (whose inverse direction is
clamped, and whose sign may differ between cells) and suns so low that the
shadow side reaches more leaves than a list holds.  And a batch of members with
and without shared walks in one launch, against the members alone.
"""
import math

import numpy as np
import pytest

from dvsrender4deepspace_gb300 import DeviceScene, EventSensor, SensorBatch, terrain, trajectory
from tests.test_gpu_batch import physic

pytestmark = pytest.mark.gpu

HAPKE = dict(b=0.3, c=0.4, hS=0.06, hC=1.0, thetap=0.349066, w=0.25, B_S0=1.0, B_C0=0.0, phi=0.3)


def bowl(n, radius):
    """A sphere open above 45 degrees, its normals inward, about the origin."""
    V, I = [], []
    for i in range(n + 1):
        theta = math.pi * (1.0 - 0.75 * i / n)  # from the bottom up
        for j in range(2 * n):
            phi = math.pi * j / n
            V.append((math.sin(theta) * math.cos(phi), math.sin(theta) * math.sin(phi), math.cos(theta)))
    for i in range(n):
        for j in range(2 * n):
            a, b = i * 2 * n + j, i * 2 * n + (j + 1) % (2 * n)
            I += [(a, b, b + 2 * n), (a, b + 2 * n, a + 2 * n)]
    V = np.array(V, np.float32)
    return V * np.float32(radius), -V, np.array(I, np.uint32)


def mesh(kind):
    if kind == "bowl":
        return bowl(40, 300.0)
    V, N, I = terrain.terrain_mesh(96, seed=4)
    V, N, I = (np.asarray(a).reshape(-1, 3) for a in (V, N, I))
    if kind == "twice":
        return np.concatenate([V, V]), np.concatenate([N, N]), np.concatenate([I, I + len(V)])
    return V, N, I


@pytest.mark.parametrize("geometry", [0, 3])
@pytest.mark.parametrize("kind,light,position,ss,cells", [
    ("bowl", trajectory.sun_direction(60, 20), (20.0, -30.0, 40.0), 4, 40),
    ("bowl", (0.0, 0.0, 1.0), (0.0, 0.0, 0.0), 3, 33),
    ("twice", trajectory.sun_direction(30, 70), (31.0, -17.0, 500.0), 2, 64),
    ("ground", (0.0, 0.0, 1.0), (31.0, -17.0, 500.0), 4, 40),
    ("ground", (1.0, 0.0, 0.0), (31.0, -17.0, 500.0), 2, 40),
    ("ground", trajectory.sun_direction(2, 40), (31.0, -17.0, 900.0), 4, 64),
])
def test_shared_walks_change_no_circuit(kind, light, position, ss, cells, geometry):
    V, N, I = mesh(kind)
    cam = dict(width=96, height=64, fx=70.0, fy=70.0, cx=48.0, cy=32.0)
    scene = DeviceScene(V, N, I, cam, ss, HAPKE, geometry=geometry)
    traj = trajectory.StraightPass(position, (60.0, 25.0, 0.0), light, 1000.0, 0.3)
    ivs = trajectory.horizons(traj, 0.0, 1e-6, cells)
    states = {}
    for cw in (4, 32):
        s = EventSensor(scene, physic(photon_shot_noise=0, threshold_std=0))
        s.set_tuning(cw, 1)
        s.initialize(traj.state(0.0), 0.0)
        s.process_many(ivs)
        st = s.stats()
        states[cw] = (s.read_state(), st["primary_rays"], st["shadow_rays"])
    (a, pa), prim_a, shad_a = states[4]
    (b, pb), prim_b, shad_b = states[32]
    assert prim_a == prim_b and shad_a == shad_b > 0
    np.testing.assert_allclose(b[:, 0], a[:, 0], rtol=0, atol=1e-9)
    np.testing.assert_array_equal(pb, pa)
    assert np.ptp(a[:, 0]) > 0.1


def test_batch_of_members_with_and_without_shared_walks():
    V, N, I = mesh("ground")
    cameras = [(dict(width=96, height=64, fx=70.0, fy=70.0, cx=48.0, cy=32.0), 4, 64),  # items of many packets
               (dict(width=40, height=30, fx=40.0, fy=40.0, cx=20.0, cy=15.0), 1, 3),   # packets of ten pixels
               (dict(width=31, height=17, fx=30.0, fy=30.0, cx=15.5, cy=8.5), 3, 12)]
    base = DeviceScene(V, N, I, cameras[0][0], 1, HAPKE)
    traj = trajectory.StraightPass((31.0, -17.0, 500.0), (60.0, 25.0, 0.0), trajectory.sun_direction(30, 70), 1000.0, 0.3)

    def members():
        out = []
        for cam, ss, _ in cameras:
            s = EventSensor(base.view(cam, ss), physic(), circuit_precision="fp32")
            s.initialize(traj.state(0.0), 0.0)
            out.append(s)
        return out
    plan, t = [], [0.0] * len(cameras)
    for step in range(2):
        row = []
        for m, (_, _, cells) in enumerate(cameras):
            ivs = trajectory.horizons(traj, t[m], 1e-6, cells)
            t[m] = ivs[-1][3]
            row.append(ivs)
        plan.append(row)
    alone, batched = members(), members()
    batch = SensorBatch(batched)
    for row in plan:
        together = batch.process(row)
        for m, s in enumerate(alone):
            single = s.process_many(row[m])
            for f in single.dtype.names:
                np.testing.assert_array_equal(together[m][f], single[f])
    for a, b in zip(alone, batched):
        np.testing.assert_array_equal(a.read_state()[0], b.read_state()[0])
        assert a.stats()["primary_rays"] == b.stats()["primary_rays"]
    batch.close()
