"""The autotuner on batches of so few cells that their trace is laid out by
poses: every packet shape would run the same kernel, so none is timed and the
sensor's stays automatic.  And adaptive windows whose fallback pixels are traced a few
cells at a time (scattered pixels by pose), against the same window in one chunk.
"""
import numpy as np
import pytest

from dvsrender4deepspace_gb300 import DeviceScene, EventSensor, terrain, trajectory
from tests.test_gpu_batch import physic

pytestmark = pytest.mark.gpu

HAPKE = dict(b=0.3, c=0.4, hS=0.06, hC=1.0, thetap=0.349066, w=0.25, B_S0=1.0, B_C0=0.0, phi=0.3)


@pytest.mark.parametrize("ss,cells,timed", [(2, 5, False), (1, 7, False), (4, 1, False), (2, 8, True)])
def test_batches_traced_by_pose_have_no_shapes_to_time(ss, cells, timed):
    V, N, I = terrain.terrain_mesh(64, seed=3)
    cam = dict(width=64, height=48, fx=60.0, fy=60.0, cx=32.0, cy=24.0)
    traj = trajectory.StraightPass((5.0, -8.0, 350.0), (80.0, 10.0, 0.0), trajectory.sun_direction(30, 40), 1000.0, 0.4)
    s = EventSensor(DeviceScene(V, N, I, cam, ss, HAPKE), physic())
    s.initialize(traj.state(0.0), 0.0)
    ivs = trajectory.horizons(traj, 0.0, 1e-6, cells)
    tuned = s.autotune(ivs)
    assert (tuned["candidates"] > 0) == timed and (tuned["best_ms"] > 0) == timed
    assert tuned["rays_per_lane"] in (1, 2, 4) and tuned["cells_per_warp"] >= 1
    assert np.isfinite(s.read_state()[0][:, 0]).all()
    s.process_many(ivs)


@pytest.mark.parametrize("ss", [1, 3])
def test_fallback_pixels_a_few_cells_at_a_time(ss):
    V, N, I = terrain.terrain_mesh(48, seed=3)
    cam = dict(width=96, height=72, fx=90.0, fy=90.0, cx=48.0, cy=36.0)
    scene = DeviceScene(V, N, I, cam, ss, HAPKE)
    traj = trajectory.StraightPass((5.0, -8.0, 350.0), (80.0, 10.0, 0.0), trajectory.sun_direction(30, 40), 1000.0, 0.4)
    ivs = [(dict(a, intensity_rate=2e8), dict(b, intensity_rate=-2e8), t0, t1)
           for a, b, t0, t1 in trajectory.horizons(traj, 0.0, 1e-5, 150)]
    got = []
    for chunk in (0, 7):
        s = EventSensor(scene, physic(photon_shot_noise=0), cells_per_chunk=chunk)
        s.initialize(traj.state(0.0), 0.0)
        events = s.process_adaptive(ivs, 1e-11)
        assert s.refinement_statistics()["fallback_pixels"] > 32 * 4864 // 32  # enough for full packets
        got.append((events, s.read_state()[0]))
    (ea, sa), (eb, sb) = got
    assert len(ea) == len(eb) > 0
    np.testing.assert_allclose(sb, sa, rtol=0, atol=1e-9)  # exact ties in hit distance only
