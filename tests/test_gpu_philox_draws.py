"""The Philox circuit's photon counts drawn ahead, a thread per pixel-cell,
against the same draws inside the circuit: a sensor alone draws ahead, as a
batch's only member it does not.  A draw depends on its pixel and cell alone, so
events and states are the same bits, for pixel and cell counts around a block's
128 threads and over several batches; with reset noise both draw in the circuit.
"""
import numpy as np
import pytest

from dvsrender4deepspace_gb300 import DeviceScene, EventSensor, SensorBatch, terrain, trajectory
from tests.test_gpu_batch import physic

pytestmark = pytest.mark.gpu

HAPKE = dict(b=0.3, c=0.4, hS=0.06, hC=1.0, thetap=0.349066, w=0.25, B_S0=1.0, B_C0=0.0, phi=0.3)


@pytest.mark.parametrize("width,height,ss,cells", [(1, 1, 2, 1), (16, 8, 1, 3), (43, 3, 1, 64), (33, 31, 2, 97)])
@pytest.mark.parametrize("reset_noise", [0, 1])
def test_draws_ahead_equal_draws_in_the_circuit(width, height, ss, cells, reset_noise):
    V, N, I = terrain.terrain_mesh(48, seed=3)
    cam = dict(width=width, height=height, fx=30.0, fy=30.0, cx=width / 2, cy=height / 2)
    base = DeviceScene(V, N, I, cam, ss, HAPKE)
    traj = trajectory.StraightPass((5.0, -8.0, 350.0), (80.0, 10.0, 0.0), trajectory.sun_direction(30, 40), 1e5, 0.4)
    phys = physic(reset_thermal_noise=reset_noise)
    got = []
    for batched in (False, True):
        s = EventSensor(base.view(cam, ss), phys, circuit_precision="fp32-philox")
        s.initialize(traj.state(0.0), 0.0)
        b = SensorBatch([s]) if batched else None
        events, t = [], 0.0
        for k in range(2):
            ivs = trajectory.horizons(traj, t, 1e-6, cells)
            t = ivs[-1][3]
            a, e = traj.state(t), traj.state(t + 2e-4)
            ivs.append((dict(a, intensity_rate=4e8), dict(e, intensity_rate=-4e8), t, t + 2e-4))
            t += 2e-4
            events.append(b.process([ivs])[0] if batched else s.process_many(ivs))
        got.append((np.concatenate(events), s.read_state()))
        if b:
            b.close()
    (ea, (sa, pa)), (eb, (sb, pb)) = got
    for f in ea.dtype.names:
        np.testing.assert_array_equal(ea[f], eb[f])
    np.testing.assert_array_equal(sa, sb)
    np.testing.assert_array_equal(pa, pb)
    assert len(ea) > 0
