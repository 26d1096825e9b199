"""Cells of no length.  An interval is cut into equal cells, and where a cell is
shorter than the spacing of doubles at its time -- steps of 0.1 us at the
seconds of a calendar clock -- both its ends round to the same double.  Such
a cell lets nothing pass: the intervals are accepted, and a sensor alone (whose
Philox counts are drawn ahead) gives the events and states of the same sensor in
a batch (drawn in the circuit), bit for bit.
"""
import numpy as np
import pytest

from dvsrender4deepspace_gb300 import DeviceScene, EventSensor, SensorBatch, terrain, trajectory
from tests.test_gpu_batch import physic

pytestmark = pytest.mark.gpu

HAPKE = dict(b=0.3, c=0.4, hS=0.06, hC=1.0, thetap=0.349066, w=0.25, B_S0=1.0, B_C0=0.0, phi=0.3)


def zero_length_cells(ivs, step):
    """How many of the intervals' cells have equal ends, as the sensor forms them."""
    zero = 0
    for _, _, t0, t1 in ivs:
        n = int(np.ceil((t1 - t0) / float(np.float32(step))))
        ends = [t0 + k * ((t1 - t0) / n) for k in range(n)] + [t1]
        zero += sum(a == b for a, b in zip(ends, ends[1:]))
    return zero


@pytest.mark.parametrize("circuit", ["fp32-philox", "fp32", "fp64"])
@pytest.mark.parametrize("start,horizon,step", [(1.7e9, 1e-6, 1e-7), (2.0 ** 33, 1e-5, 1e-6)])
def test_cells_of_no_length_pass(circuit, start, horizon, step):
    V, N, I = terrain.terrain_mesh(48, seed=3)
    cam = dict(width=33, height=21, fx=30.0, fy=30.0, cx=16.5, cy=10.5)
    base = DeviceScene(V, N, I, cam, 2, HAPKE)
    traj = trajectory.StraightPass((5.0, -8.0, 350.0), (0.0, 0.0, 0.0), trajectory.sun_direction(30, 40), 1e5, 0.4)
    ivs = trajectory.horizons(traj, start, horizon, 20)
    assert zero_length_cells(ivs, step) > 20
    pulse = traj.state(ivs[-1][3])
    ivs.append((dict(pulse, intensity_rate=4e8), dict(pulse, intensity_rate=-4e8), ivs[-1][3], ivs[-1][3] + 2e-4))
    got = []
    for batched in (False, True):
        s = EventSensor(base.view(cam, 2), physic(circuit_step=step), circuit_precision=circuit)
        s.initialize(traj.state(0.0), start)
        if batched:
            b = SensorBatch([s])
            events = b.process([ivs])[0]
            b.close()
        else:
            events = s.process_many(ivs)
        got.append((events, s.read_state()))
    (ea, (sa, pa)), (eb, (sb, pb)) = got
    for f in ea.dtype.names:
        np.testing.assert_array_equal(ea[f], eb[f])
    np.testing.assert_array_equal(sa, sb)
    np.testing.assert_array_equal(pa, pb)
    assert np.isfinite(sa[:, 0]).all() and len(ea) > 0
