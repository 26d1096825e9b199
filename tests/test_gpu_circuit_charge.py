"""The FP64 circuit's receptor step for either sign of the charge scale (a
negative temperature or subthreshold slope makes it negative; the parameters
are accepted) against the receptor's closed form
1/x' = 1/r + (1/x - 1/r) e^-K, K = r T / charge, on both sides of the step's
two forms in |K| per cell, and through the refinement's verdicts, which use the
same step.  Tolerance as in test_gpu_circuit_run.py.
"""
import numpy as np
import pytest

from dvsrender4deepspace_gb300 import DeviceScene, EventSensor
from dvsrender4deepspace_gb300.raycast import derive_parameters
from tests.test_gpu_batch import physic
from tests.test_gpu_parity import plane_mesh
from tests.test_oracle_golden import DAVIS_HAPKE, POSE

pytestmark = pytest.mark.gpu

CAM = dict(width=16, height=12, fx=30.0, fy=30.0, cx=8.0, cy=6.0)


def sensors(temperature, **over):
    V, N, I = plane_mesh()
    scene = DeviceScene(V, N, I, CAM, 1, DAVIS_HAPKE)
    phys = physic(**dict(dict(photon_shot_noise=0, threshold_std=0, threshold_pos=1e3, threshold_neg=1e3,
                              dark_current_a=0, temperature_k=temperature), **over))

    def sensor(intensity):
        s = EventSensor(scene, phys)
        s.initialize(dict(POSE, intensity=intensity), 0.0)
        return s
    return sensor, derive_parameters(phys)["charge_scale"]


@pytest.mark.parametrize("temperature,share", [(-300, 0.02), (300, 0.02), (-300, 0.5), (300, 0.5)])
def test_receptor_step_of_either_charge(temperature, share):
    sensor, charge = sensors(temperature)
    assert (charge < 0) == (temperature < 0)
    base = np.exp(sensor(1000.0).read_state()[0][:, 0])  # electrons a second at intensity 1000
    cells, step = 8, float(np.float32(1e-6))
    after = 1000.0 * share * abs(charge) / (step * base.mean())  # |K| of a cell is about `share`
    u0 = sensor(0.5 * after).read_state()[0][:, 0]
    rate = np.exp(np.longdouble(1) * sensor(after).read_state()[0][:, 0])
    s, st = sensor(0.5 * after), dict(POSE, intensity=after)
    assert len(s.process_many([(st, st, k * step, (k + 1) * step) for k in range(cells)])) == 0
    K = rate * np.longdouble(cells * step) / np.longdouble(charge)
    want = -np.log(1 / rate + (np.exp(-u0.astype(np.longdouble)) - 1 / rate) * np.exp(-K))
    assert np.abs(K).min() > 0.1
    np.testing.assert_allclose(s.read_state()[0][:, 0], want.astype(np.float64), rtol=0, atol=7e-13)


def test_refinement_sees_a_negative_charge():
    """A light that doubles in the window moves the receptors apart under a charge of either sign, so the
    initial probes do not do for it."""
    for temperature in (300, -300):
        sensor, charge = sensors(temperature, threshold_pos=0.05, threshold_neg=0.05)
        s = sensor(1000.0)
        ivs = [(dict(POSE, intensity_rate=8e6), dict(POSE, intensity_rate=-8e6), 0.0, 2e-3)]
        try:
            s.process_adaptive(ivs, 10.0)
        except RuntimeError:
            assert temperature < 0  # the circuit itself may leave the range of the log
        assert s.refinement_statistics()["traced_pixel_samples"] > 5 * 192
