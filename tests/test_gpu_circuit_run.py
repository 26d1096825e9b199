"""The FP64 circuit over runs of cells without events, against the receptor's
closed form: u(T) = -log(e^-K / e^u0 + (1 - e^-K) / r), K = r T / charge, at a
constant rate r, and u0 - log1p(e^u0 T / charge) without light, whatever the
cells T is cut into.  Each cell rounds about ten FP64 operations (1e-15
relative), so 640 cells stay within 7e-13 of it.  The light sets K per cell on
both sides of the step's two forms (the series below 0.35).
"""
import numpy as np
import pytest

from dvsrender4deepspace_gb300 import DeviceScene, EventSensor, terrain, trajectory
from dvsrender4deepspace_gb300.raycast import derive_parameters
from tests.test_gpu_batch import physic

pytestmark = pytest.mark.gpu

HAPKE = dict(b=0.3, c=0.4, hS=0.06, hC=1.0, thetap=0.349066, w=0.25, B_S0=1.0, B_C0=0.0, phi=0.3)


@pytest.mark.parametrize("before,after,cells", [
    (1000.0, 3000.0, 640), (3000.0, 1000.0, 1), (2e5, 5e5, 640), (1e6, 4e7, 33), (4e7, 1e3, 640), (1e5, 0.0, 640)])
def test_receptor_follows_its_closed_form(before, after, cells):
    V, N, I = terrain.terrain_mesh(48, seed=3)
    cam = dict(width=24, height=17, fx=30.0, fy=30.0, cx=12.0, cy=8.5)
    scene = DeviceScene(V, N, I, cam, 2, HAPKE)
    phys = physic(photon_shot_noise=0, threshold_std=0, threshold_pos=1e3, threshold_neg=1e3, dark_current_a=0)
    pose = trajectory.StraightPass((5.0, -8.0, 350.0), (0.0, 0.0, 0.0), trajectory.sun_direction(30, 40), 1.0, 0.4).state(0)

    def sensor(intensity):
        s = EventSensor(scene, phys)
        s.initialize(dict(pose, intensity=intensity), 0.0)
        return s
    u0 = sensor(before).read_state()[0][:, 0]
    rate = np.exp(np.longdouble(1) * sensor(after).read_state()[0][:, 0]) if after else np.zeros(len(u0), np.longdouble)
    lit = u0 > 0
    assert lit.sum() > 50
    s, t, step = sensor(before), 0.0, float(np.float32(1e-6))
    for n in (cells // 2, cells - cells // 2):  # two batches: the run is cut once
        if n:
            st = dict(pose, intensity=after)
            assert len(s.process_many([(st, st, t + k * step, t + (k + 1) * step) for k in range(n)])) == 0
            t += n * step
    got = s.read_state()[0][:, 0]
    charge = np.longdouble(derive_parameters(phys)["charge_scale"])
    x, T = np.exp(np.longdouble(1) * u0[lit]), np.longdouble(t)
    if after:
        K = rate[lit] * T / charge
        want = -np.log(np.exp(-K) / x - np.expm1(-K) / rate[lit])
    else:
        want = -np.log(1 / x + T / charge)
    np.testing.assert_allclose(got[lit].astype(np.float64), want.astype(np.float64), rtol=0, atol=7e-13)
