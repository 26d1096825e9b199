"""Per-vertex albedo through every sampler that reads it, against the FP64
oracle's image of the same mesh: frames (one and several sub-rays a pixel), the
temporal packets of an exposure, a sensor's cells traced in items with and
without a shared walk, and the adaptive solver's probes.  The albedo runs over
0.05..0.95 with some values outside [0, 1], which fall back to the material's.
Radiance within the stated 1e-5 outside the oracle's margin classes; log
voltages, whose static light the receptor holds, within 2e-5.
"""
import numpy as np
import pytest

from dvsrender4deepspace_gb300 import CamRayCaster, DeviceScene, EventSensor, terrain, trajectory
from oracle import oracle as O
from tests.test_gpu_batch import physic

pytestmark = pytest.mark.gpu

HAPKE = dict(b=0.3, c=0.4, hS=0.06, hC=1.0, thetap=0.349066, w=0.25, B_S0=1.0, B_C0=0.0, phi=0.3)
POSE = trajectory.StraightPass((5.0, -8.0, 350.0), (0.0, 0.0, 0.0), trajectory.sun_direction(40, 40), 1000.0, 0.4).state(0)


def ground():
    V, N, I = terrain.terrain_mesh(48, seed=3)
    albedo = np.random.default_rng(5).uniform(0.05, 0.95, len(np.asarray(V).reshape(-1, 3))).astype(np.float32)
    albedo[::17] = -1.0
    albedo[::29] = 1.5
    return V, N, I, albedo


@pytest.mark.parametrize("ss,geometry", [(1, 0), (2, 3), (5, 1), (6, 2)])
def test_albedo_through_frames_sensors_and_probes(ss, geometry):
    V, N, I, albedo = ground()
    cam = dict(width=43, height=31, fx=40.0, fy=40.0, cx=21.5, cy=15.5)
    scene = DeviceScene(V, N, I, cam, ss, HAPKE, albedos=albedo, geometry=geometry)
    want, _, flags = O.OracleScene(V, N, I, cam, ss, HAPKE, albedos=albedo, fp64=True).render_margin(POSE)
    plain, lit = flags == 0, want > 0
    assert (plain & lit).sum() > 300
    uniform = O.OracleScene(V, N, I, cam, ss, HAPKE, fp64=True).render(POSE)[0]
    assert np.median(np.abs(uniform[plain & lit] / want[plain & lit] - 1)) > 0.2
    caster = CamRayCaster(scene)
    frame = np.asarray(caster.render_state(POSE)[0]).ravel()
    exposure = np.asarray(caster.render_blur([POSE] * 8, [1.0] + [0.0] * 7)).ravel()
    for image in (frame, exposure):
        np.testing.assert_allclose(image[plain], want[plain], rtol=1e-5, atol=0)
    np.testing.assert_allclose(exposure, frame, rtol=1e-6, atol=0)

    # under constant light the receptor stays where the frame's radiance put it, whichever way the cells are traced
    phys = physic(photon_shot_noise=0, threshold_std=0)
    ivs = trajectory.horizons(trajectory.StraightPass((5.0, -8.0, 350.0), (0.0, 0.0, 0.0),
                                                      trajectory.sun_direction(40, 40), 1000.0, 0.4), 0.0, 1e-6, 64)
    states = []
    for tuning in (None, (4, 1), (32, 1)):
        s = EventSensor(scene, phys)
        s.initialize(POSE, 0.0)
        start = s.read_state()[0][:, 0]
        if tuning:
            s.set_tuning(*tuning)
            s.process_many(ivs)
        else:
            # a pulse within the window makes the solver probe between the horizons' ends
            a = dict(POSE, intensity_rate=1e7)
            b = dict(POSE, intensity_rate=-1e7)
            s.process_adaptive(ivs[:32] + [(a, b, ivs[31][3], ivs[31][3] + 1e-4)], 1e-3)
            assert s.refinement_statistics()["traced_pixel_samples"] > 6 * 43 * 31
            native = EventSensor(scene, phys)
            native.initialize(POSE, 0.0)
            native.process_many(ivs[:32] + [(a, b, ivs[31][3], ivs[31][3] + 1e-4)])
            np.testing.assert_allclose(s.read_state()[0][:, 0], native.read_state()[0][:, 0], rtol=0, atol=1e-3)
            continue
        np.testing.assert_allclose(s.read_state()[0][plain, 0], start[plain], rtol=0, atol=2e-5)
        states.append(s.read_state()[0][:, 0])
    np.testing.assert_allclose(states[1], states[0], rtol=0, atol=1e-9)
