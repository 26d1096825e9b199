"""The adaptive solver's refinement, one warp per pixel: a sensor against its
own row bands, whose pixels meet other warps, other neighbours and a shorter
last block.  Knots, exact segments, fallbacks and probe counts belong to a
pixel alone, so the bands' statistics add up to the sensor's and every pixel's
circuit state is the same bits, whether its window takes five probes, many
bisections, exact segments or more knots than fit.
"""
import numpy as np
import pytest

from dvsrender4deepspace_gb300 import DeviceScene, EventSensor, terrain, trajectory
from tests.test_gpu_batch import physic

pytestmark = pytest.mark.gpu

HAPKE = dict(b=0.3, c=0.4, hS=0.06, hC=1.0, thetap=0.349066, w=0.25, B_S0=1.0, B_C0=0.0, phi=0.3)


def run(scene, traj, phys, ivs, tolerance, rows):
    s = EventSensor(scene, phys, row_begin=rows[0], row_end=rows[1])
    s.initialize(traj.state(0.0), 0.0)
    assert s.process_adaptive(ivs, tolerance) is not None
    return s.read_state()[0], s.refinement_statistics()


@pytest.mark.parametrize("ss,geometry,horizons,pulse,tolerance", [
    (1, 0, 40, 0.0, 1e-2),      # nothing to bisect
    (1, 3, 100, 2e7, 1e-2),     # two rays a split
    (3, 2, 60, 2e7, 1e-3),      # packets that straddle probes
    (4, 0, 60, 2e7, 1e-2),      # a split is one packet
    (5, 1, 30, 2e7, 1e-2),      # more sub-rays than are summed at a time
    (2, 0, 190, 2e7, 1e-11),    # more knots than fit: fallback pixels
])
def test_bands_refine_as_the_whole_sensor(ss, geometry, horizons, pulse, tolerance):
    V, N, I = terrain.terrain_mesh(48, seed=3)
    cam = dict(width=31, height=9, fx=30.0, fy=30.0, cx=15.5, cy=4.5)
    scene = DeviceScene(V, N, I, cam, ss, HAPKE, geometry=geometry)
    traj = trajectory.StraightPass((5.0, -8.0, 350.0), (80.0, 10.0, 0.0), trajectory.sun_direction(30, 40), 1000.0, 0.4)
    ivs = trajectory.horizons(traj, 0.0, 1e-5, horizons - 1)
    a, b = traj.state(ivs[-1][3]), traj.state(ivs[-1][3] + 1e-5)
    ivs.append((dict(a, intensity_rate=pulse), dict(b, intensity_rate=-pulse), ivs[-1][3], ivs[-1][3] + 1e-5))
    phys = physic(photon_shot_noise=0)
    whole, stats = run(scene, traj, phys, ivs, tolerance, (0, 9))
    bands = [run(scene, traj, phys, ivs, tolerance, rows) for rows in ((0, 2), (2, 3), (3, 9))]
    np.testing.assert_array_equal(np.concatenate([b[0] for b in bands]), whole)
    for k in ("traced_pixel_samples", "fallback_pixels", "exact_segments", "native_cell_queries"):
        assert sum(b[1][k] for b in bands) == stats[k], k
    assert max(b[1]["maximum_knots"] for b in bands) == stats["maximum_knots"]
    if tolerance == 1e-11:
        assert stats["fallback_pixels"] > 0


@pytest.mark.parametrize("capacity_reached", [True, False])
def test_rays_are_the_probes_rays(capacity_reached):
    """Over gentle ground under a high sun every ray through a pixel's centre hits and casts a shadow ray (the native
    run shows it; with many sub-rays a few slip through Moeller-Trumbore's edges), so the rays of a window are twice
    its counted probes, exact cells and fallback pixels' native cells: probes that the depth-first walk does not
    reach before a pixel's knots overflow are in neither count."""
    ss = 1
    x = 10.0 * np.arange(64)
    height = 2.0 * np.sin(x[None, :] / 50.0) + 2.0 * np.cos(x[:, None] / 60.0)
    V, N, I = terrain.mesh_from_heightfield(height.astype(np.float32), 10.0)
    cam = dict(width=31, height=9, fx=30.0, fy=30.0, cx=15.5, cy=4.5)
    scene = DeviceScene(V, N, I, cam, ss, HAPKE, geometry=0)
    traj = trajectory.StraightPass((5.0, -8.0, 350.0), (80.0, 10.0, 0.0), trajectory.sun_direction(60, 40), 1000.0, 0.4)
    ivs = trajectory.horizons(traj, 0.0, 1e-5, 190 if capacity_reached else 20)
    phys = physic(photon_shot_noise=0)
    rays = []
    tolerance = 1e-11 if capacity_reached else 1e-4
    for process in (lambda s: s.process_many(ivs), lambda s: s.process_adaptive(ivs, tolerance)):
        s = EventSensor(scene, phys)
        s.initialize(traj.state(0.0), 0.0)
        before = s.stats()
        assert process(s) is not None
        after = s.stats()
        rays.append(sum(after[k] - before[k] for k in ("primary_rays", "shadow_rays")))
    pixels, stats = 31 * 9, s.refinement_statistics()
    assert rays[0] % (pixels * 2 * ss * ss) == 0
    cells = rays[0] // (pixels * 2 * ss * ss)
    samples = stats["traced_pixel_samples"] + stats["native_cell_queries"] + stats["fallback_pixels"] * cells
    assert (stats["fallback_pixels"] > 0) == capacity_reached
    assert rays[1] == 2 * ss * ss * samples
