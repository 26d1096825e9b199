"""The adaptive solver's refinement against the depth-first walk it stands for
(src/cuda/optical_sampler.cu:39-84), restated here for one pixel: a stack of 16
segments, each judged when it is popped, the knots counted as they are written.
The kernel opens several pending segments of a pixel at a time, so what it has
to reproduce is the walk's order: how many probes, knots, exact segments, and
whether the knots overflow, for every pixel.

A walk's light comes from sensors initialized at the probed times (the log
of the light is their receptor's state).  It differs from the kernel's own probe
in the last bits of a ray's direction, 1e-7 of the light, so a pixel with a
verdict within 1e-6 of its bound is left out.
"""
import ctypes as C
import math

import numpy as np
import pytest

from dvsrender4deepspace_gb300 import DeviceScene, EventSensor, terrain, trajectory
from dvsrender4deepspace_gb300.raycast import derive_parameters
from oracle import oracle as O
from tests.test_gpu_batch import physic

pytestmark = pytest.mark.gpu

HAPKE = dict(b=0.3, c=0.4, hS=0.06, hC=1.0, thetap=0.349066, w=0.25, B_S0=1.0, B_C0=0.0, phi=0.3)
ROWS, STACK, MARGIN = 48, 16, 1e-6


def receptor_log_at(u, rate, dt, charge):
    k = rate * dt / charge
    return -math.log(math.exp(-k) / math.exp(u) - math.expm1(-k) / rate)


def walk(rate_at, v0, budget, start, end, step, charge, tolerance, capacity):
    """(samples, knots, exact segments, fallback) of one pixel; None where a verdict is too near its bound."""
    light = [rate_at(start + (end - start) * j * .25) for j in range(5)]
    stack = [(.5, 1.0, light[2], light[3], light[4]), (0.0, .5, light[0], light[1], light[2])]
    samples, written, exact = 5, 1, 0
    while stack:
        a, b, left, middle, right = stack.pop()
        estimate, length = (left + right) * .5, (b - a) * (end - start)
        residual = abs(math.log(middle / estimate))
        error = abs(receptor_log_at(v0, middle, length, charge) - receptor_log_at(v0, estimate, length, charge))
        photons = max(middle, estimate) * length
        if min(abs(residual - tolerance), abs(error - budget), abs(photons - 1.0)) < MARGIN:
            return None
        if error <= budget and (residual <= tolerance or photons < 1.0):
            if written + 2 > capacity:
                return samples, written, exact, True
            written += 2
        elif length <= step or len(stack) + 2 > STACK:
            if written >= capacity:
                return samples, written, exact, True
            written += 1
            exact += 1
        else:
            mid = (a + b) * .5
            samples += 2
            lower = rate_at(start + (end - start) * (a + mid) * .5)
            upper = rate_at(start + (end - start) * (mid + b) * .5)
            stack += [(mid, b, middle, upper, right), (a, mid, left, lower, middle)]
    return samples, written, exact, False


def pulses(traj, count, length, rate):
    """`count` intervals, each with a pulse that adds up to rate * length / 4 to the light's 1000."""
    return [(dict(a, intensity_rate=rate), dict(b, intensity_rate=-rate), t0, t1)
            for a, b, t0, t1 in trajectory.horizons(traj, 0.0, length, count)]


def jumps(traj, length, at):
    """A window of constant light that jumps at the given fractions of it."""
    ends = [0.0] + [length * f for f in at] + [length]
    ivs = []
    for k, (t0, t1) in enumerate(zip(ends, ends[1:])):
        level = dict(intensity=1000.0 * (1 + k % 2))
        ivs.append((dict(traj.state(t0), **level), dict(traj.state(t1), **level), t0, t1))
    return ivs


@pytest.mark.parametrize("case,tolerance,refractory", [
    ("one pulse", 1e-3, 5e-5),
    ("many pulses", 1e-3, 5e-5),       # more knots than fit
    ("some pulses", 1e-2, 5e-5),
    ("jumps", 1e-2, 5e-3),             # exact segments at the stack's depth
    ("late jump", 1e-2, 5e-3),
])
def test_refinement_is_the_depth_first_walk(case, tolerance, refractory):
    x = 10.0 * np.arange(64)
    height = 2.0 * np.sin(x[None, :] / 50.0) + 2.0 * np.cos(x[:, None] / 60.0)
    V, N, I = terrain.mesh_from_heightfield(height.astype(np.float32), 10.0)
    cam = dict(width=1, height=ROWS, fx=60.0, fy=60.0, cx=0.5, cy=ROWS / 2)
    scene = DeviceScene(V, N, I, cam, 2, HAPKE)
    traj = trajectory.StraightPass((5.0, -8.0, 350.0), (80.0, 10.0, 0.0), trajectory.sun_direction(60, 40), 1000.0, 0.4)
    ivs = {"one pulse": lambda: pulses(traj, 1, 2e-3, 8e6), "many pulses": lambda: pulses(traj, 190, 1e-5, 2e8),
           "some pulses": lambda: pulses(traj, 7, 2e-4, 2e7), "jumps": lambda: jumps(traj, 0.1, (0.2, 0.37, 0.61, 0.83)),
           "late jump": lambda: jumps(traj, 0.1, (0.93,))}[case]()
    phys = physic(photon_shot_noise=0, threshold_std=0, refractory_time=refractory)
    params = derive_parameters(phys)
    start, end = ivs[0][2], ivs[-1][3]
    packed, library, table = O.intervals_array(ivs), O.load(False), {}

    def light(t):
        """The log of every pixel's light at time t."""
        if t not in table:
            i = next(k for k, iv in enumerate(ivs) if t <= iv[3])
            state = O.ostate()
            library.oracle_optical_state_at(C.byref(packed[i]), t, C.byref(state))
            s = EventSensor(scene, phys)
            p, l = state.position, state.light
            s.initialize(dict(position=(p.x, p.y, p.z), light=(l.x, l.y, l.z), rotation=tuple(state.rotation),
                              intensity=state.intensity), 0.0)
            table[t] = s.read_state()[0][:, 0]
        return table[t]

    compared, fallbacks, exact_segments, most = 0, 0, 0, 0
    for row in range(ROWS):
        s = EventSensor(scene, phys, row_begin=row, row_end=row + 1)
        s.initialize(ivs[0][0], start)
        state = s.read_state()[0][0]
        assert s.process_adaptive(ivs, tolerance) is not None
        got = s.refinement_statistics()
        want = walk(lambda t: math.exp(light(t)[row]), state[0], 1e-3 * min(state[3], state[4]), start, end,
                    params["integration_step"], params["charge_scale"], tolerance, s.adaptive_cache_capacity())
        if want is None:
            continue
        samples, knots, exact, fallback = want
        compared += 1
        fallbacks += fallback
        exact_segments += exact
        most = max(most, knots)
        assert got["traced_pixel_samples"] == samples, row
        assert got["fallback_pixels"] == fallback, row
        assert got["exact_segments"] == exact, row
        if not fallback:
            assert got["maximum_knots"] == knots, row
    assert compared >= ROWS // 6 and most > 20
    assert (fallbacks > 0) == (case == "many pulses")
    if "jump" in case:
        assert exact_segments > 0
