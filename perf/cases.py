"""The work a user has this framework do, as measurable cases.

Every case goes through the public entry points (DeviceScene and its views,
CamRayCaster, EventSensor, SensorBatch, EventReadout).  Terrains are resident
on the GPU and shared by the jobs over them, as in a rendering service; what
differs from job to job -- trajectory, sun, flicker of the light, sensor seed,
event streams -- is made from the seed.

An event-sensor pass is one whole job: a sensor is created over a resident
terrain, initialized, given its batches of horizons, drained, read out and
closed.  Its outputs are the events and the pixel-circuit state.
"""
import math
import random

import numpy as np
import torch

from dvsrender4deepspace_gb300 import _capi, terrain, trajectory
from dvsrender4deepspace_gb300.raycast import (CamRayCaster, DeviceScene, EventReadout, EventSensor, SensorBatch,
                                               interval_array)

HAPKE = dict(b=0.3, c=0.4, hS=0.06, hC=1.0, thetap=0.349066, w=0.25, B_S0=1.0, B_C0=0.0, phi=0.3)
PHYSIC = dict(threshold_pos=0.2, threshold_neg=0.2, refractory_time=200e-6, readout_bandwidth=5e6,
              readout_latency=18e-9, threshold_std=0.03, threshold_min=0.01, wavelength_nm=550,
              quantum_efficiency=0.3, pixel_pitch_um=15, fill_factor=0.2, f_number=2.0, lens_transmission=0.8,
              radiance_scale=0.001, temperature_k=300, subthreshold_kappa=0.8, receptor_capacitance_f=1e-15,
              reset_capacitance_f=20e-15, dark_current_a=1e-18, reset_leakage_a=0, circuit_step=1e-6,
              photon_shot_noise=1, reset_thermal_noise=0, random_seed=114514, max_events_per_step=16,
              readout_queue_capacity=1000000)
# device rays one pass of the largest listed case traces (primary and shadow): a drawn case stays below
MOST_RAYS = 1280 * 720 * 64 * 64 * 2
RAY_FLOPS = 250        # ray set-up, one box and one triangle test, interpolation and shading of one ray
CELL_FLOPS = 120       # one circuit cell: photon count, receptor step, comparison


def listed():
    """name, and what it stands for:
    cam_davis       one DAVIS346 frame, one ray a pixel: the smallest render, latency and copies
    cam_hd_ss16     one 1280x720 frame with 16 x 16 sub-rays in the precision geometry (config/prophesee.yaml)
    blur_davis      one motion-blur exposure of 8 poses (the configs' blur resolution)
    job_64x48       the smallest serving job: launches, host work and the sensor's own set-up
    job_davis_fp64  the plain method: 346x260, one ray a pixel, FP64 circuit, 640 cells
    job_davis_orbit one trajectory of the batching workload: 16 sub-rays, FP32 circuit
    job_ragged      odd sizes: 637x479, 9 sub-rays, 50 horizons of three cells, bright enough for dense events
    job_hd          the 1280x720 precision sensor: FP16 bounds, watertight test, Philox noise
    adaptive_davis  the adaptive solver the app uses for long sequences: 200 horizons a window
    batch_64x48     16 uneven small trajectories advanced together, as a server batches small jobs
    readout_hd      a busy 1280x720 sensor's batch put in (t, y, x) order (no bus)
    readout_merge   runs of four sensors merged through one finite bus, small ragged batches
    """
    return [
        dict(name="cam_davis", kind="cam", grid=256, width=346, height=260, fx=300.0, ss=1, geometry=0),
        dict(name="cam_hd_ss16", kind="cam", grid=1024, width=1280, height=720, fx=1000.0, ss=16, geometry=3),
        dict(name="blur_davis", kind="blur", grid=1024, width=346, height=260, fx=300.0, ss=4, geometry=0, poses=8),
        dict(name="job_64x48", kind="job", grid=512, width=64, height=48, fx=56.0, ss=1, geometry=0,
             circuit="fp32-philox", horizons=64, step_us=1.0, batches=2, intensity=1000.0),
        dict(name="job_davis_fp64", kind="job", grid=256, width=346, height=260, fx=300.0, ss=1, geometry=0,
             circuit="fp64", horizons=64, step_us=10.0, batches=2, intensity=1000.0),
        dict(name="job_davis_orbit", kind="job", grid=1024, width=346, height=260, fx=300.0, ss=4, geometry=0,
             circuit="fp32", horizons=64, step_us=10.0, batches=1, intensity=1000.0),
        dict(name="job_ragged", kind="job", grid=512, width=637, height=479, fx=550.0, ss=3, geometry=2,
             circuit="fp64", horizons=50, step_us=2.5, batches=2, intensity=20000.0),
        dict(name="job_hd", kind="job", grid=2048, width=1280, height=720, fx=1000.0, ss=8, geometry=3,
             circuit="fp32-philox", horizons=64, step_us=1.0, batches=1, intensity=1000.0),
        dict(name="adaptive_davis", kind="adaptive", grid=1024, width=346, height=260, fx=300.0, ss=4, geometry=0,
             circuit="fp64", horizons=200, step_us=10.0, batches=1, intensity=1000.0),
        dict(name="batch_64x48", kind="batch", grid=512, width=64, height=48, fx=56.0, ss=1, geometry=0,
             circuit="fp32", horizons=64, step_us=1.0, batches=4, members=16, intensity=20000.0),
        dict(name="readout_hd", kind="readout", width=1280, height=720, events=1 << 20, window_us=64.0, batches=1,
             bandwidth=0.0),
        dict(name="readout_merge", kind="readout", width=346, height=260, events=3001, window_us=640.0, batches=6,
             bandwidth=2e7),
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _rays(c):
    """Primary and shadow rays of one pass."""
    px = c["width"] * c["height"] * c["ss"] ** 2
    if c["kind"] == "cam":
        return 2 * px
    if c["kind"] == "blur":
        return 2 * px * c["poses"]
    if c["kind"] == "adaptive":
        return 2 * px * c["batches"] * 24  # five probes a pixel, and bisections
    return 2 * px * _cells(c) * c["batches"] * c.get("members", 1)


def _cells(c):
    """Circuit cells of one batch: ceil(step / 1 us) a horizon (the circuit step is a float)."""
    step = float(np.float32(PHYSIC["circuit_step"]))
    return c["horizons"] * math.ceil(float(np.float32(c["step_us"] * 1e-6)) / step)


def draw(rng):
    kind = rng.choice(["cam", "blur", "job", "job", "job", "adaptive", "batch", "readout"])
    if kind == "readout":
        bus = rng.random() < 0.5
        return dict(kind=kind, width=rng.choice([346, 640, 1280]), height=rng.choice([260, 480, 720]),
                    events=int(_log_uniform(rng, 50, 60_000 if bus else 1 << 20)),
                    window_us=rng.choice([64.0, 640.0, 10000.0]), batches=rng.randint(2, 6) if bus else 1,
                    bandwidth=_log_uniform(rng, 1e7, 1e9) if bus else 0.0)
    while True:
        w = int(_log_uniform(rng, 64, 1280))
        c = dict(kind=kind, grid=rng.choice([256, 512, 1024]), width=w, height=max(9, int(w * rng.uniform(0.55, 0.8))),
                 fx=round(w * rng.uniform(0.75, 1.0), 2), ss=rng.choice([1, 1, 2, 3, 4, 5, 8, 16]),
                 geometry=rng.choice([0, 0, 1, 2, 3]))
        if kind == "blur":
            c["poses"] = rng.randint(2, 40)
        if kind in ("job", "adaptive", "batch"):
            c.update(circuit=rng.choice(["fp64", "fp32", "fp32-philox"]), horizons=rng.randint(9, 64),
                     step_us=rng.choice([1.0, 2.5, 5.0, 10.0]), batches=rng.randint(1, 3),
                     intensity=rng.choice([1000.0, 1000.0, 5000.0, 20000.0]))
        if kind == "adaptive":
            c.update(circuit=rng.choice(["fp64", "fp32"]), horizons=rng.randint(20, 200), step_us=10.0, ss=min(c["ss"], 4),
                     batches=1)
        if kind == "batch":
            c.update(members=rng.randint(2, 24), width=rng.randint(40, 128), height=rng.randint(32, 96),
                     fx=rng.uniform(40.0, 110.0), ss=min(c["ss"], 4))
        cells = c["width"] * c["height"] * _cells(c) * c["batches"] if "horizons" in c else 0
        slow = 4 if c.get("circuit") == "fp64" else 1
        if _rays(c) + 8 * slow * cells * c.get("members", 1) <= MOST_RAYS // 2:
            return c


# ---- inputs ---------------------------------------------------------------------------
_terrains = {}  # resident terrains: (grid, geometry) -> DeviceScene
_meshes = {}


def _mesh(grid):
    if grid not in _meshes:
        _meshes[grid] = terrain.terrain_mesh(grid, seed=20260000 + grid)
    return _meshes[grid]


def _camera(c):
    return dict(width=c["width"], height=c["height"], fx=c["fx"], fy=c["fx"], cx=c["width"] / 2, cy=c["height"] / 2)


def _view(c):
    key = (c["grid"], c["geometry"])
    if key not in _terrains:
        V, N, I = _mesh(c["grid"])
        _terrains[key] = DeviceScene(V, N, I, dict(width=64, height=48, fx=56.0, fy=56.0, cx=32.0, cy=24.0), 1, HAPKE,
                                     geometry=c["geometry"])
    return _terrains[key].view(_camera(c), c["ss"])


class _Flicker:
    """An orbit whose light flickers (a tumbling reflector, an exposure lamp): what makes a slow pass give events."""

    def __init__(self, rng, grid, intensity=1000.0):
        half = 10.0 * (grid - 1) / 2
        elevation = math.radians(rng.uniform(20.0, 60.0))
        self.orbit = trajectory.Orbit((rng.uniform(-.3, .3) * half, rng.uniform(-.3, .3) * half),
                                      _log_uniform(rng, 700.0, 2500.0), rng.uniform(10.0, 200.0),
                                      rng.uniform(0, 2 * math.pi), math.radians(rng.uniform(-5.0, 5.0)),
                                      trajectory.sun_direction(math.degrees(elevation), rng.uniform(0.0, 360.0)),
                                      intensity)
        self.w = 2 * math.pi / rng.uniform(0.8e-3, 1.6e-3)
        self.phase = rng.uniform(0, 2 * math.pi)

    def state(self, t):
        s = self.orbit.state(t)
        a = self.w * t + self.phase
        s["intensity"] = self.orbit.intensity * (1.0 + 0.7 * math.sin(a))
        s["intensity_rate"] = self.orbit.intensity * 0.7 * self.w * math.cos(a)
        return s


def _states(c, seed):
    """The poses of a frame or an exposure (20 ms) of a seeded orbit."""
    rng = random.Random(seed)
    traj = _Flicker(rng, c["grid"])
    n = c.get("poses", 1)
    return [dict(traj.state(0.02 * j / max(1, n - 1)), intensity=1000.0, intensity_rate=0.0) for j in range(n)]


def _job(c, rng, short=1.0):
    """A job's start pose and batches of horizon intervals; `short` of the horizons."""
    traj = _Flicker(rng, c["grid"], c["intensity"])
    n = max(1, int(round(c["horizons"] * short)))
    step, batches, t = c["step_us"] * 1e-6, [], 0.0
    for _ in range(c["batches"]):
        ivs = trajectory.horizons(traj, t, step, n)
        batches.append(interval_array(ivs))
        t = ivs[-1][3]
    physic = dict(PHYSIC, random_seed=rng.randint(1, 1 << 30))
    return dict(pose=traj.state(0.0), batches=batches, physic=physic)


def _events(c, rng, t0, n):
    r = np.random.default_rng(rng.randint(0, 1 << 30))
    ev = np.zeros(n, _capi.EVENT_DTYPE)
    ev["timestamp"] = t0 + r.uniform(0.0, c["window_us"] * 1e-6, n)
    ev["x"] = r.integers(0, c["width"], n)
    ev["y"] = r.integers(0, c["height"], n)
    ev["polarity"] = r.integers(0, 2, n)
    ev["depth"] = r.uniform(500.0, 3000.0, n).astype(np.float32)
    return ev


def prepare(case, seed):
    c = dict(case)
    rng = random.Random(seed)
    s = dict(case=c)
    if c["kind"] in ("cam", "blur"):
        s["view"] = _view(c)
        s["caster"] = CamRayCaster(s["view"])
        s["states"] = _states(c, seed)
        n = c.get("poses", 1)
        s["weights"] = np.full(n, 1.0 / n, np.float32)
    elif c["kind"] in ("job", "adaptive"):
        s["view"] = _view(c)
        s["job"] = _job(c, rng)
    elif c["kind"] == "batch":
        # uneven lengths: member m flies a part of the horizons
        s["views"] = [_view(c) for _ in range(c["members"])]
        s["jobs"] = [_job(c, rng, rng.uniform(0.25, 1.0)) for _ in range(c["members"])]
    else:
        t, s["batches"] = 1.0, []
        for b in range(c["batches"]):
            s["batches"].append((_events(c, rng, t, max(1, c["events"] - 37 * b)), t + c["window_us"] * 1e-6))
            t += c["window_us"] * 1e-6
        if c["bandwidth"] == 0:  # an ordering stage keeps nothing between batches: one handle for the program's life
            s["readout"] = EventReadout(0.0, 0.0, 1000, device=True, max_batch=c["events"])
    if c["kind"] in ("job", "adaptive", "batch"):
        # the program's event buffer: as many as a pixel's refractory time lets through
        jobs = s["jobs"] if "jobs" in s else [s["job"]]
        most = math.ceil(c["horizons"] * c["step_us"] * 1e-6 * c["batches"] / PHYSIC["refractory_time"]) + 2
        n = len(jobs) * c["width"] * c["height"] * most
        s["out"] = {f: np.zeros(n, _capi.EVENT_DTYPE[f]) for f in _FIELDS}
        s["filled"] = 0
    return s


# ---- one pass -------------------------------------------------------------------------
_FIELDS = ("timestamp", "x", "y", "polarity", "depth")


def _fields(chunks):
    ev = chunks[0] if len(chunks) == 1 else np.concatenate(chunks)
    return {f: np.ascontiguousarray(ev[f]) for f in _FIELDS}


def _store(state, chunks):
    """The events into the program's buffer, field by field; the slots a longer earlier pass filled are cleared."""
    n = sum(len(ev) for ev in chunks)
    for f in _FIELDS:
        out, at = state["out"][f], 0
        for ev in chunks:
            out[at:at + len(ev)] = ev[f]
            at += len(ev)
        out[n:state["filled"]] = 0
    state["filled"] = n
    return dict(state["out"], count=n)


def run(state):
    c = state["case"]
    if c["kind"] == "cam":
        image, depth = state["caster"].render_state(state["states"][0])
        return {"image": image, "depth": depth}
    if c["kind"] == "blur":
        return {"image": state["caster"].render_blur(state["states"], state["weights"])}
    if c["kind"] in ("job", "adaptive"):
        job = state["job"]
        sensor = EventSensor(state["view"], job["physic"], circuit_precision=c["circuit"])
        sensor.initialize(job["pose"], 0.0)
        if c["kind"] == "job":
            chunks = [sensor.process_many(b) for b in job["batches"]]
        else:
            chunks = [sensor.process_adaptive(b, 1e-2) for b in job["batches"]]
        chunks.append(sensor.drain())
        circuit, pending = sensor.read_state()
        sensor.close()
        return dict(_store(state, chunks), state=circuit, pending=pending)
    if c["kind"] == "batch":
        sensors = [EventSensor(v, j["physic"], circuit_precision=c["circuit"])
                   for v, j in zip(state["views"], state["jobs"])]
        for s, j in zip(sensors, state["jobs"]):
            s.initialize(j["pose"], 0.0)
        batch = SensorBatch(sensors)
        chunks = [[] for _ in sensors]
        for b in range(c["batches"]):
            for m, ev in enumerate(batch.process([j["batches"][b] for j in state["jobs"]])):
                chunks[m].append(ev)
        states = []
        for m, s in enumerate(sensors):
            chunks[m].append(s.drain())
            states.append(s.read_state()[0])
        batch.close()
        for s in sensors:
            s.close()
        return dict(_store(state, [e for m in chunks for e in m]), state=np.concatenate(states))
    readout = state.get("readout")
    if readout is None:
        readout = EventReadout(c["bandwidth"], 18e-9, 1_000_000, device=True, max_batch=c["events"])
    chunks = [readout.submit(ev, now) for ev, now in state["batches"]]
    if c["bandwidth"]:
        chunks.append(readout.drain())
    return _fields(chunks)


def work(case):
    c = dict(case)
    if c["kind"] == "readout":
        return {"bytes": 2 * 17.0 * c["events"] * c["batches"], "flops": 0.0}
    px = c["width"] * c["height"]
    # every triangle and shading record in view read once, at most one a sub-ray
    scene = 112.0 * min(2 * (c["grid"] - 1) ** 2, px * c["ss"] ** 2)
    if c["kind"] == "cam":
        return {"bytes": scene + 8.0 * px, "flops": float(RAY_FLOPS) * _rays(c)}
    if c["kind"] == "blur":
        return {"bytes": scene + 4.0 * px, "flops": float(RAY_FLOPS) * _rays(c)}
    members = c.get("members", 1)
    cells = px * _cells(c) * c["batches"] * members
    return {"bytes": scene + members * px * 2 * 41.0,
            "flops": float(RAY_FLOPS) * _rays(c) + float(CELL_FLOPS) * cells}


# ---- the same in 64 bits ----------------------------------------------------------------
def _exact_hapke(ci, ce, cg):
    """The Hapke reflectance of the scene's material at incidence, emission and phase cosines (torch, FP64)."""
    h = {k: float(np.float32(v)) for k, v in HAPKE.items()}
    pi = math.pi
    ci, ce, cg = ci.clamp(0, 1), ce.clamp(0, 1), cg.clamp(-1, 1)
    si, se = (1 - ci * ci).clamp_min(0).sqrt(), (1 - ce * ce).clamp_min(0).sqrt()
    tg = torch.tan((torch.acos(cg) / 2).clamp(-pi / 2 + 1e-6, pi / 2 - 1e-6))
    cpsi = ((cg - ci * ce) / (si * se + 1e-6)).clamp(-1, 1)
    psi = torch.acos(cpsi)
    b, c, w = h["b"], h["c"], h["w"]
    p = ((1 + c) / 2 * (1 - b * b) / (1 - 2 * b * cg + b * b) ** 1.5
         + (1 - c) / 2 * (1 - b * b) / (1 + 2 * b * cg + b * b) ** 1.5)
    bs = 1 / (1 + tg / h["hS"])
    q = 1.209 * h["phi"] ** (2 / 3)
    K = -math.log(1 - q) / q
    tt = math.tan(h["thetap"])
    chi = 1 / math.sqrt(1 + pi * tt * tt)

    def e12(cy, sy):
        cot = cy / sy.clamp_min(1e-6) / tt
        return torch.exp(-2 / pi * cot), torch.exp(-cot * cot / pi)
    e1i, e2i = e12(ci, si)
    e1e, e2e = e12(ce, se)
    eta_i = chi * (ci + si * tt * e2i / (2 - e1i))
    eta_e = chi * (ce + se * tt * e2e / (2 - e1e))
    s2 = torch.sin(psi / 2) ** 2
    f = torch.exp(-2 * torch.tan(psi / 2))
    low = ci >= ce
    d = 2 - torch.where(low, e1e, e1i) - psi / pi * torch.where(low, e1i, e1e)
    mu0 = chi * (ci + si * tt * torch.where(low, cpsi * e2e + s2 * e2i, e2i - s2 * e2e) / d)
    mue = chi * (ce + se * tt * torch.where(low, e2e - s2 * e2i, cpsi * e2i + s2 * e2e) / d)
    S = mue / eta_e * ci / eta_i * chi / (1 - f + f * chi * torch.where(low, ci / eta_i, ce / eta_e))
    r0 = (1 - math.sqrt(1 - w)) / (1 + math.sqrt(1 - w))

    def H(x):
        return torch.where(x <= 1e-8, torch.ones_like(x),
                           1 / (1 - w * x * (r0 + (1 - 2 * r0 * x) * 0.5 * torch.log(1 + 1 / x))))
    M = H(mu0 / K) * H(mue / K) - 1
    return w / (4 * pi) * mu0 / (mu0 + mue + 1e-6) * K * (p * (1 + bs * h["B_S0"]) + M) * S


def _nearest(o, d, v0, e1, e2, self_tri=None):
    """Nearest Moller-Trumbore hit of every ray with every triangle: (t, triangle, u, v), t = inf for a miss."""
    n = len(o)
    best = torch.full((n,), math.inf, dtype=torch.float64, device=o.device)
    tri = torch.zeros(n, dtype=torch.long, device=o.device)
    bu, bv = torch.zeros_like(best), torch.zeros_like(best)
    ray_chunk = 4096
    for r in range(0, n, ray_chunk):
        O, D = o[r:r + ray_chunk], d[r:r + ray_chunk]
        # triangles near the chunk's rays: the box of their segments down to the terrain's height range
        lo_z, hi_z = float(v0[:, 2].min()) - 700.0, float(v0[:, 2].max()) + 700.0
        dz = torch.where(D[:, 2].abs() < 1e-9, torch.full_like(D[:, 2], 1e-9), D[:, 2])
        ts = torch.stack([((lo_z - O[:, 2]) / dz).clamp(0, 3e4), ((hi_z - O[:, 2]) / dz).clamp(0, 3e4)], 1)
        ends = O[:, None, :2] + ts[:, :, None] * D[:, None, :2]
        box_lo, box_hi = ends.amin((0, 1)) - 15.0, ends.amax((0, 1)) + 15.0
        near = ((v0[:, :2] >= box_lo) & (v0[:, :2] <= box_hi)).all(1).nonzero().flatten()
        for k in range(0, len(near), 4096):
            ids = near[k:k + 4096]
            a, f, g = v0[ids], e1[ids], e2[ids]
            pv = torch.linalg.cross(D[:, None, :], g[None])
            det = (f[None] * pv).sum(-1)
            tv = O[:, None, :] - a[None]
            u = (tv * pv).sum(-1) / det
            qv = torch.linalg.cross(tv, f[None].expand_as(tv))
            v = (D[:, None, :] * qv).sum(-1) / det
            t = (g[None] * qv).sum(-1) / det
            ok = (det.abs() >= 1e-6) & (u >= 0) & (v >= 0) & (u + v <= 1) & (t > 1e-6)
            if self_tri is not None:
                ok &= ids[None] != self_tri[r:r + ray_chunk, None]
            t = torch.where(ok, t, torch.full_like(t, math.inf))
            m, j = t.min(1)
            win = m < best[r:r + ray_chunk]
            rows = torch.arange(len(O), device=o.device)
            for dst, src in ((best, m), (tri, ids[j]), (bu, u[rows, j]), (bv, v[rows, j])):
                dst[r:r + ray_chunk] = torch.where(win, src, dst[r:r + ray_chunk])
    return best, tri, bu, bv


def _exact_image(c, state):
    """One frame in FP64: radiance and depth of every pixel (None where it takes too long)."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    V, N, I = _mesh(c["grid"])
    V, N = (torch.tensor(x, dtype=torch.float64, device=dev) for x in (V, N))
    I = torch.tensor(I.astype(np.int64), device=dev)
    v0, e1, e2 = V[I[:, 0]], V[I[:, 1]] - V[I[:, 0]], V[I[:, 2]] - V[I[:, 0]]
    f32 = lambda v: torch.tensor(np.asarray(v, np.float32).astype(np.float64), device=dev)  # noqa: E731
    q, light = f32(state["rotation"]), f32(state["light"])
    light = light / light.norm()
    cam, ss = _camera(c), c["ss"]
    # pixels in 32 x 32 tiles, so that a chunk of rays sees few triangles
    ys, xs = torch.meshgrid(torch.arange(c["height"], device=dev), torch.arange(c["width"], device=dev), indexing="ij")
    order = torch.argsort(((ys // 32) * 10000 + xs // 32).flatten(), stable=True)
    x, y = xs.flatten()[order].double(), ys.flatten()[order].double()
    radiance, depth, hits = torch.zeros_like(x), torch.zeros_like(x), torch.zeros_like(x)
    for sy in range(ss):
        for sx in range(ss):
            px = (x + (sx + .5) / ss - .5 - float(np.float32(cam["cx"]))) / float(np.float32(cam["fx"]))
            py = (y + (sy + .5) / ss - .5 - float(np.float32(cam["cy"]))) / float(np.float32(cam["fy"]))
            v = torch.stack([px, -py, -torch.ones_like(px)], 1)
            qv = q[:3].expand_as(v)
            t2 = 2 * torch.linalg.cross(qv, v)
            d = v + q[3] * t2 + torch.linalg.cross(qv, t2)
            d = d / d.norm(dim=1, keepdim=True)
            o = f32(state["position"]).expand_as(d)
            t, tri, bu, bv = _nearest(o, d, v0, e1, e2)
            hit = t.isfinite()
            depth += torch.where(hit, t, torch.zeros_like(t))
            hits += hit
            n = (N[I[tri, 0]] * (1 - bu - bv)[:, None] + N[I[tri, 1]] * bu[:, None] + N[I[tri, 2]] * bv[:, None])
            n = n / n.norm(dim=1, keepdim=True)
            ci, ce, cg = n @ light, -(n * d).sum(1), -(d @ light)
            lit = (hit & (ci > 0) & (ce > 0)).nonzero().flatten()
            point = v0[tri[lit]] + bu[lit, None] * e1[tri[lit]] + bv[lit, None] * e2[tri[lit]]
            blocked = _nearest(point, light.expand_as(point), v0, e1, e2, tri[lit])[0].isfinite()
            lit = lit[~blocked]
            value = _exact_hapke(ci[lit], ce[lit], cg[lit]).clamp_min(0) * float(np.float32(state["intensity"]))
            radiance[lit] += value / (1 + px[lit] ** 2 + py[lit] ** 2) ** 2
    depth = torch.where(hits > 0, depth / hits.clamp_min(1), torch.full_like(depth, -1.0))
    image, dep = torch.empty_like(radiance), torch.empty_like(depth)
    image[order], dep[order] = radiance / ss ** 2, depth
    return image.cpu().numpy(), dep.cpu().numpy()


def exact(case, seed):
    c = dict(case)
    if c["kind"] in ("cam", "blur"):
        states = _states(c, seed)
        if c["width"] * c["height"] * c["ss"] ** 2 * len(states) > 200_000 or c["grid"] > 512:
            return None
        frames = [_exact_image(c, st) for st in states]
        if c["kind"] == "cam":
            return {"image": frames[0][0], "depth": frames[0][1]}
        return {"image": sum(f[0] for f in frames) / len(frames)}
    if c["kind"] == "readout":
        s = prepare(dict(c, kind="readout", bandwidth=c["bandwidth"] or -1.0), seed)  # the streams, without a handle
        if c["bandwidth"] == 0:
            ev = s["batches"][0][0]
            ev = ev[np.lexsort((ev["x"], ev["y"], ev["timestamp"]))]
            return {"timestamp": ev["timestamp"], "x": None, "y": None, "polarity": None, "depth": ev["depth"].astype(np.float64)}
        times, depths, free = [], [], 0.0
        for ev, _ in s["batches"]:
            ev = ev[np.lexsort((ev["x"], ev["y"], ev["timestamp"]))]
            k = np.arange(len(ev)) / c["bandwidth"]
            done = np.maximum(free, np.maximum.accumulate(ev["timestamp"] - k)) + k + 1 / c["bandwidth"]
            free = done[-1]
            times.append(done + 18e-9)
            depths.append(ev["depth"].astype(np.float64))
        return {"timestamp": np.concatenate(times), "x": None, "y": None, "polarity": None, "depth": np.concatenate(depths)}
    # jobs draw photon noise from device streams that 64-bit arithmetic alone does not give
    return None
