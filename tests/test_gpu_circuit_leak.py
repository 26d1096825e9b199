"""A reference that leaks upward (reset_leakage_a < 0) as well as downward, in
the FP64 circuit's runs of cells: the leak moves the reference in every cell,
quiet ones too.  Under constant light the leak alone makes the events, so the
adaptive solver's knots carry the exact light; a pulse adds crossings of both
signs to the native cells.  Against the FP64 oracle, whose margin classes name
the pixels that rounding may decide; times within the stated 1 us.
"""
import pytest

from dvsrender4deepspace_gb300 import DeviceScene, EventSensor
from oracle import oracle as O
from tests.test_gpu_parity import compare_event_streams, plane_mesh
from tests.test_oracle_golden import DAVIS, DAVIS_HAPKE, POSE, davis_physic

pytestmark = pytest.mark.gpu

CROP = dict(DAVIS, width=32, height=24, cx=DAVIS["cx"] - 157, cy=DAVIS["cy"] - 118)
PULSE = [(POSE, POSE, 0, 0.001), (dict(POSE, intensity_rate=8e6), dict(POSE, intensity_rate=-8e6), 0.001, 0.003)]
STATIC = [(POSE, POSE, 0, 0.001), (POSE, POSE, 0.001, 0.002)]


@pytest.mark.parametrize("circuit,solver,leakage", [
    ("fp64", "native", -1.3e-14), ("fp64", "native", 1.3e-14), ("fp32", "native", -1.3e-14),
    ("fp64", "static", -1.3e-12), ("fp64", "adaptive", -1.3e-12), ("fp64", "adaptive", 1.3e-12)])
def test_leak_of_either_sign_against_the_oracle(circuit, solver, leakage):
    V, N, I = plane_mesh()
    phys = davis_physic(threshold_std=0, photon_shot_noise=0, max_events_per_step=64, readout_bandwidth=0,
                        readout_latency=0, random_seed=42, reset_leakage_a=leakage)  # 20 or 2000 /s
    ivs = PULSE if solver == "native" else STATIC
    s = EventSensor(DeviceScene(V, N, I, CROP, 1, DAVIS_HAPKE), phys, circuit_precision=circuit)
    s.initialize(POSE, 0)
    ev = s.process_adaptive(ivs, 1e-3) if solver == "adaptive" else s.process_many(ivs)
    oracle = O.OracleSensor(O.OracleScene(V, N, I, CROP, 1, DAVIS_HAPKE, fp64=True), phys, margin=True)
    oracle.initialize(POSE, 0)
    want = oracle.process(ivs)
    assert len(want) > 700
    report = compare_event_streams(ev, want, oracle.margins(), CROP["width"])
    assert report["unclassified_mismatches"] == 0, report
    assert report["max_timestamp_error_s"] < 1e-6, report
