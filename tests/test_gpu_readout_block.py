"""Small batches through the one-cluster readout against the host FIFO, at the
sizes where one block (512), the cluster's shares (8 x 512) and their padding end, with
ties in t that (y, x) decide and events equal in all three, whose arrival order
stays.  Order, fields, drops and peak are exact; delivery times are the same
FP64 sums grouped as a scan (1 ns, as in test_gpu_readout.py).
"""
import numpy as np
import pytest

from dvsrender4deepspace_gb300 import EventSensor
from dvsrender4deepspace_gb300.raycast import EventReadout
from tests.test_gpu_parity import plane_sensor
from tests.test_gpu_readout import random_events, same_stream
from tests.test_oracle_golden import POSE

pytestmark = pytest.mark.gpu

SIZES = (1, 0, 2, 3, 31, 255, 256, 257, 511, 512, 513, 514, 1000, 2048, 4095, 4096, 4097, 5, 8191, 300)


@pytest.mark.parametrize("bandwidth,latency,capacity", [(0.0, 0.0, 1000), (5e6, 18e-9, 1_000_000), (2e6, 1e-6, 500)])
@pytest.mark.parametrize("window,ties", [(64e-6, False), (0.01, False), (64e-6, True)])
def test_block_readout_equals_the_host_fifo(bandwidth, latency, capacity, window, ties):
    rng = np.random.default_rng(31)
    dev = EventReadout(bandwidth, latency, capacity, device=True, max_batch=10_000)
    host = EventReadout(bandwidth, latency, capacity)
    t = 1.0
    for n in SIZES:
        ev = random_events(rng, n, t, t + window)
        if ties and bandwidth == 0:  # few instants and pixels: equal events in arrival order (told apart by their depth)
            ev["timestamp"] = t + rng.integers(0, 4, n) * 1e-6
            ev["x"], ev["y"] = rng.integers(0, 3, n), rng.integers(0, 2, n)
        t += window
        same_stream(dev.submit(ev, t), host.submit(ev, t), bandwidth > 0)
        assert dev.dropped() == host.dropped() and dev.peak_queue() == host.peak_queue()
    same_stream(dev.drain(), host.drain(), bandwidth > 0)


def test_a_burst_after_quiet_batches():
    """The cluster sized by a quiet batch takes the burst that follows it through the radix passes."""
    scene, phys = plane_sensor(readout_bandwidth=2e7, readout_latency=1e-6, readout_queue_capacity=500_000,
                               threshold_pos=0.05, threshold_neg=0.05)
    start, end = dict(POSE, intensity_rate=8e6), dict(POSE, intensity_rate=-8e6)
    dev, host = EventSensor(scene, phys), EventSensor(scene, phys, host_readout=True)
    for s in (dev, host):
        s.initialize(POSE, 0)
    sizes = []
    for iv in [(POSE, POSE, 0, 0.001), (start, end, 0.001, 0.003), (POSE, POSE, 0.003, 0.004)]:
        a, b = dev.process(iv), host.process(iv)
        same_stream(a, b, True)
        sizes.append(len(b))
    same_stream(dev.drain(), host.drain(), True)
    assert sizes[0] == 0 and dev.stats()["events_generated"] > 4096
