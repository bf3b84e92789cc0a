"""The autotuner on a network that otherwise runs whole ticks in one kernel:
every probe takes the launched kernels, the only ones its knobs shape, and its
time covers all of its ticks."""

import numpy as np
import pytest

from snncuda_gb300.connectome import Connectome
from snncuda_gb300.simulation import Simulation, default_config

pytestmark = pytest.mark.gpu


def test_busy_tick_inside_a_probe(gpu_lib):
    n, s = 2000, 4000
    rng = np.random.default_rng(1)
    net = Connectome(
        threshold=np.full(n, 1e6, np.float32), pattern_window_ticks=np.full(n, 9, np.uint64),
        similarity_threshold=np.full(n, 0.9, np.float32), max_reference_patterns=np.full(n, 1, np.uint64),
        source=rng.integers(0, n, s, dtype=np.uint32), target=rng.integers(0, n, s, dtype=np.uint32),
        weight=np.full(s, 0.1, np.float32), max_weight=np.full(s, 1, np.float32), delay_ticks=np.ones(s, np.uint32),
        compartment=np.ones(s, np.uint8), receptor=np.zeros(s, np.uint8), plasticity_enabled=np.ones(s, np.uint8))
    sim = Simulation(net, default_config(gpu_lib), gpu_lib)
    # the first probe runs 16 ticks untimed and then 64: the second of those
    # has more events due than the one kernel takes
    sim.inject(np.tile(np.arange(n, dtype=np.uint32), 5), np.full(5 * n, 17, np.uint64), np.full(5 * n, 0.1, np.float32))
    tuning = sim.autotune(probe_ticks=64)
    # seven dependent kernels a tick, at least 1 us each
    assert tuning["ms_per_tick_before"] > 0.004
    assert tuning["max_slot_events"] == 5 * n
    sim.close()
