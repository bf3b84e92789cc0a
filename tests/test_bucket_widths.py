"""Large networks of few synapses have wider buckets (128 or 256 targets, by
neuron count and synapses): counts on both sides of each width, random traffic
and a group of busy neighbours whose buckets are taken in parts, exact against
the CPU oracle."""

import numpy as np
import pytest

from snncuda_gb300.connectome import Connectome
from snncuda_gb300.simulation import Simulation, default_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,fanout", [(389_119, 1), (389_120, 1), (778_240, 1), (778_300, 2), (390_007, 200)])
def test_widths(gpu_lib, port_lib, n, fanout):
    rng = np.random.default_rng(n)
    sources = min(n, 2_000_000 // fanout)  # 2e6 random synapses at most,
    group = np.arange(n - 700, n - 500)    # and 60,000 to 200 neighbours
    source = np.concatenate([np.repeat(rng.permutation(n)[:sources], fanout), rng.integers(0, n, 60_000)])
    target = np.concatenate([rng.integers(0, n, sources * fanout), rng.choice(group, 60_000)])
    s = source.size
    net = Connectome(
        threshold=np.ones(n, np.float32), pattern_window_ticks=np.full(n, 2, np.uint64),
        similarity_threshold=np.full(n, 0.9, np.float32), max_reference_patterns=np.full(n, 1, np.uint64),
        source=source.astype(np.uint32), target=target.astype(np.uint32), weight=rng.uniform(0.05, 0.4, s).astype(np.float32),
        max_weight=np.full(s, 0.5, np.float32), delay_ticks=rng.integers(1, 3, s, dtype=np.uint32),
        compartment=rng.integers(0, 4, s, dtype=np.uint8), receptor=rng.integers(0, 2, s, dtype=np.uint8),
        plasticity_enabled=np.ones(s, np.uint8))
    out = []
    for lib in (gpu_lib, port_lib):
        sim = Simulation(net, default_config(lib, raster_capacity=1 << 21, slot_event_capacity=1 << 20), lib)
        for tick in (0, 2):
            sim.inject(np.arange(tick, n, 3), np.full(len(range(tick, n, 3)), tick), np.full(len(range(tick, n, 3)), 1.5))
        sim.run_until(6)
        c, r = sim.counters(), sim.raster()
        out.append(([c[k] for k in ("delivered_spikes", "fired_spikes", "pending_events", "max_slot_events")],
                    [x.tolist() for x in r], sim.digest()))
        sim.close()
    assert out[0] == out[1]
    assert out[0][0][1] > n // 2
