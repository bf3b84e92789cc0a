"""Buckets with more events than a block of the tick kernel holds are taken in
parts of their targets, a block each: event counts at the edges of the numbers
of parts, spread over a bucket's targets, on a few of them and mostly on one (a
part that does not fit either), a last bucket that is not full, targets with
one and with several reference patterns.  Exact against the CPU oracle."""

import numpy as np
import pytest

from snncuda_gb300.connectome import Connectome
from snncuda_gb300.simulation import Simulation, default_config

pytestmark = pytest.mark.gpu

TARGETS = 75  # two full buckets of 32 and a part of a third


def _network(events, spread, patterns, seed):
    """`events` sources (neurons 0 ..) with a synapse each to the last TARGETS neurons."""
    rng = np.random.default_rng(seed)
    bucket = [(0, 32), (32, 64), (64, TARGETS)][seed % 3]
    to = rng.integers(*bucket, events)
    if spread == "few":
        to = rng.choice([bucket[0], bucket[0] + 7, bucket[1] - 1], events)
    elif spread == "one":
        to = np.where(rng.random(events) < 0.7, bucket[0] + 3, to)
    first = -(-events // 32) * 32 + 32  # the targets start at a bucket
    n = first + TARGETS
    threshold = np.ones(n, np.float32)
    threshold[first:] = rng.uniform(0.2, 2.0, TARGETS)
    ptr = np.zeros(events + 1, np.uint64)
    ptr[1:] = np.cumsum(np.where(rng.random(events) < 0.02, 2, 1))  # some synapses twice in the tick
    return events, Connectome(
        threshold=threshold, pattern_window_ticks=np.full(n, 6, np.uint64), similarity_threshold=np.full(n, 0.9, np.float32),
        max_reference_patterns=np.full(n, patterns, np.uint64), source=rng.permutation(events).astype(np.uint32),
        target=(first + to).astype(np.uint32), weight=rng.uniform(0.001, 0.02, events).astype(np.float32),
        max_weight=np.full(events, 0.05, np.float32), delay_ticks=np.ones(events, np.uint32),
        compartment=rng.integers(0, 4, events, dtype=np.uint8), receptor=rng.integers(0, 2, events, dtype=np.uint8),
        plasticity_enabled=np.ones(events, np.uint8), code_offset_ptr=ptr, code_offsets=np.zeros(int(ptr[-1]), np.uint32))


def _run(lib, sources, net, advance):
    cfg = default_config(lib, raster_capacity=1 << 20)
    cfg.max_weight = 1.0
    sim = Simulation(net, cfg, lib)
    for tick in (0, 2, 3):
        sim.inject(np.arange(sources), np.full(sources, tick), np.full(sources, 1.5, np.float32))
    getattr(sim, advance)(6)
    keep = ("delivered_spikes", "fired_spikes", "synaptic_events", "pending_events", "max_slot_events")
    counters, raster = sim.counters(), sim.raster()
    out = ({k: counters[k] for k in keep}, raster[0].tolist(), raster[1].tolist(), sim.digest())
    sim.close()
    return out


@pytest.mark.parametrize("events", [1255, 1281, 1570, 1610, 3140, 6400, 25_700])
@pytest.mark.parametrize("spread", ["even", "few", "one"])
@pytest.mark.parametrize("patterns", [1, 3])
def test_parts(gpu_lib, port_lib, events, spread, patterns):
    seed = events + patterns + len(spread)
    sources, net = _network(events, spread, patterns, seed)
    # the profiled ticks take the large networks' kernels whatever the size
    assert _run(gpu_lib, sources, net, "profile") == _run(port_lib, sources, net, "run_until")
