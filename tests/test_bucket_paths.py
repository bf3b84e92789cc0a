"""The tick kernel's blocks hold a bucket's events in shared memory, rank each
target's events there, and fall back to global memory when a bucket or a
target has too many.  Networks whose busy target and busy bucket lie at those
limits, with and without fires, against the CPU oracle bit for bit."""

import numpy as np
import pytest

from snncuda_gb300.connectome import Connectome
from snncuda_gb300.simulation import Simulation, default_config

pytestmark = pytest.mark.gpu


def _fan_in(hub_events, other_events, threshold, patterns, codes, seed):
    """Sources 64.. fire together; `hub_events` synapses end at neuron 5 and
    `other_events` at the 30 neurons of its bucket that follow it."""
    rng = np.random.default_rng(seed)
    sources = hub_events + other_events
    n = 64 + sources
    target = np.concatenate([np.full(hub_events, 5), rng.integers(6, 31, other_events)]).astype(np.uint32)
    source = (64 + rng.permutation(sources)).astype(np.uint32)
    order = rng.permutation(sources)  # Connectome order differs from both
    s = sources
    ptr = np.zeros(s + 1, np.uint64)
    counts = rng.integers(1, codes + 1, s)
    ptr[1:] = np.cumsum(counts)
    thr = np.ones(n, np.float32)
    thr[:64] = threshold
    return n, Connectome(
        threshold=thr, pattern_window_ticks=np.full(n, 6, np.uint64), similarity_threshold=np.full(n, 0.9, np.float32),
        max_reference_patterns=np.full(n, patterns, np.uint64), source=source[order], target=target[order],
        weight=rng.uniform(0.001, 0.02, s).astype(np.float32), max_weight=np.full(s, 0.05, np.float32),
        delay_ticks=rng.integers(1, 3, s, dtype=np.uint32), compartment=rng.integers(0, 4, s, dtype=np.uint8),
        receptor=rng.integers(0, 2, s, dtype=np.uint8), plasticity_enabled=np.ones(s, np.uint8),
        code_offset_ptr=ptr, code_offsets=rng.integers(0, 2, int(ptr[-1]), dtype=np.uint32))


def _run(lib, n, net, advance):
    cfg = default_config(lib, raster_capacity=1 << 20)
    cfg.max_weight = 1.0
    sim = Simulation(net, cfg, lib)
    for tick in (0, 3, 4):
        sim.inject(np.arange(64, n), np.full(n - 64, tick), np.full(n - 64, 1.5, np.float32))
        sim.inject([5, 5, 7], [tick + 2] * 3, [0.01, -0.02, 0.3])
    getattr(sim, advance)(9)
    keep = ("delivered_spikes", "fired_spikes", "synaptic_events", "pending_events", "max_slot_events")
    counters = sim.counters()
    raster = sim.raster()
    out = ({k: counters[k] for k in keep}, raster[0].tolist(), raster[1].tolist(), sim.digest())
    sim.close()
    return out


# about 1.5 delays x codes per tick: each case reaches its limit in some tick;
# 257, 1024 and 1025 are edges of the rows that post-spike STDP reads at once
@pytest.mark.parametrize("hub,other", [(0, 40), (33, 5), (257, 0), (511, 0), (700, 100), (1023, 300), (1024, 0),
                                       (1025, 0), (1400, 1300), (4000, 0)])
@pytest.mark.parametrize("threshold,patterns,codes", [(1e6, 1, 1), (0.8, 1, 4), (0.8, 3, 6)])
def test_busy_targets(gpu_lib, port_lib, hub, other, threshold, patterns, codes):
    n, net = _fan_in(hub, other, threshold, patterns, codes, hub + other)
    want = _run(port_lib, n, net, "run_until")
    # the profiled ticks take the large networks' kernels whatever the size
    assert _run(gpu_lib, n, net, "profile") == want
    assert _run(gpu_lib, n, net, "run_until") == want
