"""Small networks run whole ticks in one cluster of eight blocks, each with an
eighth of the targets.  Networks at the edges of that split, ticks with more
events than it takes (the other kernels finish the run), more fires than it
places at a time, many delivery delays, injections beyond the wheel and runs
in pieces: counters, rasters and state digests equal the CPU oracle's."""

import numpy as np
import pytest

from snncuda_gb300 import synthetic
from snncuda_gb300.connectome import Connectome
from snncuda_gb300.simulation import SNNCudaError, Simulation, default_config

pytestmark = pytest.mark.gpu


def _random(n, fanout, delays, patterns=1, codes=1, weight=(0.05, 0.4), seed=1):
    rng = np.random.default_rng(seed)
    s = n * fanout
    ptr = np.zeros(s + 1, np.uint64)
    ptr[1:] = np.cumsum(rng.integers(1, codes + 1, s))
    return Connectome(
        threshold=np.ones(n, np.float32), pattern_window_ticks=np.full(n, 9, np.uint64),
        similarity_threshold=np.full(n, 0.9, np.float32), max_reference_patterns=np.full(n, patterns, np.uint64),
        source=np.repeat(np.arange(n, dtype=np.uint32), fanout), target=rng.integers(0, n, s, dtype=np.uint32),
        weight=rng.uniform(*weight, s).astype(np.float32), max_weight=np.full(s, 0.5, np.float32),
        delay_ticks=rng.choice(delays, s).astype(np.uint32), compartment=rng.integers(0, 4, s, dtype=np.uint8),
        receptor=rng.integers(0, 4, s, dtype=np.uint8), plasticity_enabled=rng.integers(0, 2, s, dtype=np.uint8),
        code_offset_ptr=ptr, code_offsets=rng.integers(0, 4, int(ptr[-1]), dtype=np.uint32))


def _run(lib, net, stops, bursts, slots=0):
    n = net.neuron_count
    cfg = default_config(lib, raster_capacity=1 << 20, slot_event_capacity=slots)
    cfg.max_weight = 1.0
    sim = Simulation(net, cfg, lib)
    rng = np.random.default_rng(n)
    for tick, share in bursts:
        who = np.flatnonzero(rng.random(n) < share).astype(np.uint32)
        sim.inject(who, np.full(who.size, tick), rng.uniform(0.4, 1.6, who.size).astype(np.float32))
    out = []
    for stop in stops:
        sim.run_until(stop)
        sim.inject([n - 1, 0], [stop + 3, stop + 900], [1.2, 1.2])
        c, r = sim.counters(), sim.raster()
        out.append(({k: c[k] for k in ("delivered_spikes", "fired_spikes", "external_events", "pending_events",
                                       "next_tick", "max_slot_events")}, r[0].tolist(), r[1].tolist(), sim.digest()))
    sim.close()
    return out


@pytest.mark.parametrize("n,fanout", [(1, 1), (7, 3), (8, 2), (9, 5), (513, 4), (4097, 2), (32768, 1)])
@pytest.mark.parametrize("patterns,codes", [(1, 2), (3, 6)])
def test_splits(gpu_lib, port_lib, n, fanout, patterns, codes):
    net = _random(n, fanout, np.arange(0, 12), patterns, codes)
    args = (net, (0, 1, 40, 41, 1100), [(0, 0.2), (3, 0.2), (30, 0.1), (990, 0.2)])
    assert _run(gpu_lib, *args) == _run(port_lib, *args)


@pytest.mark.parametrize("delays", [np.arange(1, 3), np.arange(1, 250)])
def test_bursts(gpu_lib, port_lib, delays):
    """Every neuron fires in one tick: 2,000 fires placed in one or several
    rounds; then more than 8,192 events come due in a tick."""
    net = _random(2000, 12, delays, weight=(0.001, 0.01))
    args = (net, (5, 300), [(2, 1.0), (4, 1.0), (150, 0.5)])
    assert _run(gpu_lib, *args) == _run(port_lib, *args)


def test_slot_overflow(gpu_lib):
    """A delivery slot without room reports the same error as ever."""
    net = _random(500, 40, [4], weight=(0.001, 0.002))
    cfg = default_config(gpu_lib, slot_event_capacity=4096)
    sim = Simulation(net, cfg, gpu_lib)
    sim.inject(np.arange(500), np.zeros(500), np.full(500, 2.0))
    with pytest.raises(SNNCudaError, match="slot capacity"):
        sim.run_until(10)
    sim.close()


def test_long_run_in_pieces(gpu_lib, port_lib):
    w = synthetic.PLAIN_1K.scaled(neurons=300, fanout=40, drive_rate_hz=20.0)
    net, drive = synthetic.build_network(w), synthetic.build_drive(w, 1300)
    out = []
    for lib, stops in ((gpu_lib, (511, 512, 1024, 1299)), (port_lib, (1299,))):
        sim = Simulation(net, default_config(lib, raster_capacity=1 << 20), lib)
        sim.inject(*drive)
        for stop in stops:
            sim.run_until(stop)
        out.append((sim.digest(), [x.tolist() for x in sim.raster()]))
        sim.close()
    assert out[0] == out[1]


@pytest.mark.parametrize("kind", ["rows", "classes", "fan-out"])
def test_costly_ticks(gpu_lib, port_lib, kind):
    """Networks whose ticks lose time in the one-kernel form (many rows of
    post-spike STDP, fires times delivery classes, one fire's events), so that
    the other kernels take over in the middle of a run."""
    rng = np.random.default_rng(4)
    if kind == "rows":  # 4,000 inputs to each of 40 outputs that fire in every tick
        n, delays = 4040, [1]
        source, target = np.repeat(np.arange(4000), 40), np.tile(np.arange(4000, 4040), 4000)
    elif kind == "classes":
        n, delays = 2500, np.arange(1, 250)
        source, target = np.repeat(np.arange(n), 2), rng.integers(0, n, 2 * n)
    else:
        n, delays = 9000, np.arange(1, 250)
        source, target = np.repeat(np.arange(3), 60_000), rng.integers(3, n, 180_000)
    s = source.size
    threshold = np.ones(n, np.float32)
    if kind == "rows":
        threshold[4000:] = 0.01
    net = Connectome(
        threshold=threshold, pattern_window_ticks=np.full(n, 9, np.uint64), similarity_threshold=np.full(n, 0.9, np.float32),
        max_reference_patterns=np.full(n, 1, np.uint64), source=source.astype(np.uint32), target=target.astype(np.uint32),
        weight=np.full(s, 0.004, np.float32), max_weight=np.full(s, 0.005, np.float32),
        delay_ticks=rng.choice(delays, s).astype(np.uint32), compartment=np.ones(s, np.uint8), receptor=np.zeros(s, np.uint8),
        plasticity_enabled=np.ones(s, np.uint8))
    out = []
    for lib in (gpu_lib, port_lib):
        sim = Simulation(net, default_config(lib, raster_capacity=1 << 20), lib)
        drive = np.random.default_rng(6)
        for tick in range(60):
            some = [tick % 3] if kind == "fan-out" and tick % 4 == 0 else [3] if kind == "fan-out" else \
                drive.choice(2500 if kind == "classes" else 4000, 60 if kind == "rows" else 900, replace=False)
            sim.inject(some, np.full(len(some), tick), np.full(len(some), 1.5, np.float32))
        for stop in (0, 1, 30, 59):
            sim.run_until(stop)
            c, r = sim.counters(), sim.raster()
            out.append(([c[k] for k in ("delivered_spikes", "fired_spikes", "external_events", "pending_events")],
                        r[0].tolist(), r[1].tolist(), sim.digest()))
        sim.close()
    assert out[:4] == out[4:]
