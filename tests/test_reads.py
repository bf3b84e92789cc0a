"""State reads unpacked on the device (from 8,192 neurons or synapses on, in
rounds of half the wheel-slot capacity): every array equals the CPU oracle's,
at sizes on both sides of the limit and of a round, for a network of its own
and for a batch member, before and after an eviction."""

import numpy as np
import pytest

from snncuda_gb300 import synthetic
from snncuda_gb300.simulation import Batch, Simulation, default_config

pytestmark = pytest.mark.gpu


def _workload(neurons, fanout, patterns=1):
    return synthetic.STDP_100K.scaled(neurons=neurons, fanout=fanout, seed=neurons, weight_scale=0.2, max_weight=0.4,
                                      max_reference_patterns=patterns, drive_rate_hz=20.0)


def _config(lib, slots=0):
    cfg = default_config(lib, slot_event_capacity=slots)
    cfg.max_weight = 1.0
    return cfg


def _same(got, want):
    assert got.keys() == want.keys()
    for k in want:
        assert got[k].dtype == want[k].dtype and np.array_equal(got[k], want[k]), k


@pytest.mark.parametrize("neurons,fanout,slots", [(2048, 4, 0), (8191, 1, 0), (8192, 1, 16384), (8200, 2, 16384),
                                                  (20001, 3, 16384)])
def test_reads(gpu_lib, port_lib, neurons, fanout, slots):
    w = _workload(neurons, fanout, 1 + neurons % 2)
    net, drive = synthetic.build_network(w), synthetic.build_drive(w, 40)
    sims = []
    for lib in (gpu_lib, port_lib):
        sim = Simulation(net, _config(lib, slots), lib)
        sim.inject(*drive)
        sim.run_until(39)
        sims.append(sim)
    gpu, port = sims
    for turn in range(2):
        _same(gpu.neurons(), port.neurons())
        _same(gpu.synapses(), port.synapses())
        a, b = gpu.counters(), port.counters()
        assert all(a[k] == b[k] for k in ("delivered_spikes", "fired_spikes", "pending_events", "next_tick"))
        if turn == 0:
            gpu.evict()
            for sim in sims:
                sim.inject([1, 2], [41, 60], [1.0, 1.0])
                sim.run_until(50)
    for sim in sims:
        sim.close()


def test_batch_member_reads(gpu_lib, port_lib):
    sizes = [(300, 5), (9000, 2), (40, 3), (8192, 1)]
    members = [_workload(n, f) for n, f in sizes]
    nets = [synthetic.build_network(w) for w in members]
    out = []
    for lib in (gpu_lib, port_lib):
        b = Batch(nets, _config(lib), lib, stdp_enabled=[True, False, True, True])
        for i, w in enumerate(members):
            b.inject(i, *synthetic.build_drive(w, 30))
        b.run_until(24)
        out.append(b)
    for i in range(len(sizes)):
        _same(out[0].neurons(i), out[1].neurons(i))
        _same(out[0].synapses(i), out[1].synapses(i))
        a, b = out[0].counters(i), out[1].counters(i)
        assert all(a[k] == b[k] for k in ("delivered_spikes", "fired_spikes", "pending_events", "external_events"))
