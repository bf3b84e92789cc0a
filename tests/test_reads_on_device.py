"""State reads at the sizes from which they are unpacked on the device (16,384
neurons, 12,288 synapses), in one round and in several, and with a wheel slot
too small for that: every array equals the CPU oracle's, for a network of its
own and for a batch member."""

import pytest

from snncuda_gb300 import synthetic
from snncuda_gb300.simulation import Batch, Simulation
from test_reads import _config, _same, _workload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("neurons,fanout,slots", [
    (12287, 1, 0), (12288, 1, 0), (16383, 1, 0), (16384, 1, 0),  # one round from these sizes on
    (33000, 2, 0), (65536, 1, 0),     # two rounds of the neurons; up to three of the synapses
    (16384, 1, 2048),                 # sixteen rounds: copied whole
    (24000, 3, 16384),                # the synapses in nine rounds, the neurons whole
    (17500, 4, 6144), (17400, 4, 6144)])  # 70,000 synapses in 23 rounds; 69,600 need 70,656
def test_reads(gpu_lib, port_lib, neurons, fanout, slots):
    w = _workload(neurons, fanout, 1 + neurons % 2).scaled(drive_rate_hz=8.0)
    net, drive = synthetic.build_network(w), synthetic.build_drive(w, 24)
    sims = []
    for lib in (gpu_lib, port_lib):
        sim = Simulation(net, _config(lib, slots), lib)
        sim.inject(*drive)
        sim.run_until(23)
        sims.append(sim)
    _same(sims[0].neurons(), sims[1].neurons())
    _same(sims[0].synapses(), sims[1].synapses())
    for sim in sims:
        sim.close()


def test_batch_member_reads(gpu_lib, port_lib):
    members = [_workload(n, f) for n, f in [(300, 5), (17001, 1), (40, 3), (16384, 2)]]
    nets = [synthetic.build_network(w) for w in members]
    out = []
    for lib in (gpu_lib, port_lib):
        b = Batch(nets, _config(lib), lib, stdp_enabled=[True, False, True, True])
        for i, w in enumerate(members):
            b.inject(i, *synthetic.build_drive(w, 30))
        b.run_until(24)
        out.append(b)
    for i in range(len(members)):
        _same(out[0].neurons(i), out[1].neurons(i))
        _same(out[0].synapses(i), out[1].synapses(i))
