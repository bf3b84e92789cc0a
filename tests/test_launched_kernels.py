"""The launched tick kernels with settings that the smaller networks of the other
tests do not bring to them (those run whole ticks in one kernel): a network
above that kernel's limit with each placement of post-spike STDP and of the
temporal patterns, a tiny placing pass and odd grids, and with staging copies
that are not waited for.  Counters, rasters and digests equal the oracle's."""

import numpy as np
import pytest

from snncuda_gb300 import synthetic
from snncuda_gb300.simulation import SNNCudaError, Simulation, default_config

pytestmark = pytest.mark.gpu

NEURONS, TICKS = 40_000, 60  # one kernel: at most 32,768 neurons
SNNCUDA_ERR_TIMEOUT = 5


@pytest.fixture(scope="module", params=[1, 3], ids=["one_pattern", "three_patterns"])
def case(request, port_lib):
    w = synthetic.STDP_100K.scaled(neurons=NEURONS, fanout=60, ticks=TICKS, seed=17, weight_scale=0.1, max_weight=0.1,
                                   drive_rate_hz=20.0, max_reference_patterns=request.param)
    net, drive = synthetic.build_network(w), synthetic.build_drive(w, TICKS)
    sim = _simulation(port_lib, net, drive)
    sim.run_until(TICKS - 1)
    want = _state(sim)
    assert want[0]["max_slot_events"] > 20_000  # several tiles for one block
    sim.close()
    return net, drive, want


def _simulation(lib, net, drive, **config):
    cfg = default_config(lib, raster_capacity=1 << 22, **config)
    cfg.max_weight = 1.0
    sim = Simulation(net, cfg, lib)
    sim.inject(*drive)
    return sim


def _state(sim):
    c, r = sim.counters(), sim.raster()
    keep = ("delivered_spikes", "fired_spikes", "synaptic_events", "external_events", "max_slot_events", "next_tick")
    return {k: c[k] for k in keep}, r[0].tolist(), r[1].tolist(), sim.digest()


TUNING = dict(grid_events=600, grid_walk=1, grid_bucket=7, grid_temporal=5, ticks_per_graph=5, block_threads=0,
              slot_event_capacity=0, scatter_pass_events=0, side_serial=0)


@pytest.mark.parametrize("changes", [dict(side_serial=1), dict(side_serial=0, scatter_pass_events=64),
                                     dict(side_serial=1, scatter_pass_events=64, grid_events=3)])
def test_tuned_runs(gpu_lib, case, changes):
    net, drive, want = case
    sim = _simulation(gpu_lib, net, drive)
    sim.run_until(9)
    sim.apply_tuning(dict(TUNING, **changes))
    sim.run_until(TICKS - 1)
    assert _state(sim) == want
    sim.close()


@pytest.mark.parametrize("grid_bucket", [1, 7])
def test_waits_that_give_up(gpu_lib, case, grid_bucket):
    """A limit of 0: k_events' copies, and at one counting block the due list's too."""
    net, drive, want = case
    sim = _simulation(gpu_lib, net, drive, stage_wait_ns=0)
    sim.apply_tuning(dict(TUNING, grid_bucket=grid_bucket))
    with pytest.raises(SNNCudaError) as err:
        sim.run_until(TICKS - 1)
    assert err.value.status == SNNCUDA_ERR_TIMEOUT
    assert _state(sim) == want
    sim.close()
