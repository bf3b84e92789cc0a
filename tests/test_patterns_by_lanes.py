"""Temporal patterns of targets with several reference patterns, in the kernel that
takes two, four or eight lanes for a target by the most patterns that any keeps:
targets with 1 up to that many side by side, exact against the CPU oracle."""

import numpy as np
import pytest

from snncuda_gb300 import synthetic
from snncuda_gb300.simulation import Simulation, default_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("most", [2, 3, 4, 5, 8, 9, 20])
def test_patterns(gpu_lib, port_lib, most):
    n = 10_007  # more than 32 lanes each would fill the GPU
    w = synthetic.STDP_100K.scaled(neurons=n, fanout=8, seed=most, weight_scale=0.3, max_weight=0.5, drive_rate_hz=40.0)
    net, drive = synthetic.build_network(w), synthetic.build_drive(w, 48)
    net.max_reference_patterns = np.random.default_rng(most).integers(1, most + 1, n).astype(np.uint64)
    net.max_reference_patterns[5] = most
    out = []
    for lib, advance in ((gpu_lib, "profile"), (port_lib, "run_until")):  # (profile: the launched kernels)
        cfg = default_config(lib, raster_capacity=1 << 20)
        cfg.max_weight = 1.0
        sim = Simulation(net, cfg, lib)
        sim.inject(*drive)
        getattr(sim, advance)(47)
        out.append((sim.digest(), sim.recognition(), [x.tolist() for x in sim.raster()]))
        sim.close()
    assert out[0] == out[1]
