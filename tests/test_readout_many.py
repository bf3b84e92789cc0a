"""One-hop readouts with enough results for a thread each: on both sides of the
number of results (262,144) and of the synapses per readout (256) where that
begins and ends, samples above and below the hash table's limit.  Weights are
powers of two, so sums in any order are exact: results equal the CPU oracle's."""

import numpy as np
import pytest

from snncuda_gb300.simulation import Readout
from test_readout_paths import _equal, _network, _samples


@pytest.mark.gpu
@pytest.mark.parametrize("samples,readouts,synapses", [(513, 511, 20_000), (512, 512, 20_000), (300, 1000, 257_000),
                                                       (300, 1000, 256_000)])
def test_many_results(gpu_lib, port_lib, samples, readouts, synapses):
    n = 5000
    rng, net = _network(n, synapses, samples)
    if synapses > 200_000:  # all of them at 1,000 readouts, 256 or 257 each
        net.target = (np.arange(synapses) % 1000).astype(np.uint32)
        chosen = rng.permutation(1000)
    else:
        chosen = rng.choice(n, readouts, replace=False)
    batch = _samples(rng, n, [int(c) for c in rng.integers(0, 40, samples - 2)] + [4097, 1])
    batch[-2] = [(int(a), b) for a, (_, b) in zip(rng.permutation(n), batch[-2])]
    _equal(Readout(net, gpu_lib).feedforward(batch, chosen), Readout(net, port_lib).feedforward(batch, chosen))
    _equal(Readout(net, gpu_lib).feedforward(batch[:-2], chosen), Readout(net, port_lib).feedforward(batch[:-2], chosen))
