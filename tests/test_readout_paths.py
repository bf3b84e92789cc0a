"""Readout kernels at the edges of their tiles: inputs at and above the hash
table's limit, top-k with ties, negative and zero events, more readouts and
hidden neurons than a block has threads, neurons that are both.  Every weight
is a power of two and the sums need few bits, so any summation order gives the
same float: results equal the CPU oracle's exactly."""

import numpy as np
import pytest

from snncuda_gb300.connectome import Connectome
from snncuda_gb300.simulation import Readout


def _network(n, synapses, seed, delays=(2, 4)):
    rng = np.random.default_rng(seed)
    return rng, Connectome(
        threshold=rng.choice([0.5, 1.0, 2.0], n).astype(np.float32), pattern_window_ticks=np.full(n, 10, np.uint64),
        similarity_threshold=np.full(n, 0.9, np.float32), max_reference_patterns=np.full(n, 1, np.uint64),
        source=rng.integers(0, n, synapses, dtype=np.uint32), target=rng.integers(0, n, synapses, dtype=np.uint32),
        weight=rng.choice([-0.5, 0.5, 1.0], synapses).astype(np.float32), max_weight=np.full(synapses, 2, np.float32),
        delay_ticks=rng.integers(delays[0], delays[1] + 1, synapses, dtype=np.uint32),
        compartment=np.ones(synapses, np.uint8), receptor=np.zeros(synapses, np.uint8),
        plasticity_enabled=np.ones(synapses, np.uint8))


def _samples(rng, n, counts):
    return [[(int(a), float(b)) for a, b in zip(rng.integers(0, n, c), rng.choice([-0.5, 0.5, 0.25, 0.0], c))]
            for c in counts]


def _equal(got, want):
    for a, b in zip(got, want):
        assert np.array_equal(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("counts", [(0, 1, 33, 300), (4096, 5), (4097, 5)])
def test_feedforward_inputs(gpu_lib, port_lib, counts):
    n = 9001
    rng, net = _network(n, 40_000, 5)
    samples = _samples(rng, n, counts)
    for s, c in zip(samples, counts):  # distinct neurons: the merged count is c
        if c > 300:
            s[:] = [(int(a), b) for a, (_, b) in zip(rng.permutation(n), s)]
    readouts = rng.choice(n, 77, replace=False)
    _equal(Readout(net, gpu_lib).feedforward(samples, readouts), Readout(net, port_lib).feedforward(samples, readouts))


@pytest.mark.gpu
@pytest.mark.parametrize("n,synapses,readouts,top_hidden,top_readouts,scores", [
    (40, 300, 1, 1, 1, 1),
    (700, 4000, 16, 5, 1, 1),      # many equal events at the boundary: the first ones win
    (700, 4000, 16, 600, 3, 1),    # fewer positive events than places: zeros and negatives fill them
    (700, 4000, 600, 20, 40, 0),   # more readouts than threads; zero scores open gates
    (1300, 9000, 513, 0, 0, 1),    # no selection, threshold gates
    (1300, 9000, 30, 699, 29, 0),
])
def test_recurrent_selection(gpu_lib, port_lib, n, synapses, readouts, top_hidden, top_readouts, scores):
    rng, net = _network(n, synapses, n + readouts)
    samples = _samples(rng, n, (0, 1, min(n, 90), 400))
    chosen = rng.choice(n, readouts, replace=False)
    options = dict(top_k_hidden=top_hidden, top_k_feedback_readouts=top_readouts, use_scores_not_spikes=scores)
    both = rng.permutation(n)[:n - n // 4]  # some readouts are hidden neurons too
    for hidden in (None, both):
        if hidden is None and readouts == n:
            continue
        got = Readout(net, gpu_lib).recurrent(samples, chosen, hidden, **options)
        want = Readout(net, port_lib).recurrent(samples, chosen, hidden, **options)
        assert got[3] == want[3]
        _equal(got[:3], want[:3])
