"""One readout handle in two host threads: each call gets its own inputs'
results, whatever the other's sizes are."""

import threading

import numpy as np
import pytest

from snncuda_gb300.simulation import Readout
from test_readout_paths import _network, _samples

pytestmark = pytest.mark.gpu


def test_two_threads(gpu_lib):
    rng, net = _network(3000, 40_000, 8)
    readout, alone = Readout(net, gpu_lib), Readout(net, gpu_lib)
    calls = []
    for count, outs in ((3, 20), (200, 300), (40, 7), (600, 64)):
        samples, chosen = _samples(rng, 3000, rng.integers(1, 60, count)), rng.choice(3000, outs, replace=False)
        calls.append(lambda h, s=samples, c=chosen: h.feedforward(s, c))
        calls.append(lambda h, s=samples[:20], c=chosen: h.recurrent(s, c, top_k_hidden=30))
    want = [call(alone) for call in calls]
    wrong = []

    def work(first):
        for k in range(60):
            i = (first + 3 * k) % len(calls)
            for a, b in zip(calls[i](readout), want[i]):
                if not np.array_equal(a, b):
                    wrong.append(i)

    threads = [threading.Thread(target=work, args=(first,)) for first in (0, 3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


def test_large_call_gives_its_memory_back(gpu_lib):
    """After a call with 400 MB of results, the handle keeps no buffer of that size."""
    import torch
    _, net = _network(9000, 9000, 2)
    readout, chosen = Readout(net, gpu_lib), np.arange(8192)
    samples = [[(i, 1.0)] for i in range(4096)]
    readout.feedforward(samples[:2], chosen[:2])
    before = torch.cuda.mem_get_info()[0]
    scores = readout.feedforward(samples, chosen)[0]
    assert before - torch.cuda.mem_get_info()[0] < 300 << 20
    assert np.array_equal(readout.feedforward(samples[:64], chosen)[0], scores[:64])
