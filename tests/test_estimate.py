"""snncuda_sim_estimate_bytes, by which the server admits jobs, covers the
buffers of a simulation that has many neurons and hardly any synapses: the
per-neuron state and the grouping's bucket counters, on both sides of the bucket
counts where the counters' share is largest.  Host code: runs without a GPU."""

import ctypes

import numpy as np
import pytest

from conftest import GPU_PATH, _ensure_built
from snncuda_gb300.connectome import Connectome
from snncuda_gb300.simulation import _network_struct

SMS = 148  # no device of this family has fewer


def _estimate(lib, n, slots):
    from snncuda_gb300.simulation import default_config
    z, u8 = np.zeros(0, np.uint32), np.zeros(0, np.uint8)
    net = Connectome(
        threshold=np.ones(n, np.float32), pattern_window_ticks=np.ones(n, np.uint64),
        similarity_threshold=np.ones(n, np.float32), max_reference_patterns=np.ones(n, np.uint64), source=z, target=z,
        weight=np.zeros(0, np.float32), max_weight=np.zeros(0, np.float32), delay_ticks=z, compartment=u8, receptor=u8,
        plasticity_enabled=u8)
    struct, keep = _network_struct(net)
    out = ctypes.c_uint64()
    cfg = default_config(lib, slot_event_capacity=slots)
    assert lib.snncuda_sim_estimate_bytes(ctypes.byref(struct), ctypes.byref(cfg), ctypes.byref(out)) == 0
    return out.value


@pytest.mark.parametrize("n", [1, 29_000, 30_000, 1_000_000, (1 << 21) - 64, 1 << 21, (1 << 21) + 1, 4_000_000])
def test_covers_the_buffers(n):
    from snncuda_gb300 import _abi
    _ensure_built()
    lib, slots, window = _abi.bind(str(GPU_PATH)), 4096, 1
    shift = 5 if n >> 6 < 3 * SMS else 6
    while shift < 8 and n >> (shift + 1) >= 20 * SMS:  # (hardly any synapses: wide buckets)
        shift += 1
    while -(-n >> shift) > 32768:
        shift += 1
    buckets = -(-n >> shift)
    fires = min(slots, max(65536, 4 * n))
    state = n * (64 + 64 + 32 + 8 * (window + 1) + 48 + 8 * (window + 1))  # parameters, records, patterns
    state += n * (8 + 8 + 4 + 4 + 8)                   # row pointers, segments, fired targets
    state += 2 * slots * 8 + slots * (8 + 3 * 16 + 4)  # wheel, events of a tick
    state += fires * 4 + fires // 8 * 12
    counters = 4 * SMS * 4 * buckets + 3 * 4 * buckets
    sorting = n * 16  # counts and offsets of creation's sorts
    assert _estimate(lib, n, slots) >= state + counters + sorting
