"""The grouping kernels at the limits of their paths: buckets at and above what
a block holds in shared memory, segments at and above the longest it ranks
there (512), the longest a warp sorts (1,024) and the radix sort's shares, one
or several long segments, a last bucket that is not full.  Exact against the
numpy restatement."""

import numpy as np
import pytest

from test_group_events import EXT, expected_grouping, make_events, run_device

pytestmark = pytest.mark.gpu


def _check(lib, ev, neurons, fn):
    rc, g, s = run_device(lib, ev, neurons, fn)
    assert rc == 0
    want_g, want_s = expected_grouping(ev, neurons)
    assert np.array_equal(s, want_s) and np.array_equal(g, want_g)


@pytest.mark.parametrize("fn", ["snncuda_group_events", "snncuda_group_events_static"])
@pytest.mark.parametrize("busy", [512, 513, 1024, 1025, 4096, 4097, 33_000])
@pytest.mark.parametrize("neurons", [1, 257, 3000])
def test_busy_targets(gpu_lib, fn, busy, neurons):
    rng = np.random.default_rng(busy + neurons)
    ev = make_events(rng, busy + 700, neurons)
    hot = rng.permutation(ev.size)[:busy]  # exactly `busy` events go to one neuron, the rest elsewhere
    ev &= ~np.uint64(0x7FFFFFFF)
    ev |= np.where(np.arange(ev.size) % neurons == neurons // 2, 0, np.arange(ev.size) % neurons).astype(np.uint64)
    ev[hot] = (ev[hot] & ~np.uint64(0x7FFFFFFF)) | np.uint64(neurons // 2)
    _check(gpu_lib, ev, neurons, fn)


def test_many_long_segments(gpu_lib):
    rng = np.random.default_rng(3)
    ev = make_events(rng, 700_000, 2000)
    target = rng.choice([3, 4, 5, 700, 1999], ev.size).astype(np.uint64)
    ev = np.where(rng.random(ev.size) < 0.6, (ev & ~np.uint64(0x7FFFFFFF)) | target, ev)
    _check(gpu_lib, ev, 2000, "snncuda_group_events")


@pytest.mark.parametrize("count", [4095, 4096, 4097])
def test_full_bucket(gpu_lib, count):
    rng = np.random.default_rng(count)
    ev = make_events(rng, count, 200)  # one bucket
    _check(gpu_lib, ev, 200, "snncuda_group_events")
    assert (ev & EXT).any()


def test_a_long_segment_for_every_warp(gpu_lib):
    """More segments above 512 events than the kernel has warps: up to 1,024
    events each is a warp's work then, more a block's."""
    neurons, rng = 6000, np.random.default_rng(9)
    sizes = rng.choice([512, 513, 600, 1024, 1025, 1300], neurons)
    ev = make_events(rng, int(sizes.sum()), neurons)
    target = rng.permutation(np.repeat(np.arange(neurons, dtype=np.uint64), sizes))
    _check(gpu_lib, (ev & ~np.uint64(0x7FFFFFFF)) | target, neurons, "snncuda_group_events")
