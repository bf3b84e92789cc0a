"""Sizes of the grouping calls' scratch, from the layout both entry points use:
the list of targets that have more events than a warp sorts fits behind the
counter rows' start for every documented size, and the arrays do not overlap.
Host code only (compiled here with g++)."""

import json
import pathlib
import shutil
import subprocess

import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]

PROGRAM = r"""
#include <cuda_runtime_api.h>
#include <cstdio>
#include "engine.h"
int main() {
    using namespace snngb;
    unsigned count, neurons;
    std::printf("[");
    for (bool first = true; std::scanf("%u %u", &count, &neurons) == 2; first = false) {
        const GroupLayout l = group_layout(count, neurons);
        std::printf("%s[%zu,%zu,%zu,%zu,%zu,%zu,%zu,%zu,%u,%u,%u,%zu]", first ? "" : ",", l.bcnt, l.btot, l.bstart,
                    l.bcur, l.grp_tmp, l.slot_count, l.ts, l.bytes, group_buckets(neurons), kWarpSortEvents, kGroupGrid,
                    sizeof(TickState));
    }
    std::printf("]");
}
"""


@pytest.fixture(scope="module")
def layouts(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    include = pathlib.Path(nvcc).resolve().parents[1] / "include"
    if shutil.which("g++") is None or not (include / "cuda_runtime_api.h").exists():
        pytest.skip("no host compiler or CUDA headers")
    work = tmp_path_factory.mktemp("layout")
    (work / "layout.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(ROOT / "snncuda_gb300" / "csrc"), "-I", str(include),
                    str(work / "layout.cpp"), "-o", str(work / "layout")], check=True)

    def run(sizes):
        out = subprocess.run([str(work / "layout")], input="\n".join(f"{c} {n}" for c, n in sizes),
                             capture_output=True, text=True, check=True)
        return json.loads(out.stdout)

    return run


def test_listed_targets_fit(layouts):
    edges = [1, 2, 255, 256, 257, (1 << 18), *(v for s in range(21, 28) for v in ((1 << s) - 1, 1 << s, (1 << s) + 1)),
             (1 << 28) - 1, 1 << 28]
    sizes = [(c, n) for n in edges for c in (0, 1, 513, 1 << 20, 1 << 27, 1_080_000_000, (1 << 31) - 1)]
    for (count, neurons), row in zip(sizes, layouts(sizes)):
        bcnt, btot, bstart, bcur, grp_tmp, slot, ts, end, buckets, warp_events, grid, ts_bytes = row
        # targets that can each hold more than `warp_events` of the events
        listed = min(neurons, count // (warp_events + 1))
        assert (btot - bcnt) // 4 >= max(listed, grid * buckets), (count, neurons)
        assert (bstart - btot) // 4 >= buckets and (bcur - bstart) // 4 >= buckets + 1, (count, neurons)
        assert (grp_tmp - bcur) // 4 >= buckets and slot - grp_tmp >= 16 * count, (count, neurons)
        assert ts - slot >= 4 and end - ts >= ts_bytes, (count, neurons)
        assert all(at % 256 == 0 for at in row[:8])
