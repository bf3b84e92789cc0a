"""Performance cases of the tick engine, the batched form, the grouping
building block and the inference readouts, through their public entry points.

Every simulation case keeps a running network (as a user's program does) and
one pass injects the next stretch of its drive, advances it and reads back what
such a program looks at.  The networks are this repository's synthetic
workloads (`snncuda_gb300.synthetic`) at several sizes, with weights scaled by
10 / fan-out (0.05 at most) so that every size stays driven by its input, as
the batched benchmark's members are.
"""

import ctypes
import math

import numpy as np
import torch

from snncuda_gb300 import synthetic
from snncuda_gb300.connectome import AMPA, BASAL, Connectome
from snncuda_gb300.simulation import Batch, Readout, Simulation, backend, default_config


def listed():
    return [
        # A closed loop around a small network: an agent injects one tick's
        # input, advances one tick and reads the fires.  The smallest call.
        {"name": "step_1k", "kind": "step", "neurons": 1000, "fanout": 100},
        # The plain 1,000-neuron network with the default neuron parameters
        # (window 500, 500 reference patterns), 100 ticks a call.
        {"name": "plain_1k", "kind": "plain", "neurons": 1000, "fanout": 100, "ticks": 100},
        # The feed-forward relay of the reference's spike throughput
        # benchmark: 288 columns of six 16-neuron layers, one-to-one, every
        # first-layer neuron stimulated, 7 ticks.
        {"name": "relay_27k", "kind": "relay", "columns": 288, "layers": 6, "width": 16},
        # Training with long spike codes and several reference patterns per
        # neuron; the weights and all other synapse state are read after
        # every presentation.
        {"name": "train_5k", "kind": "train", "neurons": 5003, "fanout": 200, "codes": 8, "patterns": 3, "ticks": 64},
        # An ordinary plastic network (the 100k network's distributions).
        {"name": "stdp_20k", "kind": "stdp", "neurons": 20000, "fanout": 1000, "ticks": 128, "stimulus": False},
        # A trained network run with plasticity and temporal learning off.
        {"name": "infer_33k", "kind": "infer", "neurons": 33331, "fanout": 500, "ticks": 100},
        # The recognition workload: 16 temporal codes over the background
        # drive, 2e8 plastic synapses.  The largest call.
        {"name": "recog_200k", "kind": "stdp", "neurons": 200000, "fanout": 1000, "ticks": 64, "stimulus": True},
        # Independent ragged networks advanced together in one handle.
        {"name": "batch_24", "kind": "batch", "networks": 24, "smallest": 211, "largest": 8009, "fanout": 100,
         "ticks": 50},
        # One tick's due list of the 1e6-neuron network regrouped by target.
        {"name": "group_13m", "kind": "group", "events": 13107211, "neurons": 1000000, "hub": 0.0, "static": False},
        # The same step inside a latency-critical loop that owns its memory.
        {"name": "group_30k", "kind": "group", "events": 30011, "neurons": 10007, "hub": 0.0, "static": True},
        # One-hop readout of a batch of samples.
        {"name": "readout_ff", "kind": "forward", "neurons": 20000, "fanout": 500, "samples": 64, "inputs": 100,
         "readouts": 100},
        # Recurrent readout: top-1 feedback, hidden selection, two iterations.
        {"name": "readout_rec", "kind": "recurrent", "neurons": 2000, "fanout": 40, "samples": 32, "inputs": 30,
         "readouts": 16, "iterations": 2, "top_k_hidden": 40},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "plain", "relay", "train", "stdp", "stdp", "infer", "batch", "group", "group", "forward",
                       "recurrent"])
    if kind == "step":
        return {"kind": kind, "neurons": _log(rng, 100, 5000), "fanout": rng.randint(20, 100)}
    if kind == "plain":
        return {"kind": kind, "neurons": _log(rng, 200, 4000), "fanout": rng.randint(40, 110), "ticks": rng.randint(20, 150)}
    if kind == "relay":
        return {"kind": kind, "columns": _log(rng, 4, 600), "layers": rng.randint(3, 8), "width": rng.randint(5, 32)}
    if kind == "train":
        return {"kind": kind, "neurons": _log(rng, 500, 6000), "fanout": rng.randint(50, 200), "codes": rng.randint(2, 8),
                "patterns": rng.randint(1, 6), "ticks": rng.randint(16, 96)}
    if kind == "stdp":
        return {"kind": kind, "neurons": _log(rng, 3000, 100000), "fanout": rng.randint(200, 1000),
                "ticks": rng.randint(32, 100), "stimulus": rng.random() < 0.5}
    if kind == "infer":
        return {"kind": kind, "neurons": _log(rng, 2000, 50000), "fanout": rng.randint(100, 700),
                "ticks": rng.randint(40, 120)}
    if kind == "batch":
        return {"kind": kind, "networks": rng.randint(3, 40), "smallest": rng.randint(60, 400),
                "largest": rng.randint(1000, 8000), "fanout": rng.randint(20, 150), "ticks": rng.randint(20, 80)}
    if kind == "group":
        static = rng.random() < 0.5
        return {"kind": kind, "events": _log(rng, 1000, 1 << 20 if static else 12000000),
                "neurons": _log(rng, 300, 200000 if static else 1500000), "hub": rng.choice([0.0, 0.0, 0.01, 0.05]),
                "static": static}
    if kind == "forward":
        return {"kind": kind, "neurons": _log(rng, 500, 20000), "fanout": rng.randint(40, 500),
                "samples": _log(rng, 1, 96), "inputs": rng.randint(10, 150), "readouts": rng.randint(2, 200)}
    return {"kind": kind, "neurons": _log(rng, 200, 2000), "fanout": rng.randint(20, 60), "samples": _log(rng, 1, 48),
            "inputs": rng.randint(5, 60), "readouts": rng.randint(2, 40), "iterations": rng.randint(1, 2),
            "top_k_hidden": rng.choice([0, 16, 40])}


# ---------------------------------------------------------------------------
# networks
# ---------------------------------------------------------------------------

def _scale(fanout):
    return min(0.05, 10.0 / fanout)


def _workload(case, seed):
    n, fanout, kind = case["neurons"], case["fanout"], case["kind"]
    if kind in ("step", "plain"):
        return synthetic.PLAIN_1K.scaled(neurons=n, fanout=fanout, seed=seed, weight_scale=min(0.3, 30.0 / fanout))
    scale = _scale(fanout)
    if kind == "train":
        # more offsets per spike: smaller weights keep the drive dominant
        return synthetic.STDP_100K.scaled(neurons=n, fanout=fanout, seed=seed, codes=(1, case["codes"]),
                                          code_offset_max=15, max_reference_patterns=case["patterns"],
                                          weight_scale=0.6 * scale, max_weight=0.6 * scale)
    base = synthetic.STDP_100K
    if case.get("stimulus"):  # its coinciding codes want the workload's own, smaller weights
        base, scale = synthetic.RECOG_1M, synthetic.RECOG_1M.weight_scale
    return base.scaled(neurons=n, fanout=fanout, seed=seed, weight_scale=scale, max_weight=scale)


def _relay(case):
    """`columns` chains of `layers` populations of `width` neurons, one-to-one."""
    cols, layers, width = case["columns"], case["layers"], case["width"]
    ids = np.arange(cols * layers * width, dtype=np.uint32).reshape(cols, layers, width)
    n, source, target = ids.size, ids[:, :-1].ravel(), ids[:, 1:].ravel()
    s = source.size
    net = Connectome(
        threshold=np.full(n, 1.0, np.float32), pattern_window_ticks=np.full(n, 16, np.uint64),
        similarity_threshold=np.full(n, 0.9, np.float32), max_reference_patterns=np.full(n, 8, np.uint64),
        source=source, target=target, weight=np.full(s, 1.0, np.float32), max_weight=np.full(s, 2.0, np.float32),
        delay_ticks=np.full(s, 1, np.uint32), compartment=np.full(s, BASAL, np.uint8),
        receptor=np.full(s, AMPA, np.uint8), plasticity_enabled=np.full(s, 1, np.uint8))
    return net, ids[:, 0].ravel()


def _fires(state, counters, room):
    """The pass's fire records, (tick, neuron) rows behind each other in a
    buffer of `room` rows (the rest stays zero)."""
    before, state["fires"] = state.get("fires", 0), counters["raster_count"]
    ticks, neurons = state["sim"].raster(before, counters["raster_count"] - before)
    rows = np.zeros((room, 2), np.int64)
    rows[:ticks.size, 0] = ticks
    rows[:ticks.size, 1] = neurons
    return rows


def _config(raster=0, **more):
    cfg = default_config(raster_capacity=raster, **more)
    cfg.max_weight = 1.0
    return cfg


def _start(sim, drive, ticks):
    """The running network a pass finds: `ticks` ticks of its drive are done."""
    n, t, w = drive
    keep = t < ticks
    sim.inject(n[keep], t[keep], w[keep])
    sim.run_until(ticks - 1)
    return ticks


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("step", "plain"):
        w = _workload(case, seed)
        # every neuron may keep its 500 patterns of 501 runs
        sim = Simulation(synthetic.build_network(w), _config(1 << 24, pattern_run_capacity=500 * 501))
        drive = synthetic.build_drive(w, 256 if kind == "step" else max(case["ticks"], 64))
        tick = _start(sim, drive, 64)
        n, t, x = drive
        if kind == "step":
            return {"kind": kind, "sim": sim, "tick": tick,
                    "drive": [(n[t == k], x[t == k]) for k in range(256)]}
        keep = t < case["ticks"]
        return {"kind": kind, "sim": sim, "tick": tick, "ticks": case["ticks"], "drive": (n[keep], t[keep], x[keep])}
    if kind == "relay":
        net, first = _relay(case)
        weights = np.random.default_rng(seed).uniform(0.9, 1.4, first.size).astype(np.float32)
        drive = (first, np.zeros(first.size, np.uint64), weights)
        return {"kind": kind, "sim": Simulation(net, _config()), "tick": 0, "ticks": case["layers"] + 1, "drive": drive}
    if kind in ("train", "stdp", "infer"):
        w = _workload(case, seed)
        more = {"slot_event_capacity": 1 << 18} if kind == "train" else {}
        sim = Simulation(synthetic.build_network(w), _config(1 << 25, **more))
        drive = synthetic.build_drive(w, max(case["ticks"], 32))
        tick = _start(sim, drive, 32)
        if kind == "infer":
            sim.set_plasticity(False)
            sim.set_temporal_learning(False)
        n, t, x = drive
        keep = t < case["ticks"]
        return {"kind": kind, "sim": sim, "tick": tick, "ticks": case["ticks"], "drive": (n[keep], t[keep], x[keep])}
    if kind == "batch":
        sizes = np.geomspace(case["smallest"], case["largest"], case["networks"]).astype(int)
        members = [synthetic.STDP_100K.scaled(neurons=int(n), fanout=case["fanout"], seed=seed + i,
                                              weight_scale=_scale(case["fanout"]), max_weight=_scale(case["fanout"]))
                   for i, n in enumerate(sizes)]
        batch = Batch([synthetic.build_network(w) for w in members], _config(),
                      stdp_enabled=[i % 2 == 0 for i in range(len(members))])
        return {"kind": kind, "batch": batch, "tick": 0, "ticks": case["ticks"],
                "drives": [synthetic.build_drive(w, case["ticks"]) for w in members]}
    if kind == "group":
        gen = torch.Generator(device="cuda").manual_seed(seed)
        count, neurons = case["events"], case["neurons"]

        def ints(high):
            return torch.randint(0, high, (count,), generator=gen, device="cuda", dtype=torch.int64)

        target = ints(neurons)
        if case["hub"] > 0:  # a hub neuron that receives this share of the events
            chance = torch.rand(count, generator=gen, device="cuda")
            target = torch.where(chance < case["hub"], torch.full_like(target, neurons // 3), target)
        external = torch.where(ints(100) == 0, 0x80000000, 0)
        events = (ints(1 << 31) << 32) | target | external
        return {"kind": kind, "lib": backend(), "static": case["static"], "neurons": neurons, "events": events,
                "grouped": torch.empty_like(events),
                "start": torch.empty(neurons + 1, dtype=torch.int32, device="cuda")}
    net, samples, readouts = _readout_case(case, seed)
    options = {}
    if kind == "recurrent":
        options = {"iterations": case["iterations"], "top_k_hidden": case["top_k_hidden"]}
    return {"kind": kind, "readout": Readout(net), "samples": samples, "readouts": readouts, "options": options}


def _readout_case(case, seed):
    """A network and samples of (neuron, weight) pairs over half of it."""
    n = case["neurons"]
    w = synthetic.STDP_100K.scaled(neurons=n, fanout=case["fanout"], seed=seed, weight_scale=0.5)
    rng = np.random.default_rng(seed)
    samples = [list(zip(rng.integers(0, n, case["inputs"]).tolist(),
                        rng.uniform(0.1, 1.0, case["inputs"]).astype(np.float32).tolist()))
               for _ in range(case["samples"])]
    return synthetic.build_network(w), samples, rng.choice(n, case["readouts"], replace=False).astype(np.uint32)


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

_COUNTERS = ("delivered_spikes", "fired_spikes", "synaptic_events", "external_events", "next_tick", "pending_events")


def _advance(state):
    """Injects the pass's drive and runs its ticks."""
    n, t, w = state["drive"]
    state["sim"].inject(n, t + np.uint64(state["tick"]), w)
    state["tick"] += state["ticks"]
    state["sim"].run_until(state["tick"] - 1)


def run(state):
    kind = state["kind"]
    if kind == "step":
        sim, tick = state["sim"], state["tick"]
        n, w = state["drive"][tick % len(state["drive"])]
        sim.inject(n, np.full(n.size, tick, np.uint64), w)
        sim.run_until(tick)
        state["tick"] = tick + 1
        counters = sim.counters()
        return {"fires": _fires(state, counters, 4 * sim.neuron_count), **{k: counters[k] for k in _COUNTERS}}
    if kind in ("plain", "stdp", "infer"):
        sim = state["sim"]
        _advance(state)
        counters = sim.counters()
        room = sim.neuron_count * (8 + state["ticks"] // 20)
        out = {"fires": _fires(state, counters, room), **{k: counters[k] for k in _COUNTERS}, **sim.neurons()}
        if kind != "plain":
            # the synapse records (64 bytes each) stay on the device while a
            # program of this size runs, which reads them once at its end (in
            # seconds, at 2e7 synapses); beside the whole neuron state their
            # checksums are compared, and the training case reads all of them
            out["checksums"] = np.array(sim.checksum(), np.uint64).view(np.int64)
        return out
    if kind == "relay":
        _advance(state)
        counters = state["sim"].counters()
        return {**{k: counters[k] for k in _COUNTERS}, **state["sim"].neurons()}
    if kind == "train":
        _advance(state)
        return {"neurons": state["sim"].neurons(), "synapses": state["sim"].synapses()}
    if kind == "batch":
        batch, base = state["batch"], np.uint64(state["tick"])
        for i, (n, t, w) in enumerate(state["drives"]):
            batch.inject(i, n, t + base, w)
        state["tick"] += state["ticks"]
        batch.run_until(state["tick"] - 1)
        counters = [batch.counters(i) for i in range(batch.count)]
        neurons = [batch.neurons(i) for i in range(batch.count)]
        sums = np.array(batch.checksums(), np.uint64).view(np.int64)
        return {"checksums": sums, "counters": np.array([[c[k] for k in _COUNTERS] for c in counters], np.int64),
                **{k: np.concatenate([a[k] for a in neurons]) for k in neurons[0]}}
    if kind == "group":
        lib = state["lib"]
        call = lib.snncuda_group_events_static if state["static"] else lib.snncuda_group_events
        rc = call(state["events"].data_ptr(), state["events"].numel(), state["neurons"], state["grouped"].data_ptr(),
                  state["start"].data_ptr(), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc != 0:
            raise RuntimeError(lib.snncuda_last_error().decode())
        return [state["grouped"], state["start"]]
    if kind == "forward":
        return list(state["readout"].feedforward(state["samples"], state["readouts"]))
    return list(state["readout"].recurrent(state["samples"], state["readouts"], **state["options"]))


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def _tick_work(neurons, fanout, ticks, offsets, rate):
    """Bytes and operations of `ticks` ticks at `rate` fires per neuron and
    tick: per event its word written at the fire and read at delivery, and its
    synapse state (weight, spike times and counts, the code window) read and
    written; per touched neuron its state read and written; the fires' own
    in-rows for the post-spike rule; the neuron state once more for the reader."""
    events = neurons * rate * fanout * offsets * ticks
    touched = min(neurons * ticks, events)
    fires = neurons * rate * ticks
    return {"bytes": int(events * (16 + 49) + touched * 96 + fires * fanout * 16 + neurons * 130),
            "flops": int(events * 20 + touched * 8 + fires * fanout * 4)}


def work(case):
    kind = case["kind"]
    if kind in ("step", "plain"):
        return _tick_work(case["neurons"], case["fanout"], case.get("ticks", 1), 1.0, 0.009)
    if kind == "relay":
        n = case["columns"] * case["layers"] * case["width"]
        return {"bytes": int(n * (16 + 49 + 96 + 130)), "flops": int(n * 28)}
    if kind == "train":
        w = _tick_work(case["neurons"], case["fanout"], case["ticks"], (1 + case["codes"]) / 2, 0.005)
        w["bytes"] += case["neurons"] * case["fanout"] * 2 * 73
        return w
    if kind in ("stdp", "infer"):
        return _tick_work(case["neurons"], case["fanout"], case["ticks"], 2.5, 0.005)
    if kind == "batch":
        neurons = int(np.geomspace(case["smallest"], case["largest"], case["networks"]).astype(int).sum())
        return _tick_work(neurons, case["fanout"], case["ticks"], 2.5, 0.005)
    if kind == "group":
        return {"bytes": 16 * case["events"] + 4 * (case["neurons"] + 1), "flops": 0}
    rows = case["readouts"] * case["fanout"]
    if kind == "forward":
        return {"bytes": 12 * rows + case["samples"] * (12 * case["inputs"] + 12 * case["readouts"]),
                "flops": 2 * case["samples"] * rows}
    steps = 20 * (1 + 2 * case["iterations"]) + 1
    return {"bytes": 24 * rows + case["samples"] * (12 * case["inputs"] + 12 * case["readouts"]),
            "flops": 4 * case["samples"] * steps * rows}


# ---------------------------------------------------------------------------
# 64-bit values of the readouts' scores
# ---------------------------------------------------------------------------

def _dense_inputs(samples, n):
    x = np.zeros((len(samples), n))
    for s, pairs in enumerate(samples):
        for neuron, weight in pairs:
            x[s, neuron] += weight
    return x


def exact(case, seed):
    if case["kind"] not in ("forward", "recurrent"):
        return None  # spikes, state words and event words: compared bit by bit
    net, samples, readouts = _readout_case(case, seed)
    n = net.neuron_count
    weight = net.weight.astype(np.float64)
    x = _dense_inputs(samples, n)
    position = np.full(n, -1)
    position[readouts] = np.arange(readouts.size)
    if case["kind"] == "forward":
        scores = np.zeros((len(samples), readouts.size))
        edges = np.flatnonzero(position[net.target] >= 0)
        column = position[net.target[edges]]
        for s in range(len(samples)):
            scores[s] = np.bincount(column, x[s, net.source[edges]] * weight[edges], readouts.size)
        return [scores, None, None]
    delay = np.maximum(net.delay_ticks, 1).astype(np.int64)
    steps = int(delay.max()) * (1 + 2 * case["iterations"]) + 1
    hidden = position < 0
    up = np.flatnonzero(hidden[net.source] & ~hidden[net.target])
    down = np.flatnonzero(~hidden[net.source] & hidden[net.target])
    scores = np.zeros((len(samples), readouts.size))
    for s in range(len(samples)):
        hid, out = np.zeros((steps, n)), np.zeros((steps, readouts.size))
        hid[0] = np.where(hidden, x[s], 0.0)
        for t in range(steps):
            if 0 < case["top_k_hidden"] < int(hidden.sum()):
                live = np.flatnonzero(hidden)
                keep = live[np.argsort(-hid[t, live], kind="stable")[:case["top_k_hidden"]]]
                kept = np.zeros(n)
                kept[keep] = hid[t, keep]
                hid[t] = kept
            e = up[t + delay[up] < steps]
            np.add.at(out, (t + delay[e], position[net.target[e]]), hid[t, net.source[e]] * weight[e])
            gate = np.zeros(readouts.size)
            best = int(np.argmax(out[t]))
            gate[best] = out[t, best]
            e = down[t + delay[down] < steps]
            np.add.at(hid, (t + delay[e], net.target[e]), 0.5 * gate[position[net.source[e]]] * weight[e])
        scores[s] = out.sum(axis=0)
    return [scores, None, None, None]
