"""Timed cases of the simulation path, through the package's public entry points.

A case names a model, a layout, a delay and how a program drives the net:

  step     one step(out=True): the spikes of one step, the reference's own calling form
           (snn::step(std::vector<int>*)), marked in the program's own vector of neurons;
           what a program that reacts to every step does
  run      run(steps), then neurons(): a simulation of which the final state is wanted
  record   run_record(steps), then neurons(): the spike raster, kept in the program's own
           array, and the final state
  weights  run(steps), then neurons() and synapses(): a plastic net whose learned weights
           are wanted
  build    a new net of the layout, then run_record(steps) and neurons(): one point of a
           parameter sweep, where every net is constructed, used briefly and dropped
  batch    many small nets of three models stepped together by Batch.run(steps), then every
           net's neurons()

`warm` steps are run while the net is prepared, past the initial transient of a net that
starts at rest. dt is 0.1 ms throughout.
"""
import math

import numpy as np

from spice_b200 import Batch, Layout, Snn

DT = 1e-4
BRUNEL = "0>1:0.1;1>1:0.1"  # Poisson and LIF halves, both projecting onto the LIF half
VA = "0>0:0.02"


def listed():
    return [
        # closed-loop use: every step's spikes handed to the host, on the small published VA net
        {"name": "va_5k_step", "entry": "step", "model": "vogels_abbott", "pops": "5000", "conns": VA, "delay": 1, "warm": 1000,
         "steps": 1, "kernel": ""},
        # the classic 4,000 + 1,000 VA benchmark net from rest, delay 1 (the shortest there is)
        {"name": "va_5k_run", "entry": "run", "model": "vogels_abbott", "pops": "5000", "conns": VA, "delay": 1, "warm": 0,
         "steps": 500, "kernel": ""},
        # an irregular circuit: odd populations, uneven densities, a delay that is no multiple
        # of anything, read out as a raster
        {"name": "brunel_ragged_record", "entry": "record", "model": "brunel", "pops": "9973,7001,5011",
         "conns": "0>1:0.07;0>2:0.033;1>1:0.05;1>2:0.11;2>1:0.2", "delay": 7, "warm": 600, "steps": 601, "kernel": ""},
        # Brunel at a tenth of the benchmark's size, raster wanted (e2e form of the benchmark)
        {"name": "brunel_1e8_record", "entry": "record", "model": "brunel", "pops": "22360,22360", "conns": BRUNEL, "delay": 15,
         "warm": 600, "steps": 1050, "kernel": ""},
        # the headline benchmark: Brunel at 1e9 synapses, 0.105 s of biological time
        {"name": "brunel_1e9_run", "entry": "run", "model": "brunel", "pops": "70710,70710", "conns": BRUNEL, "delay": 15,
         "warm": 600, "steps": 1050, "kernel": ""},
        # the reference's published VA size: 1e9 synapses, sparser, delay 8
        {"name": "va_1e9_run", "entry": "run", "model": "vogels_abbott", "pops": "223607", "conns": VA, "delay": 8, "warm": 600,
         "steps": 400, "kernel": ""},
        # the reference's sparse 1e9 net: 800,641 neurons of out-degree 1,249, delay 1
        {"name": "synth_1e9_run", "entry": "run", "model": "synth", "pops": "800641", "conns": "0>0:0.00156", "delay": 1, "warm": 50,
         "steps": 100, "kernel": ""},
        # STDP at the published size: 5e8 plastic synapses, the spike raster wanted
        {"name": "brunel_plus_5e8_record", "entry": "record", "model": "brunel_with_plasticity", "pops": "50000,50000",
         "conns": BRUNEL, "delay": 15, "warm": 300, "steps": 300, "kernel": ""},
        # STDP on a small net, the learned weights wanted
        {"name": "brunel_plus_1e6_weights", "entry": "weights", "model": "brunel_with_plasticity", "pops": "2236,2236",
         "conns": BRUNEL, "delay": 15, "warm": 300, "steps": 2000, "kernel": ""},
        # the generic kernel, which runs every model of a user's own
        {"name": "brunel_ordered_run", "entry": "run", "model": "brunel", "pops": "15811,15811", "conns": BRUNEL, "delay": 15,
         "warm": 300, "steps": 300, "kernel": "ordered"},
        # a parameter sweep's mix of small nets sharing the GPU
        {"name": "batch_24", "entry": "batch", "model": "mixed", "pops": "24", "conns": "", "delay": 0, "warm": 300, "steps": 600,
         "kernel": ""},
        # one point of a sweep over nets of 1e8 synapses: construction, 150 steps, gone
        {"name": "brunel_1e8_build", "entry": "build", "model": "brunel", "pops": "22360,22360", "conns": BRUNEL, "delay": 15,
         "warm": 0, "steps": 150, "kernel": ""},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _halves(syn, rng):
    """Two populations of about N / 2, N = sqrt(syn / 0.05), one of them a little off."""
    half = max(64, int(math.sqrt(syn / 0.05) / 2))
    return f"{half},{half + rng.randrange(0, 37)}"


def draw(rng):
    """A case of the listed ones' ranges: the same models and entries, sizes log-uniform,
    odd populations, other densities and delays."""
    kind = rng.choice(["step", "va", "brunel", "ragged", "brunel", "synth", "plastic", "weights", "ordered", "batch", "build"])
    case = {"entry": "run", "model": "brunel", "conns": BRUNEL, "delay": rng.choice([1, 3, 7, 8, 15, 15, 15, 20]), "warm": 600,
            "steps": rng.randrange(150, 1000), "kernel": ""}
    if kind == "step":
        model = rng.choice(["vogels_abbott", "brunel"])
        syn = _log(rng, 2e5, 5e7)
        case.update(entry="step", model=model, steps=1, warm=1000)
        if model == "brunel":
            case.update(pops=_halves(syn, rng))
        else:
            case.update(pops=str(int(math.sqrt(syn / 0.02)) + rng.randrange(0, 7)), conns=VA, delay=rng.choice([1, 1, 8]))
    elif kind == "va":
        case.update(model="vogels_abbott", pops=str(int(math.sqrt(_log(rng, 2e5, 7e8) / 0.02)) + rng.randrange(0, 7)), conns=VA,
                    delay=rng.choice([1, 8, 8, 12]), steps=rng.randrange(150, 400))
    elif kind == "brunel":
        case.update(entry=rng.choice(["run", "record"]), pops=_halves(_log(rng, 1e6, 8e8), rng))
    elif kind == "ragged":
        k = rng.randrange(2, 6)
        size = _log(rng, 2e3, 6e4)
        pops = [max(50, int(size * rng.uniform(0.2, 1.0))) for _ in range(k)]
        conns = [f"{a}>{b}:{round(rng.uniform(0.01, 0.2), 4)}" for a in range(k) for b in range(1, k) if a == 0 or b == a or rng.random() < 0.4]
        case.update(entry=rng.choice(["run", "record"]), pops=",".join(map(str, pops)), conns=";".join(conns),
                    delay=rng.choice([2, 5, 7, 11, 16]))
    elif kind == "synth":
        n = int(_log(rng, 5e4, 8e5))
        case.update(model="synth", pops=str(n), conns=f"0>0:{round(1249.0 / n * rng.uniform(0.5, 1.0), 6)}",
                    delay=rng.choice([1, 1, 2, 6]), warm=50, steps=100)
    elif kind == "plastic":
        case.update(entry=rng.choice(["run", "record"]), model="brunel_with_plasticity", pops=_halves(_log(rng, 1e6, 3e8), rng),
                    delay=rng.choice([8, 15, 15, 20]), warm=300, steps=rng.randrange(100, 300))
    elif kind == "weights":
        case.update(entry="weights", model="brunel_with_plasticity", pops=_halves(_log(rng, 2e5, 5e6), rng), delay=15, warm=300,
                    steps=rng.randrange(500, 2000))
    elif kind == "ordered":
        case.update(model=rng.choice(["brunel", "vogels_abbott"]), kernel="ordered", warm=300, steps=rng.randrange(100, 300))
        syn = _log(rng, 1e6, 1e8)
        if case["model"] == "brunel":
            case.update(pops=_halves(syn, rng))
        else:
            case.update(pops=str(int(math.sqrt(syn / 0.02))), conns=VA, delay=8)
    elif kind == "batch":
        case.update(entry="batch", model="mixed", pops=str(rng.randrange(6, 25)), conns="", delay=0, warm=300, steps=rng.randrange(150, 600))
    else:
        model = rng.choice(["brunel", "vogels_abbott", "brunel_with_plasticity"])
        syn = _log(rng, 1e6, 2e8 if model != "brunel_with_plasticity" else 2e7)
        case.update(entry="build", model=model, warm=0, steps=rng.randrange(200, 400))  # VA from rest is silent for 138 steps
        if model == "vogels_abbott":
            case.update(pops=str(int(math.sqrt(syn / 0.02))), conns=VA, delay=8)
        else:
            case.update(pops=_halves(syn, rng), delay=15)
    return case


# ---------------------------------------------------------------------------------------
# nets
# ---------------------------------------------------------------------------------------
def _pops(case):
    return [int(x) for x in case["pops"].split(",")]


def _conns(case):
    out = []
    for c in case["conns"].split(";"):
        ends, p = c.split(":")
        a, b = ends.split(">")
        out.append((int(a), int(b), float(p)))
    return out


def _batch_specs(case, seed):
    """The nets of a batch: models in turn, synapses log-uniform over 1e5 to 2e7 (the sizes
    belong to the case; the seed sets the nets' graphs and Poisson streams)."""
    count = int(case["pops"])
    rng = np.random.RandomState(count)
    specs = []
    for i in range(count):
        model = ("vogels_abbott", "brunel", "brunel_with_plasticity")[i % 3]
        syn = math.exp(rng.uniform(math.log(1e5), math.log(2e7)))
        if model == "vogels_abbott":
            pops, conns, delay = [max(64, int((syn / 0.02) ** 0.5))], [(0, 0, 0.02)], 8
        else:
            half = max(32, int((syn / 0.05) ** 0.5) // 2)
            pops, conns, delay = [half, half], [(0, 1, 0.1), (1, 1, 0.1)], 15
        specs.append((model, pops, conns, delay, 100 * seed + i + 1, 100 * seed + 50 + i))
    return specs


def _net(case, seed):
    options = {"kernel": case["kernel"]} if case["kernel"] else None
    return Snn(case["model"], Layout(_pops(case), _conns(case)), dt=DT, delay=case["delay"], seed=seed + 1, graph_seed=seed + 1337,
               options=options)


def prepare(case, seed):
    entry = case["entry"]
    state = {"case": case, "seed": seed}
    if entry in ("record", "build"):  # the program's raster: as many ids as run_record makes room for
        state["ids"] = np.full(case["steps"] * max(1, sum(_pops(case)) // 20), -1, dtype=np.int32)
        state["filled"] = 0
    if entry == "build":
        return state
    if entry == "batch":
        from spice_b200.autotune import layout_work, tile_targets

        specs = _batch_specs(case, seed)
        targets = tile_targets([layout_work(Layout(pops, conns)) for _, pops, conns, _, _, _ in specs], 148, 2.0)
        batch, nets = Batch(), []
        for (model, pops, conns, delay, s, g), tiles in zip(specs, targets):
            net = Snn(model, Layout(pops, conns), dt=DT, delay=delay, seed=s, graph_seed=g)
            net.set_tile_target(tiles)
            batch.add(net)
            nets.append(net)
        batch.run(case["warm"])
        batch.sync()
        return dict(state, batch=batch, nets=nets)
    net = _net(case, seed)
    net.run(case["warm"])
    net.sync()
    if entry == "step":
        state["fired"] = np.zeros(net.num_neurons(), dtype=np.uint8)
    return dict(state, net=net)


def run(state):
    case = state["case"]
    entry, steps = case["entry"], case["steps"]
    if entry == "step":
        fired = state["fired"]
        fired[:] = 0
        fired[state["net"].step(out=True)] = 1
        return {"fired": fired}
    if entry == "batch":
        state["batch"].run(steps)
        state["batch"].sync()
        got = [net.neurons() for net in state["nets"]]
        return {"real": np.concatenate([a for arrays in got for a in arrays if a.dtype == np.float32]),
                "whole": np.concatenate([a for arrays in got for a in arrays if a.dtype != np.float32])}
    net = _net(case, state["seed"]) if entry == "build" else state["net"]
    out = {}
    if entry in ("record", "build"):
        out["counts"], ids = net.run_record(steps)
        kept = state["ids"]
        kept[:ids.size] = ids
        kept[ids.size:state["filled"]] = -1
        state["filled"] = ids.size
        out["ids"] = kept
    else:
        net.run(steps)
    out["neurons"] = net.neurons()
    if entry == "weights":
        out["synapses"] = net.synapses()
    if entry == "build":
        net.close()
    return out


# ---------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------
# spikes per neuron and step at steady state
RATE = {"vogels_abbott": 0.0025, "brunel": 0.0025, "brunel_with_plasticity": 0.0025, "synth": 0.005}
ATTRS = {"vogels_abbott": 4, "brunel": 2, "brunel_with_plasticity": 2, "synth": 1}


def _net_work(model, pops, conns, steps):
    """Bytes and operations of `steps` steps: every spiking neuron's row once per spike
    (per synapse the smaller of a 4-byte index and 1 / p bits of a target bitmap; its
    weight read and written where the net learns), the state in and out, the raster out;
    one addition per arriving synapse and a handful of operations per neuron and step."""
    n = sum(pops)
    spikes = RATE[model] * n * steps
    per_spike = events = 0.0
    for a, b, p in conns:
        share = pops[a] / n
        targets = pops[b] * p
        per_spike += share * targets * (min(4.0, 1.0 / (8.0 * p)) + (8.0 if model == "brunel_with_plasticity" else 0.0))
        events += share * targets
    return {"bytes": spikes * per_spike + 8.0 * ATTRS[model] * n + 4.0 * spikes, "flops": spikes * events + 8.0 * n * steps}


def work(case):
    if case["entry"] == "batch":
        parts = [_net_work(m, pops, conns, case["steps"]) for m, pops, conns, _, _, _ in _batch_specs(case, 0)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    pops, conns = _pops(case), _conns(case)
    w = _net_work(case["model"], pops, conns, case["steps"])
    syn = sum(pops[a] * pops[b] * p for a, b, p in conns)
    if case["entry"] == "weights":
        w["bytes"] += 12.0 * syn
    if case["entry"] == "build":
        w["bytes"] += 4.0 * syn  # the adjacency rows written
    return w


# ---------------------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------------------
def _philox(c0, c1, c2, c3, key):
    """Philox-4x32-10 (Salmon, Moraes, Dror and Shaw, SC'11) over arrays of counters."""
    m32 = np.uint64(0xFFFFFFFF)
    c = [np.asarray(x, dtype=np.uint64) for x in (c0, c1, c2, c3)]
    k0, k1 = key & 0xFFFFFFFF, key >> 32
    for _ in range(10):
        a, b = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        c = [(b >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), b & m32, (a >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), a & m32]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c


def _rows(n, edges, width, seed):
    """Every neuron's targets: one Bernoulli draw per candidate, at most `width` of a row."""
    rows = [[] for _ in range(n)]
    for ci, (s0, s1, d0, d1, p) in enumerate(edges):
        threshold = math.floor(float(np.float32(p)) * 4294967296.0)
        blocks = np.arange((d1 - d0 + 3) // 4)
        for s in range(s0, s1):
            r = np.stack(_philox(np.full(blocks.size, s), blocks, np.full(blocks.size, ci), np.full(blocks.size, 0x47524150), seed), 1)
            hit = np.flatnonzero(r.reshape(-1)[:d1 - d0] < threshold)
            rows[s].append(hit + d0)
    return [np.concatenate(r)[:width] if r else np.zeros(0, dtype=np.int64) for r in rows]


def exact(case, seed):
    """The Vogels-Abbott net from rest in 64 bits: V and the two conductances (the
    refractory counters are whole numbers). Spiking nets are chaotic, so a 64-bit run
    says what a 32-bit one should give only while their spikes agree: the first 500 steps
    of a small net that starts at rest. None for all others."""
    if case["entry"] != "run" or case["model"] != "vogels_abbott" or case["warm"] or case["steps"] > 500 or int(case["pops"]) > 6000:
        return None
    n, delay = int(case["pops"]), case["delay"]
    p = float(np.float32(_conns(case)[0][2]))
    width = (int(n * p + 3 * math.sqrt(n * p * (1 - p))) + 31) // 32 * 32
    rows = _rows(n, [(0, n, 0, n, p)], width, seed + 1337)
    n_exc = int(np.float32(0.8) * np.float32(n))
    w_exc, w_inh = 0.4 * 16e6 / n / n, 5.1 * 16e6 / n / n
    v, gex, gin, wait = np.full(n, -0.06), np.zeros(n), np.zeros(n), np.zeros(n, dtype=np.int64)
    fired = []
    for t in range(case["steps"]):
        if t >= delay and fired[t - delay].size:
            for ids, g, w in ((fired[t - delay][fired[t - delay] < n_exc], gex, w_exc), (fired[t - delay][fired[t - delay] >= n_exc], gin, w_inh)):
                if ids.size:
                    g += w * np.bincount(np.concatenate([rows[i] for i in ids]), minlength=n)
        wait -= 1
        spike = (wait <= 0) & (v > -0.05)
        free = (wait <= 0) & ~spike
        v = np.where(free, v + ((-0.06 - v) + gex * (0.0 - v) + gin * (-0.08 - v) + 0.02) * (DT / 0.02), v)
        v[spike] = -0.06
        wait[spike] = 50
        gex -= gex * (DT / 0.005)
        gin -= gin * (DT / 0.01)
        fired.append(np.flatnonzero(spike))
    return {"neurons": [v, gex, gin, None]}
