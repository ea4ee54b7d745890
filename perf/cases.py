"""The work that users of this simulator have it do, as measurable cases.

A case is a dict of plain values; its ``kind`` names the entry point:

  faults  one circuit with its fault list: new patterns, ``Simulator.run``,
          per-fault results (count mode, drop mode, tuned sweep shape)
  good    the good machine alone (no faults) and the last round's values
  batch   many small circuits, new patterns each, in one ``Batch.run``
  serve   a burst of requests against the resident circuits of a ``Server``
  load    a .ckt text read into a handle: element order, levels, types

Circuits and fault lists come from the repository's generator, the same for
every seed of a case (but for ``load``); patterns and samples of fault lists
come from the seed.
Sizes are those of the repository's workloads (c1 to c5), tests and smoke run.
All outputs are whole numbers.
"""
import math

import numpy as np
import torch

from lsim_b200 import Simulator, gen
from lsim_b200.batch import Batch
from lsim_b200.serve import Server

# Fault-list sizes of the generator, per gate, and the share of the gates
# whose flip needs a sweep of its own; only work() uses them.
FAULTS_PER_GATE = {"outputs": 2.0, "collapsed": 3.7, "pins": 6.4}
STEMS_PER_GATE = 0.54


def listed():
    return [
        # the smallest call: the smoke run's circuit, one round of 64 patterns
        dict(name="one_round", kind="faults", gates=400, io=16, levels=14, fan3=0.5, types="bench",
             hubs=0.0, faults="collapsed", max_faults=0, patterns=64, drop=False, n_detect=0, tune=False),
        # the small workload c1
        dict(name="small", kind="faults", gates=2000, io=64, levels=30, fan3=0.5, types="bench",
             hubs=0.0, faults="outputs", max_faults=0, patterns=4096, drop=False, n_detect=0, tune=False),
        # the median circuit of the batched workload on its own, with a
        # pattern count that is no multiple of the word or the tile
        dict(name="median_ragged", kind="faults", gates=6586, io=205, levels=61, fan3=0.5, types="bench",
             hubs=0.0, faults="outputs", max_faults=0, patterns=10001, drop=False, n_detect=0, tune=False),
        # c2s, the c2 shape at 50,000 gates, two tiles, sweep shape tuned as
        # long runs do
        dict(name="large_tuned", kind="faults", gates=50000, io=1000, levels=38, fan3=0.6, types="bench",
             hubs=0.0, faults="collapsed", max_faults=0, patterns=4096, drop=False, n_detect=0, tune=True),
        # c2, the headline circuit and its whole fault list, one tile of its
        # patterns, default options
        dict(name="headline_tile", kind="faults", gates=200000, io=1000, levels=150, fan3=0.6, types="bench",
             hubs=0.0, faults="collapsed", max_faults=0, patterns=2048, drop=False, n_detect=0, tune=False),
        # MUX gates: one exact sweep per fault instead of one per stem
        dict(name="mux_exact", kind="faults", gates=20000, io=300, levels=40, fan3=0.5, types="all",
             hubs=0.0, faults="outputs", max_faults=0, patterns=1000, drop=False, n_detect=0, tune=False),
        # test generation: drop mode on a c3-like circuit (hubs, biased
        # patterns), eight tiles
        dict(name="drop_hubs", kind="faults", gates=30000, io=750, levels=60, fan3=0.6, types="bench",
             hubs=0.1, faults="collapsed", max_faults=0, patterns=16384, drop=True, n_detect=1, tune=False),
        # levels too wide for shared memory: the global-memory sweep, a
        # sample of the fault list
        dict(name="wide_levels", kind="faults", gates=200000, io=1000, levels=4, fan3=0.6, types="bench",
             hubs=0.0, faults="collapsed", max_faults=3000, patterns=256, drop=False, n_detect=0, tune=False),
        # the reference's GPU program: the good machine over all patterns of c2
        dict(name="good_machine", kind="good", gates=200000, io=1000, levels=150, fan3=0.6, types="bench",
             hubs=0.0, patterns=65536),
        # the batched workload at circuits that do not fill the GPU alone
        dict(name="batch_small", kind="batch", circuits=48, gates_lo=500, gates_hi=5000,
             patterns_lo=1024, patterns_hi=16384, types="bench"),
        # the served workload: a burst of requests over circuits of several sizes
        dict(name="serve_burst", kind="serve", circuits=6, gates_lo=1000, gates_hi=100000, requests=24,
             faults_lo=1000, faults_hi=20000, patterns_lo=64, patterns_hi=8192),
        # reading the headline circuit
        dict(name="load_circuit", kind="load", gates=200000, io=1000, levels=150, fan3=0.6, types="bench",
             hubs=0.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _shape(rng, lo, hi):
    """Gates, levels (at most c2's level width, 1,333 gates, or c3's) and PIs of a drawn circuit."""
    g = _log(rng, lo, hi)
    levels = max(rng.randint(10, 150), -(-g // rng.choice([1333, 1333, 5000])))
    return dict(gates=g, levels=max(2, min(levels, g // 4)), io=min(1000, max(16, g // 32)) + rng.randint(0, 3))


def draw(rng):
    kind = rng.choices(["faults", "good", "batch", "serve", "load"], [10, 1, 2, 2, 1])[0]
    if kind == "good":
        return dict(kind=kind, **_shape(rng, 1000, 200000), fan3=0.6, types=rng.choice(["bench", "all"]),
                    hubs=0.0, patterns=_log(rng, 64, 65536))
    if kind == "load":
        return dict(kind=kind, **_shape(rng, 2000, 400000), fan3=0.6, types=rng.choice(["bench", "all"]),
                    hubs=rng.choice([0.0, 0.1]))
    if kind == "batch":
        types = rng.choice(["bench", "bench", "all"])
        lo = _log(rng, 300, 2000 if types == "bench" else 500)
        return dict(kind=kind, circuits=rng.randint(3, 56), gates_lo=lo, gates_hi=rng.randint(3, 8) * lo,
                    patterns_lo=64, patterns_hi=_log(rng, 500, 16384), types=types)
    if kind == "serve":
        return dict(kind=kind, circuits=rng.randint(1, 8), gates_lo=1000, gates_hi=_log(rng, 3000, 100000),
                    requests=rng.choice([1, rng.randint(2, 40)]), faults_lo=500, faults_hi=_log(rng, 1000, 20000),
                    patterns_lo=64, patterns_hi=_log(rng, 100, 8192))
    c = dict(kind=kind, **_shape(rng, 400, 100000), fan3=rng.choice([0.3, 0.5, 0.6]),
             types=rng.choice(["bench", "bench", "all"]), hubs=rng.choice([0.0, 0.0, 0.1]),
             faults=rng.choice(["outputs", "collapsed", "pins"]), max_faults=rng.choice([0, 0, _log(rng, 200, 20000)]),
             patterns=_log(rng, 64, 16384), drop=rng.random() < 0.25, n_detect=0, tune=rng.random() < 0.2)
    if c["drop"]:
        c["n_detect"] = rng.choice([1, 3, 40])
    if c["types"] == "all":  # one sweep per fault
        c["gates"] = min(c["gates"], 20000 + c["gates"] % 1000)
        c["levels"] = min(c["levels"], c["gates"] // 4)
    elif rng.random() < 0.1:  # levels too wide for shared memory, sampled faults
        c["gates"] = rng.randint(100000, 200000)
        c.update(levels=rng.randint(3, 5), max_faults=rng.randint(200, 3000), tune=False)
    # no more than a tenth of the headline tile's gate-word evaluations
    while _evaluations(c) > 3.5e10:
        c["patterns"] = (c["patterns"] + 1) // 2
        if c["patterns"] <= 2048:
            c["max_faults"] = (c["max_faults"] or 40000) // 2 + 1
    return c


def _evaluations(c):
    """Gate-word evaluations of the sweeps: each runs the gates above its root, half of them on average."""
    flips = (FAULTS_PER_GATE[c["faults"]] if c["types"] == "all" else STEMS_PER_GATE) * c["gates"]
    if c["max_faults"]:
        flips = min(flips, c["max_faults"])
    return flips * c["gates"] / 2 * -(-c["patterns"] // 64)


# ------------------------------------------------------------------ inputs
def _circuit_text(c, seed=0):
    return gen.circuit(c["gates"], c["io"], c["io"], c["levels"], p_fanin3=c["fan3"],
                       type_mask=gen.ALL_TYPES if c["types"] == "all" else gen.BENCH_TYPES, seed=seed,
                       hub_frac=c["hubs"])


def _words(rng, rows, n_pi, patterns, biased=False):
    """Pattern words [rows][n_pi]; half of the PIs at P(1) = 1/4 when biased."""
    w = rng.integers(0, 1 << 64, (rows, n_pi), dtype=np.uint64)
    if biased:
        w[:, ::2] &= rng.integers(0, 1 << 64, (rows, (n_pi + 1) // 2), dtype=np.uint64)
    if patterns % 64:
        w[-1] &= np.uint64((1 << (patterns % 64)) - 1)
    return w


def _rows(patterns):
    return -(-patterns // 64)


def _fault_inputs(c, seed):
    """Circuit text, fault text, indices of the sampled faults (None: all) and pattern words."""
    rng = np.random.default_rng(seed)
    ckt = _circuit_text(c)
    flst = gen.faults(ckt, c["faults"])
    words = _words(rng, _rows(c["patterns"]), c["io"], c["patterns"], biased=c["hubs"] > 0)
    pick = None
    if c["max_faults"]:
        head = flst.split(None, 2)
        pick = np.sort(rng.permutation(int(head[head[0] == "@pins"]))[: c["max_faults"]])
    return ckt, flst, pick, words


def prepare(case, seed):
    c = case
    rng = np.random.default_rng(seed)
    if c["kind"] == "faults":
        ckt, flst, pick, words = _fault_inputs(c, seed)
        sim = Simulator(0)
        sim.load_circuit(ckt)
        sim.set_fault_text(flst)
        if pick is not None:
            site, pin, value = sim.faults()
            sim.set_faults(site[pick], pin[pick], value[pick])
        return dict(kind="faults", sim=sim, words=words, patterns=c["patterns"],
                    options=dict(drop=c["drop"], n_detect=c["n_detect"], tune=c["tune"]))
    if c["kind"] == "good":
        sim = Simulator(0)
        sim.load_circuit(_circuit_text(c))
        sim.set_faults([], [], [])
        return dict(kind="good", sim=sim, patterns=c["patterns"],
                    words=_words(rng, _rows(c["patterns"]), c["io"], c["patterns"]))
    if c["kind"] == "batch":
        batch, members = Batch(0), []
        for cfg in gen.batch_configs(c["circuits"], gates=(c["gates_lo"], c["gates_hi"]),
                                     patterns=(c["patterns_lo"], c["patterns_hi"]),
                                     type_mask=gen.ALL_TYPES if c["types"] == "all" else gen.BENCH_TYPES):
            P = cfg.pop("n_patterns")
            kind = cfg.pop("faults")
            ckt = gen.circuit(**cfg)
            sim = Simulator(-1)
            sim.load_circuit(ckt)
            sim.set_fault_text(gen.faults(ckt, kind))
            members.append((sim, _words(rng, _rows(P), cfg["n_pi"], P), P))
            batch.add(sim)
        return dict(kind="batch", batch=batch, members=members)
    if c["kind"] == "serve":
        server = Server(0, slot_bytes=1 << 30)
        ids = []
        for cfg in gen.serve_configs(c["circuits"], gates=(c["gates_lo"], c["gates_hi"]), levels=(20, 150)):
            kind = cfg.pop("faults")
            ckt = gen.circuit(**cfg)
            host = Simulator(-1)
            host.load_circuit(ckt)
            host.set_fault_text(gen.faults(ckt, kind))
            P = c["patterns_hi"]
            ids.append((server.add_circuit(ckt, _words(rng, _rows(P), cfg["n_pi"], P), P), host.faults()))
        requests = []
        sizes = np.random.default_rng(c["requests"])
        for _ in range(c["requests"]):
            cid, (site, pin, value) = ids[sizes.integers(len(ids))]
            n = int(np.exp(sizes.uniform(np.log(c["faults_lo"]), np.log(c["faults_hi"]))))
            P = int(np.exp(sizes.uniform(np.log(c["patterns_lo"]), np.log(c["patterns_hi"]))))
            pick = np.sort(rng.permutation(len(site))[:n])
            requests.append((cid, site[pick], value[pick], pin[pick], P))
        return dict(kind="serve", server=server, requests=requests)
    return dict(kind="load", sim=Simulator(0), text=_circuit_text(c, seed).encode())


# ------------------------------------------------------------------ one pass
def _whole(results):
    """The 32-byte result records as [faults][4] words: flags, first pattern, count, last round."""
    return results.view(np.int64).reshape(-1, 4)


def run(state):
    if state["kind"] == "faults":
        sim = state["sim"]
        sim.set_patterns(state["words"], state["patterns"])
        sim.run(**state["options"])
        return _whole(sim.results())
    if state["kind"] == "good":
        sim = state["sim"]
        sim.set_patterns(state["words"], state["patterns"])
        sim.run()
        return sim.good_values().view(np.int64)
    if state["kind"] == "batch":
        for sim, words, patterns in state["members"]:
            sim.set_patterns(words, patterns)
        state["batch"].run()
        return [_whole(sim.results()) for sim, _, _ in state["members"]]
    if state["kind"] == "serve":
        server = state["server"]
        tickets = [server.submit(cid, site, value, pin, n_patterns=P)
                   for cid, site, value, pin, P in state["requests"]]
        return [_whole(server.wait(t)) for t in tickets]
    sim = state["sim"]
    sim.load_circuit(state["text"])
    return dict(order=sim.gate_idx_to_tpg_order_idx().view(np.int64), levels=sim.levels().view(np.int64),
                types=sim.types())


# ------------------------------------------------------------------ work
def work(case):
    """Bytes: circuit (edges and types), pattern words and results, once each.
    Operations: one per gate-word evaluation (64 patterns of one gate)."""
    c = case
    if c["kind"] == "load":  # a wire line and a gate line per gate, about 31 bytes in all
        return dict(bytes=31.0 * c["gates"] + 17.0 * c["gates"], flops=0)
    if c["kind"] == "batch":
        g = (c["gates_hi"] - c["gates_lo"]) / math.log(c["gates_hi"] / c["gates_lo"])
        g2 = (c["gates_hi"] ** 2 - c["gates_lo"] ** 2) / 2 / math.log(c["gates_hi"] / c["gates_lo"])
        rows = (c["patterns_lo"] + c["patterns_hi"]) / 128
        return dict(bytes=c["circuits"] * (g * 9 + rows * g / 4 + 64 * g),
                    flops=c["circuits"] * STEMS_PER_GATE * g2 / 2 * rows)
    if c["kind"] == "serve":
        g = (c["gates_hi"] - c["gates_lo"]) / math.log(c["gates_hi"] / c["gates_lo"])
        f = (c["faults_hi"] - c["faults_lo"]) / math.log(c["faults_hi"] / c["faults_lo"])
        rows = (c["patterns_hi"] - c["patterns_lo"]) / math.log(c["patterns_hi"] / c["patterns_lo"]) / 64
        return dict(bytes=c["requests"] * f * 40, flops=c["requests"] * f / 2 * g / 2 * rows)
    rows = _rows(c["patterns"])
    circuit = 9.0 * c["gates"]
    if c["kind"] == "good":
        return dict(bytes=circuit + rows * c["io"] * 8 + (c["gates"] + 2 * c["io"]) * 8, flops=c["gates"] * rows)
    faults = c["max_faults"] or FAULTS_PER_GATE[c["faults"]] * c["gates"]
    return dict(bytes=circuit + rows * c["io"] * 8 + faults * 40,
                flops=_evaluations(c) / (min(rows, 32) if c["drop"] else 1))


# ------------------------------------------------------------------ exact
GATES = ["INV", "AND", "OR", "XOR", "NAND", "NOR", "XNOR", "MUX", "CLKBUF"]


def _netlist(ckt, io):
    """Gate types and inputs (in pin order) by file id -- PIs, POs, gates --
    and the ids of the gates in an order of evaluation."""
    tok = list(map(int, ckt.split()))
    n_gates, n_wires = tok[2], tok[3]
    n = 2 * io + n_gates
    pins, at = [{} for _ in range(n)], 4
    for _ in range(n_wires):
        src, k = tok[at], tok[at + 2]
        for j in range(at + 3, at + 3 + 2 * k, 2):
            pins[tok[j]][3 if tok[j + 1] == 5 else tok[j + 1]] = src
        at += 3 + 2 * k
    types = [""] * (2 * io) + [GATES[t] for t in tok[at: at + n_gates]]
    inputs = [[p[q] for q in sorted(p)] for p in pins]
    order = []
    readers, missing = [[] for _ in range(n)], [len(x) for x in inputs]
    for e in range(io, n):
        for s in inputs[e]:
            readers[s].append(e)
    ready = list(range(io))
    while ready:
        e = ready.pop()
        if e >= 2 * io:
            order.append(e)
        for r in readers[e]:
            missing[r] -= 1
            if not missing[r]:
                ready.append(r)
    return types, inputs, order


def _gate(t, x):
    """One gate on 64-bit words; a MUX tests its whole select word."""
    if t == "MUX":
        return (x[2] & x[1]) | (x[0] & (x[2] == 0).to(torch.int64))
    r = x[0]
    for y in x[1:]:
        r = r & y if t in ("AND", "NAND") else r | y if t in ("OR", "NOR") else r ^ y
    return ~r if t in ("INV", "NAND", "NOR", "XNOR") else r


def exact(case, seed):
    """The result records of a small count-mode case, every fault simulated in
    the whole circuit with 64-bit operations; None where that takes too long
    and where the outputs follow the reference's element order."""
    c = case
    if c["kind"] != "faults" or c["drop"]:
        return None
    rows = _rows(c["patterns"])
    n_faults = c["max_faults"] or FAULTS_PER_GATE[c["faults"]] * c["gates"]
    if n_faults * c["gates"] * rows > 2e10:
        return None
    ckt, flst, pick, words = _fault_inputs(c, seed)
    io, dev = c["io"], "cuda" if torch.cuda.is_available() else "cpu"
    types, inputs, order = _netlist(ckt, io)
    tok = flst.split()
    if tok[0] == "@pins":
        faults = np.array(tok[2:], dtype=np.int64).reshape(-1, 3)
    else:
        faults = np.array(tok[1:], dtype=np.int64).reshape(-1, 2)
        faults = np.concatenate([faults, np.zeros((len(faults), 1), np.int64)], 1)
    if pick is not None:
        faults = faults[pick]
    pi = torch.from_numpy(words.T.copy().view(np.int64)).to(dev)
    valid = torch.full((rows,), -1, dtype=torch.int64, device=dev)
    if c["patterns"] % 64:
        valid[-1] = (1 << (c["patterns"] % 64)) - 1

    def machine(chunk):
        """PO words [POs][faults + 1][rows]; machine 0 has no fault."""
        at = {}
        for i, (site, value, pin) in enumerate(chunk):
            at.setdefault(int(site), []).append((i + 1, -int(value), int(pin)))
        n = len(chunk) + 1
        vals = [None] * len(types)
        for e in list(range(io)) + order:
            v = pi[e].expand(n, rows) if e < io else _gate(types[e], [vals[s] for s in inputs[e]])
            if e in at:
                v = v.clone()
                for i, value, pin in at[e]:
                    if pin:
                        x = [vals[s][i] for s in inputs[e]]
                        x[pin - 1] = torch.full_like(x[0], value)
                        v[i] = _gate(types[e], x)
                    else:
                        v[i] = value
            vals[e] = v
        return [vals[inputs[e][0]] for e in range(io, 2 * io)]

    out = np.zeros((len(faults), 4), np.int64)
    out[:, 3] = rows - 1
    shifts = torch.arange(63, -1, -1, device=dev)
    per = max(1, int(4e9 / 8 / (len(types) * rows)))
    for f0 in range(0, len(faults), per):
        chunk = faults[f0: f0 + per]
        diff = torch.zeros((len(chunk), rows), dtype=torch.int64, device=dev)
        for po in machine(chunk):
            diff |= (po[1:] ^ po[:1]) & valid
        count = torch.zeros(len(chunk), dtype=torch.int64, device=dev)
        first = torch.full((len(chunk),), -1, dtype=torch.int64, device=dev)
        for r in range(rows - 1, -1, -1):
            bits = (diff[:, r, None] >> shifts) & 1  # highest bit first: pattern order
            count += bits.sum(1)
            width = 64 if r < rows - 1 or c["patterns"] % 64 == 0 else c["patterns"] % 64
            pos = bits.argmax(1)
            first = torch.where(bits.any(1), r * 64 + pos - (64 - width), first)
        k = slice(f0, f0 + len(chunk))
        last = (diff[:, -1] != 0).to(torch.int64)
        out[k, 0] = ((count > 0).to(torch.int64) + 256 * last).cpu().numpy()
        out[k, 1], out[k, 2] = first.cpu().numpy(), count.cpu().numpy()
    return out
