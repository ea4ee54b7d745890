"""Circuits with many PO drivers on one level, whose values need no room
beyond the level, against the oracle."""
import numpy as np
import pytest

from lsim_b200 import Server, Simulator, gen
from lsim_b200.batch import Batch
from tests.oracle_lib import Oracle

pytestmark = pytest.mark.gpu


def circuit(drivers, pis=40, rows=3, width=100, types=(1, 2, 3, 4, 5, 6), seed=0):
    """`rows` levels of `width` two-input gates, then one level of `drivers`
    gates of one to four inputs, each driving a PO of its own."""
    rng = np.random.default_rng(seed)
    g0 = pis + drivers
    gates = rows * width + drivers
    sinks = [[] for _ in range(g0 + gates)]
    prev = list(range(pis))
    kinds = []
    for r in range(rows + 1):
        row = [g0 + r * width + i for i in range(width if r < rows else drivers)]
        for i, e in enumerate(row):
            t = int(rng.choice(types))
            n = 2 if r < rows else 1 + i % 4
            if n == 1:
                t = 0 if i % 8 else 8
            elif t == 7:
                n = 3
            for k in range(n):
                src = prev[int(rng.integers(len(prev)))]
                sinks[src].append((e, 5 if t == 7 and k == 2 else k + 1))
            kinds.append(t)
            if r == rows:
                sinks[e].append((pis + i, 1))
        prev = row
    wires = ["%d 1 %d %s" % (e, len(s), " ".join("%d %d" % x for x in s)) for e, s in enumerate(sinks) if s]
    return "%d %d %d %d\n%s\n%s\n" % (pis, drivers, gates, len(wires), "\n".join(wires),
                                      "\n".join(str(t) for t in kinds))


def work(drivers, patterns, pis=40, rows=3, width=100, **kw):
    """Circuit text, fault list (outputs of half of the rows' gates and of 200
    drivers) and pattern text."""
    ckt = circuit(drivers, pis, rows, width, **kw)
    rng = np.random.default_rng(drivers)
    g0 = pis + drivers
    sites = np.concatenate([g0 + rng.permutation(rows * width)[: rows * width // 2],
                            g0 + rows * width + rng.permutation(drivers)[:200]])
    flst = "%d\n%s\n" % (len(sites), "\n".join("%d %d" % (e, i % 2) for i, e in enumerate(sites)))
    return ckt, flst, gen.patterns(pis, patterns, seed=3)


def same(got, ref):
    assert np.array_equal(got["detected"], ref["detected"])
    assert np.array_equal(got["first_pattern"], ref["first"])
    assert np.array_equal(got["count"], ref["count"])
    assert np.array_equal(got["ref_last_round_flag"], ref["ref_flag"])


@pytest.mark.parametrize("drivers", [4000, 29000, 40000])
def test_default_and_tuned_runs(drivers):
    ckt, flst, ptn = work(drivers, 300)
    ref = Oracle(ckt, flst, ptn).simulate()
    for tune in (False, True):
        sim = Simulator(0)
        sim.read_text(ckt, flst, ptn)
        sim.run(tune=tune)
        same(sim.results(), ref)


@pytest.mark.parametrize("types", [(1, 2, 3, 4, 5, 6), (1, 3, 7)])
@pytest.mark.parametrize("drivers", [4000, 29000, 40000])
def test_every_shape_batches_and_servers(drivers, types):
    """Shapes that the gates' live values (some 200 here) leave room for."""
    patterns = 4500 if drivers == 4000 else 1100
    ckt, flst, ptn = work(drivers, patterns, types=types)
    ref = Oracle(ckt, flst, ptn).simulate()
    sim = Simulator(0)
    sim.read_text(ckt, flst, ptn)
    for shape in [dict()] + [dict(words_per_item=m) for m in (1, 2, 4, 8)] + \
            [dict(words_per_item=8, ctas_per_sm=2, block_threads=256), dict(sweep_variant="shared"),
             dict(sweep_variant="global")]:
        sim.run(**shape)
        same(sim.results(), ref)
    with Batch(0) as b:
        host = Simulator(-1)
        host.read_text(ckt, flst, ptn)
        b.add(host)
        for opts in (dict(), dict(tune=True), dict(words_per_item=8)):
            b.run(**opts)
            same(host.results(), ref)
    site, pin, value = host.faults()
    with Server(0, slot_bytes=1 << 30) as s:
        cid = s.add_circuit(ckt, host.patterns(), patterns)
        same(s.wait(s.submit(cid, site, value, pin, n_patterns=patterns)), ref)
