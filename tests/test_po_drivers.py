"""Slots of circuits whose PO drivers, or folded gates' inputs, would keep
more values than the gates alone, and their sweeps on the CPU (standard
library checks and the address sanitizer on)."""
import os
import subprocess

import pytest

from lsim_b200 import build
from tests.test_gpu_po_drivers import circuit

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
ANY_SHAPE = 384  # slots that every launch shape has room for


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("po") / "po_driver_check")
    src = [os.path.join(build.CSRC, f) for f in ("fsimb_netlist.cpp", "fsimb_plan.cpp")]
    subprocess.check_call(["/usr/bin/g++", "-std=c++17", "-O2", "-D_GLIBCXX_ASSERTIONS", "-fsanitize=address",
                           os.path.join(ROOT, "tests", "cpp", "po_driver_check.cpp")] + src + ["-o", exe])

    def run(tmp_path, text, sweeps):
        path = tmp_path / "c.ckt"
        path.write_text(text)
        r = subprocess.run([exe, str(path), str(sweeps)], capture_output=True, text=True, timeout=600)
        assert r.returncode == 0, r.stderr[-2000:]
        lines = [[int(x) for x in s.split()] for s in r.stdout.split("\n") if s]
        live, direct, folded = lines[0]
        assert len(lines) == 5
        for g, slots, compared in lines[1:]:
            assert slots <= -(-max(live, ANY_SHAPE) // g) * g
            assert compared > 0
        return live, direct, folded

    return run


@pytest.mark.parametrize("types", [(1, 2, 3, 4, 5, 6), (1, 3, 7)])
@pytest.mark.parametrize("drivers", [100, 500, 4000, 29000, 40000])
def test_po_drivers_need_no_slots(check, tmp_path, drivers, types):
    live, direct, _ = check(tmp_path, circuit(drivers, types=types), 400000 // drivers + 20)
    assert live <= 500
    assert direct == (drivers if drivers > ANY_SHAPE else 0)


@pytest.mark.parametrize("gates", [50, 1000])
@pytest.mark.parametrize("buffers", [0, 1])
def test_folded_gates_do_not_outnumber_the_gates_live_values(check, tmp_path, gates, buffers):
    """A chain; every link gives an XOR pair, ANDed at once and used by a gate
    at the end only: folding the AND would keep both XORs to the end.  With
    buffers, the ANDs are read through a BUF and an INV."""
    pis, n = 8, gates
    pos = 2 * n
    g0 = pis + pos
    kinds, sinks = [], []

    def add(t, *inputs):
        e = g0 + len(kinds)
        kinds.append(t)
        for k, s in enumerate(inputs):
            sinks.append((s, e, k + 1))
        return e

    link, ands = 0, []
    for i in range(n):
        link = add(4 if i % 2 else 5, link, 1 + i % 3)  # NAND, NOR
        a, b = add(3, link, 4), add(6, link, 5)  # XOR, XNOR
        ands.append(add(1, a, b))
    end = add(3, link, 6)
    for i, a in enumerate(ands):
        last = [add(1, a, end)] if not buffers else [add(1, add(8, a), end), add(2, add(0, a), end)]
        for j, e in enumerate(last):
            sinks.append((e, pis + 2 * i + j, 1))
        if not buffers:
            sinks.append((add(0, end), pis + 2 * i + 1, 1))
    out = {}
    for s, e, k in sinks:
        out.setdefault(s, []).append("%d %d" % (e, k))
    text = "%d %d %d %d\n%s\n%s\n" % (pis, pos, len(kinds), len(out), "\n".join(
        "%d 1 %d %s" % (s, len(x), " ".join(x)) for s, x in sorted(out.items())), "\n".join(map(str, kinds)))
    live, _, folded = check(tmp_path, text, 40)
    assert live >= n
    if not buffers:
        assert (folded == 0) == (n == 1000)
