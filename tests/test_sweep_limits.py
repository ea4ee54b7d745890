"""Schedules at the limits of what the sweep's records can hold, on the CPU
with the standard library's checks switched on."""
import os
import subprocess

import pytest

from lsim_b200 import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
MAX_SLOTS = {16: 32767, 8: 1 << 14, 4: 1 << 14, 2: 1 << 14}


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("limits") / "sweep_limits_check")
    src = [os.path.join(build.CSRC, f) for f in ("fsimb_netlist.cpp", "fsimb_plan.cpp")]
    subprocess.check_call(["/usr/bin/g++", "-std=c++17", "-O2", "-D_GLIBCXX_ASSERTIONS",
                           os.path.join(ROOT, "tests", "cpp", "sweep_limits_check.cpp")] + src + ["-o", exe])

    def run(tmp_path, text):
        path = tmp_path / "c.ckt"
        path.write_text(text)
        r = subprocess.run([exe, str(path)], capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr
        lines = r.stdout.split("\n")
        live = int(lines[0].split()[1])
        return live, {int(g): (int(n), s if s == "refused" else int(s))
                      for g, n, s in (x.split() for x in lines[1:] if x)}

    return run


def _two_rows(n):
    """n XORs of neighbouring PIs (16 of them); n ANDs, each of two of the
    XORs, each with a PO: every XOR is read twice, so all n live at once."""
    pis = 16
    g0 = pis + n
    sinks = [[] for _ in range(g0 + 2 * n)]
    for i in range(n):
        sinks[i % pis].append((g0 + i, 1))
        sinks[(i + 1 + i // pis % (pis - 1)) % pis].append((g0 + i, 2))
        sinks[g0 + i].append((g0 + n + i, 1))
        sinks[g0 + (i + 1) % n].append((g0 + n + i, 2))
        sinks[g0 + n + i].append((pis + i, 1))
    wires = ["%d 1 %d %s" % (e, len(s), " ".join("%d %d" % x for x in s)) for e, s in enumerate(sinks) if s]
    return "%d %d %d %d\n%s\n%s\n" % (pis, n, 2 * n, len(wires), "\n".join(wires), "\n".join(["3"] * n + ["1"] * n))


@pytest.mark.parametrize("n", [1000, 16000, 17000, 33000])
def test_a_schedule_beyond_the_slot_fields_is_refused(check, tmp_path, n):
    live, got = check(tmp_path, _two_rows(n))
    assert live >= n
    assert set(got) == set(MAX_SLOTS)
    for g, (slots, packed) in got.items():
        assert slots >= n
        if slots > MAX_SLOTS[g]:
            assert packed == "refused"
        else:
            assert packed >= 2 * n
    if n == 33000:
        assert all(packed == "refused" for _, packed in got.values())


@pytest.fixture(scope="module")
def shape(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("shape") / "sweep_shape_check")
    lib = build.build()
    subprocess.check_call(["/usr/bin/g++", "-std=c++17", "-O2", "-I/usr/local/cuda/include",
                           os.path.join(ROOT, "tests", "cpp", "sweep_shape_check.cpp"), lib,
                           "-Wl,-rpath," + os.path.dirname(lib), "-o", exe])

    def run(tmp_path, text, smem, words):
        path = tmp_path / "c.ckt"
        path.write_text(text)
        r = subprocess.run([exe, str(path), str(smem), str(words)], capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr
        lines = [[int(x) for x in s.split()] for s in r.stdout.split("\n") if s and s != "none"]
        return (None if r.stdout.startswith("none") else lines[0]), lines[0 if r.stdout.startswith("none") else 1:]

    return run


@pytest.mark.parametrize("n", [1000, 17000, 33000])
@pytest.mark.parametrize("smem", [16 << 10, 64 << 10, 227 << 10])
@pytest.mark.parametrize("words", [1, 32])
def test_the_default_shape_fits_or_there_is_none(shape, tmp_path, n, smem, words):
    got, likely = shape(tmp_path, _two_rows(n), smem, words)
    room = smem - 1536  # what the launch's own use leaves
    if got is None:
        assert (2 * n + 16) * 8 > room  # not one word of every gate's value
    else:
        m, threads, slots = got
        assert slots * m * 8 <= room and slots <= MAX_SLOTS[16 // m]
        assert 32 <= threads <= 1024 and threads % 32 == 0
    for m, _ in likely:
        assert n * m * 8 <= room
    assert n != 33000 or got is None
