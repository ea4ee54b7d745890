"""Sweep schedules (clusters of single-consumer gates, slots, live-in lists)
run on the CPU against a plain evaluation of the netlist: gates of every
type with 1 to 4 inputs, repeated inputs, MUX, shallow circuits (levels
ordered by record kind) and deep ones."""
import os
import subprocess

import pytest

from lsim_b200 import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("sweep") / "sweep_net_check")
    src = [os.path.join(build.CSRC, f) for f in ("fsimb_netlist.cpp", "fsimb_plan.cpp")]
    subprocess.check_call(["/usr/bin/g++", "-std=c++17", "-O2", os.path.join(ROOT, "tests", "cpp", "sweep_net_check.cpp")]
                          + src + ["-o", exe])
    return exe


@pytest.mark.parametrize("seed", range(4))
@pytest.mark.parametrize("gates,inputs,mux,window,near", [
    (3, 2, 0, 8, 4), (60, 2, 0, 12, 4), (200, 3, 0, 60, 4), (200, 4, 0, 200, 4), (200, 4, 1, 40, 4),
    (300, 3, 1, 300, 4), (250, 1, 0, 9, 4), (9000, 3, 0, 9000, 9000), (9000, 4, 1, 9000, 9000)])
def test_schedules_equal_plain_evaluation(check, seed, gates, inputs, mux, window, near):
    r = subprocess.run([check] + [str(x) for x in (seed, gates, inputs, mux, window, near)], capture_output=True,
                       text=True, timeout=120)
    assert r.returncode == 0, r.stderr
    assert int(r.stdout.split()[0]) > 0
