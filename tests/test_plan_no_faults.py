"""The plan of the good machine alone (no faults)."""
import os
import subprocess

from lsim_b200 import build, gen

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_a_plan_without_faults_is_bare(tmp_path):
    exe = str(tmp_path / "plan_no_faults_check")
    src = [os.path.join(build.CSRC, f) for f in ("fsimb_netlist.cpp", "fsimb_plan.cpp")]
    subprocess.check_call(["/usr/bin/g++", "-std=c++17", "-O2",
                           os.path.join(ROOT, "tests", "cpp", "plan_no_faults_check.cpp")] + src + ["-o", exe])
    path = tmp_path / "c.ckt"
    path.write_text(gen.circuit(5000, 40, 30, 20, type_mask=gen.ALL_TYPES))
    r = subprocess.run([exe, str(path)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
