"""What a refused CUDA call leaves behind (host only)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = "/usr/local/cuda"


def test_a_reported_error_is_cleared(tmp_path):
    exe = str(tmp_path / "cuda_error_check")
    subprocess.check_call(["/usr/bin/g++", "-std=c++17", "-O1", "-I" + CUDA + "/include",
                           os.path.join(ROOT, "tests", "cpp", "cuda_error_check.cpp"), "-o", exe])
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
