"""Index arithmetic of the sampling kernels (birp_cpp_gb300/csrc/point_index.h)
for calls of up to 2^31 - 1 points, on the host."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_point_index(tmp_path):
    exe = str(tmp_path / "point_index")
    src = os.path.join(ROOT, "tests", "cpp", "point_index_test.cpp")
    subprocess.run(["g++", "-O2", "-std=c++17", src, "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
