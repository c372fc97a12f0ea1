"""The device blocks kept between cubes (birp_cpp_gb300/csrc/block_cache.h): what is kept, what a request gets, the
bound, the device they belong to and threads, on the host."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_block_cache(tmp_path):
    exe = str(tmp_path / "block_cache")
    src = os.path.join(ROOT, "tests", "cpp", "block_cache_test.cpp")
    subprocess.run(["g++", "-O2", "-std=c++17", "-Wall", "-pthread", src, "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
