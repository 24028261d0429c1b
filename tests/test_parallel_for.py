"""The host loop of the set-up tables (common.hpp, parallel_for) when threads or
memory run out, on the CPU (tests/parallel_for_check.cpp)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_running_out_of_memory_or_threads(tmp_path):
    exe = tmp_path / "parallel_for_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-I", os.path.join(ROOT, "fvmpor_b200", "csrc"),
                    os.path.join(ROOT, "tests", "parallel_for_check.cpp"), "-o", str(exe)], check=True)
    for _ in range(3):
        r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
        assert r.returncode == 0, r.stdout + r.stderr
