"""The block factor's layout for the triangular sweeps, on the CPU: what the
device's lanes read (tests/ilu_layout_check.cpp walks it lane by lane) gives the
triangular solves, stays inside the arrays and hits different banks, and the
window is little larger than the factor, rows of many neighbours among them."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def walk(tmp_path_factory):
    exe = tmp_path_factory.mktemp("ilu") / "ilu_layout_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-I", os.path.join(ROOT, "fvmpor_b200", "csrc"),
                    os.path.join(ROOT, "tests", "ilu_layout_check.cpp"), "-o", str(exe)], check=True)

    def run(*args):
        r = subprocess.run([str(exe)] + [str(a) for a in args], capture_output=True, text=True)
        assert r.returncode == 0, r.stdout
        return float(r.stdout)

    return run


@pytest.mark.parametrize("rows,per_row,hubs,hub_len", [
    (1, 0, 0, 0), (2, 2, 0, 0), (3, 0, 0, 0), (5, 4, 0, 0), (31, 6, 0, 0), (33, 6, 0, 0), (128, 12, 0, 0), (700, 12, 0, 0),
    (150, 4, 1, 63), (150, 4, 1, 64), (150, 4, 1, 65), (150, 4, 1, 66), (400, 6, 2, 300), (1500, 6, 1, 1400), (200, 150, 0, 0)])
def test_sweeps_of_the_layout(walk, rows, per_row, hubs, hub_len):
    for seed in range(4):
        walk(rows, per_row, hubs, hub_len, seed)


def test_a_row_of_many_neighbours_widens_nothing_else(walk):
    # 1,500 rows, one coupled to 1,400 others: at most a group of kIluWide = 64 by
    # four lanes beside its own entries, of about 12,000
    assert walk(1500, 8, 1, 1400, 0) < walk(1500, 8, 0, 0, 0) + 0.05
