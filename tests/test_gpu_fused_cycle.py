"""The fused GMRES cycle (assembled FP32 operator, blocks resident in shared
memory) over the calls of one context: the dimension is the call's own, whatever
workspace an earlier call has left, also where only the smaller one's cycle fits
the shared memory; and a cycle in which a wait ran out after it had converged
fails by itself and leaves nothing to the next one."""
import os
import shutil
import subprocess

import numpy as np
import pytest
import torch

import fvmpor_b200 as fb

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def box(nx, ny, nz):
    return fb.make_problem("richards3d", nx=nx, ny=ny, nz=nz, Lx=float(nx), Ly=float(ny), Lz=float(nz))


def replay(ph, cuda, n_steps=3, **opts):
    """state, statistics and kernel launches of the first steps of one sequence"""
    y0 = torch.empty(ph.problem.n_nodes, dtype=torch.float64, device=cuda)
    ph.initial_head(y0)
    steps = np.zeros(n_steps, dtype=[("h", "f8"), ("order", "i4")])
    steps["h"], steps["order"] = [600.0, 600.0, 1200.0][:n_steps], [1, 2, 2][:n_steps]
    rep = fb.Integrator(ph, max_restarts=40, **opts)
    ye = torch.empty_like(y0)
    before = ph.counters()["launches"]
    rc, st = rep.replay(0.0, y0, 600.0, steps, ye, newton_tol=1e-5)
    assert rc == 0
    return ye.cpu().numpy(), st, ph.counters()["launches"] - before


@pytest.mark.parametrize("nx,ny,nz,per_sm,first,then", [
    (46, 43, 19, 0, 60, 6),
    # blocks of about 1,796 rows: a cycle of 30 steps fits an SM, one of 60 does not
    (112, 111, 20, 1, 60, 30)])
@pytest.mark.parametrize("variant", [0, 1])
def test_dimension_is_the_call_s_own(nx, ny, nz, per_sm, first, then, variant, cuda):
    p = box(nx, ny, nz)
    out = []
    for dims in ((first, then), (then,)):
        ph = fb.Physics(p)
        assert fb.lib().fvm_set_krylov_variant(ph._c, variant) == 0
        if per_sm:
            fb.Preconditioner(ph).set_blocks_per_sm(per_sm)
        for m in dims:
            res = replay(ph, cuda, n_steps=2, krylov_dim=m, precision=1, krylov_operator=1)
        out.append(res)
        ph.close()
    assert out[0][1]["nli"] == out[1][1]["nli"]
    assert np.array_equal(out[0][0], out[1][0])


def test_late_failure_is_seen_when_it_happens(cuda, tmp_path):
    exe, lib = tmp_path / "late_failure_check", os.path.join(ROOT, "fvmpor_b200")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "--expt-relaxed-constexpr",
                    "-I", os.path.join(lib, "csrc"), os.path.join(ROOT, "tests", "late_failure_check.cu"), "-o", str(exe),
                    "-L", lib, "-lfvmpor_b200", "-Xlinker", "-rpath=" + lib], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
