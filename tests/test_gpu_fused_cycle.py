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


N_STEPS = 100


def steps_of_a_run(ph, cuda, n_steps=N_STEPS):
    """first step size and accepted steps of an adaptive run: long enough that the
    last solves take a few dozen Krylov steps"""
    y0 = torch.empty(ph.problem.n_nodes, dtype=torch.float64, device=cuda)
    ph.initial_head(y0)
    run = fb.Integrator(ph, krylov_dim=40, max_order=5, max_steps=n_steps, precision=1, krylov_operator=1)
    rc, st = run.integrate(0.0, 30 * 86400.0, y0, torch.empty_like(y0))
    assert rc == 1 and st["nst"] == n_steps
    tr = run.trace()
    return float(tr["h"][0]), tr


def replay(ph, cuda, steps, **opts):
    """final state and statistics of the sequence, every corrector solved tightly"""
    y0 = torch.empty(ph.problem.n_nodes, dtype=torch.float64, device=cuda)
    ph.initial_head(y0)
    rep = fb.Integrator(ph, max_order=5, max_restarts=60, **opts)
    ye = torch.empty_like(y0)
    rc, st = rep.replay(0.0, y0, steps[0], steps[1], ye, newton_tol=1e-5)
    assert rc == 0
    return ye.cpu().numpy(), st


@pytest.mark.parametrize("nx,ny,nz,per_sm,first,then", [
    (46, 43, 19, 0, 60, 6),
    # blocks of about 1,796 rows: a cycle of 30 steps fits an SM, one of 60 does not
    (112, 111, 20, 1, 60, 30)])
@pytest.mark.parametrize("variant", [0, 1])
def test_dimension_is_the_call_s_own(nx, ny, nz, per_sm, first, then, variant, cuda):
    p = box(nx, ny, nz)
    out, steps = [], None
    for dims in ((first, then), (then,)):
        ph = fb.Physics(p)
        assert fb.lib().fvm_set_krylov_variant(ph._c, variant) == 0
        if per_sm:
            fb.Preconditioner(ph).set_blocks_per_sm(per_sm)
        if steps is None:
            other = fb.Physics(p)
            steps = steps_of_a_run(other, cuda)
            other.close()
        for m in dims:
            res = replay(ph, cuda, steps, krylov_dim=m, precision=1, krylov_operator=1)
        out.append(res)
        ph.close()
    assert out[0][1]["nli"] == out[1][1]["nli"]
    assert np.array_equal(out[0][0], out[1][0])


@pytest.mark.parametrize("nx,ny,nz", [(46, 43, 19), (104, 102, 20)])
@pytest.mark.parametrize("variant", [0, 1])
def test_the_fused_cycle_runs(nx, ny, nz, variant, cuda):
    """Blocks of about 274 and 1,534 rows, cycles that converge and cycles that end
    with a full basis: a fused solve waits once per cycle, and once more for its
    Newton update when it restarted (the separate kernels wait twice per cycle
    and for every update); the Newton iteration does not depend on the dimension."""
    ph = fb.Physics(box(nx, ny, nz))
    assert fb.lib().fvm_set_krylov_variant(ph._c, variant) == 0
    steps = steps_of_a_run(ph, cuda)
    nni = {}
    for m in (40, 4):
        _, st = replay(ph, cuda, steps, krylov_dim=m, precision=1, krylov_operator=1)
        cycles = st["nps"] - st["nli"]   # one apply for each Krylov step, one at a cycle's start
        assert st["nli"] > 5 * st["nni"]   # solves of more than a step or two
        assert m == 40 or cycles > 2 * st["nni"]
        assert st["nsync"] <= 2 * cycles - st["nni"] + 4
        nni[m] = st["nni"]
    assert abs(nni[4] - nni[40]) <= 0.1 * nni[40]
    ph.close()


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe, lib = tmp_path_factory.mktemp("fused") / "fused_cycle_check", os.path.join(ROOT, "fvmpor_b200")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "--expt-relaxed-constexpr",
                    "-I", os.path.join(lib, "csrc"), os.path.join(ROOT, "tests", "fused_cycle_check.cu"), "-o", str(exe),
                    "-L", lib, "-lfvmpor_b200", "-Xlinker", "-rpath=" + lib], check=True)

    def run(what):
        r = subprocess.run([str(exe), what], capture_output=True, text=True, timeout=120)
        assert r.returncode == 0, r.stdout + r.stderr

    return run


def test_late_failure_is_seen_when_it_happens(cuda, check):
    check("late")


def test_restarted_solves_meet_their_tolerance(cuda, check):
    check("restart")


def test_solves_with_a_node_of_many_neighbours(cuda, check):
    check("wide")
