"""fvm_integrate_batch: several contexts integrated side by side from host threads.
Their fused cycles (cooperative launches, programmatic dependents of the kernel
ahead) compete for the SMs, and their set-up tables are built by several
threads each at the same time; every member's run is the one it takes alone, bit
by bit."""
import numpy as np
import pytest
import torch

import fvmpor_b200 as fb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("opts", [dict(precision=1, krylov_operator=1), dict(precision=1)])
def test_members_run_as_if_alone(opts, cuda):
    # three boxes of 148 blocks, of which two fit the SMs at once, and planes of
    # one to ten blocks
    problems = [fb.make_problem("richards3d", nx=70, ny=70, nz=20, Lx=70.0, Ly=70.0, Lz=20.0, seed=s) for s in (1, 2, 3)]
    problems += [fb.make_problem("richards2d", nx=nx, ny=ny) for nx, ny in ((21, 11), (81, 41), (151, 93), (60, 50), (99, 71))]
    t_end, kw = 7200.0, dict(krylov_dim=30, max_restarts=5, max_order=5, **opts)

    def start():
        phs = [fb.Physics(p) for p in problems]
        y0 = [torch.empty(ph.N, dtype=torch.float64, device=cuda) for ph in phs]
        for ph, y in zip(phs, y0):
            ph.initial_head(y)
        return phs, y0

    alone = []
    phs, y0 = start()
    for ph, y in zip(phs, y0):
        ye = torch.empty_like(y)
        rc, st = fb.Integrator(ph, **kw).integrate(0.0, t_end, y, ye)
        assert rc == 0
        alone.append((ye.cpu().numpy(), st))
        ph.close()
    phs, y0 = start()
    ye = [torch.empty_like(y) for y in y0]
    rc, status, stats = fb.integrate_batch(phs, 0.0, t_end, y0, ye, n_threads=len(phs), **kw)
    assert rc == 0 and all(s == 0 for s in status)
    for m, (ref, st) in enumerate(alone):
        for key in ("nst", "nni", "nli", "npe", "nsync"):
            assert stats[m][key] == st[key], (m, key)
        assert np.array_equal(ye[m].cpu().numpy(), ref), m
    for ph in phs:
        ph.close()
