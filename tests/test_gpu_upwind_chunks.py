"""The step's upwind directions formed chunk by chunk (meshes of 59 chunks of 512
elements or more; smaller ones go edge by edge) against the CPU oracle:
the residual with the frozen directions.

Tolerance as in test_gpu_parity.py for residuals: 1e-10 of the largest entry.
The heads are noisy enough that no edge's flux is near zero, so a direction that
differs shows as an error of the flux's own size."""
import numpy as np
import pytest
import torch

import fvmpor_b200 as fb
from oracle.pyoracle import Oracle

pytestmark = pytest.mark.gpu

# 59 chunks (the least that go chunk by chunk) to 311, a full last chunk, one and
# two zones, rebuilt and stored geometry
CASES = [("richards2d", dict(nx=123, ny=123), 0), ("richards2d", dict(nx=401, ny=200), 0),
         ("richards3d", dict(nx=31, ny=33, nz=25), 0), ("richards3d", dict(nx=17, ny=16, nz=19), fb.FLAG_STORED_GEOMETRY),
         ("richards3d", dict(nx=32, ny=33, nz=24), 0)]


@pytest.mark.parametrize("case", range(len(CASES)))
def test_begin_step_then_residual(case, cuda):
    name, size, flags = CASES[case]
    p = fb.make_problem(name, **size)
    ph = fb.Physics(p, flags=flags) if flags else fb.Physics(p)
    orc = Oracle(p)
    z = p.arrays()["coords"][:, 1 if name == "richards2d" else 2]
    rng = np.random.default_rng(case)
    y = p.water_table - z + 0.05 * rng.standard_normal(p.n_nodes)
    yp = 1e-7 * rng.standard_normal(p.n_nodes)
    yt, ypt = torch.as_tensor(y, device=cuda), torch.as_tensor(yp, device=cuda)
    F = torch.empty_like(yt)
    for shift in (0.0, 0.3):   # a second step on the same context
        ph.begin_step(0.0, yt + shift, ypt)
        orc.begin_step(0.0, y + shift, yp)
        ph.residual(0.0, yt + shift, ypt, F)
        ref = orc.residual(0.0, y + shift, yp)
        assert np.abs(F.cpu().numpy() - ref).max() < 1e-10 * np.abs(ref).max()
