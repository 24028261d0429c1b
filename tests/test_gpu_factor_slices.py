"""The sliced block factor at the sizes where its layout can go wrong (blocks of
a few rows, rows that do not fill a slice, several blocks, levels wider than the
CTA's warps; the largest blocks of the fused cycle), against the CPU oracle's
factorisation of the same matrix in the same order.

Tolerances: the FP64 apply differs from the oracle's by rounding only (1e-10 of
the result, as in test_gpu_configs.py); the FP32 factor by FP32 rounding through
two sweeps (2e-4)."""
import numpy as np
import pytest
import torch

import fvmpor_b200 as fb
from oracle.pyoracle import Oracle, factor_given

pytestmark = pytest.mark.gpu

MESHES = [dict(name="richards2d", nx=3, ny=2), dict(name="richards2d", nx=8, ny=4), dict(name="richards2d", nx=11, ny=3),
          dict(name="richards2d", nx=61, ny=49), dict(name="richards3d", nx=1, ny=1, nz=1),
          dict(name="richards3d", nx=7, ny=5, nz=3), dict(name="richards3d", nx=22, ny=17, nz=9)]


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("mesh", range(len(MESHES)))
def test_apply_matches_the_oracle(mesh, precision, cuda):
    m = dict(MESHES[mesh])
    p = fb.make_problem(m.pop("name"), **m)
    ph, orc = fb.Physics(p), Oracle(p)
    a = p.arrays()
    rng = np.random.default_rng(mesh)
    z = a["coords"][:, 1 if "nz" not in m else 2]
    y = p.water_table - z + 0.05 * rng.standard_normal(p.n_nodes)
    yp = 1e-7 * rng.standard_normal(p.n_nodes)
    T = lambda v: torch.as_tensor(v, device=cuda)
    yt, ypt = T(y), T(yp)
    ph.begin_step(0.0, yt, ypt)
    orc.begin_step(0.0, y, yp)
    F0 = orc.residual(0.0, y, yp)
    ewt = 1.0 / (1e-6 * np.abs(y) + 1e-6)
    pc = fb.Preconditioner(ph)
    # the other precision first: its factor must not show in this one's
    assert pc.setup(0.0, 1e-3, 400.0, yt, ypt, T(F0), T(ewt), 1 - precision) == 0
    assert pc.setup(0.0, 2e-3, 500.0, yt, ypt, T(F0), T(ewt), precision) == 0
    nb = pc.info()["nblocks"]
    assert orc.psetup(0.0, 2e-3, 500.0, y, yp, F0, ewt, nb) == 0
    assert factor_given(orc, pc.jacobian()[2], nb) == 0
    r = rng.standard_normal(p.n_nodes)
    zt = torch.empty_like(yt)
    pc.apply(T(r), zt)
    ref = orc.psolve(r)
    err = np.abs(zt.cpu().numpy() - ref).max() / np.abs(ref).max()
    assert err < (1e-10 if precision == 0 else 2e-4), err


@pytest.mark.parametrize("nx,ny,nz", [(46, 43, 19), (104, 102, 20)])
def test_fused_cycle_smallest_and_largest_blocks(nx, ny, nz, cuda):
    """Blocks of about 274 and 1,534 rows: the two orthogonalisations replay
    the same steps to the same state (1e-10, as in test_gpu_krylov_variants.py)."""
    p = fb.make_problem("richards3d", nx=nx, ny=ny, nz=nz, Lx=float(nx), Ly=float(ny), Lz=float(nz))
    ph = fb.Physics(p)
    y0 = torch.empty(p.n_nodes, dtype=torch.float64, device=cuda)
    ph.initial_head(y0)
    steps = np.zeros(3, dtype=[("h", "f8"), ("order", "i4")])
    steps["h"], steps["order"] = [600.0, 600.0, 1200.0], [1, 2, 2]
    out = []
    for v in (0, 1):
        assert fb.lib().fvm_set_krylov_variant(ph._c, v) == 0
        rep = fb.Integrator(ph, krylov_dim=40, precision=1, krylov_operator=1, max_restarts=5)
        ye = torch.empty_like(y0)
        rc, st = rep.replay(0.0, y0, 600.0, steps, ye, newton_tol=1e-5)
        assert rc == 0
        out.append(ye.cpu().numpy())
    assert np.abs(out[0] - out[1]).max() < 1e-10 * np.abs(out[0]).max()
    ph.close()
