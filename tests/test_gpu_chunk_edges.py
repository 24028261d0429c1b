"""Kernels that take the elements in chunks, on meshes whose element counts
fall on, just under and just over whole chunks (192 elements of the quotient
Jacobian), against the FP64 oracle and, for FP32 quotients, the device's FP64
ones.

Tolerances: the FP64 Jacobian as in test_gpu_parity.py (1e-6 of the row
maximum, plus the residual's rounding over the shift).  Each FP32 quotient is
rounded once (2^-24 relative), an entry sums at most 24 of them (the tetrahedra
around a node of the boxes), none larger than a small multiple of the row's
diagonal: 4 x 24 x 2^-24 of the row maximum."""
import numpy as np
import pytest
import torch

import fvmpor_b200 as fb
from oracle.pyoracle import Oracle

pytestmark = pytest.mark.gpu

# (mesh, elements): 6 per box cell, 2 per plane cell
MESHES = {
    "3d_one_cell": (("3d", dict(nx=1, ny=1, nz=1)), 6),
    "3d_whole": (("3d", dict(nx=4, ny=4, nz=2)), 192),
    "3d_one_over": (("3d", dict(nx=11, ny=3, nz=1)), 198),
    "3d_two_under": (("3d", dict(nx=9, ny=7, nz=1)), 378),
    "3d_two_whole": (("3d", dict(nx=8, ny=4, nz=2)), 384),
    "2d_one_under": (("2d", dict(nx=96, ny=2)), 190),
    "2d_whole": (("2d", dict(nx=13, ny=9)), 192),
    "2d_over": (("2d", dict(nx=98, ny=2)), 194),
}


def problem(name):
    (kind, kw), n_elements = MESHES[name]
    if kind == "3d":
        kw = dict(kw, Lx=float(kw["nx"]), Ly=float(kw["ny"]), Lz=float(kw["nz"]))
    p = fb.make_problem("richards" + kind, **kw)
    assert p.n_elements == n_elements
    return p


def state(p, seed):
    a = p.arrays()
    vert = a["coords"][:, 1 if p.mesh.dim == 2 else 2]
    rng = np.random.default_rng(seed)
    return p.water_table - vert + 0.05 * rng.standard_normal(p.n_nodes), 1e-6 * rng.standard_normal(p.n_nodes)


def T(x, dev):
    return torch.as_tensor(np.ascontiguousarray(x, np.float64), device=dev)


@pytest.mark.parametrize("flags", [fb.FLAG_STORED_GEOMETRY, fb.FLAG_RECOMPUTE_GEOMETRY])
@pytest.mark.parametrize("name", list(MESHES))
def test_quotient_jacobian(name, flags, cuda):
    p = problem(name)
    if flags == fb.FLAG_RECOMPUTE_GEOMETRY and p.mesh.dim == 2:
        pytest.skip("geometry recompute is a 3D variant")
    ph, orc = fb.Physics(p, flags), Oracle(p)
    pc = fb.Preconditioner(ph)
    y, yp = state(p, 5)
    ewt = 1.0 / (1e-6 * np.abs(y) + 1e-6)
    cj, h = 2e-3, 500.0
    yt, ypt = T(y, cuda), T(yp, cuda)
    for frozen in (False, True):   # averaged face weights, then upwind ones
        if frozen:
            ph.begin_step(0.0, yt, ypt)
            orc.begin_step(0.0, y, yp)
        F0 = orc.residual(0.0, y, yp)
        assert pc.setup(0.0, cj, h, yt, ypt, T(F0, cuda), T(ewt, cuda), 0) == 0
        assert orc.psetup(0.0, cj, h, y, yp, F0, ewt, pc.info()["nblocks"]) == 0
        rp, col, val = pc.jacobian()
        orp, ocol, oval, _ = orc.jacobian()
        assert np.array_equal(rp, orp) and np.array_equal(col, ocol)
        rows = np.repeat(np.arange(p.n_nodes), np.diff(rp))
        rmax = np.maximum.reduceat(np.abs(oval), rp[:-1])
        d = np.sqrt(np.finfo(float).eps) * np.maximum(np.abs(y), np.maximum(np.abs(h * yp), 1.0 / ewt))
        S = np.abs(F0) + 1e-3 * np.abs(F0).max() + np.abs(orc.ahh() * yp)
        assert (np.abs(val - oval) / (1e-6 * rmax[rows] + 5e-13 * S[rows] / d[col])).max() < 1.0
        assert pc.setup(0.0, cj, h, yt, ypt, T(F0, cuda), T(ewt, cuda), 1) == 0
        val32 = pc.jacobian()[2]
        assert (np.abs(val32 - val) / (4 * 24 * 2.0**-24 * rmax[rows])).max() < 1.0
