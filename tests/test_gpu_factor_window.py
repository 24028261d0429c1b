"""What the block factor's window must leave room for (shared memory of a CTA and
of an SM), and rows that it holds apart: the applies against the CPU oracle's
of the same matrix in the same order.

* The Schur-coupled apply in FP64 on boxes of one block per SM and of two, where
  the factor with its forward result fills most of the shared memory, and on one
  whose factor fits unpadded only (read in place); in FP32 with four per SM.
* The block-Jacobi apply of blocks too large to be staged.
* Nodes of 63 to 400 neighbours (rows of more than 64 entries beside the
  diagonal are stored apart), both applies.

Tolerances as in test_gpu_factor_slices.py: FP64 differs by rounding (1e-10 of the
result), FP32 by FP32 rounding through the sweeps (2e-4)."""
import numpy as np
import pytest
import torch

import fvmpor_b200 as fb
from oracle.pyoracle import Oracle, factor_given

pytestmark = pytest.mark.gpu


def check_apply(p, precision, cuda, schur=-1, per_sm=0, seed=0):
    ph, orc = fb.Physics(p), Oracle(p)
    rng = np.random.default_rng(seed)
    z = p.arrays()["coords"][:, 1 if p.mesh.dim == 2 else 2]
    y = p.water_table - z + 0.05 * rng.standard_normal(p.n_nodes)
    yp = 1e-7 * rng.standard_normal(p.n_nodes)
    T = lambda v: torch.as_tensor(v, device=cuda)
    yt, ypt = T(y), T(yp)
    ph.begin_step(0.0, yt, ypt)
    orc.begin_step(0.0, y, yp)
    F0 = orc.residual(0.0, y, yp)
    ewt = 1.0 / (1e-6 * np.abs(y) + 1e-6)
    pc = fb.Preconditioner(ph)
    if per_sm:
        pc.set_blocks_per_sm(per_sm)
    pc.set_schur(schur)
    assert pc.setup(0.0, 2e-3, 500.0, yt, ypt, T(F0), T(ewt), precision) == 0
    nb = pc.info()["nblocks"]
    if schur >= 0:
        assert pc.schur_info()["fp32" if precision else "fp64"]
        orc.set_schur(schur)
    assert orc.psetup(0.0, 2e-3, 500.0, y, yp, F0, ewt, nb) == 0
    assert factor_given(orc, pc.jacobian()[2], nb) == 0
    r = rng.standard_normal(p.n_nodes)
    zt = torch.empty_like(yt)
    pc.apply(T(r), zt)
    ref = orc.psolve(r)
    ph.close()
    err = np.abs(zt.cpu().numpy() - ref).max() / np.abs(ref).max()
    assert err < (1e-10 if precision == 0 else 2e-4), err


def box(nx, ny, nz):
    return fb.make_problem("richards3d", nx=nx, ny=ny, nz=nz, Lx=float(nx), Ly=float(ny), Lz=float(nz))


@pytest.mark.parametrize("nx,ny,nz,per_sm,precision", [
    (100, 100, 20, 1, 0), (100, 100, 20, 2, 0), (105, 105, 20, 2, 0), (100, 100, 20, 4, 1), (13, 13, 14, 0, 0),
    (30, 30, 20, 0, 0)])
def test_schur_apply_where_the_factor_fits(nx, ny, nz, per_sm, precision, cuda):
    check_apply(box(nx, ny, nz), precision, cuda, schur=2, per_sm=per_sm)


@pytest.mark.parametrize("precision", [0, 1])
def test_blocks_too_large_to_stage(precision, cuda):
    # about 2,940 rows
    check_apply(box(130, 128, 25), precision, cuda, per_sm=1)


def fan(sectors):
    """a disc of `sectors` sectors, two rings around one node in the middle of
    the node order"""
    a = 2.0 * np.pi * np.arange(sectors) / sectors
    ring = np.stack([np.cos(a), np.sin(a), 0.0 * a], axis=1)
    xyz = np.concatenate([ring, [[0.0, 0.0, 0.0]], 2.0 * ring])
    i, j = np.arange(sectors), (np.arange(sectors) + 1) % sectors
    o = sectors + 1
    tri = np.concatenate([np.stack([i, j, np.full(sectors, sectors)], 1), np.stack([i, o + i, o + j], 1),
                          np.stack([i, o + j, j], 1)])
    zone = fb.Zone(1e-5, 1e-5, 1e-5, 0.4, 2.0, 1.8, 0.1)
    none = np.zeros(0, np.int32)
    return fb.Problem.from_arrays(2, xyz, tri, np.zeros(len(tri), np.int32), none, none, none,
                                  np.zeros(len(xyz), np.int32), [zone], [fb.BC(1, 1, 0.0, 0.0, 0.0)], water_table=-1.0)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("sectors", [63, 64, 65, 66, 400, 1600])
def test_a_node_of_many_neighbours(sectors, precision, cuda):
    check_apply(fan(sectors), precision, cuda)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("sectors", [65, 1600])
def test_schur_apply_with_a_node_of_many_neighbours(sectors, precision, cuda):
    # (65 sectors: one block, no interface; 1,600: three blocks)
    check_apply(fan(sectors), precision, cuda, schur=2)
