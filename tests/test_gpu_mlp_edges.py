"""The MLP kernels at the edges of their tiles (128 rows, a few hundred CTAs,
several tiles per CTA) against the numpy oracle, with the tolerances of
test_gpu_mlp.py: the device rounds to BF16 at the same points as the oracle but
sums in another order, so an activation can land one BF16 ulp away."""
import numpy as np
import pytest
import torch

import fvmpor_b200 as fb
from oracle import mlp_ref

pytestmark = pytest.mark.gpu


def network(seed):
    rng = np.random.default_rng(seed)
    mu = rng.normal(0, 1, 8).astype(np.float32)
    sd = (rng.random(8) + 0.5).astype(np.float32)
    ph = fb.Physics(fb.make_problem("richards2d", nx=21, ny=11))
    net = fb.Predictor(ph)
    P = mlp_ref.init_params(seed, mu, sd)
    net.set_params(P)
    return ph, net, P, mu, sd, rng


@pytest.mark.parametrize("n", [1, 127, 129, 148 * 4 * 128 + 5])
def test_forward_edges(n, cuda):
    _, net, P, mu, sd, rng = network(11)
    X = (mu + sd * rng.standard_normal((n, 8))).astype(np.float32)
    out = torch.full((n + 8,), 7.0, dtype=torch.float32, device=cuda)
    assert net.forward(torch.as_tensor(X, device=cuda), out[:n]) == 0
    ref = mlp_ref.forward(P, X)
    # 0.3: the size of the outputs of such a network
    assert np.abs(out[:n].cpu().numpy() - ref).max() < 1e-2 * max(np.abs(ref).max(), 0.3)
    assert (out[n:] == 7.0).all()   # nothing past the last row


@pytest.mark.parametrize("n", [1, 127, 129, 148 * 128 + 7, 148 * 256 + 1])
def test_gradient_and_step_edges(n, cuda):
    """The gradient against the oracle's, and one full-batch Adam step against
    the step that this gradient gives."""
    _, net, P, mu, sd, rng = network(12)
    X = (mu + sd * rng.standard_normal((n, 8))).astype(np.float32)
    Y = rng.standard_normal(n).astype(np.float32)
    Xt, Yt = torch.as_tensor(X, device=cuda), torch.as_tensor(Y, device=cuda)
    g, loss, rc = net.grad(Xt, Yt)
    assert rc == 0
    g0, loss0 = mlp_ref.grad(P, X, Y)
    assert abs(loss - loss0) < 2e-2 * loss0
    off = [mlp_ref.OFF_W1, mlp_ref.OFF_B1, mlp_ref.OFF_W2, mlp_ref.OFF_B2, mlp_ref.OFF_W3, mlp_ref.OFF_B3,
           mlp_ref.OFF_W4, mlp_ref.OFF_B4, mlp_ref.N_TRAIN]
    for a, b in zip(off, off[1:]):
        assert np.linalg.norm(g[a:b] - g0[a:b]) < 5e-2 * np.linalg.norm(g0[a:b]), (a, b)
    rc, hist = net.train(Xt, Yt, epochs=1, batch=n, lr=1e-3)
    assert rc == 0 and abs(hist[0] - loss) < 1e-6 * loss
    step = net.get_params()[:mlp_ref.N_TRAIN] - P[:mlp_ref.N_TRAIN]
    gd = np.asarray(g[:mlp_ref.N_TRAIN], dtype=np.float64)
    # m / (1 - b1) = g and v / (1 - b2) = g^2 up to FP32 rounding (1e-5 of the
    # step covers the few operations), the sum rounded to FP32
    want = -1e-3 * gd / (np.abs(gd) + 1e-8)
    big = np.abs(gd) > 1e-15   # below, g^2 leaves the FP32 range
    assert (np.abs(step - want)[big] < 1e-8 + 1.2e-7 * (np.abs(P[:mlp_ref.N_TRAIN]) + 1e-3)[big]).all()
    # the step's BF16 operands: the oracle's forward with the new parameters
    out = torch.empty(n, dtype=torch.float32, device=cuda)
    assert net.forward(Xt, out) == 0
    ref = mlp_ref.forward(net.get_params(), X)
    assert np.abs(out.cpu().numpy() - ref).max() < 1e-2 * max(np.abs(ref).max(), 1.0)
