"""Training batch by batch: the launches of an epoch's batches overlap, so an epoch
is compared with the same batches trained one call at a time, each on a copy of
its samples written by the kernel ahead of the call.  The same kernels on the
same numbers in the same order: bit for bit."""
import numpy as np
import pytest
import torch

import fvmpor_b200 as fb
from oracle import mlp_ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,batch", [(300, 128), (5000, 257), (70000, 8192), (200000, 148 * 256)])
def test_epoch_equals_its_batches(n, batch, cuda):
    rng = np.random.default_rng(n)
    mu, sd = rng.normal(0, 1, 8).astype(np.float32), (rng.random(8) + 0.5).astype(np.float32)
    P = mlp_ref.init_params(3, mu, sd)
    X = torch.as_tensor((mu + sd * rng.standard_normal((n, 8))).astype(np.float32), device=cuda)
    Y = torch.as_tensor(rng.standard_normal(n).astype(np.float32), device=cuda)
    ph = [fb.Physics(fb.make_problem("richards2d", nx=21, ny=11)) for _ in range(2)]
    whole, single = (fb.Predictor(q) for q in ph)
    whole.set_params(P)
    single.set_params(P)
    rc, hist = whole.train(X, Y, epochs=2, batch=batch, lr=1e-3)
    assert rc == 0
    for epoch in range(2):
        loss = 0.0
        for b in range(0, n, batch):
            xb, yb = X[b:b + batch].clone(), Y[b:b + batch].clone()
            rc, h = single.train(xb, yb, epochs=1, batch=batch, lr=1e-3)
            assert rc == 0
            loss += float(h[0]) * len(yb)
        # (sums of FP32 batch losses, each rounded once more here)
        assert abs(loss / n - hist[epoch]) < 1e-6 * hist[epoch]
    assert np.array_equal(whole.get_params(), single.get_params())
