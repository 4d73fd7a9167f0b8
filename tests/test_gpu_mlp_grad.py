"""Sensor-network gradient kernel at the edges of its 64-sample tiles, every input width, against the FP64 numpy
restatement.  Bound: a pre-activation is a sum of at most 57 FP32 terms of order one (rounding 57 * 2^-24 = 3.4e-6),
which the two layers pass on with weights of Glorot size; the gradient's norm follows to the same order: 1e-5."""
import numpy as np
import pytest

from dgkernel_b200 import sensor as SN
from oracle import mlp_ref as MR

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nin", [4, 10, 20, 35, 56])
@pytest.mark.parametrize("n", [1, 63, 64, 65, 1000, 40001])
def test_gradient_tiles(nin, n):
    import torch
    rng = np.random.default_rng(nin * 100003 + n)
    p = SN.init_params(nin, seed=n % 97)
    X = rng.normal(size=(n, nin)).astype(np.float32)
    X /= np.linalg.norm(X, axis=1, keepdims=True)
    y = rng.uniform(size=n).astype(np.float32)
    net = SN.SensorNet(nin, p)
    loss, g = net.loss_grad(torch.tensor(X, device="cuda"), torch.tensor(y, device="cuda"))
    lw, gw = MR.loss_grad(p, X, y, nin)
    assert abs(loss - lw) <= 1e-5 * lw
    assert np.linalg.norm(g.cpu().numpy() - gw) <= 1e-5 * np.linalg.norm(gw)
