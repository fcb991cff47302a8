"""The MLP's layer products (64 x 64 tiles, inner chunks of 16, rows of a
weight gradient in ranges of 128) at sizes that leave remainders in every one,
against the FP64 restatement.  FP32 sums of up to a few thousand terms of
random sign: 1e-5 of the result's norm."""
import numpy as np
import pytest

from oracle import mlp_oracle
from tailor_gb300 import learned

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,n", [
    ((3, 17, 1, 5), 1), ((1, 64, 2, 65), 63), ((5, 33, 3, 2), 257), ((3, 256, 4, 80), 2050),
    ((70, 130, 2, 70), 1000),
])
def test_gradients_and_forward(gpu_lib, shape, n):
    net = learned.MLP(*shape, seed=3)
    rng = np.random.default_rng(n)
    X = rng.standard_normal((n, shape[0])).astype(np.float32)
    Y = rng.standard_normal((n, shape[3])).astype(np.float32)
    p = net.get_params().astype(np.float64)
    for _ in range(2):  # the counters and partial sums are ready for another batch
        loss, g = net.gradients(X, Y)
        loss_ref, g_ref = mlp_oracle.loss_and_grad(p, X, Y, shape)
        assert abs(loss - loss_ref) <= 1e-5 * abs(loss_ref)
        assert np.linalg.norm(g - g_ref) <= 1e-5 * np.linalg.norm(g_ref)
    y_ref, _, _ = mlp_oracle.forward(p, X, shape)
    assert np.linalg.norm(net.forward(X) - y_ref) <= 1e-5 * np.linalg.norm(y_ref)
    net.close()
