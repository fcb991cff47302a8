"""The MLP's layer products at batch sizes on both sides of every tile: a row of a
forward pass is the same sums in the same order whatever the batch, so its bits do
not depend on the tile; gradients against the FP64 restatement with the tolerance of
FP32 sums of random sign (1e-5 of the norm)."""
import numpy as np
import pytest

from oracle import mlp_oracle
from tailor_gb300 import learned

pytestmark = pytest.mark.gpu

SHAPE = (5, 130, 2, 70)


def test_forward_bits_do_not_depend_on_the_tile(gpu_lib):
    net = learned.MLP(*SHAPE, seed=2)
    X = np.random.default_rng(1).standard_normal((4100, 5)).astype(np.float32)
    tiles = {gpu_lib.tlr_mlp_tile(n, 130, 1, 152) for n in (17, 700, 4100)}
    assert tiles == {16, 32, 64}
    whole = net.forward(X)
    for n in (1, 15, 16, 17, 33, 65, 700):
        assert np.array_equal(net.forward(X[:n]), whole[:n])
    net.close()


@pytest.mark.parametrize("n", [1, 16, 17, 31, 33, 64, 65, 190, 320])
def test_gradients(gpu_lib, n):
    net = learned.MLP(*SHAPE, seed=3)
    rng = np.random.default_rng(n)
    X = rng.standard_normal((n, 5)).astype(np.float32)
    Y = rng.standard_normal((n, 70)).astype(np.float32)
    p = net.get_params().astype(np.float64)
    loss, g = net.gradients(X, Y)
    loss_ref, g_ref = mlp_oracle.loss_and_grad(p, X, Y, SHAPE)
    assert abs(loss - loss_ref) <= 1e-5 * abs(loss_ref)
    assert np.linalg.norm(g - g_ref) <= 1e-5 * np.linalg.norm(g_ref)
    net.close()
