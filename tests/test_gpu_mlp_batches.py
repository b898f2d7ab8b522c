"""The weight gradients of batches above 256, whose product goes through the staging ring more than
once (its K is the batch padded to 64; the ring holds four chunks of 64), layer by layer against the CPU
oracle with the same BF16 rounding points (1e-2 relative L2, as in test_gpu_surrogate), and the same
bits in a second call: the sums' order is fixed, so a chunk multiplied before it has arrived would show."""
import numpy as np
import pytest

from helpers import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [257, 320, 321, 1000, 1024, 2048, 4096])
def test_weight_gradients_of_large_batches(fwt, B):
    from fastweavturb_b200.surrogate import MLP
    from oracle import mlp_oracle as MO

    rng = np.random.default_rng(B)
    net = MLP(n_in=5, width=256, depth=2, n_out=45, batch_max=4096, seed=4)
    p = net.params().astype(np.float64)
    X = rng.uniform(-1, 1, (B, 5)).astype(np.float32)
    T = rng.normal(0, 1, (B, 45)).astype(np.float32)
    _, gp, gx = net.loss_grad(X, T)
    _, gpo, gxo = MO.loss_grad(p, net.widths, X, T)
    assert rel_l2(gx, gxo) <= 1e-2
    for (W, b), (Wo, bo) in zip(MO.unflatten(gp, net.widths), MO.unflatten(gpo, net.widths)):
        assert rel_l2(W, Wo) <= 1e-2
        assert rel_l2(b, bo) <= 1e-2
    for _ in range(3):
        _, again, _ = net.loss_grad(X, T)
        assert np.array_equal(again, gp)
    net.close()
