"""The network's fused products at the edges of their tiles: batches around the 64-row padding and
the 128-row tile, widths around the 32-column tile, one hidden layer and more layers than one
launch holds, against the CPU oracle with the same BF16 rounding points (loss 1e-3, gradients 1e-2
relative L2, as in test_gpu_surrogate: an FP32 sum on the other side of a BF16 rounding boundary
moves one element by 2^-8)."""
import numpy as np
import pytest

from helpers import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_in,width,depth,n_out,B", [(5, 16, 1, 1, 1), (5, 48, 2, 45, 64), (64, 32, 3, 33, 65),
                                                      (5, 256, 4, 45, 129), (1, 80, 9, 256, 300)])
def test_network_matches_oracle_at_tile_edges(fwt, n_in, width, depth, n_out, B):
    from fastweavturb_b200.surrogate import MLP
    from oracle import mlp_oracle as MO

    rng = np.random.default_rng(width + B)
    net = MLP(n_in=n_in, width=width, depth=depth, n_out=n_out, batch_max=300, seed=2)
    p = net.params().astype(np.float64)
    X = rng.uniform(-1, 1, (B, n_in)).astype(np.float32)
    T = rng.normal(0, 1, (B, n_out)).astype(np.float32)
    Y = net.forward(X)
    Yo, _, _ = MO.forward(p, net.widths, X)
    assert rel_l2(Y, Yo) <= 1e-3
    loss, gp, gx = net.loss_grad(X, T)
    lo, gpo, gxo = MO.loss_grad(p, net.widths, X, T)
    assert loss == pytest.approx(lo, rel=1e-3)
    assert rel_l2(gp, gpo) <= 1e-2
    assert rel_l2(gx, gxo) <= 1e-2
    # one step moves every parameter by lr times the sign of its gradient (Adam's first step)
    assert net.train_step(X, T, 1e-3) == pytest.approx(lo, rel=1e-3)
    move = net.params().astype(np.float64) - p
    big = np.abs(gp) > 1e-2 * np.abs(gp).max()
    assert np.allclose(move[big], -1e-3 * np.sign(gp[big]), rtol=1e-2)
    net.close()
