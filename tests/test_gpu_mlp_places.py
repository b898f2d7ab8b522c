"""The forward pass where the outputs' place in the exchange buffer follows inputs of 1, 2, 3 and 0
floats modulo four: outputs of a multiple of four columns leave 16 bytes a store, which have to start on
16 bytes.  Against the CPU oracle with the same BF16 rounding points (1e-3, as in test_gpu_surrogate);
the loss and its gradients read their targets from the same place."""
import numpy as np
import pytest

from helpers import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_in,n_out,B", [(3, 16, 1), (5, 48, 3), (7, 64, 65), (5, 64, 2), (1, 16, 2), (4, 16, 1),
                                          (3, 17, 5), (63, 256, 63), (1, 256, 1)])
def test_outputs_after_any_input_size(fwt, n_in, n_out, B):
    from fastweavturb_b200.surrogate import MLP
    from oracle import mlp_oracle as MO

    rng = np.random.default_rng(100 * n_in + B)
    net = MLP(n_in=n_in, width=64, depth=2, n_out=n_out, batch_max=65, seed=6)
    p = net.params().astype(np.float64)
    X = rng.uniform(-1, 1, (B, n_in)).astype(np.float32)
    T = rng.normal(0, 1, (B, n_out)).astype(np.float32)
    w = rng.uniform(0.5, 2.0, n_out).astype(np.float32)
    Y = net.forward(X)
    Yo, _, _ = MO.forward(p, net.widths, X)
    assert rel_l2(Y, Yo) <= 1e-3
    loss, gp, gx = net.loss_grad(X, T, w_out=w)
    lo, gpo, gxo = MO.loss_grad(p, net.widths, X, T, w_out=w)
    assert loss == pytest.approx(lo, rel=1e-3)
    assert rel_l2(gp, gpo) <= 1e-2
    assert rel_l2(gx, gxo) <= 1e-2
    net.close()


@pytest.mark.parametrize("B", [409, 410, 4096])
def test_outputs_on_both_sides_of_the_single_copy(fwt, B):
    """Outputs and inputs of up to 2^19 bytes come back in one copy, larger ones apart."""
    from fastweavturb_b200.surrogate import MLP
    from oracle import mlp_oracle as MO

    net = MLP(n_in=64, width=64, depth=1, n_out=256, batch_max=4096, seed=6)
    X = np.random.default_rng(B).uniform(-1, 1, (B, 64)).astype(np.float32)
    Yo, _, _ = MO.forward(net.params().astype(np.float64), net.widths, X)
    assert rel_l2(net.forward(X), Yo) <= 1e-3
    net.close()
