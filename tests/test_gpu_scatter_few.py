"""The tile-free path with fewer pieces than warps, about as many, and enough for whole chunks: a chunk
holds one to four pieces by their number.  Against the same lines through the tiles (the same tests and
arithmetic: 2e-6 relative L2), and without a twist against the FP64 oracle (1e-5, as in test_gpu_parity).
With one, these rough lines have points beyond sharp bends where the reference extrapolates a section's
quintic by a thousand times its length; no FP32 path follows it there."""
import numpy as np
import pytest

from helpers import gpu_params, oracle_inputs, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tubes,nodes", [(1, 16), (1, 128), (3, 1024), (9, 1024), (12, 1024)])
@pytest.mark.parametrize("sigma_ratio,eta", [(1.0, 0.0), (2.0, 0.4)])
def test_few_pieces(fwt, orc, tubes, nodes, sigma_ratio, eta):
    from fastweavturb_b200.configs import Level, Workload
    N = 64
    cells = 6.0 if nodes < 1024 else 2.5
    sigma = cells * 2 * np.pi / N / 3 / sigma_ratio
    w = Workload("few", N, [Level(tubes=tubes, nodes=nodes, sigma=sigma, Gamma=1.0, H=0.7, dB=0.5)], seed=nodes,
                 sigma_ratio=sigma_ratio, eta_t=eta)
    p, cl = oracle_inputs(orc, w)
    ref, _ = orc.deposit(p, cl)
    fields = []
    for limit in (None, 0.0):
        ctx = fwt.Context(gpu_params(fwt, w))
        if limit is not None:
            ctx.set_scatter_radius_limit(limit)
        ctx.set_centerlines(cl.npoint, cl.xyz, p.sigma, p.Gamma, p.n_T)
        ctx.deposit(1, tubes)
        fields.append(ctx.field(0).copy())
        ctx.close()
    assert np.abs(ref).max() > 0
    assert eta != 0.0 or rel_l2(fields[0], ref) <= 1e-5
    assert rel_l2(fields[0], fields[1]) <= 2e-6
