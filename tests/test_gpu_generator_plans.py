"""The generator's kept transform plans and their shared work area: one context asked for other shapes
call after call, levels in growing and falling order and more of them than plans are kept, gives the bits
that a fresh context gives for each call."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CALLS = [([4], [256]),
         ([2, 3, 5], [128, 256, 512]),
         ([7, 1], [1024, 64]),
         ([0, 3], [256, 128]),
         ([1 + k for k in range(20)], [2 ** (1 + k % 10) for k in range(20)]),   # 40 plans of 32 kept
         ([2, 3, 5], [128, 256, 512])]


def _generate(ctx, tubes, nodes):
    import torch

    n = int(np.dot(tubes, nodes))
    xyz = torch.zeros(3, n, dtype=torch.float64, device="cuda")
    ctx.fbb_generate(9, tubes, nodes, [0.4 + 0.02 * k for k in range(len(tubes))], [0.5] * len(tubes),
                     *(x.data_ptr() for x in xyz))
    return xyz.cpu().numpy()


def test_one_context_gives_what_fresh_ones_give(fwt):
    kept = fwt.Context(fwt.Params(N=32, N_downsample=32))
    for tubes, nodes in CALLS:
        a = _generate(kept, tubes, nodes)
        fresh = fwt.Context(fwt.Params(N=32, N_downsample=32))
        b = _generate(fresh, tubes, nodes)
        fresh.close()
        assert np.isfinite(a).all() and np.abs(a).max() > 0
        assert np.array_equal(a, b)
    kept.close()
