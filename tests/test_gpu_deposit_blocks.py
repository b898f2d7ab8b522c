"""The tile-owned FP32 deposition at the sizes where its tiles and stores can go wrong, against the
FP64 oracle on every grid point (FP32 path: 1e-5 relative L2, as in test_gpu_parity)."""
import numpy as np
import pytest

from helpers import gpu_params, oracle_inputs, rel_l2

pytestmark = pytest.mark.gpu

TOL32 = 1e-5


@pytest.mark.parametrize("N", [22, 42])
@pytest.mark.parametrize("piece_cells", [None, 0.0])
def test_rows_that_do_not_start_on_16_bytes(fwt, orc, N, piece_cells):
    """N a multiple of 2 but not of 4: the rows of omega start on 8 bytes, where a 16-byte store
    is not allowed; tubes thick enough for the tile kernels (sub-segments, and pieces at 0.2)."""
    from fastweavturb_b200.configs import small
    w = small(N=N, seed=3, nlev=2, tubes0=2, nodes0=64, sigma0=0.35)
    p, cl = oracle_inputs(orc, w)
    ctx = fwt.Context(gpu_params(fwt, w))
    ctx.set_centerlines(cl.npoint, cl.xyz, p.sigma, p.Gamma, p.n_T)
    if piece_cells is not None:
        ctx.set_piece_radius_limit(piece_cells)
    ctx.set_scatter_radius_limit(0.0)
    ctx.deposit(1, w.ntubes)
    vor = ctx.field(0).copy()
    ctx.close()
    ref, _ = orc.deposit(p, cl)
    assert np.abs(vor).max() > 0
    assert rel_l2(vor, ref) <= TOL32
