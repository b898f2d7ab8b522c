"""Thin FP32 tubes in a context whose memory cap leaves no room for the tile-free path's sums (32 bytes a
grid point): the lines go through the tiles, which need them only where a pair is handed to FP64."""
import numpy as np
import pytest

from helpers import rel_l2

pytestmark = pytest.mark.gpu

N = 64


def _deposit(fwt, p, cl, mem_cap, scatter_cells=None):
    ctx = fwt.Context(fwt.Params(N=N, N_downsample=N, line_s=1, line_e=len(cl.npoint), sigma_ratio=1.0,
                                 mem_cap=mem_cap))
    try:
        if scatter_cells is not None:
            ctx.set_scatter_radius_limit(scatter_cells)
        ctx.set_centerlines(cl.npoint, cl.xyz, p.sigma, p.Gamma, p.n_T)
        ctx.deposit(1, len(cl.npoint))
        return ctx.field(0).copy()
    finally:
        ctx.close()


def test_lines_without_room_for_the_sums_take_the_tiles(fwt, orc):
    # straight tubes of 6 grid spacings along x, their chords' planes 0.3 spacings off the grid points
    dx = 2 * np.pi / N
    x = (np.arange(32) * 2 + 0.3) * dx - np.pi
    lines = [np.stack([x, np.full(32, y), np.full(32, z)], axis=1) for y, z in ((0.41, -0.23), (-1.7, 1.37))]
    p = orc.Params(N=N, N_downsample=N, line_s=1, line_e=2, sigma_ratio=1.0, sigma=np.full(2, 2 * dx),
                   Gamma=np.array([1.0, -0.6]), n_T=np.ones(2, dtype=np.int32), if_filter=np.zeros(2, dtype=np.int32))
    cl = orc.Centerlines(npoint=np.array([32, 32], dtype=np.int64), xyz=np.concatenate(lines))
    for cap in range(4 << 20, 64 << 20, 1 << 20):   # the least memory that the tiles take
        try:
            tiles = _deposit(fwt, p, cl, cap, 0.0)
            break
        except fwt.FwtError as e:
            assert "memory cap" in str(e)
    field = _deposit(fwt, p, cl, cap)
    ref, _ = orc.deposit(p, cl)
    assert np.array_equal(field, tiles)
    assert rel_l2(field, ref) <= 1e-5          # FP32 path, as in test_gpu_parity
    assert rel_l2(_deposit(fwt, p, cl, 0), ref) <= 1e-5
