"""Thin tubes deposited piece by piece (without tiles) against the same pieces searched tile by
tile: both apply the same test and arithmetic to every point, so the counts are identical and
the fields agree to the rounding of the tile path's second FP32 addition (pairs redone in FP64
are added apart).  Lines whose chords meet every case of the row geometry: along an axis (planes
parallel to two families of rows), along face and space diagonals, long straight chords, tight
turns, and lines that cross the periodic boundary."""

import numpy as np
import pytest

from helpers import gpu_params, rel_l2

pytestmark = pytest.mark.gpu


def _lines():
    s = np.linspace(-np.pi, np.pi, 48, endpoint=False)
    out = []
    for d in ([1, 0, 0], [0, 1, 0], [0, 0, 1], [1, 1, 0], [0, -1, 1], [1, 1, 1], [-1, 2, 1]):
        p = np.outer(d, s) + np.array([[0.3], [-1.1], [2.9]])
        out.append(p)
    for r, n in ((0.25, 40), (1.3, 24)):   # circles: tight turns, and few long chords
        a = np.linspace(0, 2 * np.pi, n, endpoint=False)
        out.append(np.stack([3.0 + r * np.cos(a), r * np.sin(a), 0.4 * r * np.sin(2 * a)]))
    return [(((p + np.pi) % (2 * np.pi)) - np.pi).T for p in out]   # (nodes, 3)


@pytest.mark.parametrize("cells", [0.55, 1.0, 1.9, 3.9, 5.0, 7.9])
@pytest.mark.parametrize("ratio,eta", [(1.0, 0.0), (2.0, 0.3)])
def test_scattered_pieces_equal_searched_pieces(fwt, cells, ratio, eta):
    from fastweavturb_b200.configs import small

    N = 64
    w = small(N=N, seed=1, nlev=1, tubes0=1, nodes0=64)
    lines = _lines()
    xyz = np.concatenate(lines)
    npoint = np.array([p.shape[0] for p in lines], dtype=np.int32)
    n = len(lines)
    sigma = np.full(n, cells * 2 * np.pi / N / 3 / ratio)   # the largest truncation radius is `cells`
    res = {}
    for scatter in (8.0, 0.0):
        ctx = fwt.Context(gpu_params(fwt, w, line_e=n, sigma_ratio=ratio, eta_t=eta))
        ctx.set_centerlines(npoint, xyz, sigma, np.ones(n), np.ones(n, dtype=np.int32))
        ctx.set_piece_radius_limit(8.0)
        ctx.set_scatter_radius_limit(scatter)
        ctx.deposit(1, n)
        k = ctx.counters()
        res[scatter] = ctx.field(0).copy(), k["accepted"], k["redone_fp64"], k["pairs"]
        ctx.close()
    assert res[8.0][3] == 0 < res[0.0][3]
    assert res[8.0][1] > 0
    assert res[8.0][1:3] == res[0.0][1:3]
    assert rel_l2(res[8.0][0], res[0.0][0]) <= 1e-6
