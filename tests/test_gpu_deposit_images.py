"""Thick FP32 tubes of a constant core (the tile-owned block kernel) on both sides of the periodic
boundary, against the FP64 oracle on every grid point (1e-5 relative L2, as in test_gpu_parity), and the
same bits in every repetition (integer sums do not depend on the order, so an image code or a record
read before it was written would show)."""
import numpy as np
import pytest

from helpers import rel_l2

pytestmark = pytest.mark.gpu

TOL32 = 1e-5


def closed_curve(rng, centre, nodes, modes, size):
    """A closed curve of `modes` Fourier modes about `centre`, wrapped into [-pi, pi)."""
    t = np.arange(nodes) / nodes * 2 * np.pi
    x = np.zeros((nodes, 3))
    for m in range(1, modes + 1):
        a, b = rng.normal(size=3), rng.normal(size=3)
        x += size / m ** 2 * (np.outer(np.cos(m * t), a) + np.outer(np.sin(m * t), b))
    return np.mod(x + centre + np.pi, 2 * np.pi) - np.pi


def deposit(fwt, p, cl, N, ntf_times, repeat=1):
    fields = []
    ctx = fwt.Context(fwt.Params(N=N, N_downsample=N, line_s=1, line_e=len(cl.npoint), sigma_ratio=1.0,
                                 ntf_times=ntf_times))
    ctx.set_piece_radius_limit(0.0)
    for _ in range(repeat):
        ctx.set_centerlines(cl.npoint, cl.xyz, p.sigma, p.Gamma, p.n_T)   # clears the field
        ctx.deposit(1, len(cl.npoint))
        fields.append(ctx.field(0).copy())
    ctx.close()
    return fields


def lines(orc, N, curves, sigma, ntf_times):
    n = len(curves)
    p = orc.Params(N=N, N_downsample=N, line_s=1, line_e=n, sigma_ratio=1.0, ntf_times=ntf_times,
                   sigma=np.full(n, sigma), Gamma=np.linspace(1.0, -0.7, n), n_T=np.ones(n, dtype=np.int32),
                   if_filter=np.zeros(n, dtype=np.int32))
    return p, orc.Centerlines(npoint=np.array([len(c) for c in curves], dtype=np.int64), xyz=np.concatenate(curves))


@pytest.mark.parametrize("N,sigma", [(32, 0.3), (48, 0.1)])
def test_images_across_every_face(fwt, orc, N, sigma):
    """Tubes about the corner, the edges, the faces and the middle of the periodic box."""
    rng = np.random.default_rng(N)
    centres = [(np.pi, np.pi, np.pi), (np.pi, np.pi, 0.3), (-np.pi, 0.2, 0.1), (0.0, 0.1, -np.pi), (0.2, -0.1, 0.3)]
    p, cl = lines(orc, N, [closed_curve(rng, c, 40, 3, 0.8) for c in centres], sigma, 50)
    fields = deposit(fwt, p, cl, N, 50, repeat=4)
    ref, _ = orc.deposit(p, cl)
    assert rel_l2(fields[0], ref) <= TOL32
    for f in fields[1:]:
        assert np.array_equal(f, fields[0])


@pytest.mark.parametrize("ntf_times", [3, 5, 6, 7, 8, 10, 50])
@pytest.mark.parametrize("sigma", [0.2, 0.35, 0.6])
@pytest.mark.parametrize("path", ["blocks", "piece tiles", "pieces without tiles"])
def test_records_on_both_sides_of_the_short_wrap_rule(fwt, orc, ntf_times, sigma, path):
    """Records take the short path (no periodic bookkeeping) where the bend of consecutive chords is below
    41 degrees, the spline's distance from its start keeps clear of a second wrap, and x - c stays below
    half a period.  Few sub-segments a turn give bends from 7 to 60 degrees; tubes of up to 1.8 in radius
    on curves along the faces reach all three limits.  A point that was wrapped wrongly is off by its whole
    value: one of at most 1e5 values of a size moves the relative L2 distance by more than 3e-3, so 1e-4
    against the FP64 oracle."""
    N = 32
    rng = np.random.default_rng(ntf_times)
    centres = [(np.pi, 0.4, -1.0), (0.3, -np.pi, np.pi), (np.pi - 0.5, np.pi + 0.4, 0.2), (0.1, 0.2, 0.3)]
    p, cl = lines(orc, N, [closed_curve(rng, c, 7 + 4 * i, 2, 0.7) for i, c in enumerate(centres)], sigma, ntf_times)
    ctx = fwt.Context(fwt.Params(N=N, N_downsample=N, line_s=1, line_e=len(centres), sigma_ratio=1.0,
                                 ntf_times=ntf_times))
    ctx.set_piece_radius_limit(0.0 if path == "blocks" else 100.0)
    ctx.set_scatter_radius_limit(100.0 if path == "pieces without tiles" else 0.0)
    ctx.set_centerlines(cl.npoint, cl.xyz, p.sigma, p.Gamma, p.n_T)
    ctx.deposit(1, len(centres))
    field = ctx.field(0)
    ctx.close()
    ref, _ = orc.deposit(p, cl)
    assert rel_l2(field, ref) <= 1e-4
