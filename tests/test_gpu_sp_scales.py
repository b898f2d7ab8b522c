"""S_p of fields and scales far from one: what is summed is (du s)^p, whose size says nothing about that of
du^p or s^p alone.  Tolerance: the sums hold 3 N^3 FP64 terms in some order, below 1e-11 of the natural
size (as in test_gpu_stats_shapes)."""
import numpy as np
import pytest

from helpers import gpu_params, oracle_inputs, sp_close

pytestmark = pytest.mark.gpu


def _sp(fwt, orc, strength, r):
    from fastweavturb_b200.configs import small
    w = small(N=24, seed=13, nlev=2, tubes0=2, nodes0=64, sigma0=0.4)
    p, cl = oracle_inputs(orc, w)
    ctx = fwt.Context(gpu_params(fwt, w, precision=64))
    ctx.set_centerlines(cl.npoint, cl.xyz, p.sigma, p.Gamma * strength, p.n_T)
    ctx.deposit(1, w.ntubes)
    ctx.biot_savart()
    ctx.cal_helicity()
    _, Sp = ctx.Sp_calculate(pmax=10, r=r)
    ctx.close()
    return Sp


@pytest.mark.parametrize("exponent", [-130, -101, 101, 130])
def test_normalised_moments_do_not_depend_on_the_circulation(fwt, orc, exponent):
    """A circulation scaled by a power of two scales every FP64 velocity by it, and S_p of u / u' not at
    all."""
    r = np.array([1, 2, 5, 11], dtype=np.int32)
    a, b = _sp(fwt, orc, 2.0 ** exponent, r), _sp(fwt, orc, 1.0, r)
    for q in range(10):
        sp_close(a, b, q, 1e-11)


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("size,scale", [(2.0 ** -100, 2.0 ** 101), (1e10, 1e28), (1e-20, 1e-25), (3.0, -0.7),
                                        (2.0, 0.0), (1.0, 1.3)])
def test_sums_of_a_block_at_any_scale(fwt, precision, size, scale):
    """fwt_sp_block takes the caller's scale: the increments are exact in FP64 and multiplied by it."""
    import torch

    N, ny, nz = 20, 6, 3
    ctx = fwt.Context(fwt.Params(N=N, N_downsample=N, precision=precision))
    dt = torch.float32 if precision == 32 else torch.float64
    g = torch.Generator(device="cuda").manual_seed(3)
    u = (torch.randn(nz, ny, N, device="cuda", generator=g, dtype=torch.float64) * size).to(dt)
    r = np.array([1, 7, 20], dtype=np.int32)
    got = ctx.sp_block(u.data_ptr(), N, ny, nz, 0, scale, r)
    x = u.double().cpu().numpy()
    for m, q in enumerate(r):
        du = (np.roll(x, -int(q), axis=2) - x) * scale
        for p in range(10):
            want, mag = (du ** (p + 1)).sum(), (np.abs(du) ** (p + 1)).sum()
            if np.isfinite(mag) and mag > 1e-290:
                assert abs(got[p, m] - want) <= 1e-11 * mag
            elif mag == 0.0:
                assert got[p, m] == 0.0
    ctx.close()
