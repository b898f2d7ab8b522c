"""S_p and the PDFs at the shapes where their kernels' splits change, against plain FP64 sums and a
literal first-match histogram of the context's own fields.

Tolerances: S_p sums n = 3 N^3 FP64 terms of each order in some order: the difference between two
orders of summation is below n 2^-53 of the sum of magnitudes, < 1e-11 (max S_2)^(p/2)-sized here;
histogram counts are integers of the same REAL(4) comparisons: equal."""
import numpy as np
import pytest

from helpers import gpu_params, oracle_inputs, sp_close

pytestmark = pytest.mark.gpu


def _ctx(fwt, orc, N, precision):
    from fastweavturb_b200.configs import small
    w = small(N=N, seed=13, nlev=2, tubes0=2, nodes0=64, sigma0=0.4)
    p, cl = oracle_inputs(orc, w)
    ctx = fwt.Context(gpu_params(fwt, w, precision=precision))
    ctx.set_centerlines(cl.npoint, cl.xyz, p.sigma, p.Gamma, p.n_T)
    ctx.deposit(1, w.ntubes)
    ctx.biot_savart()
    ctx.cal_helicity()
    return ctx


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("N,pmax,nr", [(8, 1, 1), (22, 4, 5), (36, 6, 33), (40, 10, 64), (64, 3, 24)])
def test_structure_functions_of_any_shape(fwt, orc, N, precision, pmax, nr):
    """Lines shorter than a warp, lines that are no multiple of it, orders between the kernel's
    variants, one separation, 64 (two grids of groups), separations of zero, of N and beyond, and
    repeated ones."""
    ctx = _ctx(fwt, orc, N, precision)
    r = np.array([(3 * k) % (2 * N + 3) for k in range(nr)], dtype=np.int32)
    _, Sp = ctx.Sp_calculate(pmax=pmax, r=r)
    up = ctx.cal_helicity()["up"]
    u = ctx.field_tensor(1).double().cpu().numpy() / up          # [c, z, y, x]
    ref = np.zeros((max(pmax, 2), nr))
    for m, q in enumerate(r):
        for d in range(3):
            du = np.roll(u[d], -int(q), axis=2 - d) - u[d]
            for p in range(ref.shape[0]):
                ref[p, m] += (du ** (p + 1)).sum()
    ref /= 3.0 * N ** 3
    for p in range(pmax):
        sp_close(Sp, ref, p, 1e-11) if pmax > 1 else np.testing.assert_allclose(Sp[0], ref[0], rtol=0, atol=1e-12)
    ctx.close()


@pytest.mark.parametrize("nbins", [1, 2, 160, 161, 2000, 8192])
@pytest.mark.parametrize("which,component", [(0, -1), (1, 1)])
def test_histograms_of_any_bin_count(fwt, orc, nbins, which, component):
    """Bin counts around the limits of the interleaved copies (32 up to 157 bins, fewer beyond)."""
    ctx = _ctx(fwt, orc, 36, 32)
    val, _, cnt = ctx.export_pdf(which, component, nbins=nbins)
    up = ctx.cal_helicity()["up"]
    f = ctx.field_tensor(0 if which else 1).cpu().numpy()
    v = (f.astype(np.float64) * (1.0 / up)).astype(np.float32)
    v = (v if component < 0 else v[component]).ravel()
    bsz = np.float32(np.float32(v.max() - v.min()) / np.float32(nbins))
    half = np.float32(np.float32(0.5) * bsz)
    lo, hi = (val - half).astype(np.float32), (val + half).astype(np.float32)
    at = np.searchsorted(hi, v, side="right")                    # first bin with v < hi
    inside = at < nbins
    inside[inside] &= lo[at[inside]] <= v[inside]
    assert np.array_equal(cnt.astype(np.int64), np.bincount(at[inside], minlength=nbins))
    ctx.close()
