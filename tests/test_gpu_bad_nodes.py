"""Centerlines whose turning angle is not a number are refused with the library's error, before any record
is built from a count, and leave the context usable."""
import numpy as np
import pytest

from helpers import gpu_params, oracle_inputs, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,mode", [(32, 0), (32, 1), (64, 0), (64, 1)])
@pytest.mark.parametrize("tubes", [1, 20])
@pytest.mark.parametrize("what", ["coincident", "all coincident", "nan", "inf"])
def test_lines_without_a_turning_angle(fwt, orc, precision, mode, tubes, what):
    from fastweavturb_b200.configs import Level, Workload

    # one line goes to the full sum at once, twenty of 256 nodes through the quadrature of 64 intervals
    w = Workload("bad", 32, [Level(tubes=tubes, nodes=256, sigma=0.15, Gamma=1.0, H=0.7, dB=0.5)], seed=3)
    p, cl = oracle_inputs(orc, w)
    xyz = cl.xyz.copy()
    if what == "coincident":
        xyz[101] = xyz[100]
    elif what == "all coincident":
        xyz[:256] = xyz[0]
    else:
        xyz[100, 1] = np.nan if what == "nan" else np.inf
    ctx = fwt.Context(gpu_params(fwt, w, precision=precision, deposit_mode=mode))
    ctx.set_centerlines(cl.npoint, xyz, p.sigma, p.Gamma, p.n_T)
    if what == "coincident":
        # the section's length is zero or, by the order of the arc length's sums, a rounding of it: refused
        # or built
        try:
            ctx.deposit(1, tubes)
        except fwt.FwtError as e:
            assert "cannot be sub-divided" in str(e) or "outside" in str(e) or "box" in str(e)
    else:
        with pytest.raises(fwt.FwtError, match="cannot be sub-divided"):
            ctx.deposit(1, tubes)
    ctx.set_centerlines(cl.npoint, cl.xyz, p.sigma, p.Gamma, p.n_T)
    ctx.deposit(1, tubes)
    ref, _ = orc.deposit(p, cl)
    assert rel_l2(ctx.field(0), ref) <= 1e-5
    ctx.close()
