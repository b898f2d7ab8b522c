"""Sub-segment counts of the sections where the quadratures of the turning angle hand over to each
other: presample counts on both sides of the line (512) from which the coarse sums are used, and
curves from smooth to rough."""

import pytest

from helpers import gpu_params, oracle_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ntf_pre", [100, 511, 512, 1000, 3001])
@pytest.mark.parametrize("H", [0.25, 0.85])
@pytest.mark.parametrize("ntf_times", [7, 50])
def test_sub_segment_counts(fwt, orc, ntf_pre, H, ntf_times):
    """The number of sub-segments, an integer, equals the oracle's FP64 sum over ntf_pre + 1
    samples, line by line (each line is deposited alone)."""
    from fastweavturb_b200.configs import Level, Workload

    lv = [Level(tubes=3, nodes=200, sigma=0.1, Gamma=1.0, H=H, dB=0.8),
          Level(tubes=3, nodes=77, sigma=0.05, Gamma=0.5, H=H, dB=0.2)]
    w = Workload("sections", 32, lv, seed=5)
    p, cl = oracle_inputs(orc, w)
    gp = gpu_params(fwt, w)
    gp.ntf_pre, gp.ntf_times = ntf_pre, ntf_times
    ctx = fwt.Context(gp)
    ctx.set_centerlines(cl.npoint, cl.xyz, p.sigma, p.Gamma, p.n_T)
    for i in range(len(cl.npoint)):
        want = int(orc.line_ntf(cl.line(i), ntf_times, ntf_pre)[0][:-1].sum())
        ctx.deposit(i + 1, i + 1)
        assert ctx.counters()["subsegments"] == want
    ctx.close()
