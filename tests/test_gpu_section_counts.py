"""Sub-segment counts on both sides of the section numbers at which the quadratures of 64 and of 256
intervals come in (4096 and 65536 slots of a batch, a line's sections and one more each)."""
import pytest

from helpers import gpu_params, oracle_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tubes,nodes", [(16, 255), (16, 256), (256, 255), (257, 255), (300, 300)])
@pytest.mark.parametrize("H", [0.3, 0.8])
def test_counts_of_a_batch(fwt, orc, tubes, nodes, H):
    """The number of sub-segments, an integer, equals the oracle's FP64 sums over 1001 samples."""
    from fastweavturb_b200.configs import Level, Workload

    w = Workload("sections", 32, [Level(tubes=tubes, nodes=nodes, sigma=0.02, Gamma=1.0, H=H, dB=0.5)], seed=tubes)
    p, cl = oracle_inputs(orc, w)
    want = sum(int(orc.line_ntf(cl.line(i))[0][:-1].sum()) for i in range(tubes))
    ctx = fwt.Context(gpu_params(fwt, w))
    ctx.set_centerlines(cl.npoint, cl.xyz, p.sigma, p.Gamma, p.n_T)
    ctx.deposit(1, tubes)
    assert ctx.counters()["subsegments"] == want
    ctx.close()
