"""FP64 deposition where a tile's records are cut into parts (small grids) and where they are not,
with and without a varying core: one call and two calls over the same lines, and the FP64
oracle within the suite's FP64 rule (four times the algorithm's own rounding floor on the workload:
a varying core's curvature term amplifies rounding)."""

import numpy as np
import pytest

from helpers import fp64_floor, gpu_params, oracle_inputs, rel_l2, tol64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [20, 64, 132])   # 18 and 256 tiles (8 parts), 2601 (1); ragged tiles
@pytest.mark.parametrize("ratio,eta", [(1.0, 0.0), (3.0, 0.0), (1.0, 0.4)])
def test_fp64_parts(fwt, orc, N, ratio, eta):
    from fastweavturb_b200.configs import small

    w = small(N=N, seed=9, nlev=2, tubes0=2, nodes0=64, sigma0=0.3 / ratio)
    w.sigma_ratio, w.eta_t = ratio, eta
    p, cl = oracle_inputs(orc, w)
    out = []
    for ranges in ([(1, w.ntubes)], [(1, 3), (4, w.ntubes)]):
        ctx = fwt.Context(gpu_params(fwt, w, precision=64))
        ctx.set_centerlines(cl.npoint, cl.xyz, p.sigma, p.Gamma, p.n_T)
        for s, e in ranges:
            ctx.deposit(s, e)
        out.append(ctx.field(0).copy())
        ctx.close()
    # the same contributions in another order: 64-bit rounding of at most a few hundred terms a point
    assert rel_l2(out[0], out[1]) <= 1e-13
    vor, _ = orc.deposit(p, cl)
    assert rel_l2(out[0], vor) <= tol64(fp64_floor(orc, p, cl)[0])
    assert np.abs(vor).max() > 0
