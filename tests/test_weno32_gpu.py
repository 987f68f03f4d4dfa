"""The FP32 level-set stages (two cells a thread) on grids of odd and even sizes, one and many cells past a
block: the interface of the FP32 grid against the FP64 one.  Tolerance: some 60 steps of FP32 roundings
(2^-24) of interface values below 8 A, without cancellation 3e-5."""

import numpy as np
import pytest

import ibim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(40, 41, 63), (41, 40, 64), (39, 45, 65), (44, 43, 34)])
def test_fp32_matches_fp64_at_the_interface(ctx, n):
    h = 0.4
    r = np.random.default_rng(sum(n))
    lo = [-h * (k - 1) / 2 for k in n]
    centers, radii = r.uniform(-1.0, 1.0, (4, 3)), r.uniform(1.0, 1.5, 4)
    grids = []
    for prec in (ibim.PRECISION_FP64, ibim.PRECISION_MIXED):
        cfg = ibim.default_config(lo=lo, h=h, n=n, band=4, init=-2.0 * max(n), probe=0.8, reinit_t=19.5 * 0.5 * h,
                                  thickness=2, precision=prec)
        g, steps = ctx.levelset(centers, radii, cfg)
        grids.append((g.download(), list(steps)))
    (a, sa), (b, sb) = grids
    assert sa == sb
    near = np.abs(a) < 2 * h
    assert near.sum() > 500
    assert np.abs(a - b)[near].max() < 3e-5
