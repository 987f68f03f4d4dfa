"""The FP32 translations of every order against the FP64 operator, over leaves of fewer and of more points than a
warp has lanes, a single leaf, and repeated products (the upward pass resets its own counters).
Tolerance: FP32 sums of at most 4 p^3 = 2,048 terms a translation leave sqrt(2048) 2^-24 of the largest value,
over a handful of translations 1e-5."""

import numpy as np
import pytest

import ibim

pytestmark = pytest.mark.gpu

H = 0.5


@pytest.mark.parametrize("order,n,leaf", [(2, 1500, 10), (3, 900, 33), (4, 60, 64), (4, 4000, 5), (5, 2500, 200),
                                          (6, 1500, 31), (7, 1200, 64), (8, 1000, 40)])
def test_mixed_matches_fp64(ctx, order, n, leaf):
    r = np.random.default_rng(order + n)
    v = r.normal(size=(n, 3))
    v /= np.linalg.norm(v, axis=1)[:, None]
    tube = ctx.tube(v * r.uniform(7.0, 8.0, (n, 1)), v, r.uniform(0.1, 1.0, n), H)
    kp = ibim.kernel_params(0.2, 80.0, 2.0, 1.0)
    dens = r.uniform(-1.0, 1.0, (4, n))
    p64, p32 = tube.plan(order, leaf, 10), tube.plan(order, leaf, 10, precision=ibim.PRECISION_MIXED)
    ref = p64.apply(ibim.KERNEL_BIE_FUSED, kp, dens)
    for _ in range(3):
        out = p32.apply(ibim.KERNEL_BIE_FUSED, kp, dens)
        again = p64.apply(ibim.KERNEL_BIE_FUSED, kp, dens)
        for o in range(4):
            top = np.abs(ref[o]).max()
            assert np.abs(out[o] - ref[o]).max() < 1e-5 * top, o
            assert np.abs(again[o] - ref[o]).max() < 4e-13 * top, o
