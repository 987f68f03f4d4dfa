"""The mixed path's CTA-pair M2L and packed FP32 near field against the FP64 operator on the same plan shape.

Orders 4 to 7 (an even and an odd number of row tiles, a last stage of K that ends early), operators with
one pair and with several chunks, leaves below, at and above a warp's 32 targets, sources that are no
multiple of four, kappa = 0.  Tolerance: FP32 sums of up to 4 p^3 products of 22-bit operands and of
a few thousand pairs, 2^-22 sqrt(4000) ~ 1.5e-5 of the largest value at worst."""

import numpy as np
import pytest

import ibim
from test_fp64_digits_gpu import H, sphere_points

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kappa", [0.0, 0.3])
@pytest.mark.parametrize("n,order,leaf", [(61, 4, 64), (700, 4, 20), (3001, 4, 33), (6000, 5, 32), (1500, 5, 150),
                                          (2500, 6, 40), (900, 7, 31)])
def test_mixed_matches_fp64(ctx, n, order, leaf, kappa):
    p, nrm, w = sphere_points(n, n + order)
    dens = np.random.default_rng(n).uniform(-1.0, 1.0, (4, n))
    t = ctx.tube(p, nrm, w, H)
    kp = ibim.kernel_params(kappa, 80.0, 2.0, 1.0)
    a = t.plan(order, leaf, 10).apply(ibim.KERNEL_BIE_FUSED, kp, dens)
    b = t.plan(order, leaf, 10, precision=ibim.PRECISION_MIXED).apply(ibim.KERNEL_BIE_FUSED, kp, dens)
    for o in range(4):
        assert np.abs(a[o] - b[o]).max() < 1.5e-5 * np.abs(a[o]).max(), o
