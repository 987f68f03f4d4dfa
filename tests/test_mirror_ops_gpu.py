"""Operators evaluated once a class of mirror images against the oracle's FMM: a cloud in a box of three different
edge lengths, lopsided so that some classes have all eight members and some one.  Order 8 takes the FP64
contraction of the operators themselves, the others their images.
Tolerance: that of the FP64 operator's other comparisons with the oracle, 2e-13 of the largest value."""

import numpy as np
import pytest

import ibim
import oracle as O

pytestmark = pytest.mark.gpu

H = 0.5


@pytest.mark.parametrize("order", [2, 5, 6, 8])
@pytest.mark.parametrize("kappa", [0.0, 0.3])
def test_lopsided_cloud(ctx, order, kappa):
    n = 900
    r = np.random.default_rng(order)
    p = r.uniform(-1.0, 1.0, (n, 3)) ** 3 * [9.0, 6.0, 4.0] + np.abs(r.normal(size=(n, 3))) * [1.0, 3.0, 0.5]
    nrm = r.normal(size=(n, 3))
    nrm /= np.linalg.norm(nrm, axis=1)[:, None]
    dens = r.uniform(-1.0, 1.0, (4, n))
    plan = ctx.tube(p, nrm, np.ones(n), H).plan(order, 20, 10)
    out = plan.apply(ibim.KERNEL_BIE_FUSED, ibim.kernel_params(kappa, 80.0, 2.0, 1.0), dens)
    ref = O.Tree(p, p, 20, 10).fmm(order, O.KParams(kappa, 80.0, 2.0, H), 16, dens)
    for o in range(4):
        assert np.abs(out[o] - ref[o]).max() < 2e-13 * np.abs(ref[o]).max(), o
