"""The FP64 operator's tensor-core M2L (digit products) and its near field against the oracle's FMM.

Orders 2 to 8 (8 digits up to 5, 9 at 6 and 7, the FP64-pipe contraction at 8), leaves of fewer and of
more points than a near-field CTA has threads, and the three forms of the pair update (kappa = 0,
screened, strongly screened).  Tolerance: both sides are FP64 sums of at most 4 p^3 = 2,048 terms a
translation over a handful of translations, so 2^-53 sqrt(2048) 10 ~ 5e-14 of the largest value,
times at most 4 for the cancellation of 1 - e^-t (1 + t) at the smallest t = kappa h: 2e-13."""

import numpy as np
import pytest

import ibim
import oracle as O

pytestmark = pytest.mark.gpu

H = 0.5


def sphere_points(n, seed):
    r = np.random.default_rng(seed)
    v = r.normal(size=(n, 3))
    v /= np.linalg.norm(v, axis=1)[:, None]
    return v * r.uniform(7.0, 8.0, (n, 1)) + 0.01, v, r.uniform(0.1, 1.0, n)


def compare(ctx, n, order, leaf, kappa, seed):
    p, nrm, w = sphere_points(n, seed)
    dens = np.random.default_rng(seed + 1).uniform(-1.0, 1.0, (4, n))
    plan = ctx.tube(p, nrm, w, H).plan(order, leaf, 10)
    out = plan.apply(ibim.KERNEL_BIE_FUSED, ibim.kernel_params(kappa, 80.0, 2.0, 1.0), dens)
    ref = O.Tree(p, p, leaf, 10).fmm(order, O.KParams(kappa, 80.0, 2.0, H), 16, dens)
    for o in range(4):
        assert np.abs(out[o] - ref[o]).max() < 2e-13 * np.abs(ref[o]).max(), o


@pytest.mark.parametrize("order", [2, 3, 4, 5, 6, 7, 8])
def test_orders(ctx, order):
    compare(ctx, 900 if order > 5 else 1500, order, 40, 0.4, order)


@pytest.mark.parametrize("kappa", [0.0, 0.5, 5.0])
@pytest.mark.parametrize("n,leaf", [(63, 64), (1100, 9), (1301, 257), (2600, 700)])
def test_leaf_sizes_and_screening(ctx, n, leaf, kappa):
    compare(ctx, n, 4, leaf, kappa, n)
