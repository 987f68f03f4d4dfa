"""A NaN or an infinity in the input of an FP64 product reaches every target that the direct sum carries it to: all
beyond the cutoff tau h of its source (inside it K2 alone remains).  Kernels that are zero without screening carry it
as well, 0 NaN being NaN.  Clouds of several levels, so that most targets see the source through the far field; digit
products at orders up to 7, the FP64 pipe's contraction at 8.  The product after it, of finite densities, is finite."""

import numpy as np
import pytest

import ibim
from test_fp64_digits_gpu import H, sphere_points

pytestmark = pytest.mark.gpu


def cloud(ctx, n, order, leaf, **kw):
    p, nrm, w = sphere_points(n, order)
    plan = ctx.tube(p, nrm, w, H).plan(order, leaf, 10, **kw)
    bad = n // 3
    outside = np.linalg.norm(p - p[bad], axis=1) >= 1.01 * H
    assert outside.sum() > 0.9 * n
    return plan, bad, outside


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("kappa", [0.0, 0.4])
@pytest.mark.parametrize("order,precision", [(3, ibim.PRECISION_FP64), (5, ibim.PRECISION_FP64), (6, ibim.PRECISION_FP64),
                                             (8, ibim.PRECISION_FP64), (5, ibim.PRECISION_MIXED)])
def test_block(ctx, order, precision, kappa, value):
    n = 1500
    plan, bad, outside = cloud(ctx, n, order, 40, precision=precision)
    kp = ibim.kernel_params(kappa, 80.0, 2.0, 1.0)
    for slot in (0, 2, 3):
        dens = np.random.default_rng(1).uniform(-1.0, 1.0, (4, n))
        assert np.isfinite(plan.apply(ibim.KERNEL_BIE_FUSED, kp, dens)).all()
        dens[slot, bad] = value
        out = plan.apply(ibim.KERNEL_BIE_FUSED, kp, dens)
        for o in range(4):
            assert not np.isfinite(out[o, outside]).any(), (slot, o)
    assert np.isfinite(plan.apply(ibim.KERNEL_BIE_FUSED, kp, np.ones((4, n)))).all()


@pytest.mark.parametrize("kappa", [0.0, 0.4])
@pytest.mark.parametrize("order", [4, 7])
def test_matvec_and_scalar_kernels(ctx, order, kappa):
    n = 1200
    plan, bad, outside = cloud(ctx, n, order, 30)
    kp = ibim.kernel_params(kappa, 80.0, 2.0, 1.0)
    for value in (np.nan, np.inf):
        for half in (0, 1):
            x = np.random.default_rng(2).uniform(-1.0, 1.0, 2 * n)
            x[half * n + bad] = value
            y = plan.matvec(kp, x)
            assert not np.isfinite(y.reshape(2, n)[:, outside]).any(), half
        for i, name in enumerate(ibim.KERNELS):
            m = np.random.default_rng(3).uniform(-1.0, 1.0, n)
            m[bad] = value
            assert not np.isfinite(plan.apply(i, kp, m)[outside]).any(), name
