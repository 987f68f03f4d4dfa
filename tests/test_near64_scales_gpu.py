"""The FP64 near field over the range of its arguments: clouds of one leaf from 1e-6 to 1e12 in size (odd and even
binary exponents of the distances), screened from not at all to e^-t of 2^-900, against the oracle.
Tolerance: sums of 300 pairs, each within 8 roundings of 2^-53 and the exponential's t 2^-53 at most 600 2^-53 where
e^-t itself counts; 1e-13 of the largest value, times at most 8 for the cancellation of 1 - e^-t (1 + t) at t = 0.1."""

import numpy as np
import pytest

import ibim
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1e-6, 1.4e-3, 1.0, 2.9e5, 1e12])
@pytest.mark.parametrize("screen", [0.0, 0.2, 3.0, 60.0])
def test_scales(ctx, scale, screen):
    n, h = 300, 0.5 * scale
    r = np.random.default_rng(7)
    p = r.uniform(-5.0, 5.0, (n, 3)) * scale
    nrm = r.normal(size=(n, 3))
    nrm /= np.linalg.norm(nrm, axis=1)[:, None]
    dens = r.uniform(-1.0, 1.0, (4, n))
    dens[3] /= scale  # gradients and potentials of one size
    kappa = screen / scale
    out = ctx.tube(p, nrm, np.ones(n), h).plan(2, 400, 10).apply(
        ibim.KERNEL_BIE_FUSED, ibim.kernel_params(kappa, 80.0, 2.0, 1.0), dens)
    ref = O.Tree(p, p, 400, 10).fmm(2, O.KParams(kappa, 80.0, 2.0, h), 16, dens)
    for o in range(4):
        assert np.abs(out[o] - ref[o]).max() < 8e-13 * np.abs(ref[o]).max(), o
