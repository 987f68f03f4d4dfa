"""The FP64 stages' reciprocals and square roots (seeds assembled from FP32 and integer parts) on signed-distance grids
of cells from 2^-20 to 2^20 in size, so over some 300 powers of two of the indicators, odd and even.
Tolerance against the oracle: that of the stages' other comparison, 1e-12 of the largest value."""

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("exp", [-20, -9, -3, 0, 1, 6, 13, 20])
def test_stages_scale(ctx, exp):
    n, h = (19, 24, 33), 0.37 * 2.0**exp
    x = np.stack(np.meshgrid(*[h * np.arange(k) for k in n], indexing="ij"), -1)
    g = 7.0 * h - np.linalg.norm(x - 0.5 * h * (np.array(n) - 1) - 0.1 * h, axis=-1)
    ref = g.copy()
    O.evolve(ref, h, 2.0 * h)
    G = ctx.grid(n, (0.0, 0.0, 0.0), h)
    G.upload(g)
    G.evolve(2.0 * h)
    assert np.abs(G.download() - ref).max() <= 1e-12 * np.abs(ref).max()
