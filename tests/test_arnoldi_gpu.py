"""GMRES with the one-launch Arnoldi step against the oracle's GMRES: vectors of fewer values than a block,
around the sizes where the registers per thread change, and beyond them (separate launches).  The sums are
FP64 in another order than the oracle's: solutions agree to 2^-53 times the condition number (below 100
here) times the square root of the length, at most 1e-10."""

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

BLOCK = 512 * 256


@pytest.mark.parametrize("n", [1, 7, 255, 1000, 2 * BLOCK, 2 * BLOCK + 1, 8 * BLOCK + 3, 16 * BLOCK, 16 * BLOCK + 5])
def test_gmres_matches_oracle(ctx, n):
    r = np.random.default_rng(n)
    d = 1.0 + 0.5 * r.random(n)
    b = r.uniform(-1.0, 1.0, n)

    def apply(x):
        return d * x + 0.2 * np.roll(x, 1)

    m = 5 if n > 7 else min(n, 5)
    x, info = ctx.gmres(apply, b, restart=m, maxiter=30, tol=1e-8)
    ref, rc, iters, mv = O.gmres(apply, b, m=m, max_iter=30, tol=1e-8)
    assert info["status"] == rc and info["iters"] == iters
    assert np.abs(x - ref).max() <= 1e-10 * np.abs(ref).max()
