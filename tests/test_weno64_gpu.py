"""The FP64 level-set stages (one reciprocal a WENO side, cells on consecutive threads) against the oracle.

Rows shorter and longer than a warp and a block, grids of fewer cells than a block, and a wall far
outside whose jump is small, large, and beyond 2^60 (where a cell takes the formulas as written).
Tolerance: a step is some 300 roundings of values no larger than the grid's, so 300 x 2^-53 x 30 stages
~ 1e-12 of the largest value if none cancelled."""

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

H = 0.3


def grid_of(n, wall):
    x = np.stack(np.meshgrid(*[H * np.arange(k) for k in n], indexing="ij"), -1)
    mid = H * (np.array(n) - 1) / 2
    d = np.linalg.norm(x - mid - 0.03, axis=-1)
    g = 0.3 * H * max(n) - d + 0.01 * np.random.default_rng(sum(n)).normal(size=n)
    g[d > 0.45 * H * max(n)] = wall
    return g


@pytest.mark.parametrize("wall", [-10.0, -300.0, -1e12, -1e40])
@pytest.mark.parametrize("n", [(3, 5, 7), (17, 9, 33), (24, 31, 65), (40, 37, 45)])
def test_stages(ctx, n, wall):
    g = grid_of(n, wall)
    ref = g.copy()
    O.evolve(ref, H, 0.2)
    G = ctx.grid(n, (0.0, 0.0, 0.0), H)
    G.upload(g)
    G.evolve(0.2)
    assert np.abs(G.download() - ref).max() <= 1e-12 * np.abs(ref).max()
    if wall < -1e3:  # the rounding next to such a wall exceeds the interface's values: nothing to reinitialise
        return
    P = ctx.grid(n, (0.0, 0.0, 0.0), H)
    P.upload(g)
    G.upload(ref)
    steps = O.reinitialize(ref, g, H, 0.4, thickness=2)
    assert G.reinitialize(P, 0.4) == steps
    assert np.abs(G.download() - ref).max() <= 1e-12 * np.abs(ref).max()
