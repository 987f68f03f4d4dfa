"""The FP64 level-set stages beside walls far outside, cell by cell: one step (three stages) against the oracle, each
cell by the largest value that its stencils reach, so that a wall's size excuses the cells that see it and no others.
Walls on both sides of 2^60 in the second differences, from where a cell takes the formulas as written.
Tolerance: a stage is some 100 roundings of sums of values of the stencil (the weights are between 0 and 1, and 2^-53
of relative error in an indicator moves a weight by at most a few 2^-53), three stages: 300 x 2^-53 = 3.4e-14 of the
largest value within reach."""

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

H, REACH = 0.3, 9  # three cells a stage


def reached_max(a):
    """max |a| over REACH cells to each side along every axis."""
    m = np.abs(a)
    for axis in range(3):
        src = np.moveaxis(m, axis, 0)
        out = src.copy()
        for s in range(1, REACH + 1):
            out[s:] = np.maximum(out[s:], src[:-s])
            out[:-s] = np.maximum(out[:-s], src[s:])
        m = np.moveaxis(out, 0, axis)
    return m


@pytest.mark.parametrize("wall", [0.0, -300.0, -1e6, -1e12, -4e17, -6e17, -3e18, -1e25, -1e40])
@pytest.mark.parametrize("n", [(44, 29, 33), (31, 40, 65)])
def test_one_step(ctx, n, wall):
    x = np.stack(np.meshgrid(*[H * np.arange(k) for k in n], indexing="ij"), -1)
    d = np.linalg.norm(x - H * (np.array(n) - 1) / 2 - 0.03, axis=-1)
    g = 0.3 * H * max(n) - d + 0.01 * np.random.default_rng(sum(n)).normal(size=n)
    if wall:
        g[:4] = wall           # a slab
        g[-2, 3, 5] = wall     # and one cell
    ref = g.copy()
    O.evolve(ref, H, 0.05)  # cfl 0.2: dt = 0.06, one step
    G = ctx.grid(n, (0.0, 0.0, 0.0), H)
    G.upload(g)
    G.evolve(0.05)
    err = np.abs(G.download() - ref)
    size = reached_max(g)
    assert not wall or (size < 100.0).sum() > 1000  # cells that no wall reaches
    assert (err <= 3.4e-14 * size).all(), (err / size).max()
