"""The FP64 operator in any unit of length and with halves of any size, against the oracle's FMM: one cloud of several
levels with its lengths (and the cutoff, kappa and psi with them) in Angstrom, in 10^3, 10^6 and 10^12 units an Angstrom
and in metres, and psi from 10^-6 to 10^12 times the dipole.  The oracle's values are those of the Angstrom (its list
building compares lengths with constants), scaled.  Tolerance: both sides are FP64 sums as in
test_fp64_digits_gpu.py, 2e-13 of the largest value (the smallest t = kappa h is 0.2: no more cancellation than there)."""

import numpy as np
import pytest

import ibim
import oracle as O
from test_fp64_digits_gpu import H, sphere_points

pytestmark = pytest.mark.gpu


def compare(ctx, order, leaf, n, unit, kappa, ratio, dens=None):
    p, nrm, w = sphere_points(n, order)
    if dens is None:
        dens = np.random.default_rng(order + 1).uniform(-1.0, 1.0, (4, n))
        dens[3] *= ratio
    ref = O.Tree(p, p, leaf, 10).fmm(order, O.KParams(kappa, 80.0, 2.0, H), 16, dens)
    dens = dens.copy()
    dens[3] /= unit
    plan = ctx.tube(p * unit, nrm, w, H * unit).plan(order, leaf, 10)
    out = plan.apply(ibim.KERNEL_BIE_FUSED, ibim.kernel_params(kappa / unit, 80.0, 2.0, 1.0), dens)
    for o in range(4):
        got = out[o] * (unit ** 2 if o == 0 else unit ** 3)
        assert np.abs(got - ref[o]).max() <= 2e-13 * np.abs(ref[o]).max(), o


@pytest.mark.parametrize("kappa", [0.0, 0.4])
@pytest.mark.parametrize("unit", [1e-10, 1e3, 1e6, 1e12])
@pytest.mark.parametrize("order,n,leaf", [(2, 1500, 20), (3, 1500, 40), (4, 1500, 30), (5, 1500, 40), (6, 1200, 40),
                                          (7, 900, 40)])
def test_units(ctx, order, n, leaf, unit, kappa):
    compare(ctx, order, leaf, n, unit, kappa, 1.0)


@pytest.mark.parametrize("unit", [1.0, 1e-10])
@pytest.mark.parametrize("kappa", [0.0, 0.4])
@pytest.mark.parametrize("ratio", [1e-6, 1e6, 1e12])
@pytest.mark.parametrize("order,leaf", [(4, 40), (5, 10), (6, 40)])
def test_halves_of_other_sizes(ctx, order, leaf, ratio, kappa, unit):
    compare(ctx, order, leaf, 1200, unit, kappa, ratio)


@pytest.mark.parametrize("kappa", [0.0, 0.4])
@pytest.mark.parametrize("half", [0, 1])
def test_one_half_alone(ctx, half, kappa):
    dens = np.random.default_rng(9).uniform(-1.0, 1.0, (4, 1500))
    dens[3:] = 0.0 if half == 0 else dens[3:]
    dens[:3] = 0.0 if half == 1 else dens[:3]
    compare(ctx, 5, 40, 1500, 1.0, kappa, 1.0, dens)


@pytest.mark.parametrize("ratio", [1.0, 1e6])
def test_negative_kappa(ctx, ratio):
    """Growing exponentials, which a product takes though a solve does not: neither kernel pair vanishes."""
    compare(ctx, 5, 40, 1200, 1.0, -0.05, ratio)
