"""The FP32 near field's work segments: the tuning table's size is the size they have, and large leaves are cut."""

import os

import numpy as np
import pytest

import ibim
from test_fp64_digits_gpu import H, sphere_points

pytestmark = pytest.mark.gpu


@pytest.fixture
def restore_table():
    yield
    ibim.lib().ibim_tuning_clear()
    if os.path.exists(ibim.TUNING_TABLE):
        ibim.lib().ibim_tuning_load(ibim.TUNING_TABLE.encode())


def test_table_sets_the_segments(ctx, restore_table):
    """Eight leaves side by side, near field only: in one segment a leaf the sources fill other tiles than in several,
    so the FP32 partial sums round otherwise, beyond the 1e-15 that the order of the FP64 adds leaves; both are within
    FP32 sums of 320 terms, 2^-23 sqrt(320) ~ 2e-6, of each other."""
    n = 320
    p, nrm, w = sphere_points(n, 1)
    dens = np.random.default_rng(2).uniform(-1.0, 1.0, (4, n))
    kp = ibim.kernel_params(0.3, 80.0, 2.0, 1.0)
    lib = ibim.lib()

    def product(rows):
        lib.ibim_tuning_clear()
        if rows:
            assert lib.ibim_tuning_set(4, 0, rows, 1 << 14, 2) == ibim.OK
        plan = ctx.tube(p, nrm, w, H).plan(4, 60, 1, precision=ibim.PRECISION_MIXED)
        assert plan.stats()["v_pairs"] == 0
        return plan.apply(ibim.KERNEL_BIE_FUSED, kp, dens)

    a, b = product(None), product(1 << 24)
    size = np.abs(a).max(1, keepdims=True)
    assert 1e-12 < (np.abs(a - b) / size).max() < 2e-6
    assert (np.abs(a - product(1 << 17)) / size).max() < 1e-14  # the default: left to the plan


@pytest.mark.parametrize("n,leaf", [(300, 400), (1100, 1200), (5003, 1300)])
def test_large_leaves_in_pieces(ctx, restore_table, n, leaf):
    """Leaves of more points than a segment's are cut: the sums round otherwise than in one segment a leaf, and agree with
    the FP64 operator as mixed products do (1.5e-5 of the largest value, test_m2l_pair_gpu.py)."""
    p, nrm, w = sphere_points(n, 2)
    dens = np.random.default_rng(3).uniform(-1.0, 1.0, (4, n))
    kp = ibim.kernel_params(0.3, 80.0, 2.0, 1.0)
    tube = ctx.tube(p, nrm, w, H)
    lib = ibim.lib()
    lib.ibim_tuning_clear()
    a = tube.plan(4, leaf, 10, precision=ibim.PRECISION_MIXED).apply(ibim.KERNEL_BIE_FUSED, kp, dens)
    assert lib.ibim_tuning_set(4, 0, 1 << 24, 1 << 14, 2) == ibim.OK
    b = tube.plan(4, leaf, 10, precision=ibim.PRECISION_MIXED).apply(ibim.KERNEL_BIE_FUSED, kp, dens)
    ref = tube.plan(4, leaf, 10).apply(ibim.KERNEL_BIE_FUSED, kp, dens)
    size = np.abs(ref).max(1, keepdims=True)
    assert 1e-12 < (np.abs(a - b) / size).max()
    assert (np.abs(a - ref) / size).max() < 1.5e-5 and (np.abs(b - ref) / size).max() < 1.5e-5
