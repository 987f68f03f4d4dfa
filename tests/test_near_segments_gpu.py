"""The FP32 near field's work segments: the tuning table's size is the size they have."""

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
