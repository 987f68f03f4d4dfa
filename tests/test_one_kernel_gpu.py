"""One scalar kernel's FP64 FMM on its own entry of the operator against the fused operator with the other
densities zero: all kernels, orders of one and of several row tiles, the forms of the pair update.
Tolerance: two FP64 evaluations, each within 2e-13 of the largest value of the oracle's (its derivation stands
with the fused operator's test)."""

import numpy as np
import pytest

import ibim

pytestmark = pytest.mark.gpu

H = 0.5
AX = "xyz"


def slot_field_sign(name):
    if name == "K2":
        return 3, 0, -1.0
    if name[:2] == "K1":
        return AX.index(name[2]), 0, 1.0
    if name[:2] == "K4":
        return 3, 1 + AX.index(name[2]), -1.0
    a, b = (AX.index(c) for c in name[2:])
    if name in ("K3yx", "K3zy", "K3xz"):
        a, b = b, a
    return a, 1 + b, 1.0


@pytest.mark.parametrize("order,n,leaf,kappa,tau", [(2, 700, 20, 0.3, 1.0), (3, 1300, 9, 0.4, 1.0), (4, 63, 64, 0.4, 1.0),
                                                    (5, 1500, 40, 0.0, 1.0), (6, 1200, 300, 0.1, 1.0),
                                                    (7, 900, 40, 2.0, 1.0), (4, 1500, 40, 0.4, 1e-16)])
def test_entry_matches_block(ctx, order, n, leaf, kappa, tau):
    r = np.random.default_rng(order)
    v = r.normal(size=(n, 3))
    v /= np.linalg.norm(v, axis=1)[:, None]
    plan = ctx.tube(v * r.uniform(7.0, 8.0, (n, 1)), v, r.uniform(0.1, 1.0, n), H).plan(order, leaf, 10)
    kp = ibim.kernel_params(kappa, 80.0, 2.0, tau)
    m = r.uniform(-1.0, 1.0, n)
    for i, name in enumerate(ibim.KERNELS):
        slot, field, sign = slot_field_sign(name)
        dens = np.zeros((4, n))
        dens[slot] = m
        ref = sign * plan.apply(ibim.KERNEL_BIE_FUSED, kp, dens)[field]
        out = plan.apply(i, kp, m)
        assert np.abs(out - ref).max() <= 4e-13 * np.abs(ref).max(), name
