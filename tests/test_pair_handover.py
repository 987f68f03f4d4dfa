"""Hand-over between the two CTAs of the pair kernels, by reading their source: what one CTA copies into its shared
memory is multiplied by an MMA that the other one's thread issues, so every arrive on the other CTA's barrier has to
release at cluster scope, and the wait for it to acquire at cluster scope.  (A weaker order shows as wrong sums on
some chip some day, not as a failing product.)"""

import os
import re

import numpy as np
import pytest

import ibim
from test_fp64_digits_gpu import H, sphere_points

SRC = os.path.join(os.path.dirname(ibim.__file__), "csrc", "m2l_tc.cu")


def kernel(name):
    text = open(SRC).read()
    start = re.search(r"\n    %s\(" % name, text).start()
    return text[start:text.index("\n}\n", start)]


def test_remote_arrivals_release_at_cluster_scope():
    arrives = re.findall(r"mbarrier\.arrive\S*\.shared::cluster\.b64", open(SRC).read())
    assert len(arrives) >= 4
    for a in arrives:
        assert a.startswith("mbarrier.arrive.release.cluster."), a


# barriers that the other CTA's threads arrive on (its commits complete through the asynchronous proxy)
REMOTE = {"k_m2l_tc2": ["peer_full"], "k_m2l_tc2h": ["peer_full"], "k_m2l_pair": ["acc_empty"]}


def test_waits_for_the_other_cta_acquire_at_cluster_scope():
    text = open(SRC).read()
    assert "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64" in text
    for name, barriers in REMOTE.items():
        body = kernel(name)
        for bar in barriers:
            waits = re.findall(r"(mbar_wait\w*)\(smem_u32\(&%s\b" % bar, body)
            assert waits and set(waits) == {"mbar_wait_cluster"}, (name, bar, waits)
    # the pair form's full barrier: the MMA thread's wait acquires the relay's arrive, the relay's its own CTA's
    assert re.findall(r"(mbar_wait\w*)\(smem_u32\(&full\b", kernel("k_m2l_pair")) == ["mbar_wait_cluster", "mbar_wait"]


@pytest.mark.gpu
@pytest.mark.parametrize("n,order,leaf", [(24000, 4, 8), (30000, 5, 12), (24000, 6, 8)])
def test_pair_form_matches_fp64(ctx, n, order, leaf):
    """Clouds with the pairs an operator that take the pair form.  Tolerance as in test_m2l_pair_gpu.py: FP32 sums of
    up to 4 p^3 products of 22-bit operands and a few thousand pairs, 2^-22 sqrt(4000) ~ 1.5e-5 of the largest value."""
    p, nrm, w = sphere_points(n, n + order)
    dens = np.random.default_rng(n).uniform(-1.0, 1.0, (4, n))
    t = ctx.tube(p, nrm, w, H)
    kp = ibim.kernel_params(0.3, 80.0, 2.0, 1.0)
    m = t.plan(order, leaf, 10, precision=ibim.PRECISION_MIXED)
    st = m.stats()
    assert st["v_pairs"] >= 128 * st["operators"]
    a = t.plan(order, leaf, 10).apply(ibim.KERNEL_BIE_FUSED, kp, dens)
    b = m.apply(ibim.KERNEL_BIE_FUSED, kp, dens)
    for o in range(4):
        assert np.abs(a[o] - b[o]).max() < 1.5e-5 * np.abs(a[o]).max(), o
