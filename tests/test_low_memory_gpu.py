"""FP64 products where the device has little memory left, each case in a process of its own that takes the rest first."""

import subprocess
import sys
import os

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)

CHILD = r"""
import sys
import numpy as np
import torch
sys.path[:0] = [{root!r}, {pkg!r}, {tests!r}]
import ibim
from test_fp64_digits_gpu import H, sphere_points

ctx = ibim.Context(0)
p, nrm, w = sphere_points(20000, 3)
tube = ctx.tube(p, nrm, w, H)
kp = ibim.kernel_params(0.4, 80.0, 2.0, 1.0)
dens = np.random.default_rng(4).uniform(-1.0, 1.0, (4, len(p)))
plan = tube.plan(5, 12, 10)
ops64 = plan.stats()["operators"] * 500 * 500 * 8  # digit images: 2.1 times that and 1.1 GB


def take(left):
    torch.cuda.synchronize()
    n = torch.cuda.mem_get_info()[0] - int(left)
    assert n > 0
    return torch.empty(n, dtype=torch.uint8, device="cuda")


def release():
    global hog
    hog = None
    torch.cuda.empty_cache()


def close(a, b):
    assert np.abs(a - b).max() < 4e-13 * np.abs(b).max()

"""


def child(body):
    code = CHILD.format(root=ROOT, pkg=os.path.join(ROOT, "ibim-levelset_gb300"), tests=HERE) + body
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


def test_product_after_an_allocation_that_failed():
    pytest.importorskip("torch")
    child(r"""
hog = take(0.5 * ops64)
for i in range(2):
    try:
        plan.apply(ibim.KERNEL_BIE_FUSED, kp, dens)
        raise SystemExit("no error")
    except ibim.IbimError as e:
        assert "out of memory" in str(e)
release()
out = plan.apply(ibim.KERNEL_BIE_FUSED, kp, dens)
ref = tube.plan(5, 12, 10).apply(ibim.KERNEL_BIE_FUSED, kp, dens)
for o in range(4):
    close(out[o], ref[o])
""")


@pytest.mark.parametrize("left", [1.6, 3.3, 6.5])
def test_product_without_room_for_its_images(left):
    """Room for the FP64 operators but not, or barely, for their digit images: the product runs all the same.  Both
    contractions are FP64 sums within 2e-13 of the oracle's (test_fp64_digits_gpu.py), so within 4e-13 of each other."""
    pytest.importorskip("torch")
    child(r"""
hog = take(%g * ops64)
m = dens[0]
out = plan.apply(ibim.KERNEL_BIE_FUSED, kp, dens)
one = [plan.apply(k, kp, m) for k in range(len(ibim.KERNELS))]
again = plan.apply(ibim.KERNEL_BIE_FUSED, ibim.kernel_params(0.5, 80.0, 2.0, 1.0), dens)
release()
fresh = tube.plan(5, 12, 10)
for o in range(4):
    close(out[o], fresh.apply(ibim.KERNEL_BIE_FUSED, kp, dens)[o])
    close(again[o], fresh.apply(ibim.KERNEL_BIE_FUSED, ibim.kernel_params(0.5, 80.0, 2.0, 1.0), dens)[o])
for k in range(len(ibim.KERNELS)):
    close(one[k], fresh.apply(k, kp, m))
""" % left)
