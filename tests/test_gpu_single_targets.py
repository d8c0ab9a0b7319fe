"""A warp with at most 32 targets left takes one target per lane instead of two: each
target's arithmetic stays the same, so both give the same bits."""
import pytest
import torch

from conftest import to_cuda
from test_gpu_split import cloud

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("leaf", [1, 31, 32, 33, 63, 64, 65, 96, 97, 130])
def test_one_and_two_targets_per_lane_agree(BT, dev, leaf):
    x, y, z, w, f = cloud(40 * leaf + 7 if leaf > 1 else 90, leaf)
    X, (ft,) = to_cuda(x, y, z, w), to_cuda(f)
    plan = dev.TreecodePlan.for_mesh(*X, theta=0.8, degree=3, source_leaf=leaf, target_leaf=leaf)
    for kernel in (BT.Kernel.YUKAWA, BT.Kernel.COULOMB):
        for sing in (BT.Singularity.SUBTRACTION, BT.Singularity.SKIPPING):
            one, two = (plan.convolve(ft, ft, kernel, [1.1], sing, precision="mixed", targets_per_thread=nt) for nt in (1, 2))
            assert torch.isfinite(one).all() and torch.equal(one, two)
    plan.close()
