"""What a convolution sets up before its field passes: kernel parameters as arguments or
copied (more than 64 orbitals) or on the device, and the weights' proxy charges of a
one-shot plan, formed with the charges.  Either way the same arithmetic, so the same bits."""
import pytest
import torch

from conftest import to_cuda
from test_gpu_split import cloud

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("norb", [1, 3, 64, 65, 130])
def test_parameters_from_host_and_device_agree(BT, dev, norb):
    x, y, z, w, _ = cloud(700, norb)
    f = torch.randn((norb, 700), generator=torch.Generator().manual_seed(norb), dtype=torch.float64).cuda()
    k = [0.4 + 0.02 * o for o in range(norb)]
    plan = dev.TreecodePlan.for_mesh(*to_cuda(x, y, z, w), theta=0.8, degree=3, source_leaf=60, target_leaf=60)
    host = plan.convolve(f, f, BT.Kernel.YUKAWA, k, BT.Singularity.SUBTRACTION, precision="mixed")
    there = plan.convolve(f, f, BT.Kernel.YUKAWA, torch.tensor(k, dtype=torch.float64, device="cuda"),
                          BT.Singularity.SUBTRACTION, precision="mixed")
    assert torch.isfinite(host).all() and torch.equal(host, there)
    plan.close()


@pytest.mark.parametrize("degree", [1, 4, 7, 8, 10])
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_one_shot_equals_kept_plan(BT, dev, degree, precision):
    n = 9001
    x, y, z, w, f = cloud(n, degree)
    (X, Y, Z, W), (ft,) = to_cuda(x, y, z, w), to_cuda(f)
    for kernel in (BT.Kernel.YUKAWA, BT.Kernel.COULOMB):
        once = dev.treecode(X, Y, Z, ft, X, Y, Z, ft, W, kernel, [0.9], BT.Singularity.SUBTRACTION, 0.8, degree, 150, 150,
                            precision=precision)
        plan = dev.TreecodePlan.for_mesh(X, Y, Z, W, theta=0.8, degree=degree, source_leaf=150, target_leaf=150)
        kept = plan.convolve(ft, ft, kernel, [0.9], BT.Singularity.SUBTRACTION, precision=precision)
        assert torch.isfinite(once).all() and torch.equal(once, kept.reshape(-1))
        plan.close()
