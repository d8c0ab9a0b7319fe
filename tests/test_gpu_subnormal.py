"""FP64 convolutions whose exponentials are subnormal numbers: the terms are kept, as numpy's FP64
exponential gives them, in the near field and through proxy charges."""
import numpy as np
import pytest

from conftest import to_cuda

pytestmark = pytest.mark.gpu
TINY = 5e-324   # spacing of subnormal numbers


@pytest.mark.parametrize("k", [700.0, 707.0, 708.5, 715.0, 730.0, 744.0, 760.0, 2000.0])
@pytest.mark.parametrize("sing", ["SUBTRACTION", "SKIPPING"])
def test_yukawa_near(BT, dev, k, sing):
    x = np.array([0.0, 0.5])       # targets at 0 and 0.5, the source 1 from the first
    z = np.zeros(2)
    s, w, f = np.array([1.0]), np.array([1.0]), np.array([1e10])
    plan = dev.TreecodePlan(*to_cuda(x, z, z), *to_cuda(s, z[:1], z[:1], w), theta=0.7, degree=2, source_leaf=10, target_leaf=10)
    got = plan.convolve(*to_cuda(z, f), BT.Kernel.YUKAWA, [k], getattr(BT.Singularity, sing), precision="fp64").cpu().numpy()
    ref = 1e10 * np.exp(-k * np.array([1.0, 0.5])) / np.array([1.0, 0.5])
    assert np.all(np.abs(got - ref) <= 1e-12 * ref + 2.0 * 1e10 * TINY), (got, ref)


@pytest.mark.parametrize("k", [715.0, 730.0])
def test_yukawa_far(BT, dev, k):
    rng = np.random.default_rng(2)
    s = 1.0e-4 * rng.uniform(-1.0, 1.0, (3, 200)) + np.array([[1.0], [0.0], [0.0]])
    w, f, z = np.ones(200), 1e10 * rng.uniform(0.5, 1.5, 200), np.zeros(1)
    plan = dev.TreecodePlan(*to_cuda(z, z, z), *to_cuda(*s, w), theta=0.7, degree=4, source_leaf=300, target_leaf=10, size_check=0.1)
    assert plan.info()["far_entries"] == 1
    got = plan.convolve(*to_cuda(z, f), BT.Kernel.YUKAWA, [k], BT.Singularity.SKIPPING, precision="fp64").cpu().numpy()
    r = np.sqrt((s**2).sum(0))
    ref = (f * np.exp(-k * r) / r).sum()
    assert abs(got[0] - ref) <= 1e-9 * ref + 200 * 2e10 * TINY, (got, ref)
