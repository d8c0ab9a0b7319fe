"""Proxy charges in mixed precision, bit for bit where one source makes them all."""
import numpy as np
import pytest

from conftest import to_cuda

pytestmark = pytest.mark.gpu


def far_plan(dev, x, w, degree=1):
    """Sources at x on the first axis, one target that sees them as one cluster."""
    z, t = np.zeros(len(x)), np.zeros(1)
    plan = dev.TreecodePlan(*to_cuda(t + 100.0 * np.abs(x).max(), t, t), *to_cuda(x, z, z, w), theta=0.7, degree=degree,
                            source_leaf=100, target_leaf=10, size_check=0.01)
    assert plan.info()["slots"] == 1
    return plan


def test_coordinates_are_rounded_quotients(dev):
    """Sources whose coordinate u in the box lies halfway between two FP32 numbers: u is the FP64
    quotient rounded to FP32 (to even), as numpy gives it, also where the product with the
    reciprocal lies on the other side of the tie."""
    one, half = np.float32(1), np.float32(0.5)
    rng = np.random.default_rng(1)
    cases = [(h, (2 * int(rng.integers(2**23, 2**24)) + 1) * 2.0**-25) for h in rng.integers(3, 2**27, 4000) | 1]
    other = [(h, t) for h, t in cases if np.float32(t * h * (1.0 / h)) != np.float32(t * h / h)]
    assert len(other) > 20
    for h, t in cases[:10] + other[:20]:
        x = np.array([-float(h), t * h, float(h)])       # t h is exact: 25 bits and 27
        plan = far_plan(dev, x, np.array([0.0, 1.0, 0.0]))
        u = np.float32(x[1] / h)
        l0, l1 = half / (u - one), -half / (u + one)      # nodes 1, -1; weights 1/2, -1/2
        s = l0 + l1
        # the other axes have u = 0: 1/2 each
        ref = np.repeat(np.array([half * (half * (l0 / s)), half * (half * (l1 / s))], np.float32), 4)
        got = plan.charges(3)[0, 0].astype(np.float32)
        plan.close()
        assert np.array_equal(got, ref), (h, t, got, ref)


@pytest.mark.parametrize("norb", [1, 3])
@pytest.mark.parametrize("big", [np.inf, -np.inf, 3e38])
def test_infinite_sums_stay_infinite(BT, dev, norb, big):
    """One infinite charge, or finite ones whose sum is beyond FP32, among positive basis values."""
    n = 70
    x = np.linspace(-1.0, 1.0, n) + 1e-3      # no source on a node but the outermost two
    plan = far_plan(dev, x, np.ones(n))
    f = np.full((norb, n), 1.0 if np.isinf(big) else big)
    f[:, 0] = f[:, -1] = 1.0
    f[:, 31] = big
    plan.convolve(*to_cuda(np.zeros((norb, 1)), f), BT.Kernel.COULOMB, [1.0], BT.Singularity.SKIPPING, precision="mixed")
    assert np.array_equal(plan.charges(2, norb)[:, 0], np.full((norb, 8), np.copysign(np.inf, big)))
    plan.close()
