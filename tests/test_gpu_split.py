"""Field items cut by targets and sources (Fields::split): every batch size around a
warp, a CTA's targets and a tile of sources, against the FP64 oracle.

The oracle's treecode uses the same lists, so FP64 results agree to 1e-12 and
mixed ones to 1e-6 (relative L2), the bounds of the other convolution tests.
"""
import numpy as np
import pytest

from conftest import rel_l2, to_cuda

pytestmark = pytest.mark.gpu

# leaf: batches of at most that many points; n: total (the last ones are ragged)
SIZES = [(33, 700), (63, 1500), (64, 1500), (65, 1531), (129, 3000), (257, 5003), (520, 9001)]


def cloud(n, seed):
    rng = np.random.default_rng(seed)
    p = rng.uniform(-1.0, 1.0, (3, n)) * np.array([[3.0], [2.0], [2.5]])
    return p[0].copy(), p[1].copy(), p[2].copy(), rng.uniform(0.5, 1.5, n) / n, rng.standard_normal(n)


@pytest.mark.parametrize("leaf,n", SIZES)
@pytest.mark.parametrize("precision,tol", [("mixed", 1e-6), ("fp64", 1e-12)])
def test_ragged_batches_match_oracle(BT, dev, oracle, leaf, n, precision, tol):
    x, y, z, w, f = cloud(n, leaf)
    degree = 2 + leaf % 3
    plan = dev.TreecodePlan.for_mesh(*to_cuda(x, y, z, w), theta=0.8, degree=degree, source_leaf=leaf, target_leaf=leaf)
    c = oracle.Plan(x, y, z, x, y, z, w, 0.8, degree, leaf, leaf, 1.0)
    (ft,) = to_cuda(f)
    for kernel in (BT.Kernel.YUKAWA, BT.Kernel.COULOMB):
        for sing in (BT.Singularity.SUBTRACTION, BT.Singularity.SKIPPING):
            ref = c.convolve(f, f, w, kernel, [1.3], sing)
            for nt in ((1, 2) if precision == "mixed" else (0,)):
                got = plan.convolve(ft, ft, kernel, [1.3], sing, precision=precision, targets_per_thread=nt)
                assert rel_l2(got.cpu().numpy(), ref) <= tol
    plan.close()


def test_targets_that_are_not_sources(BT, dev, oracle):
    x, y, z, w, f = cloud(4001, 5)
    tx, ty, tz, _, tv = cloud(611, 6)
    plan = dev.TreecodePlan(*to_cuda(tx, ty, tz), *to_cuda(x, y, z, w), theta=0.8, degree=3, source_leaf=100,
                            target_leaf=130)
    c = oracle.Plan(tx, ty, tz, x, y, z, w, 0.8, 3, 100, 130, 1.0)
    ref = c.convolve(tv, f, w, BT.Kernel.YUKAWA, [0.9], BT.Singularity.SUBTRACTION)
    for precision, tol in (("mixed", 1e-6), ("fp64", 1e-12)):
        got = plan.convolve(*to_cuda(tv, f), BT.Kernel.YUKAWA, [0.9], BT.Singularity.SUBTRACTION, precision=precision)
        assert rel_l2(got.cpu().numpy(), ref) <= tol


@pytest.mark.parametrize("scale", [1e-22, 1e-3, 1.0, 60.0, 1e4, 1e21])
@pytest.mark.parametrize("name,k", [("YUKAWA", 0.7), ("COULOMB", 1.1)])
@pytest.mark.parametrize("sing", ["SUBTRACTION", "SKIPPING"])
def test_fp64_pairs_over_the_distance_range(BT, dev, scale, name, k, sing):
    """Distances from far below to far above FP32's squared range, exponents past
    underflow, coincident points: the sums of numpy's FP64 functions to 1e-12 of
    the sum of the terms' magnitudes."""
    rng = np.random.default_rng(3)
    p = rng.uniform(-1.0, 1.0, (3, 150)) * scale
    p[:, 70:75] = p[:, 10:15]                      # coincident pairs are left out
    w, f = rng.uniform(0.5, 1.5, 150), rng.standard_normal(150)
    d2 = ((p[:, :, None] - p[:, None, :]) ** 2).sum(0)
    with np.errstate(divide="ignore", invalid="ignore", over="ignore", under="ignore"):
        r = np.sqrt(d2)
        if name == "YUKAWA":
            t = (f[None, :] - (f[:, None] if sing == "SUBTRACTION" else 0.0)) * w[None, :] * np.exp(-k * r) / r
        else:
            t = w[None, :] * (f[None, :] - (f[:, None] * np.exp(-k * k * d2) if sing == "SUBTRACTION" else 0.0)) / r
    t[d2 == 0.0] = 0.0
    own = f * (4.0 if name == "YUKAWA" else 2.0) * np.pi / k ** 2 if sing == "SUBTRACTION" else 0.0 * f
    got = dev.TreecodePlan.for_mesh(*to_cuda(*p, w), theta=0.7, degree=2, source_leaf=200, target_leaf=200).convolve(
        *to_cuda(f, f), getattr(BT.Kernel, name), [k], getattr(BT.Singularity, sing), precision="fp64").cpu().numpy()
    assert np.all(np.abs(got - (t.sum(1) + own)) <= 1e-12 * (np.abs(t).sum(1) + np.abs(own)) + 1e-300)


@pytest.mark.parametrize("degree", range(1, 11))
def test_rows_of_every_degree(BT, dev, oracle, degree):
    """Odd and even proxy rows, alone and beside another degree in one launch, one
    orbital per item and groups: the far kernels' loops of each length."""
    x, y, z, w, _ = cloud(9001, degree)
    leaf = 130
    F = np.random.default_rng(degree).standard_normal((5, 9001))
    k = np.linspace(0.6, 1.4, 5)
    plan = dev.TreecodePlan.for_mesh(*to_cuda(x, y, z, w), theta=0.8, degree=degree, source_leaf=leaf, target_leaf=leaf,
                                     size_check=0.05)
    assert plan.info()["far_entries"] > 0
    c = oracle.Plan(x, y, z, x, y, z, w, 0.8, degree, leaf, leaf, 0.05)
    (Ft,) = to_cuda(F)
    ref = np.stack([c.convolve(F[o], F[o], w, BT.Kernel.YUKAWA, [k[o]], BT.Singularity.SUBTRACTION) for o in range(5)])
    for og in (1, 4, 8, 16):
        got = plan.convolve(Ft, Ft, BT.Kernel.YUKAWA, k, BT.Singularity.SUBTRACTION, precision="mixed",
                            orbitals_per_item=og)
        assert rel_l2(got.cpu().numpy(), ref) <= 1e-6
    other = dev.TreecodePlan.for_mesh(*to_cuda(x, y, z, w), theta=0.8, degree=11 - degree, source_leaf=leaf,
                                      target_leaf=leaf, size_check=0.05)
    for og in (1, 4):
        S = dev.Systems([plan, other], (5, 5), BT.Kernel.YUKAWA, orbitals_per_item=og)
        got = S.convolve([Ft, Ft], [Ft, Ft], [k, k], BT.Singularity.SUBTRACTION)[0]
        assert rel_l2(got.cpu().numpy(), ref) <= 1e-6
        S.close()
    other.close()
    plan.close()
