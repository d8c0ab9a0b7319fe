"""Meshes far from the origin, seen through ordinary near ranges alone (targets beside the sources,
no cluster accepted; target values of zero, so that nothing cancels): coordinates relative to the
batch centers are exact in FP64, so moving everything must not change the error against the FP64
direct sum."""
import numpy as np
import pytest

from conftest import rel_l2, to_cuda

pytestmark = pytest.mark.gpu


def clouds(shift):
    rng = np.random.default_rng(4)
    q = lambda p: np.round(p * 2.0**20) * 2.0**-20   # exact at every shift
    s = q(rng.uniform(-1.0, 1.0, (3, 1503)))
    t = q(rng.uniform(-1.0, 1.0, (3, 701)))
    t[0] += 3.0
    s[0] += shift
    t[0] += shift
    s[1] -= shift
    t[1] -= shift
    return t, s, rng.uniform(0.5, 1.5, 1503) / 1503, np.zeros((5, 701)), rng.standard_normal((5, 1503))


@pytest.mark.parametrize("name,sing,kw", [
    ("YUKAWA", "SUBTRACTION", dict(orbitals_per_item=1, targets_per_thread=1)),
    ("YUKAWA", "SKIPPING", dict(orbitals_per_item=1, targets_per_thread=2)),
    ("COULOMB", "SUBTRACTION", dict(targets_per_thread=1)),
    ("COULOMB", "SKIPPING", dict(targets_per_thread=2)),
    ("YUKAWA", "SUBTRACTION", dict(orbitals_per_item=4)),
    ("YUKAWA", "SUBTRACTION", dict(orbitals_per_item=8)),
    ("YUKAWA", "SKIPPING", dict(orbitals_per_item=16)),
])
def test_error_does_not_grow_with_the_shift(BT, dev, oracle, name, sing, kw):
    k = np.linspace(0.6, 1.4, 5)
    kernel, sg = getattr(BT.Kernel, name), getattr(BT.Singularity, sing)
    err = []
    # the last one lies between two FP32 numbers, 128 apart there
    for shift in (0.0, 2.0**12, 2.0**20, 2.0**30 + 53.75):
        t, s, w, tv, sv = clouds(shift)
        plan = dev.TreecodePlan(*to_cuda(*t), *to_cuda(*s, w), theta=0.05, degree=3, source_leaf=150, target_leaf=130)
        info = plan.info()
        assert info["far_entries"] == 0 and info["near_close_pairs"] == 0
        got = plan.convolve(*to_cuda(tv, sv), kernel, k, sg, precision="mixed", **kw).cpu().numpy()
        ref = np.stack([oracle.direct(*t, tv[o], *s, sv[o], w, kernel, [k[o]], sg) for o in range(5)])
        err.append(rel_l2(got, ref))
        plan.close()
    # the inputs of the kernels are the same FP32 numbers at every shift but for rounding ties
    assert max(err) <= 1.5 * err[0], err
