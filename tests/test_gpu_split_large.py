"""Mixed single-orbital kernels on meshes above 131,072 targets (four warps per CTA, two or more
of which share a target's sources below 1.2 million) and on small meshes beside large ones:
selected batches against the FP64 oracle, and the same bits for one and two targets per
thread, and for a mesh alone and in a launch of several."""
import numpy as np
import pytest
import torch

from conftest import rel_l2, to_cuda
from test_gpu_split import cloud

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,leaf,degree", [(131073, 333, 3), (180001, 65, 2), (1200001, 500, 1)])
def test_large_meshes(BT, dev, oracle, n, leaf, degree):
    x, y, z, w, f = cloud(n, leaf)
    plan = dev.TreecodePlan.for_mesh(*to_cuda(x, y, z, w), theta=0.8, degree=degree, source_leaf=leaf, target_leaf=leaf)
    c = oracle.Plan(x, y, z, x, y, z, w, 0.8, degree, leaf, leaf, 1.0)
    lists, tree = c.lists(), c.tree(1)
    nb = len(lists["batch_node"])
    sel = np.unique(np.linspace(0, nb - 1, 12).astype(np.int32))
    rows = np.concatenate([tree["perm"][tree["begin"][v]:tree["end"][v]] for v in lists["batch_node"][sel]])
    (ft,) = to_cuda(f)
    for kernel in (BT.Kernel.YUKAWA, BT.Kernel.COULOMB):
        for sing in (BT.Singularity.SUBTRACTION, BT.Singularity.SKIPPING):
            one, two = (plan.convolve(ft, ft, kernel, [1.3], sing, precision="mixed", targets_per_thread=nt) for nt in (1, 2))
            assert torch.isfinite(one).all() and torch.equal(one, two)
            ref = oracle.convolve_batches(c, f, f, w, kernel, [1.3], sing, sel)[0]
            assert rel_l2(one.cpu().numpy()[rows], ref[rows]) <= 1e-6
    plan.close()


@pytest.mark.parametrize("nt", [0, 1, 2])
@pytest.mark.parametrize("name", ["YUKAWA", "COULOMB"])
def test_small_mesh_beside_a_large_one(BT, dev, name, nt):
    kernel, SS = getattr(BT.Kernel, name), BT.Singularity.SUBTRACTION
    plans, F = [], []
    for n, leaf, norb in ((20001, 130, 3), (150001, 400, 1), (700, 60, 2)):
        x, y, z, w, _ = cloud(n, n)
        plans.append(dev.TreecodePlan.for_mesh(*to_cuda(x, y, z, w), theta=0.8, degree=3, source_leaf=leaf, target_leaf=leaf))
        F.append(torch.randn((norb, n), generator=torch.Generator().manual_seed(n), dtype=torch.float64).cuda())
    k = [np.linspace(0.8, 1.2, len(f)) for f in F]
    S = dev.Systems(plans, [len(f) for f in F], kernel, orbitals_per_item=1, targets_per_thread=nt)
    got = S.convolve(F, F, k, SS)
    for p, f, ki, g in zip(plans, F, k, got):
        alone = p.convolve(f, f, kernel, ki, SS, precision="mixed", orbitals_per_item=1)
        assert torch.isfinite(g).all() and torch.equal(g, alone.reshape(g.shape))
    S.close()
