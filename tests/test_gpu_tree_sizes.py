"""Trees and lists of more points than the other tests have, where other branches build them:
sorts of more than 131,072 keys and of more than 1,024 tiles, trees built a level at a time,
scans of several tiles, and lists walked by a thread per batch."""
import numpy as np
import pytest
import torch

from conftest import to_cuda
from test_gpu_tree import _compare, _plans

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,leaf", [(30011, 9), (140003, 12), (262145, 40)])
def test_small_leaves_match_oracle(dev, oracle, n, leaf):
    rng = np.random.default_rng(n)
    pts = rng.normal(0.0, 1.0, (n, 3))
    g, c = _plans(dev, oracle, pts, pts, np.ones(n), 0.8, 2, leaf, leaf, sc=0.5)
    assert g.info()["batches"] > 8192
    _compare(g, c)


def test_lists_on_both_sides_of_the_walk_switch(dev, oracle):
    """The warps' walk and the threads' walk meet at 8,192 batches."""
    counts = []
    for n, leaf in ((30011, 5), (30011, 10), (30011, 16)):
        rng = np.random.default_rng(3)
        pts = rng.uniform(-1.0, 1.0, (n, 3))
        g, c = _plans(dev, oracle, pts, pts, np.ones(n), 0.7, 1, leaf, leaf, sc=1.0)
        counts.append(g.info()["batches"])
        _compare(g, c)
    assert min(counts) < 8192 < max(counts)


def test_sort_of_more_than_1024_tiles(dev):
    n = 4300001
    gen = torch.Generator(device="cuda").manual_seed(5)
    x, y, z = (torch.randint(0, 600, (n,), generator=gen, device="cuda").double() for _ in range(3))
    p = dev.TreecodePlan.for_mesh(x, y, z, torch.ones_like(x), theta=0.7, degree=1, source_leaf=20000, target_leaf=20000)
    t = p.tree(0)
    codes, perm = t["codes"], t["perm"].astype(np.int64)
    assert np.array_equal(np.sort(perm), np.arange(n))
    assert np.all(codes[1:] >= codes[:-1])
    same = codes[1:] == codes[:-1]
    assert same.any() and np.all(perm[1:][same] > perm[:-1][same])   # stable
    # equal points have equal codes, and only they: the codes follow the points through the sort
    key = (x * 600 + y) * 600 + z
    key = key.cpu().numpy()[perm]
    assert np.array_equal(same, key[1:] == key[:-1])
