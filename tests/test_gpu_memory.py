"""Memory that the library keeps between calls: bounded, given back on request, taken anew after."""
import pytest
import torch

from conftest import to_cuda
from test_gpu_split import cloud

pytestmark = pytest.mark.gpu


def test_kept_memory_is_bounded_and_given_back(BT, dev):
    n = 300000
    x, y, z, w, f = cloud(n, 1)
    (X, Y, Z, W), (ft,) = to_cuda(x, y, z, w), to_cuda(f)
    call = lambda: dev.treecode(X, Y, Z, ft, X, Y, Z, ft, W, BT.Kernel.YUKAWA, [0.9], BT.Singularity.SUBTRACTION, 0.8, 3, 2000, 2000)
    free = lambda: torch.cuda.mem_get_info()[0]
    dev.release_memory()
    before = free()
    one = call()
    kept = before - free()
    assert 0 < kept <= (1 << 30) + (256 << 20)      # the pool's bound, and its last block
    dev.release_memory()
    assert before - free() < kept
    assert torch.equal(one, call())
