"""A GEMM whose pipeline gives up a wait says so: the status is read and cleared by tagi_mlp_check,
the Python trainer's check raises, and GEMMs run on afterwards."""
import ctypes
import importlib

import pytest
import torch

pytestmark = pytest.mark.gpu
PKG = "treecode-accelerated-green-iteration_gb300"


def test_a_wait_that_runs_out_is_reported(native):
    learned = importlib.import_module(PKG + ".learned")
    L = native.lib()
    s = torch.cuda.Stream()
    net = learned.MLP(27, 64, 1e-3, 0, stream=s)
    net.check()                                    # nothing to report
    native.check(L.tagi_mlp_wait_probe(3, ctypes.c_void_p(s.cuda_stream)))
    with pytest.raises(native.TagiError, match="wait ran out"):
        net.check()
    net.check()                                    # cleared
    X = torch.randn(300, net.ldx, device="cuda").bfloat16()
    torch.cuda.synchronize()
    Y = net.forward(X, 300)
    net.check()
    assert torch.isfinite(Y).all()
    assert L.tagi_mlp_wait_probe(-1, None) != 0    # refused
