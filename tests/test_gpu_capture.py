"""Stream capture with the work lists that earlier calls on the plan left: any call on these orbitals
will do, whatever its targets per thread and, where the precision's own arrays exist, its precision."""
import pytest
import torch

from conftest import to_cuda
from test_gpu_split import cloud

pytestmark = pytest.mark.gpu


def make(dev, n, leaf):
    x, y, z, w, _ = cloud(n, n)
    plan = dev.TreecodePlan.for_mesh(*to_cuda(x, y, z, w), theta=0.8, degree=3, source_leaf=leaf, target_leaf=leaf)
    f = torch.randn((3, n), generator=torch.Generator().manual_seed(n), dtype=torch.float64).cuda()
    return plan, f, torch.tensor([0.7, 0.9, 1.1], dtype=torch.float64, device="cuda")


def captured(dev, plan, BT, F, k, **kw):
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    out = torch.zeros_like(F)
    with dev.Graph.capture(s) as g:
        plan.convolve(F, F, BT.Kernel.COULOMB, k, BT.Singularity.SUBTRACTION, out=out, stream=s, **kw)
    g.replay(s)
    torch.cuda.synchronize()
    return out, g


@pytest.mark.parametrize("n,leaf", [(3001, 130), (9001, 520), (140003, 1000)])
@pytest.mark.parametrize("before,then", [
    (dict(precision="mixed"), dict(precision="mixed", targets_per_thread=1)),
    (dict(precision="mixed"), dict(precision="mixed", targets_per_thread=2)),
    (dict(precision="mixed", targets_per_thread=2), dict(precision="mixed")),
    (dict(precision="fp64"), dict(precision="mixed")),
    (dict(precision="fp64"), dict(precision="mixed", targets_per_thread=2)),
    (dict(precision="mixed", targets_per_thread=1), dict(precision="fp64")),
    (dict(precision="mixed", targets_per_thread=2), dict(precision="fp64")),
])
def test_lists_of_other_settings_serve(BT, dev, n, leaf, before, then):
    plan, F, k = make(dev, n, leaf)
    call = lambda F, k, **kw: plan.convolve(F, F, BT.Kernel.COULOMB, k, BT.Singularity.SUBTRACTION, **kw)
    if then["precision"] == "fp64":   # the FP64 weight charges come with any FP64 call
        call(F[:1], k[:1], precision="fp64")
    call(F, k, **before)
    got, g = captured(dev, plan, BT, F, k, **then)
    assert torch.isfinite(got).all() and torch.equal(got, call(F, k, **then))
    g.close()
    plan.close()


def test_calls_in_other_forms_leave_a_captured_list_alone(BT, dev):
    """A plan keeps the lists of four orbital counts whatever forms each is called in: a graph over
    one of them stays valid while the other three are called in both precisions and with one and
    two targets per thread, and gives the captured call's result on new values."""
    x, y, z, w, _ = cloud(2001, 7)
    plan = dev.TreecodePlan.for_mesh(*to_cuda(x, y, z, w), theta=0.8, degree=3, source_leaf=130, target_leaf=130)
    gen = torch.Generator().manual_seed(7)
    F = torch.randn((4, 2001), generator=gen, dtype=torch.float64).cuda()
    k = torch.tensor([0.7, 0.9, 1.1, 1.3], dtype=torch.float64, device="cuda")
    SS = BT.Singularity.SUBTRACTION
    s = torch.cuda.Stream()
    G, out = F.clone(), torch.zeros_like(F)
    plan.convolve(G, G, BT.Kernel.COULOMB, k, SS, precision="mixed", out=out)
    torch.cuda.synchronize()
    with dev.Graph.capture(s) as g:
        plan.convolve(G, G, BT.Kernel.COULOMB, k, SS, precision="mixed", out=out, stream=s)
    for norb in (1, 2, 3, 4):
        for kw in (dict(precision="fp64"), dict(precision="mixed", targets_per_thread=1),
                   dict(precision="mixed", targets_per_thread=2)):
            plan.convolve(F[:norb], F[:norb], BT.Kernel.COULOMB, k[:norb], SS, **kw)
    G.copy_(2.0 * F)
    torch.cuda.synchronize()
    g.replay(s)
    torch.cuda.synchronize()
    assert torch.equal(out, plan.convolve(2.0 * F, 2.0 * F, BT.Kernel.COULOMB, k, SS, precision="mixed"))
    g.close()
    plan.close()
