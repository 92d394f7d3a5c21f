"""A wait of the training kernels that runs out: the results are NaN, and the next
step is as if it had not been."""
import pytest
import torch

from cochlearmodel_gb300 import native, warmstart

pytestmark = pytest.mark.gpu
D = "cuda:0"


# one record a CTA, and several
@pytest.mark.parametrize("n", [1, 40, 700])
def test_wait_runs_out(n):
    g = torch.Generator(device=D).manual_seed(n)
    net = warmstart.WarmStartNet(D, seed=n)
    feat = torch.zeros(n, 280, 8, dtype=torch.bfloat16, device=D)
    feat[:, 8:264] = torch.randn(n, 256, 8, generator=g, device=D).to(torch.bfloat16)
    target = torch.randn(n, 256, generator=g, device=D)
    buf = net.buffers(n)
    loss, grad = (t.clone() for t in net.gradients(feat, target, buf))
    assert torch.isfinite(loss) and torch.isfinite(grad).all()
    native.check(net.lib.cgb_ws_set_fault_injection(1), "fault injection")
    try:
        bad_loss, bad_grad = net.gradients(feat, target, buf)
        torch.cuda.synchronize()
    finally:
        native.check(net.lib.cgb_ws_set_fault_injection(0), "fault injection")
    assert torch.isnan(bad_loss) and torch.isnan(bad_grad).all()
    for k in ("out", "dout", "dpre"):  # (dout: the output's channel)
        t = buf[k][..., 0] if k == "dout" else buf[k]
        assert torch.isnan(t.float()).all(), k
    again, grad2 = net.gradients(feat, target, buf)
    assert torch.equal(again, loss) and torch.equal(grad2, grad)
