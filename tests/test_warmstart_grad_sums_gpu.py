"""Weight gradients over many records of one sign: as accurate as one record's."""
import ctypes as C

import pytest
import torch

from cochlearmodel_gb300 import native, warmstart

pytestmark = pytest.mark.gpu
D = "cuda:0"


def _rows64(x):
    r = torch.arange(256, device=x.device)[:, None]
    c = torch.arange(8, device=x.device)[None, :] ^ (r & 7)
    return x.reshape(*x.shape[:-1], 8, 8)[..., r, c, :].reshape(x.shape).contiguous()


def _products(dpre, inp):
    """[5, out, in] of dpre [n, 256, out], inp [n, 256, in], in blocks of records."""
    out = 0.0
    for a, b in zip(dpre.split(128), inp.split(128)):
        p = torch.nn.functional.pad(b.double(), (0, 0, 2, 2))
        out = out + torch.stack([torch.einsum("npo,npi->oi", a.double(), p[:, t:t + 256])
                                 for t in range(5)])
    return out


# one slot; rows for some, all and none of the slots' low parts; many records a slot
@pytest.mark.parametrize("n, parts", [(300, 1), (130, 60), (256, 256), (2560, 304), (2560, 50)])
def test_same_sign(n, parts):
    g = torch.Generator(device=D).manual_seed(n + parts)
    pos = lambda *s: torch.rand(*s, generator=g, device=D).to(torch.bfloat16) + 1  # noqa: E731
    feat = torch.zeros(n, 280, 8, dtype=torch.bfloat16, device=D)
    feat[:, 8:264] = pos(n, 256, 8)
    hid, dpre = pos(3, n, 256, 64), pos(3, n, 256, 64)
    dout = torch.zeros(n, 256, 8, dtype=torch.bfloat16, device=D)
    dout[:, :, 0] = pos(n, 256)
    lib = native.load()
    count = lib.cgb_ws_param_count()
    partial = torch.full((parts, count), float("nan"), device=D)
    grad = torch.full((count,), float("nan"), device=D)
    p = native.ptr
    k_hid, k_dpre = _rows64(hid), _rows64(dpre)
    native.check(lib.cgb_ws_wgrad_dev(p(feat), p(k_hid), p(k_dpre), p(dout), n, p(partial), parts,
                                      p(grad), C.c_void_p(torch.cuda.current_stream().cuda_stream)),
                 "cgb_ws_wgrad_dev")
    want = []
    for o, i in zip([*dpre, dout[:, :, :1]], [feat[:, 8:264], *hid]):
        want += [_products(o, i).reshape(-1), o.double().sum(dim=(0, 1))]
    want = torch.cat(want)
    # the products are exact in FP32; a record's sum takes one rounding (or cut, 2^-23) per
    # term of a step's 16 and per step of 17, its slot's one more and the last sum one
    tol = (16 + 17 + 2) * 2.0 ** -23
    err = ((grad.double() - want).abs() / want).max().item()
    assert err <= tol, (err, tol)


@pytest.mark.parametrize("n, parts", [(120, 100), (120, 40), (10, 10)])
def test_out_of_range(n, parts):
    """A product past the FP32 range is an infinity in its gradients and nothing elsewhere."""
    feat = torch.zeros(n, 280, 8, dtype=torch.bfloat16, device=D)
    hid = torch.ones(3, n, 256, 64, dtype=torch.bfloat16, device=D)
    dpre = torch.ones(3, n, 256, 64, dtype=torch.bfloat16, device=D)
    dout = torch.zeros(n, 256, 8, dtype=torch.bfloat16, device=D)
    hid[0, n // 2, 100, 5], dpre[1, n // 2, 100, 7] = 4.0, 3e38  # layer 2, the middle tap
    lib = native.load()
    count = lib.cgb_ws_param_count()
    partial = torch.zeros(parts, count, device=D)
    grad = torch.zeros(count, device=D)
    p = native.ptr
    k_hid, k_dpre = _rows64(hid), _rows64(dpre)
    native.check(lib.cgb_ws_wgrad_dev(p(feat), p(k_hid), p(k_dpre), p(dout), n, p(partial), parts,
                                      p(grad), C.c_void_p(torch.cuda.current_stream().cuda_stream)),
                 "cgb_ws_wgrad_dev")
    w2 = grad[5 * 64 * 8 + 64:][:5 * 64 * 64].reshape(5, 64, 64)
    assert w2[2, 7, 5].item() == float("inf")
    w2[2, 7, 5] = 0.0
    assert torch.isfinite(grad).all()


@pytest.mark.parametrize("n", [64, 256, 1000])
def test_slots_of_the_network(n):
    """gradients() gives the slots room for both parts, and no more."""
    net = warmstart.WarmStartNet(D, seed=n)
    feat = torch.zeros(n, 280, 8, dtype=torch.bfloat16, device=D)
    target = torch.zeros(n, 256, device=D)
    buf = net.buffers(n)
    net.gradients(feat, target, buf)
    sms = torch.cuda.get_device_properties(D).multi_processor_count
    assert buf["partial"].shape[0] == min(n, 2 * (sms // 3))
