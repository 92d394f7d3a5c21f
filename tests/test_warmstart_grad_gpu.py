"""Weight gradients of the warm-start network against FP64 sums of the same
BF16 factors."""
import ctypes as C

import numpy as np
import pytest
import torch

from cochlearmodel_gb300 import native

pytestmark = pytest.mark.gpu
D = "cuda:0"


def rows64(x):
    """[..., 256, 64] as the kernels keep it: chunk c of row r at c ^ (r & 7)."""
    r = torch.arange(256, device=x.device)[:, None]
    c = torch.arange(8, device=x.device)[None, :] ^ (r & 7)
    return x.reshape(*x.shape[:-1], 8, 8)[..., r, c, :].reshape(x.shape).contiguous()


def products(dpre, inp):
    """[5, out, in] of dpre [n, 256, out], inp [n, 256, in]."""
    p = torch.nn.functional.pad(inp, (0, 0, 2, 2))
    return torch.stack([torch.einsum("npo,npi->oi", dpre, p[:, t:t + 256]) for t in range(5)])


# one record; fewer and more records than slots; odd numbers of records a slot
@pytest.mark.parametrize("n, parts", [(0, 2), (1, 1), (1, 304), (2, 1), (7, 3), (51, 304), (103, 50)])
def test_weight_gradients_match_fp64(n, parts):
    g = torch.Generator(device=D).manual_seed(n + parts)
    rnd = lambda *s: torch.randn(*s, generator=g, device=D).to(torch.bfloat16)  # noqa: E731
    feat = torch.zeros(n, 280, 8, dtype=torch.bfloat16, device=D)
    feat[:, 8:264] = rnd(n, 256, 8)
    hid, dpre = rnd(3, n, 256, 64).relu(), rnd(3, n, 256, 64)
    dout = torch.zeros(n, 256, 8, dtype=torch.bfloat16, device=D)
    dout[:, :, 0] = rnd(n, 256)
    lib = native.load()
    count = lib.cgb_ws_param_count()
    partial = torch.full((parts, count), float("nan"), device=D)
    grad = torch.full((count,), float("nan"), device=D)
    k_hid, k_dpre = rows64(hid), rows64(dpre)
    one = torch.zeros(16, dtype=torch.uint8, device=D)  # (an empty tensor has no address)
    p = lambda t: native.ptr(t if t.numel() else one)  # noqa: E731
    native.check(lib.cgb_ws_wgrad_dev(p(feat), p(k_hid), p(k_dpre), p(dout), n, p(partial), parts,
                                      p(grad), C.c_void_p(torch.cuda.current_stream().cuda_stream)),
                 "cgb_ws_wgrad_dev")
    d = dpre.double()
    inputs = [feat[:, 8:264].double(), *hid.double()]
    outs = [*d, dout[:, :, :1].double()]
    want, size = [], []
    for o, i in zip(outs, inputs):
        want += [products(o, i).reshape(-1), o.sum(dim=(0, 1))]
        size += [products(o.abs(), i.abs()).reshape(-1), o.abs().sum(dim=(0, 1))]
    want, size = torch.cat(want).cpu().numpy(), torch.cat(size).cpu().numpy()
    # the products are exact in FP32; a sum takes one rounding (or truncation, 2^-23)
    # per term of a step's 16 and per step, and one per slot
    tol = (16 + 17 * max(n, 1) + parts) * 2.0 ** -23 * size
    got = grad.double().cpu().numpy()
    assert np.all(np.abs(got - want) <= tol), np.max(np.abs(got - want) / np.maximum(tol, 1e-30))
