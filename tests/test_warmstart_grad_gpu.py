"""Training kernels of the warm-start network: weight gradients and the backward
pass against FP64 sums of the same BF16 factors, the forward pass against the
fused inference."""
import ctypes as C

import numpy as np
import pytest
import torch

from cochlearmodel_gb300 import native, warmstart

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


# fewer records than SMs, one more, and several for each
@pytest.mark.parametrize("n", [1, 2, 153, 500])
def test_forward_and_backward_layers(n):
    g = torch.Generator(device=D).manual_seed(n)
    net = warmstart.WarmStartNet(D, seed=n)
    net.params += 0.05 * torch.randn(net.n_params, generator=g, device=D)
    net.pack()
    feat = torch.zeros(n, 280, 8, dtype=torch.bfloat16, device=D)
    feat[:, 8:264] = torch.randn(n, 256, 8, generator=g, device=D).to(torch.bfloat16)
    buf = net.buffers(n)
    out = net.forward(feat, buf)
    assert torch.equal(out.view(torch.int32), net.infer(feat).view(torch.int32))

    w = net.params.to(torch.bfloat16).double()
    size = [2560, 64, 20480, 64, 20480, 64, 320, 1]
    W1, b1, W2, b2, W3, b3, W4, b4 = torch.split(w, size)
    bias = dict(zip((1, 2, 3), torch.split(net.params.double(), size)[1:6:2]))
    eps = 2.0 ** -8 + 2.0 ** -16  # BF16 half ulp; a sum of 320 products in FP32 on top:
    acc = 340 * 2.0 ** -23

    def close(got, want, size):
        return bool(((got - want).abs() <= eps * want.abs() + acc * size).all())

    # each hidden layer from the one before as the kernel stored it
    h = [feat[:, 8:264].double(), *rows64(buf["hid"]).double()]
    for layer, W, cin in ((1, W1, 8), (2, W2, 64), (3, W3, 64)):
        W = W.reshape(5, 64, cin)
        sums = lambda x, w: sum(  # noqa: E731
            torch.nn.functional.pad(x, (0, 0, 2, 2))[:, t:t + 256] @ w[t].T for t in range(5))
        assert close(h[layer], (sums(h[layer - 1], W) + bias[layer]).relu(),
                     sums(h[layer - 1].abs(), W.abs()) + bias[layer].abs()), layer

    buf["dout"][:, :, 0] = torch.randn(n, 256, generator=g, device=D).to(torch.bfloat16)
    p = native.ptr
    native.check(net.lib.cgb_ws_backward_dev(
        p(net.blobT), p(buf["dout"]), p(buf["hid"]), n, p(buf["dpre"]),
        C.c_void_p(torch.cuda.current_stream().cuda_stream)), "cgb_ws_backward_dev")
    d = [*rows64(buf["dpre"]).double(), buf["dout"][:, :, :1].double()]
    for layer, W, cout in ((2, W4, 1), (1, W3, 64), (0, W2, 64)):
        W = W.reshape(5, cout, 64)
        sums = lambda x, w: sum(  # noqa: E731
            torch.nn.functional.pad(x, (0, 0, 2, 2))[:, 4 - t:260 - t] @ w[t] for t in range(5))
        on = h[layer + 1] > 0
        assert close(d[layer], sums(d[layer + 1], W) * on,
                     sums(d[layer + 1].abs(), W.abs()) * on), layer


@pytest.mark.parametrize("n", [1, 129, 700])
def test_mean_loss(n):
    g = torch.Generator(device=D).manual_seed(n)
    net = warmstart.WarmStartNet(D, seed=n)
    feat = torch.zeros(n, 280, 8, dtype=torch.bfloat16, device=D)
    feat[:, 8:264] = torch.randn(n, 256, 8, generator=g, device=D).to(torch.bfloat16)
    target = torch.randn(n, 256, generator=g, device=D)
    buf = net.buffers(n)
    loss, grad = net.gradients(feat, target, buf)
    e = net.s_out * buf["out"] - target  # FP32, as the kernel forms it
    want = float(np.sum(np.square(e.cpu().numpy().astype(np.float64)))) / (n * 256)
    # an FP32 product and difference (two roundings) per term, or one if contracted
    assert abs(float(loss) - want) <= 2.0 ** -21 * want
    assert abs(float(loss) - float(buf["loss"].sum()) / (n * 256)) <= (n + 16) * 2.0 ** -52 * want


@pytest.mark.parametrize("n", [1, 151, 153, 400])
def test_overlapped_step_is_the_separate_calls(n):
    """The one-call step, whose kernels overlap, on changing inputs and from a
    graph, against its kernels called one by one: the same bits."""
    g = torch.Generator(device=D).manual_seed(n)
    net = warmstart.WarmStartNet(D, seed=n)
    feat = torch.zeros(n, 280, 8, dtype=torch.bfloat16, device=D)
    target = torch.zeros(n, 256, device=D)
    buf, ref = net.buffers(n), net.buffers(n)
    net.gradients(feat, target, buf)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        net.gradients(feat, target, buf)
    ref["partial"] = torch.zeros_like(buf["partial"])
    parts = buf["partial"].shape[0]
    p = native.ptr
    for i in range(8):
        feat[:, 8:264] = torch.randn(n, 256, 8, generator=g, device=D).to(torch.bfloat16)
        target.normal_(generator=g)
        graph.replay() if i % 2 else net.gradients(feat, target, buf)
        st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        net.forward(feat, ref)
        native.check(net.lib.cgb_ws_loss_dev(p(ref["out"]), p(target), n, net.s_out,
                                             p(ref["dout"]), p(ref["loss"]), st), "loss")
        native.check(net.lib.cgb_ws_backward_dev(p(net.blobT), p(ref["dout"]), p(ref["hid"]), n,
                                                 p(ref["dpre"]), st), "backward")
        native.check(net.lib.cgb_ws_wgrad_dev(p(feat), p(ref["hid"]), p(ref["dpre"]),
                                              p(ref["dout"]), n, p(ref["partial"]), parts,
                                              p(ref["grad"]), st), "wgrad")
        for k in ("hid", "out", "dout", "dpre", "loss", "grad"):
            assert torch.equal(buf[k], ref[k]), (i, k)
