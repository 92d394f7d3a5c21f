"""The JND kernels' two ways to fetch their windows (asynchronous copies for few
intervals, registers for many), window lengths around their blocks of rows, and
rate planes that allow 16-byte copies or not."""
import ctypes as C

import numpy as np
import pytest

from cochlearmodel_gb300 import native

pytestmark = pytest.mark.gpu

F_REL_FP64 = 1e-6  # FP32 terms, compensated sums


def _sums(lam, rows, n_int, nodes, head, length, dA, ref):
    """cgb_jnd_dev on rate planes [3][rows][256] at any address."""
    import torch
    lib = native.load()
    d = lam.device
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(d)
    dA_d, ref_d, nihc = t(dA), t(ref), t(np.full(256, 117.1875))
    W = np.asarray([0.61, 0.23, 0.16], np.float32)
    ra = torch.zeros((3, n_int), dtype=torch.float64, device=d)
    ai, mr = torch.zeros_like(ra), torch.zeros((3, n_int, 256), dtype=torch.float64, device=d)
    native.check(lib.cgb_jnd_dev(
        native.ptr(lam), rows, n_int, nodes, head, length, native.ptr(dA_d), native.ptr(ref_d),
        native.ptr(nihc), native.ptr(W), 1e5, 2e4, native.ptr(ra), native.ptr(ai),
        native.ptr(mr), C.c_void_p(torch.cuda.current_stream(d).cuda_stream)), "cgb_jnd_dev")
    return ra.cpu().numpy(), ai.cpu().numpy(), mr.cpu().numpy()


@pytest.mark.parametrize("length", [1, 7, 8, 31, 32, 33, 129, 500])
def test_fetches_agree(length):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    n, nodes, head = 3, length + 5, 2
    rng = np.random.default_rng(length)
    lam = rng.uniform(0.1, 400.0, (3, n * nodes, 256)).astype(np.float32)
    dA, ref = np.array([1e-3, 2e-2, 0.0]), np.array([2, 2, 2], np.int32)
    d = torch.from_numpy(lam).to("cuda:0")
    few = _sums(d, n * nodes, n, nodes, head, length, dA, ref)

    # the planes one float further: no 16-byte copies
    off = torch.empty(d.numel() + 1, dtype=torch.float32, device=d.device)[1:]
    off.copy_(d.reshape(-1))
    assert off.data_ptr() % 16 == 4
    for a, b in zip(few, _sums(off, n * nodes, n, nodes, head, length, dA, ref)):
        assert np.array_equal(a, b)

    # the same intervals many times over: past the rule, loads to registers
    reps = 200
    many = d.repeat(1, reps, 1)
    refs = np.concatenate([ref + i * n for i in range(reps)]).astype(np.int32)
    big = _sums(many, n * nodes * reps, n * reps, nodes, head, length, np.tile(dA, reps), refs)
    for a, b in zip(few, big):
        assert np.array_equal(np.broadcast_to(a[:, None], (3, reps) + a.shape[1:]),
                              b.reshape((3, reps) + a.shape[1:]))

    # and both against 64 bits
    win = lam.reshape(3, n, nodes, 256)[:, :, head:head + length].astype(np.float64)
    W = np.asarray([0.61, 0.23, 0.16], np.float32).astype(np.float64)
    T = 2e4 / 1e5
    for i in range(2):
        c, r = win[:, i], win[:, 2]
        m, mr = c.mean(1), r.mean(1)
        want_ra = W * (117.1875 * T * ((m - mr) / dA[i]) ** 2 / mr).sum(1)
        want_ai = W * (117.1875 * (T / (length / 1e5)) * ((c - r) ** 2 / r).sum(1) /
                       (1e5 * dA[i] ** 2)).sum(1)
        assert np.abs(few[0][:, i] / want_ra - 1).max() <= F_REL_FP64
        assert np.abs(few[1][:, i] / want_ai - 1).max() <= F_REL_FP64
        assert np.abs(few[2][:, i] / m - 1).max() <= F_REL_FP64
    assert not few[0][:, 2].any() and not few[1][:, 2].any()
