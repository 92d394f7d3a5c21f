"""The IHC stage's FP32 kernel, which takes the filters that the tensor kernel does not
(fewer than 64 taps, a DC filter whose taps differ): run lengths, the tables' upload, host
mirrors and the entry point that allocates nothing, bit for bit the oracle's."""
import ctypes as C

import numpy as np
import pytest

from cochlearmodel_gb300 import ihc, native
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

ROWS = 9000


def _stage(kind):
    n = 255 if kind == "uneven DC" else 48
    t = np.sinc(0.016 * (np.arange(n) - (n - 1) / 2)) * np.hamming(n)
    stage = ihc.IHCStage("cuda:0", ac_taps=(t / t.sum()).astype(np.float32))
    if kind == "uneven DC":
        stage.dc = np.hanning(202)[1:-1].astype(np.float32) / np.float32(100.5)
    return stage


def _velocity():
    rng = np.random.default_rng(8)
    t = np.arange(ROWS)[:, None] / 1e5
    f = (300 + 30 * np.arange(256))[None, :]
    return (1e-3 * np.sin(2 * np.pi * f * t) * (1 + rng.random((1, 256)))).astype(np.float32)


def _frames():
    fr = np.zeros(2, ihc.FRAME_DTYPE)
    fr[0] = (0, 0, 5000, 5000, 1000, 5000, ihc.round64(5000), 0)
    fr[1] = (5000, 5000, 4000, 4000, 4000, 4000, ihc.round64(4000), 0)
    return fr


@pytest.fixture(scope="module", params=["48 taps", "uneven DC"])
def case(request):
    stage, v, fr = _stage(request.param), _velocity(), _frames()
    want = np.concatenate([orc.ihc_lambda(
        v[f["v_row0"]:f["v_row0"] + f["rows"]], int(f["seg"]), int(f["frdp"]), int(f["total"]),
        int(f["lam_rows"]), stage.ac.astype(np.float64), stage.dc.astype(np.float64),
        stage.prm.scale, stage.nerve.eta_AC, stage.nerve.eta_DC,
        stage.dmg_host[0].astype(np.float64), stage.nerve.aihc(),
        np.asarray(stage.nerve.spontRate, np.float32), stage.nerve.Lambda_SAT, mode=2)[1]
        for f in fr], axis=1)
    return stage, v, fr, want


def _same(lam, want):
    assert np.array_equal(np.asarray(lam).view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("run", [0, 1, 3, 8, 32])
def test_run_lengths(case, run):
    stage, v, fr, want = case
    lib = native.load()
    native.check(lib.cgb_ihc_set_run_length(run), "run length")
    try:
        _same(stage.run(v, fr, ROWS)[0], want)
    finally:
        native.check(lib.cgb_ihc_set_run_length(0), "run length")


def test_launch_keeps_the_upload(case):
    """A launch after the run length was changed takes the one of its upload."""
    import torch
    stage, v, fr, want = case
    lib, d_v = native.load(), torch.from_numpy(v).cuda()
    try:
        for run in (8, 1):
            chunk, = stage.upload_chunks([fr], ROWS, ROWS)
            native.check(lib.cgb_ihc_set_run_length(run), "run length")
            lam = torch.full((3, ROWS, 256), np.nan, device="cuda:0")
            stage.launch_chunk(d_v, chunk, lam, torch.cuda.current_stream())
            _same(lam.cpu().numpy(), want)
    finally:
        native.check(lib.cgb_ihc_set_run_length(0), "run length")


def test_host_mirror(case):
    import torch
    stage, v, fr, want = case
    chunk, = stage.upload_chunks([fr], ROWS, ROWS)
    lam = torch.full((3, ROWS, 256), np.nan, device="cuda:0")
    mirror = torch.full((3, ROWS, 256), np.nan, pin_memory=True)
    stage.launch_chunk(torch.from_numpy(v).cuda(), chunk, lam, torch.cuda.current_stream(), mirror)
    torch.cuda.synchronize()
    _same(lam.cpu().numpy(), want)
    _same(mirror.numpy(), want)


def test_noalloc(case):
    import torch
    stage, v, fr, want = case
    d_v = torch.from_numpy(v).cuda()
    lam = torch.full((3, ROWS, 256), np.nan, device="cuda:0")
    status = torch.zeros(4, dtype=torch.int32, device="cuda:0")
    p = native.ptr
    native.check(native.load().cgb_ihc_lambda_noalloc_dev(
        p(d_v), ROWS, p(fr), len(fr), p(stage.ac), len(stage.ac), p(stage.dc), len(stage.dc),
        C.byref(stage.prm), p(stage.dmg), int(stage.dmg.shape[0]), p(stage.aihc), p(lam), ROWS, None,
        p(status), C.c_void_p(torch.cuda.current_stream().cuda_stream)), "noalloc")
    _same(lam.cpu().numpy(), want)
    assert int(status[0].item()) == 0
