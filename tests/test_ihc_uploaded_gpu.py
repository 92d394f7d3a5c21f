"""A launch on uploaded IHC tables: those of its own filters and frames, or an error."""
import numpy as np
import pytest

from cochlearmodel_gb300 import ihc, native

pytestmark = pytest.mark.gpu


def _taps(n, tilt=0.0):
    t = np.sinc(0.016 * (np.arange(n) - (n - 1) / 2)) * np.hamming(n)
    t = t * (1.0 + tilt * np.arange(n))
    return (t / t.sum()).astype(np.float32)


def _frames(*lengths):
    fr = np.zeros(len(lengths), ihc.FRAME_DTYPE)
    at = 0
    for i, n in enumerate(lengths):
        fr[i] = (at, at, n, n, n, n, ihc.round64(n), 0)
        at += n
    return fr


def _uploaded(n_ac, frames):
    stage = ihc.IHCStage("cuda:0", ac_taps=_taps(n_ac))
    rows = int(frames["rows"].sum())
    return stage, stage.upload_chunks([frames], rows, rows)[0]


def _launch(stage, chunk, v):
    import torch
    lam = torch.full((3, v.shape[0], 256), np.nan, device="cuda:0")
    stage.launch_chunk(v, chunk, lam, torch.cuda.current_stream())
    torch.cuda.synchronize()
    assert int(stage.status[0].item()) == 0
    return lam


def _velocity(rows):
    import torch
    g = torch.Generator(device="cuda:0").manual_seed(rows)
    return 1e-3 * torch.randn(rows, 256, generator=g, device="cuda:0")


# both kernels, shorter and longer filters than uploaded, to the other kernel and not
@pytest.mark.parametrize("uploaded,launched", [(255, 128), (64, 257), (255, 300), (255, 63),
                                               (63, 40), (63, 255), (300, 301)])
def test_other_ac_length(uploaded, launched):
    stage, chunk = _uploaded(uploaded, _frames(512))
    stage.ac = _taps(launched)
    with pytest.raises(native.CGBError, match="not the filters|scratch buffer too small"):
        _launch(stage, chunk, _velocity(512))


@pytest.mark.parametrize("n_ac", [255, 63])
@pytest.mark.parametrize("n_dc", [199, 100])
def test_other_dc_length(n_ac, n_dc):
    stage, chunk = _uploaded(n_ac, _frames(512))
    stage.dc = stage.dc[:n_dc].copy()
    with pytest.raises(native.CGBError, match="not the filters"):
        _launch(stage, chunk, _velocity(512))


@pytest.mark.parametrize("n_ac", [255, 63])
@pytest.mark.parametrize("other", [(512,), (512, 512, 512), (512, 4000)])
def test_other_frames(n_ac, other):
    stage, chunk = _uploaded(n_ac, _frames(512, 512))
    with pytest.raises(native.CGBError, match="not the frames|scratch buffer too small"):
        _launch(stage, (_frames(*other), *chunk[1:]), _velocity(5000))


@pytest.mark.parametrize("n_ac", [255, 63])
def test_taps_are_the_uploaded_ones(n_ac):
    """The order that a symmetric filter is summed in follows the uploaded taps, not
    those that the launch names."""
    stage, chunk = _uploaded(n_ac, _frames(700, 700))
    v = _velocity(1400)
    want = _launch(stage, chunk, v)
    stage.ac = _taps(n_ac, tilt=0.01)
    assert np.array_equal(_launch(stage, chunk, v).cpu().numpy(), want.cpu().numpy())
