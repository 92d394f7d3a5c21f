"""The IHC / lambda stage with its AC filter as digit products on the tensor
cores: bit for bit the oracle's compensated FIR, at the edges of the kernel's
tiles, segments and filter lengths and on inputs that make its scales fail."""
import numpy as np
import pytest

from cochlearmodel_gb300 import ihc, native
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

ROWS = 1100


def _stage(taps=None, scale=1.0):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    nerve = ihc.NerveConfig(scale=scale)
    return ihc.IHCStage("cuda:0", nerve, ihc_profiles=np.stack(
        [np.full(256, 8.0, np.float32), np.linspace(8, 5, 256, dtype=np.float32)]), ac_taps=taps)


def _taps(n, asymmetric=False):
    t = np.sinc(2 * 800.0 / 1e5 * (np.arange(n) - (n - 1) / 2)) * (0.54 - 0.46 * np.cos(
        2 * np.pi * np.arange(n) / (n - 1)))
    if asymmetric:
        t = t * (1.0 + 0.3 * np.arange(n) / (n - 1))
    return (t / t.sum()).astype(np.float32)


def _velocity(kind):
    rng = np.random.default_rng(7)
    t = np.arange(ROWS)[:, None] / 1e5
    f = 300 + 40 * np.arange(256)[None, :]
    v = 1e-3 * np.sin(2 * np.pi * f * t) * (1 + rng.random((1, 256)))
    if kind == "noise":
        v = rng.standard_normal((ROWS, 256)) * 1e-2
    elif kind == "wide":  # magnitudes over ten decades from row to row
        v = rng.standard_normal((ROWS, 256)) * np.exp(rng.uniform(-20, 3, (ROWS, 256)))
    elif kind == "steps":  # silence, a drop by 1e-20, subnormal sections
        v[300:420] = 0.0
        v[600:] *= 1e-20
        v[:, 9] = 1e-40
    return v.astype(np.float32)


def _check(stage, v, frames):
    fr = np.zeros(len(frames), ihc.FRAME_DTYPE)
    for i, x in enumerate(frames):
        fr[i] = x
    lam_rows = int((fr["lam_row0"] + fr["lam_rows"]).max())
    lam, pot = stage.run(v, fr, lam_rows, want_ihc=True)
    for f in fr:
        r0, n = int(f["lam_row0"]), int(f["lam_rows"])
        o_ihc, o_lam = orc.ihc_lambda(
            v[f["v_row0"]:f["v_row0"] + f["rows"]], int(f["seg"]), int(f["frdp"]),
            int(f["total"]), n, stage.ac.astype(np.float64), stage.dc.astype(np.float64),
            stage.prm.scale, stage.nerve.eta_AC, stage.nerve.eta_DC,
            stage.dmg_host[f["ihc_profile"]].astype(np.float64), stage.nerve.aihc(),
            np.asarray(stage.nerve.spontRate, np.float32), stage.nerve.Lambda_SAT, mode=2)
        assert np.array_equal(pot[r0:r0 + n].view(np.uint32), o_ihc[:n].view(np.uint32))
        assert np.array_equal(lam[:, r0:r0 + n].view(np.uint32), o_lam.view(np.uint32))


@pytest.mark.parametrize("n", [63, 64, 128, 254, 255, 256, 257, 258])
@pytest.mark.parametrize("asymmetric", [False, True])
def test_filter_lengths(n, asymmetric):
    """The shortest and longest filters of the kernel and their neighbours on
    the FP32 pipe, odd and even, symmetric or not."""
    _check(_stage(_taps(n, asymmetric)), _velocity("tones"),
           [(0, 0, 700, 700, 350, 700, 704, 0), (700, 700, 400, 300, 400, 300, 448, 1)])


@pytest.mark.parametrize("seg,frdp,rows,lam_rows", [
    (128, 512, 512, 512), (127, 500, 520, 500), (129, 640, 700, 640), (1, 300, 300, 300),
    (64, 200, 300, 280), (500, 1000, 1100, 1000), (1000, 1000, 1100, 1100), (255, 257, 260, 257),
    (1100, 1100, 1100, 1)])
def test_segments_and_tiles(seg, frdp, rows, lam_rows):
    """Segments shorter and longer than a tile, ends inside a tile, the rule's
    switch to the frame total."""
    _check(_stage(), _velocity("tones"),
           [(0, 0, rows, lam_rows, seg, frdp, ihc.round64(rows), 0)])


@pytest.mark.parametrize("kind", ["noise", "wide", "steps"])
@pytest.mark.parametrize("scale", [1.0, 0.37])
def test_magnitudes(kind, scale):
    _check(_stage(scale=scale), _velocity(kind),
           [(0, 0, 1100, 1100, 1100, 1100, 1152, 0)])


def test_infinities_and_nan():
    """Values that no scale holds take the compensated FIR: infinities, NaN and
    products past the FP32 range."""
    v = _velocity("tones")
    v[400, 3], v[500, 100], v[450, 200] = np.inf, np.nan, 3e38
    _check(_stage(), v, [(0, 0, 1100, 1100, 1100, 1100, 1152, 0)])


@pytest.mark.parametrize("seg", [1100, 300])
@pytest.mark.parametrize("decades", [6, 12])
def test_onsets(seg, decades):
    """Velocity that grows from nothing by many orders of magnitude within a
    segment's first tiles, as a solved one does: more points below the digits'
    resolution than the list holds, beside rows that the products do give."""
    rise = np.minimum((np.arange(ROWS) % seg) / 150.0, 1.0)[:, None] - 1.0
    v = _velocity("tones") * 10.0 ** (decades * rise * (np.arange(256)[None, :] / 255))
    _check(_stage(), v.astype(np.float32), [(0, 0, 1100, 1100, seg, 1100, 1152, 0)])


def test_launch_of_other_filters_than_uploaded():
    """A launch on tables that were uploaded for another filter, longer than the
    kernel's: an error, and no launch."""
    import torch
    stage = _stage()
    fr = np.array([(0, 0, 512, 512, 512, 512, 512, 0)], ihc.FRAME_DTYPE)
    chunk, = stage.upload_chunks([fr], 512, 512)
    v = torch.zeros((512, 256), device="cuda:0")
    lam = torch.zeros((3, 512, 256), device="cuda:0")
    stage.ac = _taps(300)
    with pytest.raises(native.CGBError, match="not the filters that were uploaded"):
        stage.launch_chunk(v, chunk, lam, torch.cuda.current_stream())
