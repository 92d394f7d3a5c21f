"""Tiles of the IHC tensor kernel that it takes without products, where nearly all sums
would have to be taken again: bit for bit the oracle's, with tiles of both kinds in turn."""
import numpy as np
import pytest

from cochlearmodel_gb300 import ihc, native
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

ROWS = 128 * 26 + 45


def _taps(n, tilt=0.0):
    t = np.sinc(0.016 * (np.arange(n) - (n - 1) / 2)) * np.blackman(n + 2)[1:-1]
    t = t * (1.0 + tilt * np.arange(n) / n)
    return (t / t.sum()).astype(np.float32)


def _velocity(kind):
    t = np.arange(ROWS)[:, None]
    rng = np.random.default_rng(3)
    v = 1e-3 * np.sin(2 * np.pi * (t * 0.02 + rng.random((1, 256)))) * (1 + rng.random((1, 256)))
    if kind == "tiny":
        v = v * 1e-27
    elif kind == "turns":  # some tiles of each
        v = v * np.where(t // 900 % 2 == 0, 1.0, 1e-27)
    elif kind == "noise then tone":
        v = np.where(t < 1000, 1e-3 * rng.standard_normal((ROWS, 256)), v)
    return v.astype(np.float32)


@pytest.mark.parametrize("kind", ["null", "tiny", "turns", "noise then tone"])
@pytest.mark.parametrize("n,tilt", [(255, 0.0), (64, 0.0), (257, 0.3)])
@pytest.mark.parametrize("frames", [[(0, ROWS, ROWS, ROWS)],
                                    [(0, 1000, 2900, 2900), (2900, ROWS - 2900, 400, 400)]])
def test_bits(kind, n, tilt, frames):
    """Whole frames; segments that end inside such tiles, a frame of few rows."""
    stage = ihc.IHCStage("cuda:0", ac_taps=_taps(n, tilt))
    v = _velocity(kind)
    fr = np.zeros(len(frames), ihc.FRAME_DTYPE)
    for i, (at, seg, rows, frdp) in enumerate(frames):
        fr[i] = (at, at, rows, rows, seg, frdp, ihc.round64(rows), 0)
    lib = native.load()
    native.check(lib.cgb_ihc_set_run_length(24), "run length")  # many tiles a CTA
    try:
        lam, pot = stage.run(v, fr, ROWS, want_ihc=True)
    finally:
        native.check(lib.cgb_ihc_set_run_length(0), "run length")
    short, _ = stage.run(v, fr, ROWS)
    for f in fr:
        r0, m = int(f["lam_row0"]), int(f["lam_rows"])
        o_pot, o_lam = orc.ihc_lambda(
            v[r0:r0 + m], int(f["seg"]), int(f["frdp"]), int(f["total"]), m,
            stage.ac.astype(np.float64), stage.dc.astype(np.float64), stage.prm.scale,
            stage.nerve.eta_AC, stage.nerve.eta_DC, stage.dmg_host[0].astype(np.float64),
            stage.nerve.aihc(), np.asarray(stage.nerve.spontRate, np.float32),
            stage.nerve.Lambda_SAT, mode=2)
        assert np.array_equal(pot[r0:r0 + m].view(np.uint32), o_pot[:m].view(np.uint32))
        assert np.array_equal(lam[:, r0:r0 + m].view(np.uint32), o_lam.view(np.uint32))
        assert np.array_equal(short[:, r0:r0 + m].view(np.uint32), o_lam.view(np.uint32))
