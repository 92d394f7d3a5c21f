"""Frames on both sides of the rule that gives them to one IHC kernel or the other: short
ones and few, segments that end inside the tiles; bit for bit the oracle's."""
import numpy as np
import pytest

from cochlearmodel_gb300 import ihc
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _taps(n):
    t = np.sinc(0.016 * (np.arange(n) - (n - 1) / 2)) * np.hamming(n)
    return (t / t.sum()).astype(np.float32)


@pytest.mark.parametrize("n_taps", [64, 255])
@pytest.mark.parametrize("count,rows,seg", [(1, 2, 2), (1, 30, 30), (40, 25, 25), (3, 100, 100),
                                            (20, 100, 100), (30, 300, 300), (1, 3000, 50),
                                            (1, 3000, 100), (1, 12000, 100), (4, 700, 130)])
def test_bits(n_taps, count, rows, seg):
    stage = ihc.IHCStage("cuda:0", ac_taps=_taps(n_taps))
    v = (1e-3 * np.random.default_rng(rows).standard_normal((count * rows, 256))).astype(np.float32)
    fr = np.zeros(count, ihc.FRAME_DTYPE)
    for i in range(count):
        fr[i] = (i * rows, i * rows, rows, rows, seg, rows, ihc.round64(rows), 0)
    lam, pot = stage.run(v, fr, count * rows, want_ihc=True)
    for i in sorted({0, count // 2, count - 1}):
        at, f = i * rows, fr[i]
        o_pot, o_lam = orc.ihc_lambda(
            v[at:at + rows], int(f["seg"]), int(f["frdp"]), int(f["total"]), rows,
            stage.ac.astype(np.float64), stage.dc.astype(np.float64), stage.prm.scale,
            stage.nerve.eta_AC, stage.nerve.eta_DC, stage.dmg_host[0].astype(np.float64),
            stage.nerve.aihc(), np.asarray(stage.nerve.spontRate, np.float32),
            stage.nerve.Lambda_SAT, mode=2)
        assert np.array_equal(pot[at:at + rows].view(np.uint32), o_pot[:rows].view(np.uint32))
        assert np.array_equal(lam[:, at:at + rows].view(np.uint32), o_lam.view(np.uint32))
