"""The AC filter on the tensor cores where its digit sums are largest and where the digits
leave most of the velocity: bit for bit the oracle's compensated sum."""
import numpy as np
import pytest

from cochlearmodel_gb300 import ihc
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

ROWS = 1500


def _check(taps, v):
    stage = ihc.IHCStage("cuda:0", ac_taps=np.asarray(taps, np.float32))
    v = np.ascontiguousarray(v, np.float32)
    rows = len(v)
    fr = np.array([(0, 0, rows, rows, rows, rows, ihc.round64(rows), 0)], ihc.FRAME_DTYPE)
    lam, pot = stage.run(v, fr, rows, want_ihc=True)
    o_pot, o_lam = orc.ihc_lambda(
        v, rows, rows, int(fr["total"][0]), rows, stage.ac.astype(np.float64),
        stage.dc.astype(np.float64), stage.prm.scale, stage.nerve.eta_AC, stage.nerve.eta_DC,
        stage.dmg_host[0].astype(np.float64), stage.nerve.aihc(),
        np.asarray(stage.nerve.spontRate, np.float32), stage.nerve.Lambda_SAT, mode=2)
    bad = np.argwhere(pot.view(np.uint32) != o_pot[:rows].view(np.uint32))
    assert len(bad) == 0, (len(bad), bad[:4])
    assert np.array_equal(lam.view(np.uint32), o_lam.view(np.uint32))


def _sinc(n, fc=800.0):
    t = np.sinc(2 * fc / 1e5 * (np.arange(n) - (n - 1) / 2)) * np.hamming(n)
    return t / t.sum()


def _slow():
    """Nearly constant: the digit sums of all rows of the window in one direction."""
    t, s = np.arange(ROWS)[:, None], np.arange(256)[None, :]
    return (0.7 + 0.29 * s / 255) * (1 + 1e-4 * np.sin(2 * np.pi * t / 900 + s))


# a moving average (digit sums past 2^24 in the second accumulator), one that the largest
# tap keeps below, the default's shape at the longest and a wider one
@pytest.mark.parametrize("taps", [
    np.full(255, 0.9979 / 255), np.full(257, 0.9979), np.full(120, 0.9979 / 120),
    np.r_[np.full(254, 0.3), 0.9979], _sinc(257), _sinc(257, 300.0), _sinc(255)],
    ids=["flat", "flat, large", "flat, short", "one large", "sinc", "wide sinc", "default"])
@pytest.mark.parametrize("sign", [1, -1])
def test_large_digit_sums(taps, sign):
    _check(taps, sign * _slow())


@pytest.mark.parametrize("taps", [_sinc(255), _sinc(128)], ids=["default", "128"])
@pytest.mark.parametrize("small", [2.0 ** -22, 2.0 ** -27, 2.0 ** -33])
def test_constant_remainders(taps, small):
    """Steady values far below the largest of their tile: what the digits leave of them has
    one sign."""
    rng = np.random.default_rng(1)
    v = np.broadcast_to(small * (1 + rng.random((1, 256))), (ROWS, 256)).copy()
    v[250::300] = 1.0
    v[400:420] = 0.3
    _check(taps, v)
