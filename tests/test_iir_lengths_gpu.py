"""The IIR AC kernel's lengths: outputs in registers up to nine coefficients, read
back above, against the oracle bit for bit, on segments around its chunk of rows."""
import numpy as np
import pytest

from cochlearmodel_gb300 import ihc
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 8, 9, 10, 17])
@pytest.mark.parametrize("seg", [23, 24, 25, 300])
def test_lengths_and_segments(n, seg):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    stage = ihc.IHCStage("cuda:0")
    rng = np.random.default_rng(n)
    v = (1e-3 * rng.standard_normal((300, 256))).astype(np.float32)
    b = rng.uniform(-0.2, 0.2, n).astype(np.float32)
    a = (rng.uniform(-0.8, 0.8, n) / max(1, n - 1)).astype(np.float32)  # sum |a| < 1: stable
    a[0] = 1.0
    fr = np.zeros(1, ihc.FRAME_DTYPE)
    fr[0] = (0, 0, 300, 290, seg, 280, ihc.round64(300), 0)
    lam, pot, ac = stage.run_iir(v, fr, 290, b, a, want_ihc=True)
    f = fr[0]
    o_ihc, o_lam, o_ac = orc.ihc_lambda_iir(
        v, int(f["seg"]), int(f["frdp"]), int(f["total"]), 290, b.astype(np.float64),
        a.astype(np.float64), stage.dc.astype(np.float64), stage.prm.scale, stage.nerve.eta_AC,
        stage.nerve.eta_DC, stage.dmg_host[0].astype(np.float64), stage.nerve.aihc(),
        np.asarray(stage.nerve.spontRate, np.float32), stage.nerve.Lambda_SAT, mode=2)
    assert np.array_equal(ac[:290].view(np.uint32), o_ac[:290].view(np.uint32))
    assert np.array_equal(pot.view(np.uint32), o_ihc[:290].view(np.uint32))
    assert np.array_equal(lam.view(np.uint32), o_lam.view(np.uint32))
