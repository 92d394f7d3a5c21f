"""The autotuner's workload key: whatever makes other kernels run makes another key."""
from types import SimpleNamespace

import numpy as np
import pytest

from cochlearmodel_gb300 import autotune, ihc, model


def _run():
    frames = np.zeros(3, ihc.FRAME_DTYPE)
    frames["rows"] = frames["lam_rows"] = frames["seg"] = 1000
    cfg = model.RunConfig()
    return SimpleNamespace(sc=model.bm_scalars(cfg, model.ModelVectors.build()),
                           units=np.zeros(5), frames=frames, d_lam=np.zeros((3, 3000, 256)),
                           ihc=SimpleNamespace(ac=np.ones(255, np.float32),
                                               dc=np.full(200, 0.005, np.float32)))


def test_same_workload_same_key():
    assert autotune.workload(_run()) == autotune.workload(_run())


@pytest.mark.parametrize("change", ["controller", "arith", "jacobi_slow", "jacobi_fast",
                                    "ac length", "ac taps", "dc taps", "segments"])
def test_other_kernels_other_key(change):
    a, b = _run(), _run()
    if change == "ac length":
        b.ihc.ac = np.ones(48, np.float32)
    elif change == "ac taps":
        b.ihc.ac = b.ihc.ac * np.float32(0.5)
    elif change == "dc taps":
        b.ihc.dc[3] = 0.006
    elif change == "segments":
        b.frames["seg"] = 100
    else:
        setattr(b.sc, change, getattr(b.sc, change) + 1)
    assert autotune.workload(a) != autotune.workload(b)
