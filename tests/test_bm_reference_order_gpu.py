"""The BM solver in the reference's order of operations (arith 1) against a recorded run.

No CPU oracle has this mode (its tanhf and fast division are the GPU's), and the
reference's own kernels are not always there to compare with.  golden/
bm_reference_order.npz holds the velocity and the counts of the warp-per-unit kernel on a
GB300, as it was when its results were compared bit for bit with the reference's compiled
BMOHC_NEW_kernel: two tones of two blocks of 1 ms with 0.5 ms overlap, an OHC profile that
falls off towards the apex."""
import os

import numpy as np
import pytest

from cochlearmodel_gb300 import native
from tests import cases

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden",
                      "bm_reference_order.npz")
COUNTS = ("substeps", "iterations", "sweeps", "failed_samples")


def _case(mv):
    _, sc, _, units, x, rows = cases.decoupled_sweep(mv, n_signals=2, decouple=2, block_ms=1.0,
                                                     overlap_ms=0.5, seed=1)
    sc = native.BMScalars.from_buffer_copy(sc)
    sc.controller = sc.arith = 1
    return sc, cases.hearing_loss_gamma()[None], units, x, rows


# four warps per unit; a warp per unit (past two units an SM)
@pytest.mark.parametrize("many", [False, True])
def test_recorded_run(mv, bm_solver, many):
    import torch
    z = np.load(GOLDEN)
    sc, gamma, units, x, rows = _case(mv)
    copies = 1
    if many:
        sms = torch.cuda.get_device_properties(bm_solver.device).multi_processor_count
        copies = 2 * sms // len(units) + 1
        units = np.concatenate([units] * copies)
        units["out_base"] += np.repeat(np.arange(copies), len(units) // copies) * rows
    v, f, st = bm_solver.run(sc, gamma, units, x, rows * copies)
    n = len(z["v"])
    for at in {0, copies // 2, copies - 1}:
        got = v[at * rows:at * rows + n]
        assert np.array_equal(got.view(np.uint32), z["v"].view(np.uint32))
        assert np.array_equal(f[at * rows:at * rows + n], z["failed"])
    for k in COUNTS:
        assert np.array_equal(st[k], np.resize(z[k], len(units))), k
