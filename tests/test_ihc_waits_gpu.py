"""A wait of the IHC kernels that runs out ends the launch with a status, whatever
the kernel has issued by then, and leaves the GPU usable."""
import numpy as np
import pytest

from cochlearmodel_gb300 import ihc, native

pytestmark = pytest.mark.gpu


def _taps(n):
    t = np.sinc(0.016 * (np.arange(n) - (n - 1) / 2)) * np.hamming(n)
    return (t / t.sum()).astype(np.float32)


# 63 taps: the FP32 kernel's staged copies; 255: the tensor kernel, whose issuing warp
# has products under way when the workers give up.  One tile of a CTA and runs of them.
@pytest.mark.parametrize("n_taps", [63, 255])
@pytest.mark.parametrize("rows", [100, 600, 30000])
def test_wait_runs_out(n_taps, rows):
    lib = native.load()
    stage = ihc.IHCStage("cuda:0", ac_taps=_taps(n_taps))
    v = (1e-3 * np.random.default_rng(rows).standard_normal((rows, 256))).astype(np.float32)
    fr = np.array([(0, 0, rows, rows, rows, rows, ihc.round64(rows), 0)], ihc.FRAME_DTYPE)
    want, _ = stage.run(v, fr, rows)
    for _ in range(2):
        native.check(lib.cgb_ihc_set_fault_injection(1), "fault injection")
        try:
            with pytest.raises(native.CGBError, match="did not complete"):
                stage.run(v, fr, rows)
        finally:
            native.check(lib.cgb_ihc_set_fault_injection(0), "fault injection")
        again, _ = stage.run(v, fr, rows)
        assert np.array_equal(again.view(np.uint32), want.view(np.uint32))
