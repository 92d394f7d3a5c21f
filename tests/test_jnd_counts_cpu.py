"""How many intervals a JND table may have, on a machine without a GPU: what is not
refused for its arguments gets as far as the launch."""
import ctypes as C

import numpy as np
import pytest
import torch

from cochlearmodel_gb300 import native

MOST = (2 ** 31 - 1) // 3


@pytest.mark.skipif(torch.cuda.is_available(), reason="the pointers are not device memory")
@pytest.mark.parametrize("n,refused", [(1, False), (2 ** 31 // 24 + 1, False), (MOST, False),
                                       (MOST + 1, True)])
def test_batch_counts(n, refused):
    lib = native.load()
    W = np.ones(3, np.float32)
    p = C.c_void_p(4096)
    rc = lib.cgb_jnd_batch_dev(p, 1, p, n, 1, p, native.ptr(W), 1e5, 1.0, p, p, None, None)
    assert rc != 0
    assert (b"too many intervals" in lib.cgb_last_error()) == refused
