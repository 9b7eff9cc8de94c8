"""Large downloads, which several threads share (download_rows in csrc/engine.cu)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,extra", [((1000, 1003), 0), ((1000, 1003), 5), ((7, 100000), 0), ((2, 300000), 3)])
def test_large_downloads(native, oracle, shape, extra):
    """Downloads above the size at which several threads share them, dense and pitched, with a last partial
    chunk and with rows longer than a chunk: every element in place, nothing written between the rows."""
    from tbb_test_b200 import _capi as K
    from tbb_test_b200.mlp import MLP
    rows, cols = shape
    w = oracle.fill_uniform(rows, cols, 3, -1, 1)
    for prec in (K.PREC_FP32, K.PREC_BF16):
        m = MLP([cols, rows], 8, precision=prec)
        m.upload_weights(0, w)
        got = np.full((rows, cols + extra), 7.0, np.float32)
        rc = m.lib.b2_download_weights(m._h, 0, got.ctypes.data_as(C.POINTER(C.c_float)), cols + extra)
        assert rc == K.OK
        assert np.array_equal(got[:, :cols], w) and (got[:, cols:] == 7.0).all()
        m.close()
