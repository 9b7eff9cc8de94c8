"""Large downloads, which several threads share (download_rows in csrc/engine.cu)."""
import ctypes as C

import os
import subprocess
import sys

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


@pytest.mark.parametrize("shape,extra", [((257, 513), 0), ((1024, 512), 0), ((1800, 2050), 0), ((1800, 2050), 7), ((4100, 4099), 0),
                                         ((300, 20000), 3)])
def test_chunks_grow_with_the_matrix(native, oracle, shape, extra):
    """Sizes on both sides of each step in threads and chunk size, one handle growing its buffers: fresh destinations
    (pages that do not exist yet) and pitched ones, every element in place, nothing written between the rows."""
    from tbb_test_b200 import _capi as K
    from tbb_test_b200.mlp import MLP
    rows, cols = shape
    m = MLP([cols, rows, 700, 800], 8)
    ws = [oracle.fill_uniform(rows, cols, 3, -1, 1), oracle.fill_uniform(700, rows, 4, -1, 1), oracle.fill_uniform(800, 700, 5, -1, 1)]
    for l, w in enumerate(ws):
        m.upload_weights(l, w)
    for l in (2, 1, 0, 2):
        r, c = ws[l].shape
        got = np.empty((r, c + extra), np.float32)
        if extra:
            got[:] = 7.0
        assert m.lib.b2_download_weights(m._h, l, got.ctypes.data_as(C.POINTER(C.c_float)), c + extra) == K.OK
        assert np.array_equal(got[:, :c], ws[l]) and (got[:, c:] == 7.0).all()
    m.close()


@pytest.mark.parametrize("shape,extra", [((1, 1), 0), ((3, 5), 2), ((127, 129), 0), ((400, 401), 7), ((700, 800), 0), ((700, 800), 1),
                                         ((1, 655360), 0), ((1, 655361), 0)])
def test_small_downloads(native, oracle, shape, extra):
    """Matrices that land in the handle's page-locked block, up to its last byte and one element beyond: alone and in several
    threads, into fresh and pitched memory, in two handles whose blocks differ."""
    from tbb_test_b200.mlp import MLP
    rows, cols = shape
    w = oracle.fill_uniform(rows, cols, 3, -1, 1)
    for other in (7, 300):
        m = MLP([cols, rows, other], 4)
        m.upload_weights(0, w)
        for _ in range(2):
            got = np.empty((rows, cols + extra), np.float32)
            got[:, cols:] = 7.0
            assert m.lib.b2_download_weights(m._h, 0, got.ctypes.data_as(C.POINTER(C.c_float)), cols + extra) == 0
            assert np.array_equal(got[:, :cols], w) and (got[:, cols:] == 7.0).all()
        m.close()


def test_a_download_behind_queued_work_waits_in_one_thread(native):
    """Six threads copy a matrix of 2.4 MB, but none of them burns a core while the GPU is still busy with earlier work: the
    processor time of the call is that of one waiting thread."""
    import time
    import torch
    from tbb_test_b200 import _capi as K
    from tbb_test_b200.mlp import MLP
    m, n = MLP([768, 768], 64), 4096
    a, c = torch.ones(n, n, device="cuda"), torch.zeros(n, n, device="cuda")
    torch.cuda.synchronize()
    m.weights(0)
    for _ in range(300):
        m.lib.b2_sgemm(m._h, K.PREC_TF32, 0, 1, n, n, n, 1.0, a.data_ptr(), n, a.data_ptr(), n, 0.0, c.data_ptr(), n)
    cpu, wall = time.process_time(), time.perf_counter()
    m.weights(0)
    cpu, wall = time.process_time() - cpu, time.perf_counter() - wall
    assert wall > 0.02 and cpu <= 2.0 * wall, (cpu, wall)
    m.close()


OUT_OF_MEMORY = """
import ctypes as C, sys
import numpy as np
from tbb_test_b200 import _capi as K
from tbb_test_b200.mlp import MLP
fake = C.CDLL(sys.argv[1])
w = np.random.default_rng(1).standard_normal((1000, 1003), dtype=np.float32)
m = MLP([1003, 1000], 8)
m.upload_weights(0, w)
got = np.full(w.shape, 7.0, np.float32)
C.c_int.in_dll(fake, "fail_new").value = 1
rc = m.lib.b2_download_weights(m._h, 0, got.ctypes.data_as(C.POINTER(C.c_float)), 1003)
C.c_int.in_dll(fake, "fail_new").value = 0
assert C.c_int.in_dll(fake, "failed").value > 0, "nothing was allocated"
assert rc == K.OK and np.array_equal(got, w)
print("all there")
"""


def test_large_download_without_memory_for_threads(native, tmp_path):
    """Where a helper thread cannot be started for want of host memory, the calling thread does the work: no exception
    leaves the C entry point, and every element arrives."""
    here = os.path.dirname(os.path.abspath(__file__))
    so = str(tmp_path / "failing_new.so")
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", "-o", so, os.path.join(here, "fake", "failing_new.cc")], check=True)
    env = dict(os.environ, LD_PRELOAD=so, PYTHONPATH=os.path.dirname(here))
    r = subprocess.run([sys.executable, "-c", OUT_OF_MEMORY, so], env=env, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "all there" in r.stdout, r.stderr[-2000:]
