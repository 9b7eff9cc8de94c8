"""Whole steps of small fp32 networks in one launch (csrc/small_step.cu) against the launch-per-GEMM schedule of the same
handle, at the edges of its tiles (16 x 32), groups of four k and layer table."""
import ctypes as C
import time

import numpy as np
import pytest

from helpers import rel_fro

pytestmark = pytest.mark.gpu

# widths, batch, keywords; what makes them edges: one row; one column; one layer; tiles exactly and one more or less; rows of
# whole 16-byte pieces and not; sums shorter than a group of four k; more tiles than the grid has blocks; the last layer count
NETS = [([16, 32], 16, {}), ([1, 1], 1, {}), ([33, 17, 5], 7, {}), ([17, 31, 33, 1], 3, {}), ([64, 64, 64], 1, {}),
        ([128, 256, 128, 64], 32, {}), ([36, 60, 4], 130, {}), ([512, 512, 512], 24, {}), ([300, 301, 95, 40], 60, {}),
        ([20] * 17, 50, {}), ([40, 24], 2048, {}), ([64, 100, 10], 33, dict(input_grad=False))]


def make(monkeypatch, nf, batch, whole, **kw):
    from tbb_test_b200 import _capi as K
    from tbb_test_b200.mlp import MLP
    monkeypatch.setenv("B2_STEP_KERNEL", "1" if whole else "0")
    m = MLP(nf, batch, precision=K.PREC_FP32, lr=0.02, **kw)
    monkeypatch.delenv("B2_STEP_KERNEL")
    rng = np.random.default_rng(3)
    for l in range(m.L):
        m.upload_weights(l, rng.uniform(-1, 1, (nf[l + 1], nf[l])).astype(np.float32) * np.float32(nf[l] ** -0.5))
    m.upload_input(rng.standard_normal((batch, nf[0])).astype(np.float32))
    m.upload_target(np.sign(rng.standard_normal((batch, nf[-1]))).astype(np.float32))
    return m


def launches(m, f):
    before = m.launch_counts()[0]
    f()
    return m.launch_counts()[0] - before


@pytest.mark.parametrize("mode", ["baseline", "ref"])
@pytest.mark.parametrize("net", NETS, ids=lambda n: f"{'-'.join(map(str, n[0][:4]))}x{len(n[0])}b{n[1]}")
def test_one_step(native, monkeypatch, net, mode):
    """Every tensor of one step. Both sides add fp32 FMAs or better in other orders: the bound of the single GEMMs (2e-5)
    over the chain of at most 32 of them (sums of up to 2048 terms; seen: 5e-7)."""
    from tbb_test_b200 import _capi as K
    nf, batch, kw = net
    kw = dict(kw, mode=K.MODE_REF if mode == "ref" else K.MODE_BASELINE)
    a, b = make(monkeypatch, nf, batch, True, **kw), make(monkeypatch, nf, batch, False, **kw)
    assert launches(a, lambda: a.step(1)) == 1 and launches(b, lambda: b.step(1)) >= 4 * a.L
    for l in range(a.L + 1):
        assert rel_fro(a.activation(l), b.activation(l)) <= 2e-5
    for l in range(a.L):
        for what in (a.dz, b.dz), (a.weight_grad, b.weight_grad), (a.weights, b.weights):
            assert rel_fro(what[0](l), what[1](l)) <= 2e-5
    if kw.get("input_grad", True):
        assert rel_fro(a.input_grad(), b.input_grad()) <= 2e-5
    assert abs(a.loss() - b.loss()) <= 1e-5 * abs(b.loss())
    a.close()
    b.close()


@pytest.mark.parametrize("mode", ["baseline", "ref"])
@pytest.mark.parametrize("net", [([128, 256, 128, 64], 32), ([33, 101, 70], 41), ([300, 301, 95, 40], 60), ([20] * 5, 17), ([64, 48], 200)],
                         ids=lambda n: f"{'-'.join(map(str, n[0][:4]))}b{n[1]}")
def test_sums_in_k_order_are_the_same_bits(native, monkeypatch, net, mode):
    """Where no layer is as narrow and no batch as short as 16: every sum is one FMA per term in k order, as in gemm_simt_kernel
    and gemm_f32_kernel, so three steps end in the bits of separate launches of those (force_simt)."""
    from tbb_test_b200 import _capi as K
    nf, batch = net
    kw = dict(mode=K.MODE_REF if mode == "ref" else K.MODE_BASELINE)
    a, b = make(monkeypatch, nf, batch, True, **kw), make(monkeypatch, nf, batch, False, force_simt=True, **kw)
    a.step(3)
    b.step(3)
    for l in range(a.L):
        for what in (a.weights, b.weights), (a.weight_grad, b.weight_grad), (a.dz, b.dz), (a.activation, b.activation):
            assert np.array_equal(what[0](l), what[1](l))
    assert np.array_equal(a.activation(a.L), b.activation(a.L)) and np.array_equal(a.input_grad(), b.input_grad())
    a.close()
    b.close()


def test_many_steps_in_few_launches(native, monkeypatch):
    """100 steps in launches of at most 64, and the same steps one by one, from one handle's weights to the other's: equal
    bits (sums have a fixed order; the loss's block sums have none)."""
    nf, batch = [48, 64, 32], 20
    a, b = make(monkeypatch, nf, batch, True), make(monkeypatch, nf, batch, True)
    assert launches(a, lambda: a.step(100)) == 2
    for _ in range(100):
        b.step(1)
    assert all(np.array_equal(a.weights(l), b.weights(l)) for l in range(2)) and abs(a.loss() - b.loss()) <= 1e-12 * abs(b.loss())
    a.set_timing(1)  # timed steps take the launch-per-GEMM schedule in between
    assert launches(a, lambda: a.step(1)) > 1
    a.set_timing(0)
    assert launches(a, lambda: a.step(3)) == 1
    b.step(4)
    assert all(rel_fro(a.weights(l), b.weights(l)) <= 2e-5 for l in range(2))
    a.close()
    b.close()


@pytest.mark.parametrize("net", [([33, 17, 5], 7, {}), ([300, 301, 95, 40], 60, {}), ([45, 30], 70, {}), ([40, 24], 30, {}),
                                 ([64, 100, 10], 33, dict(input_grad=False)), ([63, 64, 9], 20, dict(input_grad=False)), ([1024, 1024, 1001], 16, {})],
                         ids=lambda n: f"{'-'.join(map(str, n[0]))}b{n[1]}")
def test_many_steps_of_other_networks(native, monkeypatch, net):
    """Rows that are not whole 16-byte pieces (copied through the L1, which the barriers have to empty), a single layer (a
    barrier more per step), no input gradient, more tiles than groups of warps: several steps in each of several launches against
    steps one by one (equal bits), and four steps in one launch against a launch per GEMM."""
    nf, batch, kw = net
    a, b, c = make(monkeypatch, nf, batch, True, **kw), make(monkeypatch, nf, batch, True, **kw), make(monkeypatch, nf, batch, False, **kw)
    for m, n in ((a, 1), (c, 5)):
        assert launches(m, lambda: m.step(4)) >= n
    assert all(rel_fro(a.weights(l), c.weights(l)) <= 2e-5 and rel_fro(a.weight_grad(l), c.weight_grad(l)) <= 1e-4 for l in range(a.L))
    assert 2 <= launches(a, lambda: a.step(150)) <= 75
    for _ in range(154):
        b.step(1)
    assert all(np.array_equal(a.weights(l), b.weights(l)) for l in range(a.L)) and abs(a.loss() - b.loss()) <= 1e-12 * abs(b.loss())
    for m in (a, b, c):
        m.close()


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 3e38], ids=str)
@pytest.mark.parametrize("net", [([128, 70, 90], 30), ([512, 9, 70], 8), ([80, 3], 100)], ids=lambda n: f"{'-'.join(map(str, n[0]))}b{n[1]}")
def test_values_that_are_not_finite(native, monkeypatch, net, value):
    """An input, a weight: the same elements of every tensor of a step end up infinite or not a number as with a launch per GEMM,
    whichever way the sums go. (Where finite values overflow, which of the two is a matter of the order: partial sums of both signs
    give no number.)"""
    from tbb_test_b200 import _capi as K
    nf, batch = net
    out = []
    for whole in (True, False):
        m = make(monkeypatch, nf, batch, whole, mode=K.MODE_REF)
        w, x = m.weights(0), np.linspace(-1, 1, batch * nf[0], dtype=np.float32).reshape(batch, nf[0])
        w[2, 7], x[3, 5] = -value, value
        m.upload_weights(0, w)
        m.upload_input(x)
        m.step(1)
        out.append([m.activation(l) for l in range(m.L + 1)] + [f(l) for l in range(m.L) for f in (m.dz, m.weight_grad, m.weights)] + [m.input_grad()])
        m.close()
    for got, want in zip(*out):
        assert np.array_equal(np.isfinite(got), np.isfinite(want))
        bad = ~np.isfinite(want)
        assert value == 3e38 or np.array_equal(got[bad], want[bad], equal_nan=True)


def test_host_fed_steps(native, monkeypatch):
    """Both input slots: steps fed from the host, two in flight, against blocking ones."""
    nf, batch = [40, 24, 12], 30
    fp = C.POINTER(C.c_float)
    rng = np.random.default_rng(4)
    data = [(rng.standard_normal((batch, 40)).astype(np.float32), np.sign(rng.standard_normal((batch, 12))).astype(np.float32)) for _ in range(5)]
    a, b = make(monkeypatch, nf, batch, True), make(monkeypatch, nf, batch, True)
    got, want = [], []
    for i, (x, t) in enumerate(data):
        px, pt = x.ctypes.data_as(fp), t.ctypes.data_as(fp)
        a.train_step_host_async(px, 40, pt, 12)
        if i:
            got.append(a.wait_loss())
        want.append(b.train_step_host(px, 40, pt, 12))
    got.append(a.wait_loss())
    assert np.allclose(got, want, rtol=1e-12) and all(np.array_equal(a.weights(l), b.weights(l)) for l in range(2))
    a.close()
    b.close()


@pytest.mark.parametrize("net", [([4096] * 5, 1), ([2048] * 3, 8), ([16384, 256, 10], 4), ([64] * 10, 1), ([128, 256, 128, 64], 32)],
                         ids=lambda n: f"{'-'.join(map(str, n[0][:3]))}b{n[1]}")
def test_launches_last_about_2_ms(native, monkeypatch, net):
    """A launch holds every SM. (64 steps at most; the estimate of a step is within 0.82 and 1.21 of its time at 1965 MHz, and a GPU
    at its power limit runs at two thirds of that.)"""
    m = make(monkeypatch, *net, True)
    n = launches(m, lambda: m.step(128))
    m.reset_timing()
    m.step(128)
    launch_ms = m.timing()[1] / n
    assert launch_ms <= 2.0 / 0.8 * 1.5 and (n == 2 or launch_ms >= 0.5), (n, launch_ms)
    m.close()


def late(monkeypatch, nf, batch):
    """A handle that counts one more arrival at the barriers than there will be: the first wait of its first launch runs out."""
    monkeypatch.setenv("B2_STEP_COUNT_AHEAD", "1")
    m = make(monkeypatch, nf, batch, True)
    monkeypatch.delenv("B2_STEP_COUNT_AHEAD")
    return m


def test_a_wait_that_runs_out(native, monkeypatch):
    """One wait limit (2 s) for any number of launches queued behind the one that gave up; the call reports it, the weights
    are as they were, and the next call runs."""
    from tbb_test_b200 import _capi as K
    nf, batch = [48, 64, 32], 20
    a, b = late(monkeypatch, nf, batch), make(monkeypatch, nf, batch, True)
    t0 = time.time()
    with pytest.raises(K.B2Error) as e:
        a.step(1000)
    assert e.value.code == K.ERR_TIMEOUT and time.time() - t0 < 6.0
    assert all(np.array_equal(a.weights(l), b.weights(l)) for l in range(2))
    a.step(130)
    b.step(130)
    assert all(np.array_equal(a.weights(l), b.weights(l)) for l in range(2))
    a.close()
    b.close()


def test_a_wait_that_runs_out_in_the_pipeline(native, monkeypatch):
    """With steps in flight every wait reports it until the pipeline has been drained, and none passes for a step."""
    from tbb_test_b200 import _capi as K
    nf, batch = [48, 64, 32], 20
    fp = C.POINTER(C.c_float)
    a, b = late(monkeypatch, nf, batch), make(monkeypatch, nf, batch, True)
    x, t = np.full((batch, 48), 0.25, np.float32), np.ones((batch, 32), np.float32)
    args = x.ctypes.data_as(fp), 48, t.ctypes.data_as(fp), 32
    t0 = time.time()
    a.train_step_host_async(*args)
    for _ in range(3):  # a loader that keeps two in flight
        a.train_step_host_async(*args)
        with pytest.raises(K.B2Error) as e:
            a.wait_loss()
        assert e.value.code == K.ERR_TIMEOUT
    with pytest.raises(K.B2Error):
        a.wait_loss()
    assert time.time() - t0 < 6.0 and all(np.array_equal(a.weights(l), b.weights(l)) for l in range(2))
    for m in (a, b):
        m.train_step_host_async(*args)
        m.train_step_host_async(*args)
        m.wait_loss(), m.wait_loss()
    assert all(np.array_equal(a.weights(l), b.weights(l)) for l in range(2))
    a.close()
    b.close()


def test_what_it_does_not_serve(native, monkeypatch):
    """More layers than its table, large networks, a large layer among small ones and serial schedules keep their paths."""
    from tbb_test_b200 import _capi as K
    from tbb_test_b200.mlp import MLP
    for nf, batch, kw in (([20] * 18, 50, {}), ([1024, 1024], 256, {}), ([64, 64], 4096, {}), ([2048] * 2 + [32] * 13, 128, {}),
                       ([64, 64], 32, dict(overlap=False))):
        m = MLP(nf, batch, precision=K.PREC_FP32, **kw)
        assert launches(m, lambda: m.step(1)) > 1
        m.close()


@pytest.mark.parametrize("lo", [-1.0, 0.0], ids=["signed", "positive"])
@pytest.mark.parametrize("net", [([512, 10], 2048), ([2048, 10], 64), ([300, 1], 100), ([512, 512, 9], 8), ([256, 512, 300], 16), ([33, 90, 5], 7),
                                 ([1, 70, 16], 71), ([76, 65], 2)], ids=lambda n: f"{'-'.join(map(str, n[0]))}b{n[1]}")
def test_short_sums_are_as_exact(native, monkeypatch, net, lo):
    """The GEMMs of narrow layers and short batches, whose sums are many partial ones in a launch of their own: the error
    against 64-bit sums of the same operands is no larger in a whole step (a tenth for the luck of the roundings)."""
    from tbb_test_b200 import _capi as K
    nf, batch = net
    err = []
    for whole in (True, False):
        m = make(monkeypatch, nf, batch, whole, mode=K.MODE_REF)
        rng = np.random.default_rng(5)
        w = [rng.uniform(lo, 1, (nf[l + 1], nf[l])).astype(np.float32) for l in range(m.L)]
        for l in range(m.L):
            m.upload_weights(l, w[l])
        m.upload_input(rng.uniform(lo, 1, (batch, nf[0])).astype(np.float32))
        m.step(1)
        act, dz = [m.activation(l).astype(np.float64) for l in range(m.L + 1)], [m.dz(l).astype(np.float64) for l in range(m.L)]
        e = {}
        for l in range(m.L):
            fi, fo = nf[l], nf[l + 1]
            if fi >= 64 and fo <= 16:
                e["forward", l] = rel_fro(act[l + 1], act[l] @ w[l].T)
            if batch >= 64 and fo <= 16:
                e["weight gradient", l] = rel_fro(m.weight_grad(l), dz[l].T @ act[l])
            if fo >= 64 and (batch <= 16 or fi == 1):
                e["input gradient", l] = rel_fro(dz[l - 1] if l else m.input_grad(), dz[l] @ w[l])
        err.append(e)
        m.close()
    assert err[0] and all(err[0][g] <= 1.1 * err[1][g] for g in err[0]), err
