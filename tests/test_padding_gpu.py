"""Row padding of bf16 matrices (csrc/engine.cu, b2_handle::ld) when values are not finite."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# a padded last hidden layer in front of a narrow output (which reads the padding of its weights), with fp32 and bf16
# gradients (update in pieces of 4 and 8 columns) and a remainder of each kind; a padded last layer
NETS = [([64, 301, 10], False), ([64, 300, 10], True), ([64, 303, 1], True), ([64, 77, 298, 12], False),
        ([64, 301, 33], False), ([61, 301, 37], True)]


def problem(O, nf, batch):
    ws = [O.fill_uniform(nf[l + 1], nf[l], 40 + l, -0.3, 0.3) for l in range(len(nf) - 1)]
    return ws, O.fill_normal(batch, nf[0], 7), O.fill_sign(batch, nf[-1], 8)


def upload(m, ws, x, t):
    for l, w in enumerate(ws):
        m.upload_weights(l, w)
    m.upload_input(x)
    m.upload_target(t)


@pytest.mark.parametrize("fused", ["1", "0"], ids=["one-launch", "launch-per-gemm"])
@pytest.mark.parametrize("poison", ["nan-target", "inf-input", "nan-lr"])
@pytest.mark.parametrize("nf,grad_bf16", NETS, ids=lambda v: "x".join(map(str, v)) if isinstance(v, list) else f"g{int(v)}")
def test_handle_recovers_from_non_finite_step(native, oracle, monkeypatch, nf, grad_bf16, poison, fused):
    """After a step that met an Inf or a NaN, uploading weights, inputs and targets brings a handle back to the
    state of a new one: the same bits in the fingerprint, the outputs, the loss and the weights of the next steps."""
    from tbb_test_b200 import _capi as K
    from tbb_test_b200.mlp import MLP
    monkeypatch.setenv("B2_STEP_KERNEL", fused)
    batch, L = 200, len(nf) - 1
    ws, x, t = problem(oracle, nf, batch)
    got = []
    for spoiled in (False, True):
        m = MLP(nf, batch, precision=K.PREC_BF16, lr=0.01, grad_bf16=grad_bf16)
        if spoiled:
            bx, bt = x.copy(), t.copy()
            if poison == "nan-target":
                bt[3, 0] = np.nan
            elif poison == "inf-input":
                bx[5, 2] = np.inf
            else:
                m._ck(m.lib.b2_set_lr(m._h, float("nan")))
            upload(m, ws, bx, bt)
            m.step(2)
            m._ck(m.lib.b2_set_lr(m._h, 0.01))
        upload(m, ws, x, t)
        out = [np.array([m.weights_fingerprint(l) for l in range(L)], np.uint64)]
        m.step(2)
        out += [m.activation(l) for l in range(1, L + 1)] + [m.dz(l) for l in range(L)]
        out += [m.weights(l) for l in range(L)] + [m.weight_grad(l) for l in range(L)] + [m.input_grad()]
        got.append((out, m.loss()))
        m.close()
    assert all(np.isfinite(a).all() for a in got[0][0])
    for i, (a, b) in enumerate(zip(got[0][0], got[1][0])):
        assert np.array_equal(a, b), i
    assert got[0][1] == pytest.approx(got[1][1], rel=1e-12)  # the loss adds doubles in any order


@pytest.mark.parametrize("nf,grad_bf16", [n for n in NETS if n[0][-1] >= 16], ids=lambda v: "x".join(map(str, v)) if isinstance(v, list) else f"g{int(v)}")
def test_non_finite_step_matches_launch_per_gemm(native, oracle, monkeypatch, nf, grad_bf16):
    """A step over an activation that overflowed: the same bits in one launch as in one launch per GEMM, the loss
    (which must not take in the padding, Inf * 0 there) and the outputs included."""
    from tbb_test_b200 import _capi as K
    from tbb_test_b200.mlp import MLP
    batch, L = 200, len(nf) - 1
    ws, x, t = problem(oracle, nf, batch)
    ws[-1] = np.abs(ws[-1]) + np.float32(0.01)  # Inf * positive: outputs of that row are Inf, not NaN
    x[5] = np.float32(3e38)
    ws[0] *= np.float32(1e-30)
    ws[0][7] = np.float32(1.0)  # overflows in row 5, unit 7, and nowhere else
    got = []
    for fused in ("0", "1"):
        monkeypatch.setenv("B2_STEP_KERNEL", fused)
        m = MLP(nf, batch, precision=K.PREC_BF16, lr=0.01, grad_bf16=grad_bf16)
        upload(m, ws, x, t)
        m.step(1)
        got.append([m.activation(l) for l in range(1, L + 1)] + [m.dz(l) for l in range(L)] +
                   [m.weights(l) for l in range(L)] + [np.array([m.loss()])])
        m.close()
    assert np.isinf(got[0][0][5, 7]) and np.isinf(got[0][L - 1][5]).all() and got[0][-1][0] == np.inf
    for i, (a, b) in enumerate(zip(*got)):
        assert np.array_equal(a, b, equal_nan=True), i


@pytest.mark.parametrize("nf", [[64, 301, 10], [64, 303, 2], [64, 298, 12]], ids=lambda v: "x".join(map(str, v)))
def test_narrow_layer_leaves_padding_out(native, oracle, monkeypatch, nf):
    """Without a ReLU between the layers an activation that overflowed has NaNs in its row's padding: the outputs of
    that row are still Inf, and the other rows are as in one launch per GEMM (fp32 sums in another order: K terms,
    2^-24 each)."""
    from tbb_test_b200 import _capi as K
    from tbb_test_b200.mlp import MLP
    ws, x, t = problem(oracle, nf, 200)
    ws[-1] = np.abs(ws[-1]) + np.float32(0.01)
    x[5] = np.float32(3e38)
    ws[0] *= np.float32(1e-30)
    ws[0][7] = np.float32(1.0)
    ys = []
    for fused in ("0", "1"):
        monkeypatch.setenv("B2_STEP_KERNEL", fused)
        m = MLP(nf, 200, precision=K.PREC_BF16, mode=K.MODE_REF, lr=1e-10)
        upload(m, ws, x, t)
        m.step(1)
        ys.append(m.activation(2))
        m.close()
    assert (ys[0][5] == np.inf).all() and (ys[1][5] == np.inf).all()
    a, b = np.delete(ys[0], 5, 0), np.delete(ys[1], 5, 0)
    assert np.isfinite(a).all() and np.allclose(a, b, rtol=0, atol=nf[1] * 2.0 ** -24 * np.abs(a).max() * 4)
