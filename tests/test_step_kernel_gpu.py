"""Whole steps as one launch (csrc/step_kernel.cu) against one launch per GEMM."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (widths, batch, options): one tile / several row blocks with a remainder / ragged widths of both operand majors /
# more tiles than SMs / one layer / every output kind the epilogue has; "narrow": last layer on the CUDA cores
NETS = [([96, 64], 40, {}), ([256] * 6, 256, {}), ([123, 77, 201, 33], 333, {}), ([784, 500, 300, 40], 1000, {}),
        ([512, 384, 640, 128], 640, {"grad_bf16": True}), ([1024, 1536, 512], 1500, {}), ([64] * 22, 130, {}),
        ([96] * 51, 200, {"lr": 1e-5}), ([64] * 53, 64, {"lr": 1e-5}), ([64] * 24, 130, {"input_grad": False}),
        ([192, 160, 64], 200, {"ref": True}), ([192, 160, 64], 200, {"input_grad": False}),
        ([160, 96, 10], 300, {}), ([256, 128, 1], 990, {"ref": True})]


def states(O, K, nf, batch, prec, steps, opts, fed=False):
    from tbb_test_b200.mlp import MLP
    L = len(nf) - 1
    mode = K.MODE_REF if opts.get("ref") else K.MODE_BASELINE
    m = MLP(nf, batch, precision=prec, mode=mode, lr=1e-6 if opts.get("ref") else opts.get("lr", 0.01),
            grad_bf16=opts.get("grad_bf16", False) and prec == K.PREC_BF16, input_grad=opts.get("input_grad", True))
    for l in range(L):
        a = (6.0 / nf[l]) ** 0.5
        m.upload_weights(l, O.fill_uniform(nf[l + 1], nf[l], 5 + l, -a, a))
    x = np.ascontiguousarray(O.fill_normal(batch, nf[0], 1))
    t = np.ascontiguousarray(O.fill_sign(batch, nf[-1], 2))
    before = m.launch_counts()[0]
    if fed:
        fp = C.POINTER(C.c_float)
        for i in range(steps):
            m.train_step_host_async(x.ctypes.data_as(fp), nf[0], t.ctypes.data_as(fp), nf[-1])
            loss = m.wait_loss()
    else:
        m.upload_input(x)
        m.upload_target(t)
        before = m.launch_counts()[0]
        m.step(steps)
        loss = m.loss()
    launches = m.launch_counts()[0] - before
    out = {"y": m.activation(L)}
    for l in range(L):
        out[f"w{l}"], out[f"dw{l}"], out[f"dz{l}"] = m.weights(l), m.weight_grad(l), m.dz(l)
        if l:
            out[f"act{l}"] = m.activation(l)
    if opts.get("input_grad", True):
        out["dinput"] = m.input_grad()
    m.close()
    return out, loss, launches


@pytest.mark.parametrize("prec", ["bf16", "tf32", "fp32tc"])
@pytest.mark.parametrize("net", NETS, ids=lambda n: "x".join(map(str, n[0][:4])) + f"b{n[1]}" + "".join(n[2]))
def test_step_kernel_matches_launch_per_gemm(native, oracle, monkeypatch, net, prec):
    """The same MMAs in the same k order and the same element-wise arithmetic: equal bits. A narrow last layer adds
    its products in another order (fp32, K terms: 1e-5), which a bf16 store may turn into one unit in the last
    place of a few elements (2^-8 each: 2e-3 of the tensors' norm, as for the other oracle that rounds alike)."""
    from tbb_test_b200 import _capi as K
    nf, batch, opts = net
    P = {"bf16": K.PREC_BF16, "tf32": K.PREC_TF32, "fp32tc": K.PREC_FP32_TC}[prec]
    for steps in (1, 3):
        monkeypatch.setenv("B2_STEP_KERNEL", "0")
        a, la, na = states(oracle, K, nf, batch, P, steps, opts)
        monkeypatch.setenv("B2_STEP_KERNEL", "1")
        b, lb, nb = states(oracle, K, nf, batch, P, steps, opts)
        f, lf, nfed = states(oracle, K, nf, batch, P, steps, opts, fed=True)
        # every GEMM but a narrow last one on the tensor cores, and no more layers than the kernel's table holds
        if (prec == "bf16" or all(n % 4 == 0 for n in nf)) and len(nf) <= 51:
            assert nb == 1, "not one launch for all steps"
            # per host-fed step, in both input slots: the launch, and the conversion of the input or its twin
            assert nfed == steps * (1 if prec == "tf32" else 2)
        else:
            assert nb == na and na >= steps * (3 * len(nf) - 4), "one launch per GEMM"
        tail = nf[-1] < 16
        for k in a:
            for o in (b, f):
                if not tail:
                    assert np.array_equal(a[k], o[k]), (k, steps)
                else:
                    d = np.linalg.norm((a[k] - o[k]).astype(np.float64))
                    assert d <= (1e-5 if k == "y" and steps == 1 else 2e-3) * max(np.linalg.norm(a[k]), 1e-30), (k, steps)
        assert abs(la - lb) <= 1e-5 * abs(la) and abs(la - lf) <= 1e-5 * abs(la)


# One tile of a pair with its second CTA empty / a remainder in rows and columns of either CTA / ragged widths (rows that
# start on 16-byte boundaries only) / both input slots, bf16 gradients / several rounds of the grid / narrow last layers / more
# layers than the small table holds. Odd widths run in bf16 alone, on padded rows.
PAIR_NETS = [([96, 64], 40, {}), ([256, 132, 388, 260], 130, {}), ([124, 76, 204, 36], 333, {}), ([123, 77, 201, 33], 333, {}),
             ([512, 384, 640, 128], 640, {"grad_bf16": True}), ([1024, 1536, 512], 3100, {}), ([64] * 24, 257, {"input_grad": False}),
             ([160, 96, 12], 300, {}), ([160, 96, 10], 300, {}), ([256, 128, 4], 990, {"ref": True}), ([256, 128, 1], 990, {"ref": True})]


@pytest.mark.parametrize("prec,net", [(p, n) for n in PAIR_NETS for p in ("bf16", "tf32", "fp32tc")
                                      if p == "bf16" or all(w % 4 == 0 for w in n[0])],
                         ids=lambda v: v if isinstance(v, str) else "x".join(map(str, v[0][:4])) + f"b{v[1]}" + "".join(v[2]))
def test_pair_tiles_match_single_cta_tiles(native, oracle, monkeypatch, capfd, net, prec):
    """256 x 128 tiles of CTA pairs, and the tiles of one CTA, add every element's products in the same order: equal
    bits, narrow last layers included. Each form is the one that runs, in one launch for all steps."""
    from tbb_test_b200 import _capi as K
    nf, batch, opts = net
    P = {"bf16": K.PREC_BF16, "tf32": K.PREC_TF32, "fp32tc": K.PREC_FP32_TC}[prec]
    monkeypatch.setenv("B2_STEP_KERNEL", "1")
    monkeypatch.setenv("B2_VERBOSE", "1")
    for steps, fed in ((1, False), (3, False), (2, True)):
        got = []
        for pair, form in (("0", "a CTA per tile"), ("1", "CTA pairs")):
            monkeypatch.setenv("B2_STEP_PAIR", pair)
            capfd.readouterr()
            got.append(states(oracle, K, nf, batch, P, steps, opts, fed=fed))
            assert f"whole steps in one launch, {form}\n" in capfd.readouterr().err
        (a, la, na), (b, lb, nb) = got
        # per host-fed step the launch, and the conversion of the input or its twin
        assert na == nb == (steps * (1 if prec == "tf32" else 2) if fed else 1)
        assert abs(la - lb) <= 1e-5 * abs(la)
        assert all(np.array_equal(a[k], b[k]) for k in a), (steps, fed)


@pytest.mark.parametrize("prec", ["bf16", "tf32", "fp32tc"])
@pytest.mark.parametrize("nf,batch", [([800, 800, 800], 8192), ([64, 8000, 64], 300), ([64, 64, 64], 20000), ([2304, 2304], 1500)],
                         ids=["many-tiles", "wide-middle", "long-sums", "large"])
def test_layers_of_many_tiles(native, oracle, monkeypatch, nf, batch, prec):
    """Layers of many more tiles than SMs run as one launch by default, with the bits of one launch per GEMM."""
    from tbb_test_b200 import _capi as K
    P = {"bf16": K.PREC_BF16, "tf32": K.PREC_TF32, "fp32tc": K.PREC_FP32_TC}[prec]
    a, la, na = states(oracle, K, nf, batch, P, 2, {"lr": 1e-5})
    monkeypatch.setenv("B2_STEP_KERNEL", "0")
    b, lb, nb = states(oracle, K, nf, batch, P, 2, {"lr": 1e-5})
    assert na <= 2 < nb and abs(la - lb) <= 1e-5 * abs(la)
    assert all(np.array_equal(a[k], b[k]) for k in a)


@pytest.mark.parametrize("pair", ["0", "1"], ids=["single", "pairs"])
@pytest.mark.parametrize("prec", ["bf16", "tf32"])
def test_two_handles_in_two_threads(native, oracle, monkeypatch, prec, pair):
    """Cooperative launches of two handles on one GPU, issued by two host threads at once, each keep their grid
    resident, in either form (a pair is a cluster of two CTAs): both finish with the weights they reach alone."""
    import threading
    from tbb_test_b200 import _capi as K
    from tbb_test_b200.mlp import MLP
    monkeypatch.setenv("B2_STEP_PAIR", pair)
    P = {"bf16": K.PREC_BF16, "tf32": K.PREC_TF32}[prec]
    nf, batch, L = [512] * 5, 512 if pair == "0" else 5000, 4  # 80 pair tiles a GEMM: the grid is full

    def make(seed):
        m = MLP(nf, batch, precision=P, lr=0.01)
        for l in range(L):
            m.upload_weights(l, oracle.fill_uniform(nf[l + 1], nf[l], seed + l, -0.1, 0.1))
        m.upload_input(oracle.fill_normal(batch, nf[0], seed + 20))
        m.upload_target(oracle.fill_sign(batch, nf[-1], seed + 30))
        return m

    alone = []
    for seed in (1, 100):
        m = make(seed)
        for _ in range(20):
            m.step(5)
        alone.append([m.weights(l) for l in range(L)])
        m.close()
    pair = [make(1), make(100)]
    errors = []

    def go(m):
        try:
            for _ in range(20):
                m.step(5)
        except Exception as e:  # reported below, on the test's own thread
            errors.append(e)

    threads = [threading.Thread(target=go, args=(m,)) for m in pair]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for m, ref in zip(pair, alone):
        for l in range(L):
            assert np.array_equal(m.weights(l), ref[l])
        m.close()


@pytest.mark.parametrize("nf,batch,steps", [([512] * 21, 2048, 64), ([1024] * 6, 1024, 50), ([64, 64, 64], 64, 130),
                                            ([64, 64, 64], 64, 65), ([64] * 5, 200000, 12), ([4096] * 3, 64, 48)],
                         ids=["deep", "c1", "small", "one-more", "long-sums", "many-weights"])
def test_steps_are_split_into_short_launches(native, oracle, monkeypatch, nf, batch, steps):
    """b2_step holds the GPU for a few ms at a time at most (the limit is 2 ms by estimate; twice that here, for a slow
    clock), whatever the number of steps, in few launches for short steps; and the split changes no bit."""
    from tbb_test_b200 import _capi as K
    from tbb_test_b200.mlp import MLP
    ws = [oracle.fill_uniform(nf[l + 1], nf[l], 5 + l, -0.1, 0.1) for l in range(len(nf) - 1)]
    x, t = oracle.fill_normal(batch, nf[0], 1), oracle.fill_sign(batch, nf[-1], 2)

    def run(fused):
        monkeypatch.setenv("B2_STEP_KERNEL", fused)
        m = MLP(nf, batch, precision=K.PREC_BF16, lr=1e-4)
        for l, w in enumerate(ws):
            m.upload_weights(l, w)
        m.upload_input(x)
        m.upload_target(t)
        before = m.launch_counts()[0]
        m.step(steps)
        launches = m.launch_counts()[0] - before
        loss, out = m.loss(), [m.weights(l) for l in range(len(ws))]
        m.reset_timing()
        m.step(steps)
        ms = m.timing()[1]
        m.close()
        return launches, loss, out, ms

    launches, loss, out, ms = run("1")
    assert ms / launches <= 4.0, (ms, launches)
    assert launches <= max(3, ms / 0.5)
    _, loss0, out0, _ = run("0")
    assert all(np.array_equal(a, b) for a, b in zip(out, out0)) and abs(loss - loss0) <= 1e-5 * abs(loss0)
