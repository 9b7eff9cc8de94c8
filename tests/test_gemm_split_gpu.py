"""fp32 GEMMs on split operands (csrc/gemm_split.cu) at the edges of their tiles, chunks and ways of reading, against
float64 sums and against the CUDA-core FMAs that a handle with force_simt runs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FORMS = {"fwd_NT": (False, True), "dgrad_NN": (False, False), "wgrad_TN": (True, False), "TT": (True, True)}
# (m, n, k): one tile, in part; one chunk of 64 k and several tiles per block; k behind whole chunks; rows of whole 32- and
# 16-byte pieces and of neither; one to three rounds of tiles
SHAPES = [(17, 17, 4000), (128, 64, 1024), (129, 65, 1001), (300, 204, 1300), (1500, 3000, 64), (1500, 2999, 65), (2048, 1100, 260),
          (1000, 1000, 1000), (640, 72, 2047)]


@pytest.fixture(scope="module")
def devs(native):
    from tbb_test_b200.mlp import MLP
    both = MLP([16, 16], 16), MLP([16, 16], 16, force_simt=True)
    yield both
    for m in both:
        m.close()


def sgemm(dev, ta, tb, a, b, c=None, alpha=1.0, beta=0.0):
    import torch
    from tbb_test_b200 import _capi as K
    m, k = a.shape[::-1] if ta else a.shape
    n = b.shape[0] if tb else b.shape[1]
    ad, bd = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    cd = torch.full((m, n), float("nan"), device="cuda") if c is None else torch.from_numpy(c).cuda()
    torch.cuda.synchronize()
    rc = dev.lib.b2_sgemm(dev._h, K.PREC_FP32, int(ta), int(tb), m, n, k, alpha, ad.data_ptr(), a.shape[1], bd.data_ptr(), b.shape[1],
                          beta, cd.data_ptr(), n)
    assert rc == K.OK and dev.lib.b2_sync(dev._h) == K.OK, dev.lib.b2_last_error(dev._h)
    return cd.cpu().numpy()


def operands(oracle, form, m, n, k, seed, lo=-1.0):
    ta, tb = FORMS[form]
    return ta, tb, oracle.fill_uniform(k if ta else m, m if ta else k, seed, lo, 1.0), oracle.fill_uniform(n if tb else k, k if tb else n, seed + 1, lo, 1.0)


@pytest.mark.parametrize("lo", [-1.0, 0.0], ids=["signed", "positive"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("form", list(FORMS))
def test_against_float64(devs, oracle, form, shape, lo):
    """Bound per element, in 2^-24 of the sum of magnitudes: within a chunk of 64 k four sums that lose up to two units
    each, one rounding per chunk, in D1 (2^-8 of the rest) two units in each of k/4 sums, and 4 for the last sums, alpha and
    beta. And over the whole matrix the error is not above that of FMAs in k order."""
    m, n, k = shape
    ta, tb, a, b = operands(oracle, form, m, n, k, 211, lo)
    c = oracle.fill_uniform(m, n, 213, -1.0, 1.0)
    ra, rb = (a.T if ta else a).astype(np.float64), (b.T if tb else b).astype(np.float64)
    ref, mag = ra @ rb, np.abs(ra) @ np.abs(rb)
    units = 8 + (k + 63) // 64 + k / 4 * 2 / 256 + 4
    got, fma = sgemm(devs[0], ta, tb, a, b), sgemm(devs[1], ta, tb, a, b)
    assert not np.array_equal(got, fma), "the FMA kernels ran"
    assert (np.abs(got - ref) <= units * 2.0 ** -24 * mag).all()
    assert np.linalg.norm(got - ref) <= np.linalg.norm(fma - ref)
    got = sgemm(devs[0], ta, tb, a, b, c.copy(), 2.0, -0.5)
    assert (np.abs(got - (2.0 * ref - 0.5 * c)) <= units * 2.0 ** -24 * (2.0 * mag + np.abs(c))).all()


@pytest.mark.parametrize("lo", [-1.0, 0.0], ids=["signed", "positive"])
@pytest.mark.parametrize("k", [64, 538, 2048])
def test_sums_do_not_shrink(devs, oracle, k, lo):
    """The error along the result, which many results combined to one number do not average out. The tensor core truncates:
    pieces of eight bits left sums 3.8e-8 (signed) to 6.6e-8 (positive) small, those of six 5.7e-9 to 1.7e-8 (so too a model of
    it in numpy: sums of 16 exact products and the accumulator, truncated to 24 bits)."""
    ta, tb, a, b = operands(oracle, "fwd_NT", 1500, 1600, k, 261, lo)
    ref = a.astype(np.float64) @ b.astype(np.float64).T
    got = sgemm(devs[0], ta, tb, a, b)
    assert not np.array_equal(got, sgemm(devs[1], ta, tb, a, b))
    assert abs(((got - ref) * ref).sum()) <= 2.2e-8 * (ref * ref).sum()


@pytest.mark.parametrize("shape", [(300, 204, 1300), (129, 65, 1001)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("form", list(FORMS))
def test_relu_and_mask(devs, oracle, form, shape):
    from tbb_test_b200 import _capi as K
    m, n, k = shape
    ta, tb, a, b = operands(oracle, form, m, n, k, 221)
    aux = oracle.fill_uniform(m, n, 223, -1.0, 1.0)
    plain = devs[0].sgemm_host(K.PREC_FP32, ta, tb, a, b)
    assert np.array_equal(devs[0].sgemm_host(K.PREC_FP32, ta, tb, a, b, epilogue=K.EPI_RELU), np.maximum(plain, 0))
    assert np.array_equal(devs[0].sgemm_host(K.PREC_FP32, ta, tb, a, b, epilogue=K.EPI_MASK, aux=aux), np.where(aux > 0, plain, 0))


@pytest.mark.parametrize("kind", ["inf", "nan", "overflow", "large", "small", "denormal", "negative_inf_beta"])
@pytest.mark.parametrize("shape", [(300, 204, 1300), (129, 65, 1001), (1500, 2999, 65)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("form", list(FORMS))
def test_values_at_the_ends_of_the_range(devs, oracle, form, shape, kind):
    """Where the FMAs give an Inf or a NaN the same one; elsewhere no larger an error."""
    m, n, k = shape
    ta, tb, a, b = operands(oracle, form, m, n, k, 231)
    beta, c = 0.0, None
    if kind == "inf":
        a[3, 5], b[7, 2] = np.inf, -np.inf
    elif kind == "nan":
        a[-1, -1] = np.nan
    elif kind == "negative_inf_beta":
        a[0, 0], beta, c = -np.inf, 0.5, oracle.fill_uniform(m, n, 233, -1.0, 1.0)
    else:
        a *= np.float32({"overflow": 3e38, "large": 1e34, "small": 1e-37, "denormal": 1e-40}[kind])
    got, fma = (sgemm(d, ta, tb, a, b, None if c is None else c.copy(), 1.0, beta) for d in devs)
    ok = np.isfinite(fma)
    assert np.array_equal(np.isfinite(got), ok)
    assert np.array_equal(got[~ok], fma[~ok], equal_nan=True)
    with np.errstate(all="ignore"):
        ref = (a.T if ta else a).astype(np.float64) @ (b.T if tb else b).astype(np.float64) + (0 if c is None else beta * c)
    if ok.any():
        assert np.linalg.norm(got[ok] - ref[ok]) <= np.linalg.norm(fma[ok] - ref[ok])


def test_the_choice_counts_the_sms_of_the_launch(native, monkeypatch):
    """A forward GEMM of 3 x 47 tiles and one chunk of k: one round on 148 SMs, where the tensor cores are estimated faster,
    but two on the 128 that are left when 20 are reserved, where FMAs are."""
    from tbb_test_b200 import _capi as K
    from tbb_test_b200.mlp import MLP
    monkeypatch.setenv("B2_STEP_KERNEL", "0")
    rng = np.random.default_rng(6)
    w, x = (rng.uniform(-1, 1, s).astype(np.float32) for s in ((2945, 64), (257, 64)))
    y = []
    for kw in (dict(), dict(comm_sms=20), dict(force_simt=True)):
        m = MLP([64, 2945], 257, precision=K.PREC_FP32, mode=K.MODE_REF, **kw)
        m.upload_weights(0, w)
        m.upload_input(x)
        m.step(1)
        y.append(m.activation(1))
        m.close()
    assert not np.array_equal(y[0], y[2]) and np.array_equal(y[1], y[2])


@pytest.mark.parametrize("form", ["fwd_NT", "dgrad_NN", "wgrad_TN"])
def test_a_diverged_job_is_not_held_up(devs, form):
    """Operands that are all NaN take the tensor cores' time and then FMAs in k order: at most 2.4 times what the CUDA-core kernels
    take for the same (1.7 to 1.8 measured)."""
    import time
    import torch
    from tbb_test_b200 import _capi as K
    ta, tb = FORMS[form]
    n = 1024
    a, b, c = (torch.full((n, n), float("nan"), device="cuda") for _ in range(3))
    torch.cuda.synchronize()

    def us(dev):
        best = float("inf")
        for _ in range(5):
            dev.lib.b2_sync(dev._h)
            t0 = time.perf_counter()
            for _ in range(20):
                dev.lib.b2_sgemm(dev._h, K.PREC_FP32, int(ta), int(tb), n, n, n, 1.0, a.data_ptr(), n, b.data_ptr(), n, 0.0, c.data_ptr(), n)
            dev.lib.b2_sync(dev._h)
            best = min(best, (time.perf_counter() - t0) / 20 * 1e6)
        return best
    assert us(devs[0]) <= 2.4 * us(devs[1])
