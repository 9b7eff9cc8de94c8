"""GPU parity of the three GEMM call forms (mlp_omp.cc:474,566,657) against the CPU
oracle, through the C ABI (b2_sgemm_host), for every precision and epilogue."""
import numpy as np
import pytest

from helpers import rel_fro

pytestmark = pytest.mark.gpu

FORMS = {"fwd_NT": (False, True), "dgrad_NN": (False, False), "wgrad_TN": (True, False)}
# (m, n, k): one tile / several tiles / ragged edges in every dimension / the 1024 layer
SHAPES = [(128, 256, 64), (256, 512, 256), (384, 320, 200), (104, 72, 136), (1024, 1024, 1024)]
# fp32: FMA order only; tf32: 10-bit operand mantissa, checked against the fp32 oracle;
# bf16: operands pre-rounded on both sides, so only accumulation order (fp32 output)
# or one final bf16 rounding (bf16 output) may differ.
TOL = {"fp32": 2e-5, "tf32": 2e-3, "bf16_f32out": 5e-5, "bf16_bf16out": 6e-3}


@pytest.fixture(scope="module")
def dev(native):
    from tbb_test_b200.mlp import MLP
    m = MLP([16, 16], 16)
    yield m
    m.close()


def operands(O, form, m, n, k, seed):
    ta, tb = FORMS[form]
    a = O.fill_uniform(k if ta else m, m if ta else k, seed, -1.0, 1.0)
    b = O.fill_uniform(n if tb else k, k if tb else n, seed + 1, -1.0, 1.0)
    return ta, tb, a, b


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("form", list(FORMS))
def test_fp32(dev, oracle, form, shape):
    from tbb_test_b200 import _capi as K
    m, n, k = shape
    ta, tb, a, b = operands(oracle, form, m, n, k, 11)
    c = dev.sgemm_host(K.PREC_FP32, ta, tb, a, b)
    ref = oracle.sgemm(ta, tb, a, b)
    assert rel_fro(c, ref) <= TOL["fp32"]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("form", list(FORMS))
def test_tf32_tensor_core(dev, oracle, form, shape):
    from tbb_test_b200 import _capi as K
    m, n, k = shape
    ta, tb, a, b = operands(oracle, form, m, n, k, 21)
    before = dev.launch_counts()[1]
    c = dev.sgemm_host(K.PREC_TF32, ta, tb, a, b)
    assert dev.launch_counts()[1] == before + 1, "tensor-core kernel was not used"
    ref = oracle.sgemm(ta, tb, a, b)
    assert rel_fro(c, ref) <= TOL["tf32"]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("form", list(FORMS))
def test_bf16_tensor_core(dev, oracle, form, shape):
    from tbb_test_b200 import _capi as K
    m, n, k = shape
    ta, tb, a, b = operands(oracle, form, m, n, k, 31)
    before = dev.launch_counts()[1]
    c = dev.sgemm_host(K.PREC_BF16, ta, tb, a, b)
    assert dev.launch_counts()[1] == before + 1, "tensor-core kernel was not used"
    ref = oracle.sgemm(ta, tb, oracle.round_bf16(a), oracle.round_bf16(b))
    assert rel_fro(c, ref) <= TOL["bf16_f32out"]


@pytest.mark.parametrize("shape", SHAPES + [(4096, 1024, 136), (2048, 512, 512)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("form", list(FORMS))
def test_fp32_class_tensor_core(dev, oracle, form, shape):
    """B2_PREC_FP32_TC: three tf32 MMAs per k-step on operands split into high and low parts;
    the fp32 bound of the CUDA-core kernel applies (and the plain tf32 kernel misses it by 30x)."""
    from tbb_test_b200 import _capi as K
    m, n, k = shape
    ta, tb, a, b = operands(oracle, form, m, n, k, 23)
    before = dev.launch_counts()[1]
    c = dev.sgemm_host(K.PREC_FP32_TC, ta, tb, a, b)
    assert dev.launch_counts()[1] == before + 1, "tensor-core kernel was not used"
    oracle.use_openblas()
    try:
        ref = oracle.sgemm(ta, tb, a, b)
    finally:
        oracle.use_builtin_gemm()
    assert rel_fro(c, ref) <= TOL["fp32"]
    row_err = np.linalg.norm(c - ref, axis=1) / np.maximum(np.linalg.norm(ref, axis=1), 1e-30)
    assert row_err.max() <= 1e-4


# Shapes wide enough for the 256-row tile mode (two accumulators per CTA sharing each
# B slab): an exact multiple of the tile grid, and a ragged one whose tile count leaves
# a partial last wave that is handed out as 128-row halves.
BIG_SHAPES = [(4096, 4096, 192), (7944, 4096, 136)]


@pytest.mark.parametrize("prec", ["bf16", "tf32"])
@pytest.mark.parametrize("shape", BIG_SHAPES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("form", list(FORMS))
def test_large_tile_mode(dev, oracle, form, shape, prec):
    from tbb_test_b200 import _capi as K
    m, n, k = shape
    ta, tb, a, b = operands(oracle, form, m, n, k, 81)
    before = dev.launch_counts()[1]
    c = dev.sgemm_host(K.PREC_BF16 if prec == "bf16" else K.PREC_TF32, ta, tb, a, b)
    assert dev.launch_counts()[1] == before + 1, "tensor-core kernel was not used"
    oracle.use_openblas()
    try:
        if prec == "bf16":
            ref = oracle.sgemm(ta, tb, oracle.round_bf16(a), oracle.round_bf16(b))
        else:
            ref = oracle.sgemm(ta, tb, a, b)
    finally:
        oracle.use_builtin_gemm()
    # per-row check as well, so that a wrong or missing 128-row block cannot hide in the norm
    assert rel_fro(c, ref) <= (TOL["bf16_f32out"] if prec == "bf16" else TOL["tf32"])
    row_err = np.linalg.norm(c - ref, axis=1) / np.maximum(np.linalg.norm(ref, axis=1), 1e-30)
    assert row_err.max() <= (1e-4 if prec == "bf16" else 4e-3)


@pytest.mark.parametrize("prec", ["fp32", "fp32tc", "tf32", "bf16"])
@pytest.mark.parametrize("shape", [(256, 512, 256), (104, 72, 136)], ids=lambda s: "x".join(map(str, s)))
def test_relu_and_mask_epilogues(dev, oracle, prec, shape):
    from tbb_test_b200 import _capi as K
    P = {"fp32": K.PREC_FP32, "fp32tc": K.PREC_FP32_TC, "tf32": K.PREC_TF32, "bf16": K.PREC_BF16}[prec]
    m, n, k = shape
    rnd = oracle.round_bf16 if prec == "bf16" else (lambda x: x)
    tol = {"fp32": TOL["fp32"], "fp32tc": TOL["fp32"], "tf32": TOL["tf32"], "bf16": TOL["bf16_bf16out"]}[prec]
    # forward with fused ReLU
    ta, tb, a, b = operands(oracle, "fwd_NT", m, n, k, 41)
    c = dev.sgemm_host(P, ta, tb, a, b, epilogue=K.EPI_RELU)
    ref = np.maximum(oracle.sgemm(ta, tb, rnd(a), rnd(b)), 0)
    assert (c >= 0).all()
    assert rel_fro(c, rnd(ref)) <= tol
    # input gradient masked by the sign of the stored activation
    ta, tb, a, b = operands(oracle, "dgrad_NN", m, n, k, 51)
    act = np.maximum(oracle.fill_uniform(m, n, 61, -1.0, 1.0), 0)
    c = dev.sgemm_host(P, ta, tb, a, b, epilogue=K.EPI_MASK, aux=act)
    ref = oracle.sgemm(ta, tb, rnd(a), rnd(b)) * (rnd(act) > 0)
    assert np.array_equal(c != 0, (ref != 0) & (c != 0))  # nothing leaks through the mask
    assert rel_fro(c, rnd(ref)) <= tol


def test_unaligned_shape_falls_back_to_cuda_cores(dev, oracle):
    """Leading dimensions that TMA cannot address (not a multiple of 16 bytes) and the
    N = 1 tail layer of the reference topology are served by the CUDA-core kernel."""
    from tbb_test_b200 import _capi as K
    for (m, n, k) in [(33, 1, 1024), (50, 30, 27)]:
        ta, tb, a, b = operands(oracle, "fwd_NT", m, n, k, 71)
        before = dev.launch_counts()[1]
        c = dev.sgemm_host(K.PREC_BF16, ta, tb, a, b)
        assert dev.launch_counts()[1] == before
        ref = oracle.sgemm(ta, tb, oracle.round_bf16(a), oracle.round_bf16(b))
        assert rel_fro(c, ref) <= TOL["bf16_f32out"]


@pytest.mark.parametrize("variant", ["B2_TC_STREAMK", "B2_TC_PAIR", "B2_TC_HALF_K"])
def test_optional_tile_schedules(dev, oracle, variant, monkeypatch):
    """The opt-in schedules of the tensor-core kernel - stream-K on the tail wave (k-blocks of
    a tile shared between CTAs through an fp32 workspace), CTA pairs (cta_group::2) and
    half-size k-blocks (64-byte swizzle) - give the same results as the default one."""
    from tbb_test_b200 import _capi as K
    monkeypatch.setenv(variant, "1")
    oracle.use_openblas()
    try:
        for form in FORMS:
            for (m, n, k) in [(4096, 4096, 192), (7944, 4096, 136), (1024, 1024, 1024), (256, 512, 2048)]:
                ta, tb, a, b = operands(oracle, form, m, n, k, 91)
                for _ in range(2):  # twice: the workspace flags must be re-armed by the first run
                    c = dev.sgemm_host(K.PREC_BF16, ta, tb, a, b)
                    ref = oracle.sgemm(ta, tb, oracle.round_bf16(a), oracle.round_bf16(b))
                    assert rel_fro(c, ref) <= TOL["bf16_f32out"], (variant, form, m, n, k)
                    row_err = np.linalg.norm(c - ref, axis=1) / np.maximum(np.linalg.norm(ref, axis=1), 1e-30)
                    assert row_err.max() <= 1e-4
    finally:
        oracle.use_builtin_gemm()


# CUDA-core kernels at the edges of their dispatch: 128/64/32-wide tiles with remainders, rows that are and are
# not whole 16-byte pieces, the narrow (N <= 16) and short (M <= 16) forms on both sides of their limits.
# Bound: the oracle adds in k order in fp32 as the tile kernel does (2e-5 covers the other order of the two
# split-K forms: K terms, unit roundoff 6e-8, observed growth sqrt(K)).
@pytest.mark.parametrize("shape", [(33, 65, 31), (129, 64, 64), (70, 1, 64), (70, 2, 63), (77, 16, 200), (77, 17, 200),
                                   (1, 70, 64), (2, 96, 129), (16, 100, 321), (17, 100, 321), (1300, 1100, 20), (500, 509, 40),
                                   (5, 3, 1), (1000, 10, 300), (10, 300, 1000)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("form", list(FORMS))
def test_cuda_core_dispatch_edges(dev, oracle, form, shape):
    from tbb_test_b200 import _capi as K
    m, n, k = shape
    ta, tb, a, b = operands(oracle, form, m, n, k, 101)
    ref = oracle.sgemm(ta, tb, a, b)
    c = dev.sgemm_host(K.PREC_FP32, ta, tb, a, b)
    assert rel_fro(c, ref) <= TOL["fp32"]
    aux = oracle.fill_uniform(m, n, 102, -1.0, 1.0)
    assert rel_fro(dev.sgemm_host(K.PREC_FP32, ta, tb, a, b, epilogue=K.EPI_RELU), np.maximum(ref, 0)) <= 2 * TOL["fp32"]
    assert rel_fro(dev.sgemm_host(K.PREC_FP32, ta, tb, a, b, epilogue=K.EPI_MASK, aux=aux),
                   ref * (aux > 0)) <= 2 * TOL["fp32"]


# fp32 on the CUDA cores at small grids and with rows that are not whole 16-byte pieces: (m, n, k) and the tile it takes
# (csrc/simt_tile.h: 1 64 x 64, 2 64 x 32, 3 32 x 32, 0 the general kernel) with such rows. One and several slabs of 32 k with
# remainders, every tile with remainders.
SMALL_GRIDS = {(33, 18, 1): 3, (65, 33, 31): 3, (64, 96, 32): 3, (31, 100, 33): 3, (300, 301, 95): 3, (129, 257, 97): 3, (500, 509, 97): 2,
               (333, 701, 31): 2, (449, 639, 1): 1, (400, 603, 1): 2, (577, 577, 33): 1, (300, 1003, 65): 1, (701, 803, 129): 1, (640, 900, 64): 0,
               (1001, 1300, 70): 0, (1537, 1003, 65): 0}


@pytest.mark.parametrize("shape", list(SMALL_GRIDS), ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("form", list(FORMS))
def test_fp32_small_grids(dev, native, oracle, form, shape):
    """Against sums in float64, with ReLU, mask and beta. Bound per element: K roundings of the sum of magnitudes, 2^-24 each,
    and two more for alpha and beta."""
    import ctypes as C
    import torch
    from tbb_test_b200 import _capi as K
    m, n, k = shape
    ta, tb, a, b = operands(oracle, form, m, n, k, 121)
    whole = a.shape[1] % 4 == 0 and b.shape[1] % 4 == 0
    host = C.CDLL(native.HOST_LIB)
    assert host.b2h_f32_tile(m, n, 0) == SMALL_GRIDS[shape]
    assert host.b2h_f32_tile(m, n, int(whole)) == (0 if whole and SMALL_GRIDS[shape] < 3 else SMALL_GRIDS[shape])
    ra, rb = (a.T if ta else a).astype(np.float64), (b.T if tb else b).astype(np.float64)
    ref, mag = ra @ rb, np.abs(ra) @ np.abs(rb)
    near = lambda got, want, extra=0.0: (np.abs(got.astype(np.float64) - want) <= (k + 2) * 2.0 ** -24 * (mag + extra) + 1e-30).all()  # noqa: E731
    assert near(dev.sgemm_host(K.PREC_FP32, ta, tb, a, b), ref)
    assert near(dev.sgemm_host(K.PREC_FP32, ta, tb, a, b, epilogue=K.EPI_RELU), np.maximum(ref, 0))
    aux = oracle.fill_uniform(m, n, 122, -1.0, 1.0)
    assert near(dev.sgemm_host(K.PREC_FP32, ta, tb, a, b, epilogue=K.EPI_MASK, aux=aux), ref * (aux > 0))
    ad, bd, cd = (torch.from_numpy(np.ascontiguousarray(t)).cuda() for t in (a, b, aux))
    torch.cuda.synchronize()
    assert dev.lib.b2_sgemm(dev._h, K.PREC_FP32, int(ta), int(tb), m, n, k, 2.0, ad.data_ptr(), a.shape[1], bd.data_ptr(), b.shape[1],
                            -0.5, cd.data_ptr(), n) == K.OK and dev.lib.b2_sync(dev._h) == K.OK
    assert near(cd.cpu().numpy(), 2.0 * ref - 0.5 * aux, mag + np.abs(aux))


@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("shape", [(128, 18, 60), (300, 33, 100), (256, 257, 61), (200, 1003, 64), (1, 301, 33), (700, 1302, 130),
                                   (300, 64, 61)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("entry", ["fp32", "tf32", "noalloc"])
def test_submatrices_of_larger_ones(dev, oracle, entry, form, shape):
    """Operands and result with longer rows than the GEMM uses: what lies between the rows is neither read (NaN there)
    nor written, also where rows end inside a 16-byte piece and where the values are not finite."""
    import torch
    from tbb_test_b200 import _capi as K
    m, n, k = shape
    ta, tb = FORMS[form]

    def framed(rows, cols, seed):
        t = torch.full((rows, (cols + 3) // 4 * 4 + 8), float("nan"))
        t[:, :cols] = torch.from_numpy(oracle.fill_uniform(rows, cols, seed, -1.0, 1.0))
        return t

    if entry == "noalloc" and (m if ta else k) % 8 or entry == "noalloc" and (k if tb else n) % 8:
        pytest.skip("rows the packed copies cannot have")
    a, b = framed(k if ta else m, m if ta else k, 111), framed(n if tb else k, k if tb else n, 112)
    for bad in (False, True):
        if bad:
            a[0, 0] = float("inf")
        c = torch.full((m, (n + 3) // 4 * 4 + 4), 7.0)
        ad, bd, cd = a.cuda(), b.cuda(), c.cuda()
        torch.cuda.synchronize()
        if entry == "noalloc":
            rc = dev.lib.b2_gemm_bf16_noalloc(int(ta), int(tb), m, n, k, ad.data_ptr(), a.shape[1], bd.data_ptr(),
                                              b.shape[1], cd.data_ptr(), c.shape[1], None)
        else:
            rc = dev.lib.b2_sgemm(dev._h, {"fp32": K.PREC_FP32, "tf32": K.PREC_TF32}[entry], int(ta), int(tb), m, n, k, 1.0,
                                  ad.data_ptr(), a.shape[1], bd.data_ptr(), b.shape[1], 0.0, cd.data_ptr(), c.shape[1])
        assert rc == K.OK and dev.lib.b2_sync(dev._h) == K.OK
        got = cd.cpu().numpy()
        assert (got[:, n:] == 7.0).all(), "columns behind the result were written"
        if bad:
            continue
        ra, rb = a[:, :m if ta else k].double(), b[:, :k if tb else n].double()
        if entry == "noalloc":
            ra, rb = ra.float().bfloat16().double(), rb.float().bfloat16().double()
        ref = ((ra.T if ta else ra) @ (rb.T if tb else rb)).numpy()
        assert rel_fro(got[:, :n], ref) <= {"fp32": TOL["fp32"], "tf32": TOL["tf32"], "noalloc": TOL["bf16_f32out"]}[entry]


@pytest.mark.parametrize("m,n,transa", [(4_194_305, 32, False), (4_200_000, 17, True), (2_100_000, 20, False)])
def test_cuda_core_gemm_of_very_many_rows(dev, m, n, transa):
    """Row blocks are the grid's second dimension (65535 at most): from 4 194 241 rows on only the 128-row tile has few
    enough, from 2 097 121 on the 32-row one has too many. Every row against a float64 sum (k = 16 terms, 2^-24 each)."""
    import torch
    from tbb_test_b200 import _capi as K
    k = 16
    g = torch.Generator(device="cuda")
    g.manual_seed(m)
    a = torch.rand((k, m) if transa else (m, k), device="cuda", generator=g) - 0.5
    b = torch.rand((k, n), device="cuda", generator=g) - 0.5
    c = torch.full((m, n), float("nan"), device="cuda")
    torch.cuda.synchronize()
    rc = dev.lib.b2_sgemm(dev._h, K.PREC_FP32, int(transa), 0, m, n, k, 1.0, a.data_ptr(), a.shape[1], b.data_ptr(), n, 0.0,
                          c.data_ptr(), n)
    assert rc == K.OK and dev.lib.b2_sync(dev._h) == K.OK, dev.lib.b2_last_error(dev._h)
    op = (a.T if transa else a).double()
    ref, mag = op @ b.double(), op.abs() @ b.double().abs()
    assert bool(((c.double() - ref).abs() <= 16 * 2.0 ** -24 * mag).all())
