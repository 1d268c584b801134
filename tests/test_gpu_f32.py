"""fp32 kernels (GEMM, GEMV, general / 1x1 / Winograd Conv2D, depthwise) against the CPU
oracle.  Two tolerances are asserted for every comparison: the reference's element-wise form
|got - ref| <= abs_err + rel_err * |ref| (ExpectTensorNear,
test/ccutils/mace/ops/testing/test_utils.h:208-233) with rel_err = 1e-4 (Winograd: 1e-3 against
the DIRECT fp32 convolution, as the 3x3 Winograd path is specified) and abs_err = rel_err *
rms(ref), and the range-normalised max |got - ref| <= tol * max |ref|.  Plus the reference's own
literal known-answer cases."""
import numpy as np
import pytest

from helpers import near_ratio

pytestmark = pytest.mark.gpu
PAD = {"VALID": 0, "SAME": 1, "FULL": 2}


@pytest.fixture(scope="module")
def ctx():
    import mace_b200
    c = mace_b200.Context(0)
    yield c
    c.close()


WORST = {}  # label -> (element-wise ratio, range-normalised error), printed by the last test


def rel_err(got, ref, tol=None, label=None):
    """Range-normalised error; with tol also asserts the element-wise form at rel_err = tol."""
    rng_err = float(np.abs(got.astype(np.float64) - ref).max() / max(np.abs(ref).max(), 1e-30))
    if tol is not None:
        ratio = near_ratio(got, ref, tol)
        if label:
            prev = WORST.get(label, (0.0, 0.0))
            WORST[label] = (max(prev[0], ratio), max(prev[1], rng_err))
        assert ratio <= 1.0, "element-wise |got - ref| <= %g * (rms + |ref|) violated: ratio %.3f" % (tol, ratio)
    return rng_err


@pytest.mark.parametrize("maj", [(0, 0, 0), (1, 0, 0), (0, 1, 0), (1, 1, 0), (0, 0, 1), (1, 1, 1)])
@pytest.mark.parametrize("shape", [(1, 5, 5, 5), (2, 47, 61, 33), (3, 64, 128, 96), (1, 1, 300, 700)])
def test_gemm_f32(ctx, orc, maj, shape):
    """Major-order combinations of test/ccunit/mace/ops/arm/fp32/gemm_test.cc:28-121."""
    batch, M, N, K = shape
    rng = np.random.Generator(np.random.PCG64(M + N))
    A = rng.standard_normal((batch, M, K)).astype(np.float32)
    B = rng.standard_normal((batch, K, N)).astype(np.float32)
    A_st = np.ascontiguousarray(np.swapaxes(A, 1, 2)) if maj[0] else A
    B_st = np.ascontiguousarray(np.swapaxes(B, 1, 2)) if maj[1] else B
    dA, dB, dC = ctx.upload(A_st), ctx.upload(B_st), ctx.alloc(batch * M * N * 4)
    ctx.gemm_f32(dA, dB, dC, batch, M, N, K, bool(maj[0]), bool(maj[1]), bool(maj[2]))
    got = ctx.download(dC, (batch * M * N,), np.float32)
    ref = orc.gemm_f32(A_st, B_st, batch, M, N, K, bool(maj[0]), bool(maj[1]), bool(maj[2]))
    assert rel_err(got, ref, 1e-4, "gemm_f32") <= 1e-4
    for b in (dA, dB, dC):
        b.free()


@pytest.mark.parametrize("shape", [(3, 64, 3200, 64), (1, 200, 1000, 40), (2, 24, 132, 260),
                                   (1, 300, 4100, 512)])
def test_gemm_f32_tensor_core(ctx, orc, shape):
    """Row-major A, B and C with 16-byte aligned rows run on the tensor cores (tf32 MMAs on
    hi/lo split operands); ragged M, N and K tails, with values of mixed magnitude."""
    batch, M, N, K = shape
    rng = np.random.Generator(np.random.PCG64(K))
    A = (rng.standard_normal((batch, M, K)) * np.exp(rng.uniform(-3, 3, (batch, M, K)))).astype(np.float32)
    B = rng.standard_normal((batch, K, N)).astype(np.float32)
    dA, dB, dC = ctx.upload(A), ctx.upload(B), ctx.alloc(batch * M * N * 4)
    before = ctx.launches_tensor_core
    ctx.gemm_f32(dA, dB, dC, batch, M, N, K)
    assert ctx.launches_tensor_core == before + 1, "tensor-core kernel did not run"
    got = ctx.download(dC, (batch * M * N,), np.float32)
    ref = orc.gemm_f32(A, B, batch, M, N, K)
    assert rel_err(got, ref, 1e-4, "gemm_f32_tensor_core") <= 1e-5  # element-wise at the specified 1e-4
    for b in (dA, dB, dC):
        b.free()


def test_gemm_f32_literals_and_one_side_batched(ctx, orc):
    a = np.arange(1, 7, dtype=np.float32)  # matmul_test.cc:55-58
    dA, dC = ctx.upload(a), ctx.alloc(16)
    ctx.gemm_f32(dA, dA, dC, 1, 2, 2, 3)
    assert ctx.download(dC, (4,), np.float32).tolist() == [22, 28, 49, 64]
    rng = np.random.Generator(np.random.PCG64(3))
    A = rng.standard_normal((1, 24, 40)).astype(np.float32)
    B = rng.standard_normal((4, 40, 56)).astype(np.float32)
    dA, dB, dC = ctx.upload(A), ctx.upload(B), ctx.alloc(4 * 24 * 56 * 4)
    ctx.gemm_f32(dA, dB, dC, 4, 24, 56, 40, a_batched=False)
    ref = orc.gemm_f32(A, B, 4, 24, 56, 40, a_batched=False)
    assert rel_err(ctx.download(dC, (4 * 24 * 56,), np.float32), ref, 1e-4, "gemm_f32") <= 1e-4


@pytest.mark.parametrize("shape", [(1, 16, 4), (3, 63, 257), (17, 65, 100), (36, 50, 260), (256, 1000, 2048)])
def test_gemv_f32(ctx, orc, shape):
    batch, rows, K = shape
    rng = np.random.Generator(np.random.PCG64(7))
    lhs = rng.standard_normal((rows, K)).astype(np.float32)
    rhs = rng.standard_normal((batch, K)).astype(np.float32)
    bias = rng.standard_normal(rows).astype(np.float32)
    dl, dr, db, do = ctx.upload(lhs), ctx.upload(rhs), ctx.upload(bias), ctx.alloc(batch * rows * 4)
    ctx.gemv_f32(dl, dr, db, do, batch, rows, K)
    ref = orc.gemv_f32(lhs, rhs, bias, batch, rows, K)
    assert rel_err(ctx.download(do, (batch * rows,), np.float32), ref, 1e-4, "gemv_f32") <= 1e-4


@pytest.mark.parametrize("batch", [65535, 65536, 140001])
@pytest.mark.parametrize("K", [5, 8])
def test_gemv_f32_matrix_per_entry_many_entries(ctx, batch, K):
    """A matrix per batch entry, more entries than a grid has blocks along y.  A sum of K <= 8 rounded products differs
    from the exact one by at most K + 1 units of 2^-24 of the products' absolute sum."""
    rows = 3
    rng = np.random.Generator(np.random.PCG64(batch))
    lhs = rng.standard_normal((batch, rows, K)).astype(np.float32)
    rhs = rng.standard_normal((batch, K)).astype(np.float32)
    dl, dr, do = ctx.upload(lhs), ctx.upload(rhs), ctx.alloc(batch * rows * 4)
    ctx.gemv_f32(dl, dr, None, do, batch, rows, K, lhs_batched=True)
    got = ctx.download(do, (batch, rows), np.float32)
    terms = lhs.astype(np.float64) * rhs[:, None, :]
    assert (np.abs(got - terms.sum(-1)) <= (K + 1) * 2.0 ** -24 * np.abs(terms).sum(-1)).all()
    for b in (dl, dr, do):
        b.free()


def _conv_inputs(shape, fshape, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    x = rng.random(shape, dtype=np.float32)
    fan_in = fshape[1] * fshape[2] * fshape[3]
    f = (rng.standard_normal(fshape) * np.sqrt(2.0 / fan_in)).astype(np.float32)
    bias = (rng.standard_normal(fshape[0]) * 0.01).astype(np.float32)
    return x, f, bias


@pytest.mark.parametrize("case", [
    # N, C, H, W, O, KH, KW, stride, dilation, padding, activation
    (1, 2, 3, 3, 1, 3, 3, 1, 1, "VALID", 0),
    (2, 16, 14, 14, 32, 1, 1, 1, 1, "VALID", 1),      # 1x1 -> batched GEMM
    (1, 3, 33, 35, 8, 7, 7, 2, 1, "SAME", 1),         # ResNet-style 7x7 stride-2 stem
    (2, 8, 15, 15, 16, 1, 1, 2, 1, "SAME", 0),        # 1x1 stride 2
    (1, 4, 12, 13, 6, 3, 3, 1, 2, "SAME", 2),         # dilated, RELUX
    (1, 5, 9, 9, 7, 5, 5, 1, 1, "FULL", 6),           # LEAKYRELU
])
def test_conv2d_f32(ctx, orc, case):
    N, C, H, W, O, KH, KW, st, dil, padding, act = case
    x, f, bias = _conv_inputs((N, C, H, W), (O, C, KH, KW), H * 3 + C)
    Ho, Wo, ph, pw = orc.calc_padding_and_output_size(H, W, KH, KW, (dil, dil), (st, st), PAD[padding])
    ref = orc.conv2d_f32(x, f, bias, (st, st), (dil, dil), (ph >> 1, pw >> 1), (Ho, Wo), act, 0.5, 0.1)
    dx, df, db, do = ctx.upload(x), ctx.upload(f), ctx.upload(bias), ctx.alloc(ref.nbytes)
    ctx.conv2d_f32(dx, df, db, do, N, C, H, W, O, KH, KW, (st, st), (dil, dil), (ph >> 1, pw >> 1),
                   (Ho, Wo), act, 0.5, 0.1)
    assert rel_err(ctx.download(do, ref.shape, np.float32), ref, 1e-4, "conv2d_f32") <= 1e-4


def test_conv2d_f32_reference_literals(ctx, kats):
    """TestNHWCSimple3x3VALID / SAME: all-ones 3x3x2 input and filter, bias 0.1 -> 18.1 ..."""
    for name in ("conv2d_f32_3x3_valid", "conv2d_f32_3x3_same"):
        k = kats[name]
        x = np.ones((1, 2, 3, 3), np.float32)
        f = np.ones((1, 2, 3, 3), np.float32)
        bias = np.array(k["bias"], np.float32)
        same = k["padding"] == "SAME"
        Ho = 3 if same else 1
        pad = (1, 1) if same else (0, 0)
        exp = np.array(k["expected"], np.float32).reshape(1, 1, Ho, Ho)
        dx, df, db, do = ctx.upload(x), ctx.upload(f), ctx.upload(bias), ctx.alloc(exp.nbytes)
        ctx.conv2d_f32(dx, df, db, do, 1, 2, 3, 3, 1, 3, 3, (1, 1), (1, 1), pad, (Ho, Ho))
        np.testing.assert_allclose(ctx.download(do, exp.shape, np.float32), exp, rtol=1e-5)
        for tile in (2, 6):
            ctx.winograd_f32(dx, df, db, do, 1, 2, 3, 3, 1, pad, (Ho, Ho), tile=tile)
            np.testing.assert_allclose(ctx.download(do, exp.shape, np.float32), exp, rtol=1e-4)


@pytest.mark.parametrize("case", [
    # N, C, H, W, O, padding, activation
    (1, 8, 9, 9, 8, "SAME", 0),        # small input -> F(2,3)
    (2, 16, 14, 17, 24, "VALID", 1),
    (1, 8, 20, 20, 16, "SAME", 0),     # larger than 16x16 -> F(6,3)
    (2, 64, 56, 56, 64, "SAME", 1),    # config-1 shape, reduced batch
    (1, 32, 31, 29, 40, "VALID", 2),   # tile tails
])
def test_winograd_f32(ctx, orc, case):
    N, C, H, W, O, padding, act = case
    x, f, bias = _conv_inputs((N, C, H, W), (O, C, 3, 3), H + C)
    Ho, Wo, ph, pw = orc.calc_padding_and_output_size(H, W, 3, 3, (1, 1), (1, 1), PAD[padding])
    direct = orc.conv2d_f32(x, f, bias, (1, 1), (1, 1), (ph >> 1, pw >> 1), (Ho, Wo), act, 0.5, 0.0)
    dx, df, db, do = ctx.upload(x), ctx.upload(f), ctx.upload(bias), ctx.alloc(direct.nbytes)
    ctx.winograd_f32(dx, df, db, do, N, C, H, W, O, (ph >> 1, pw >> 1), (Ho, Wo), act, 0.5, 0.0)
    got = ctx.download(do, direct.shape, np.float32)
    assert rel_err(got, direct, 1e-3, "winograd_vs_direct") <= 1e-3
    # against the oracle's Winograd restatement (same algorithm, same tile rule): tighter
    wino = orc.winograd_f32(x, f, bias, (ph >> 1, pw >> 1), (Ho, Wo), act, 0.5, 0.0)
    assert rel_err(got, wino, 1e-4, "winograd_vs_oracle_winograd") <= 1e-4
    # cached transformed filter gives the same result
    tile = 6 if (H > 16 and W > 16) else 2
    dU = ctx.alloc((tile + 2) ** 2 * O * C * 4)
    ctx.winograd_transform_filter(df, dU, C, O, tile)
    ctx.winograd_f32(dx, None, db, do, N, C, H, W, O, (ph >> 1, pw >> 1), (Ho, Wo), act, 0.5, 0.0,
                     transformed=dU)
    assert np.array_equal(ctx.download(do, direct.shape, np.float32), got)
    # the one-thread-per-tile output transform computes the same values as the plane-at-a-time one
    ctx.set_option("wino_plane", 0)
    try:
        ctx.winograd_f32(dx, df, db, do, N, C, H, W, O, (ph >> 1, pw >> 1), (Ho, Wo), act, 0.5, 0.0)
    finally:
        ctx.set_option("wino_plane", 1)
    assert np.array_equal(ctx.download(do, direct.shape, np.float32), got)


@pytest.fixture(params=[(0, 0), (64, 1), (64, 8), (128, 2)], ids=str)
def gather(ctx, request):
    """The self-fetching kernel wherever it can run, at a tile width and number of depth runs (0: by rule)."""
    ctx.set_option("f32_gather", 2)
    ctx.set_option("f32_bn", request.param[0])
    ctx.set_option("f32_splits", request.param[1])
    yield
    for name in ("f32_gather", "f32_bn", "f32_splits"):
        ctx.set_option(name, 0)


@pytest.mark.parametrize("case", [
    # N, C, H, W, O, kernel, stride, dilation, padding: odd maps and channel counts, tails of pixels (also over
    # several images), of channels and of the depth, every kind of window
    (2, 35, 9, 11, 73, (5, 5), 1, 1, "SAME"), (3, 33, 7, 7, 130, (3, 3), 2, 1, "SAME"), (1, 3, 30, 31, 64, (7, 7), 2, 1, "SAME"),
    (2, 64, 13, 14, 64, (1, 1), 1, 1, "SAME"), (2, 70, 15, 13, 40, (1, 1), 2, 1, "VALID"), (1, 20, 17, 19, 65, (3, 3), 1, 2, "SAME"),
    (5, 16, 6, 5, 33, (1, 5), 1, 1, "SAME"), (1, 200, 8, 8, 129, (3, 3), 1, 1, "VALID")])
@pytest.mark.parametrize("residual", [False, True])
def test_conv2d_f32_without_column_matrix(ctx, orc, gather, case, residual):
    N, C, H, W, O, k, s, d, pad = case
    rng = np.random.Generator(np.random.PCG64(C + O))
    x = rng.standard_normal((N, C, H, W)).astype(np.float32)
    f = rng.standard_normal((O, C) + k).astype(np.float32)
    bias = rng.standard_normal(O).astype(np.float32)
    ho, wo, ph, pw = orc.calc_padding_and_output_size(H, W, k[0], k[1], (d, d), (s, s), PAD[pad])
    dx, df, db = ctx.upload(x), ctx.upload(f), ctx.upload(bias)
    do = ctx.alloc(N * O * ho * wo * 4)
    before = ctx.launches_tensor_core
    args = (N, C, H, W, O, k[0], k[1], (s, s), (d, d), (ph >> 1, pw >> 1), (ho, wo), 1)
    if residual:
        r = rng.standard_normal((N, O, ho, wo)).astype(np.float32)
        dr = ctx.upload(r)
        ctx.conv2d_f32_residual(dx, df, db, dr, do, *args)
        ref = np.maximum(orc.conv2d_f32(x, f, bias, (s, s), (d, d), (ph >> 1, pw >> 1), (ho, wo), 0) + r, 0)
        dr.free()
    else:
        ctx.conv2d_f32(dx, df, db, do, *args)
        ref = orc.conv2d_f32(x, f, bias, (s, s), (d, d), (ph >> 1, pw >> 1), (ho, wo), 1)
    assert ctx.launches_tensor_core == before + 1
    assert rel_err(ctx.download(do, ref.shape, np.float32), ref, 1e-4, "conv2d_f32 without columns") <= 5e-5
    for b in (dx, df, db, do):
        b.free()


@pytest.mark.parametrize("maj", [(0, 0, 0), (1, 0, 0), (0, 1, 0), (1, 1, 0), (0, 0, 1), (0, 1, 1), (1, 1, 1)])
@pytest.mark.parametrize("shape", [(1, 5, 5, 5), (2, 130, 61, 33), (3, 64, 128, 96), (1, 1, 300, 701), (2, 200, 67, 520)])
def test_gemm_f32_of_any_layout_on_tensor_cores(ctx, orc, gather, maj, shape):
    batch, M, N, K = shape
    rng = np.random.Generator(np.random.PCG64(M + N))
    A = rng.standard_normal((batch, M, K)).astype(np.float32)
    B = rng.standard_normal((batch, K, N)).astype(np.float32)
    A_st = np.ascontiguousarray(np.swapaxes(A, 1, 2)) if maj[0] else A
    B_st = np.ascontiguousarray(np.swapaxes(B, 1, 2)) if maj[1] else B
    dA, dB, dC = ctx.upload(A_st), ctx.upload(B_st), ctx.alloc(batch * M * N * 4)
    before = ctx.launches_tensor_core
    ctx.gemm_f32(dA, dB, dC, batch, M, N, K, bool(maj[0]), bool(maj[1]), bool(maj[2]))
    assert ctx.launches_tensor_core == before + 1
    ref = orc.gemm_f32(A_st, B_st, batch, M, N, K, bool(maj[0]), bool(maj[1]), bool(maj[2]))
    assert rel_err(ctx.download(dC, (batch * M * N,), np.float32), ref, 1e-4, "gemm_f32 of any layout") <= 5e-5
    for b in (dA, dB, dC):
        b.free()


def _norm_err(got, exact):
    return float(np.linalg.norm(got.astype(np.float64) - exact) / np.linalg.norm(exact))


def _with_options(ctx, call, **options):
    for k, v in options.items():
        ctx.set_option(k, v)
    try:
        return call()
    finally:
        for k in options:
            ctx.set_option(k, 1 if k == "tensor_cores" else 0)


# depths on both sides of every line of the rule, and long ones
@pytest.mark.parametrize("K", [16, 47, 48, 64, 65, 72, 96, 200, 383, 384, 1024, 3000])
@pytest.mark.parametrize("positive", [False, True])
def test_gemm_f32_is_as_accurate_as_fmas(ctx, K, positive):
    """A product in a layout that only the self-fetching kernel and the CUDA cores take: by rule its error against float64
    is no larger than that of the CUDA cores' chain of fp32 FMAs (2 %: both are taken from 130 000 values)."""
    batch, M, N = 2, 200, 333
    rng = np.random.Generator(np.random.PCG64(K))
    draw = rng.random if positive else rng.standard_normal
    A, B = draw((batch, M, K)).astype(np.float32), draw((batch, N, K)).astype(np.float32)
    exact = A.astype(np.float64) @ np.swapaxes(B, 1, 2).astype(np.float64)
    dA, dB, dC = ctx.upload(A), ctx.upload(B), ctx.alloc(batch * M * N * 4)

    def run():
        ctx.gemm_f32(dA, dB, dC, batch, M, N, K, b_col_major=True)
        return _norm_err(ctx.download(dC, (batch, M, N), np.float32), exact)

    fma = _with_options(ctx, run, tensor_cores=0)
    assert run() <= 1.02 * fma
    if mb_f32_gather_run(K):   # the other tile width, and the depth cut
        for bn, splits in ((64, 1), (64, 8), (128, 1)):
            assert _with_options(ctx, run, f32_gather=2, f32_bn=bn, f32_splits=splits) <= 1.02 * fma, (bn, splits)
    for b in (dA, dB, dC):
        b.free()


def mb_f32_gather_run(K):
    """As in gemm_f32_gather.cuh."""
    return 0 if K < 48 or 64 < K < 72 else 1 if K < 384 else 2


@pytest.mark.parametrize("case", [
    # few results, little work, 1x1 with rows that TMA does not take: kernel, N, C, HW, O, stride
    (3, 1, 64, 4, 80, 1), (3, 1, 16, 14, 16, 1), (1, 2, 75, 28, 60, 1), (5, 1, 40, 7, 33, 2), (1, 1, 35, 12, 40, 1)])
def test_small_conv2d_f32_is_as_accurate_as_fmas(ctx, orc, case):
    k, N, C, HW, O, s = case
    rng = np.random.Generator(np.random.PCG64(C))
    x = rng.standard_normal((N, C, HW, HW)).astype(np.float32)
    f = rng.standard_normal((O, C, k, k)).astype(np.float32)
    ho, wo, ph, pw = orc.calc_padding_and_output_size(HW, HW, k, k, (1, 1), (s, s), PAD["SAME"])
    padded = np.zeros((N, C, HW + 2 * k, HW + 2 * k))
    padded[:, :, ph >> 1:(ph >> 1) + HW, pw >> 1:(pw >> 1) + HW] = x
    exact = sum(np.einsum("ncyx,oc->noyx", padded[:, :, i:i + s * ho:s, j:j + s * wo:s], f[:, :, i, j].astype(np.float64))
                for i in range(k) for j in range(k))
    dx, df, do = ctx.upload(x), ctx.upload(f), ctx.alloc(exact.size * 4)

    def run():
        ctx.conv2d_f32(dx, df, None, do, N, C, HW, HW, O, k, k, (s, s), (1, 1), (ph >> 1, pw >> 1), (ho, wo))
        return _norm_err(ctx.download(do, exact.shape, np.float32), exact)

    fma = _with_options(ctx, run, tensor_cores=0)
    assert run() <= 1.1 * fma  # (a few thousand values only)
    for b in (dx, df, do):
        b.free()


@pytest.mark.parametrize("positive", [False, True])
@pytest.mark.parametrize("C,O", [(48, 20), (64, 18), (64, 5), (80, 14)])
def test_short_conv2d_f32_is_as_accurate_as_fmas(ctx, C, O, positive):
    """1x1 convolutions of 14 x 15 pixels with too little work for a column matrix, at the depths of three accumulators.
    (6 %: from a few thousand values.)"""
    rng = np.random.Generator(np.random.PCG64(C + O))
    draw = rng.random if positive else rng.standard_normal
    x, f = draw((1, C, 14, 15)).astype(np.float32), draw((O, C, 1, 1)).astype(np.float32)
    exact = np.einsum("nchw,oc->nohw", x.astype(np.float64), f[:, :, 0, 0].astype(np.float64))
    dx, df, do = ctx.upload(x), ctx.upload(f), ctx.alloc(exact.size * 4)

    def run():
        ctx.conv2d_f32(dx, df, None, do, 1, C, 14, 15, O, 1, 1, (1, 1), (1, 1), (0, 0), (14, 15))
        return _norm_err(ctx.download(do, exact.shape, np.float32), exact)

    fma = _with_options(ctx, run, tensor_cores=0)
    before = ctx.launches_tensor_core
    assert run() <= 1.06 * fma
    assert ctx.launches_tensor_core == before + 1
    for b in (dx, df, do):
        b.free()


@pytest.mark.parametrize("case,tensor_core", [
    # kernel, C, HW, O: a single pixel, a few, on both sides of the depth from which the tensor cores are accurate enough
    ((1, 100, 1, 10), 1), ((1, 64, 4, 16), 1), ((3, 16, 3, 4), 1), ((1, 48, 2, 8), 1), ((1, 47, 2, 8), 0), ((3, 5, 9, 9), 0)])
def test_smallest_conv2d_f32(ctx, orc, case, tensor_core):
    """A chain of K FMAs differs from the exact sum by at most K units of 2^-24 of the sum of the products' absolute
    values (to first order: one more for the rest); the tensor cores' short runs by less."""
    k, C, HW, O = case
    K = C * k * k
    rng = np.random.Generator(np.random.PCG64(K))
    x = rng.standard_normal((1, C, HW, HW)).astype(np.float32)
    f = rng.standard_normal((O, C, k, k)).astype(np.float32)
    pad = (k - 1) // 2
    padded = np.pad(x.astype(np.float64), ((0, 0), (0, 0), (pad, pad), (pad, pad)))
    windows = np.lib.stride_tricks.sliding_window_view(padded, (k, k), (2, 3))
    dx, df, do = ctx.upload(x), ctx.upload(f), ctx.alloc(O * HW * HW * 4)
    before = ctx.launches_tensor_core
    ctx.conv2d_f32(dx, df, None, do, 1, C, HW, HW, O, k, k, (1, 1), (1, 1), (pad, pad), (HW, HW))
    assert ctx.launches_tensor_core - before == tensor_core
    got = ctx.download(do, (1, O, HW, HW), np.float32)
    exact = np.einsum("nchwij,ocij->nohw", windows, f.astype(np.float64))
    terms = np.einsum("nchwij,ocij->nohw", np.abs(windows), np.abs(f.astype(np.float64)))
    assert (np.abs(got - exact) <= (K + 1) * 2.0 ** -24 * terms).all()
    for b in (dx, df, do):
        b.free()


@pytest.mark.parametrize("shape", [(9, 300, 256), (31, 200, 1000), (33, 300, 1001)])
def test_gemv_f32_of_a_few_vectors_is_as_accurate_as_one_by_one(ctx, shape):
    batch, rows, K = shape
    rng = np.random.Generator(np.random.PCG64(batch))
    w = rng.standard_normal((rows, K)).astype(np.float32)
    x = rng.standard_normal((batch, K)).astype(np.float32)
    exact = x.astype(np.float64) @ w.T.astype(np.float64)
    dw, dx, do = ctx.upload(w), ctx.upload(x), ctx.alloc(batch * rows * 4)
    ctx.gemv_f32(dw, dx, None, do, batch, rows, K)
    together = _norm_err(ctx.download(do, (batch, rows), np.float32), exact)
    one = np.empty((batch, rows), np.float32)
    for b in range(batch):
        d1 = ctx.upload(x[b])
        ctx.gemv_f32(dw, d1, None, do, 1, rows, K)
        one[b] = ctx.download(do, (rows,), np.float32)
        d1.free()
    assert together <= 1.02 * _norm_err(one, exact)
    for b in (dw, dx, do):
        b.free()


@pytest.mark.parametrize("shape", [
    # N, C, HW, O: 3x3 convolutions that the rule may take from the Winograd kernels, F(2,3) and F(6,3)
    (1, 16, 7, 16), (3, 33, 9, 65), (7, 130, 14, 130), (1, 256, 14, 256), (1, 512, 7, 512), (2, 64, 56, 64), (9, 96, 17, 96)])
def test_conv3x3_f32_is_as_accurate_as_winograd(ctx, orc, shape):
    N, C, HW, O = shape
    rng = np.random.Generator(np.random.PCG64(C))
    x = rng.standard_normal((N, C, HW, HW)).astype(np.float32)
    f = (rng.standard_normal((O, C, 3, 3)) * np.sqrt(2.0 / (9 * C))).astype(np.float32)
    padded = np.pad(x.astype(np.float64), ((0, 0), (0, 0), (1, 1), (1, 1)))
    exact = sum(np.einsum("ncyx,oc->noyx", padded[:, :, i:i + HW, j:j + HW], f[:, :, i, j].astype(np.float64), optimize=True)
                for i in range(3) for j in range(3))
    tile = 6 if HW > 16 else 2
    dx, df, do = ctx.upload(x), ctx.upload(f), ctx.alloc(exact.size * 4)
    dt = ctx.alloc((tile + 2) ** 2 * O * C * 4)
    ctx.winograd_transform_filter(df, dt, C, O, tile)

    def run():
        ctx.winograd_f32(dx, df, None, do, N, C, HW, HW, O, (1, 1), (HW, HW), tile=tile, transformed=dt)
        return _norm_err(ctx.download(do, exact.shape, np.float32), exact)

    winograd = _with_options(ctx, run, f32_gather=1)
    assert run() <= 1.05 * winograd
    assert _with_options(ctx, run, f32_gather=2) <= 1.05 * winograd  # the direct convolution, whatever the rule says
    for b in (dx, df, do, dt):
        b.free()


@pytest.mark.parametrize("what", ["large product", "transposed", "direct", "stem", "small product", "small convolution"])
def test_f32_results_do_not_depend_on_a_rows_range(ctx, what):
    """By rule, whatever kernel: a column (channel) 1e6 times larger, whose weights are as much smaller or zero."""
    rng = np.random.Generator(np.random.PCG64(4))
    if what in ("large product", "transposed", "small product"):
        M, N, K = {"large product": (256, 76800, 512), "transposed": (1024, 1024, 1024), "small product": (64, 192, 320)}[what]
        a, b = rng.standard_normal((1, M, K)).astype(np.float32), rng.standard_normal((1, K, N)).astype(np.float32)

        def run():
            col = what == "transposed"
            da, db, dc = ctx.upload(a), ctx.upload(b.transpose(0, 2, 1) if col else b), ctx.alloc(M * N * 4)
            ctx.gemm_f32(da, db, dc, 1, M, N, K, b_col_major=col)
            got = ctx.download(dc, (M, N), np.float32)[:, :2000]
            for d in (da, db, dc):
                d.free()
            return _norm_err(got, a[0].astype(np.float64) @ b[0, :, :2000].astype(np.float64))
    else:
        n, C, HW, O, k, st = {"direct": (16, 64, 28, 64, 3, 1), "stem": (24, 3, 224, 64, 7, 2), "small convolution": (1, 40, 9, 30, 3, 1)}[what]
        b, a = rng.standard_normal((n, C, HW, HW)).astype(np.float32), rng.standard_normal((O, C, k, k)).astype(np.float32)
        ho = HW // st

        def run():
            db, da, dc = ctx.upload(b), ctx.upload(a), ctx.alloc(n * O * ho * ho * 4)
            ctx.conv2d_f32(db, da, None, dc, n, C, HW, HW, O, k, k, (st, st), (1, 1), (k // 2, k // 2), (ho, ho))
            got = ctx.download(dc, (n, O, ho, ho), np.float32)[:1]
            for d in (da, db, dc):
                d.free()
            padded = np.pad(b[:1].astype(np.float64), ((0, 0), (0, 0), (k // 2,) * 2, (k // 2,) * 2))
            exact = sum(np.einsum("ncyx,oc->noyx", padded[:, :, i:i + st * ho:st, j:j + st * ho:st], a[:, :, i, j].astype(np.float64),
                                  optimize=True) for i in range(k) for j in range(k))
            return _norm_err(got, exact)

    plain = run()
    b[:, 1] *= np.float32(1e6)
    a[(np.s_[:], np.s_[:], 1) if a.ndim == 3 else (np.s_[:], 1)] *= np.float32(1e-6)
    assert run() <= 1.1 * plain
    a[(np.s_[:], np.s_[:], 1) if a.ndim == 3 else (np.s_[:], 1)] = 0
    assert run() <= 1.1 * plain


@pytest.mark.parametrize("shape", [(32, 64, 56, 64), (1, 64, 14, 64)])
def test_conv3x3_f32_without_the_transformed_filter(shape):
    """Where the transformed filter is not read it need not be made; where it is read the call makes it."""
    import mace_b200
    L = mace_b200.lib()
    N, C, HW, O = shape
    rng = np.random.Generator(np.random.PCG64(C))
    c = mace_b200.Context(0)
    dx, do = c.upload(rng.standard_normal((N, C, HW, HW)).astype(np.float32)), c.alloc(N * O * HW * HW * 4)
    df = c.upload((rng.standard_normal((O, C, 3, 3)) * np.sqrt(2.0 / (9 * C))).astype(np.float32))
    tile = 6 if HW > 16 else 2
    dt = c.alloc((tile + 2) ** 2 * O * C * 4)
    c.winograd_transform_filter(df, dt, C, O, tile)

    def asked():
        return L.mb_conv3x3_winograd_f32_reads_transformed(c.h, dx.ptr, df.ptr, N, C, HW, HW, O, 1, 1, HW, HW, tile)

    def run(transformed):
        c.winograd_f32(dx, df, None, do, N, C, HW, HW, O, (1, 1), (HW, HW), tile=tile, transformed=transformed)
        return c.download(do, (N, O, HW, HW), np.float32)

    try:
        assert asked() == 0
        assert np.array_equal(run(df), run(dt))
        c.set_option("f32_gather", 1)
        c.set_option("f32_direct", 1)
        assert asked() == 1
        assert np.array_equal(run(df), run(dt))
        c.set_option("f32_direct", 2)
        assert asked() == 0
        assert np.array_equal(run(df), run(dt))
    finally:
        L.mb_set_runtime_failure_ratio(0.0)
        c.close()


@pytest.mark.parametrize("maj", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("c_col", [False, True])
@pytest.mark.parametrize("shape", [(1, 1, 1, 1), (2, 63, 65, 31), (1, 64, 64, 32), (3, 65, 130, 33), (1, 130, 61, 65), (70000, 2, 3, 5)])
def test_gemm_f32_on_cuda_cores(ctx, maj, c_col, shape):
    """Edges of the 64 x 64 x 32 tiles in every layout.  A chain of K FMAs differs from the exact sum by at most K units of
    2^-24 of the sum of the products' absolute values (to first order: one more for the rest)."""
    batch, M, N, K = shape
    rng = np.random.Generator(np.random.PCG64(M))
    A = rng.standard_normal((batch, M, K)).astype(np.float32)
    B = rng.standard_normal((batch, K, N)).astype(np.float32)
    dA = ctx.upload(np.ascontiguousarray(np.swapaxes(A, 1, 2)) if maj[0] else A)
    dB = ctx.upload(np.ascontiguousarray(np.swapaxes(B, 1, 2)) if maj[1] else B)
    dC = ctx.alloc(batch * M * N * 4)
    ctx.gemm_f32(dA, dB, dC, batch, M, N, K, bool(maj[0]), bool(maj[1]), c_col)
    got = ctx.download(dC, (batch, N, M) if c_col else (batch, M, N), np.float32)
    got = np.swapaxes(got, 1, 2) if c_col else got
    A, B = A.astype(np.float64), B.astype(np.float64)
    # (more entries than a grid has blocks along z: the tensor cores take them, three tf32 products)
    units = K + 1 if batch <= 65535 else 32
    assert (np.abs(got - A @ B) <= units * 2.0 ** -24 * (np.abs(A) @ np.abs(B))).all()
    for b in (dA, dB, dC):
        b.free()


@pytest.mark.parametrize("maj", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("width,splits", [(64, 1), (64, 8), (128, 1)])
@pytest.mark.parametrize("shape", [(1, 5, 63, 48), (2, 129, 65, 64), (1, 130, 129, 72), (1, 127, 200, 97), (20, 200, 300, 129),
                                   (1, 128, 128, 384), (2, 140, 70, 449)])
def test_gemm_f32_in_short_runs(ctx, maj, width, splits, shape):
    """The forms whose sums leave the tensor core every few steps, at the edges of tiles, steps and runs, with several tiles
    per CTA.  Per product 2^-22 from the split; per MMA of a run of at most 8 two units of 2^-23 from the accumulator; one of
    2^-24 per run from the sums."""
    batch, M, N, K = shape
    rng = np.random.Generator(np.random.PCG64(K))
    A = rng.standard_normal((batch, M, K)).astype(np.float32)
    B = rng.standard_normal((batch, K, N)).astype(np.float32)
    dA = ctx.upload(np.ascontiguousarray(np.swapaxes(A, 1, 2)) if maj[0] else A)
    dB = ctx.upload(np.ascontiguousarray(np.swapaxes(B, 1, 2)) if maj[1] else B)
    dC = ctx.alloc(batch * M * N * 4)
    before = ctx.launches_tensor_core
    _with_options(ctx, lambda: ctx.gemm_f32(dA, dB, dC, batch, M, N, K, bool(maj[0]), bool(maj[1])), f32_gather=2, f32_bn=width,
                  f32_splits=splits)
    assert ctx.launches_tensor_core == before + 1
    got = ctx.download(dC, (batch, M, N), np.float32)
    A, B = A.astype(np.float64), B.astype(np.float64)
    bound = 2.0 ** -22 + 8 * 2 * 2.0 ** -23 + (K // 32 + 1) * 2.0 ** -24
    if maj == (0, 0) and N % 4 == 0:  # (in TMA's layout: one run)
        bound = 2.0 ** -21 + 3 * (K // 8 + 1) * 2 * 2.0 ** -23
    assert (np.abs(got - A @ B) <= bound * (np.abs(A) @ np.abs(B))).all()
    for b in (dA, dB, dC):
        b.free()


INF_CASES = [("inf", np.inf), ("-inf", -np.inf), ("largest", np.finfo(np.float32).max), ("nan", np.nan)]


@pytest.mark.parametrize("name,value", INF_CASES)
@pytest.mark.parametrize("maj", [(0, 1), (1, 0)])
@pytest.mark.parametrize("shape", [(1, 30, 37, 20), (2, 130, 70, 64), (1, 140, 200, 100), (1, 129, 65, 1000)])
def test_gemm_f32_of_infinite_operands(ctx, maj, shape, name, value):
    """Infinities, values at the end of the range and NaNs give what IEEE arithmetic gives, at every tile width and with
    the depth cut.  (The other operands are small powers of two, exact in every split, and no finite sum overflows.)"""
    batch, M, N, K = shape
    rng = np.random.Generator(np.random.PCG64(M))
    A = rng.choice(np.float32([-0.5, -0.25, 0.25, 0.5]), (batch, M, K))
    B = rng.choice(np.float32([-0.5, -0.25, 0.25, 0.5]), (batch, K, N))
    A[0, M - 1, K // 2] = value      # a row with one of them,
    A[0, 3, 1], B[0, 1, 5] = value, 0  # one that meets a zero,
    B[-1, K - 1, N - 1] = value      # and a column
    B[0, [K // 2, 1], N - 1] = A[0, [M - 1, 3], K - 1] = 0.25  # (where both meet, nothing cancels)
    dA = ctx.upload(np.ascontiguousarray(np.swapaxes(A, 1, 2)) if maj[0] else A)
    dB = ctx.upload(np.ascontiguousarray(np.swapaxes(B, 1, 2)) if maj[1] else B)
    dC = ctx.alloc(batch * M * N * 4)
    with np.errstate(all="ignore"):
        exact = np.einsum("bmk,bkn->bmn", A.astype(np.float64), B.astype(np.float64))
    settings = [{}] + ([dict(f32_gather=2, f32_bn=64, f32_splits=8), dict(f32_gather=2, f32_bn=128, f32_splits=1)]
                       if mb_f32_gather_run(K) else [])
    for options in settings:
        _with_options(ctx, lambda: ctx.gemm_f32(dA, dB, dC, batch, M, N, K, bool(maj[0]), bool(maj[1])), **options)
        got = ctx.download(dC, (batch, M, N), np.float32)
        assert np.array_equal(np.isnan(got), np.isnan(exact)), options
        with np.errstate(all="ignore"):
            near = np.isnan(exact) | (got == exact) | (np.abs(got - exact) <= 1e-6 * (np.abs(exact) + K))
        assert near.all(), options
    for b in (dA, dB, dC):
        b.free()


@pytest.mark.parametrize("splits", [0, 1, 4])
def test_conv2d_f32_of_an_infinite_pixel(ctx, orc, splits):
    """A small convolution (padding taps left out, bias, activation, residual) around one infinite pixel and one infinite
    weight."""
    N, C, HW, O = 1, 32, 5, 70
    rng = np.random.Generator(np.random.PCG64(0))
    x = rng.choice(np.float32([-0.5, 0.25, 0.5]), (N, C, HW, HW))
    f = rng.choice(np.float32([-0.5, 0.25, 0.5]), (O, C, 3, 3))
    bias, r = rng.standard_normal(O).astype(np.float32), rng.standard_normal((N, O, HW, HW)).astype(np.float32)
    x[0, 3, 0, 1], f[7, 2, 0, 0] = np.inf, -np.inf
    ref = np.fmax(orc.conv2d_f32(x, f, bias, (1, 1), (1, 1), (1, 1), (HW, HW), 0) + r, 0)  # (a NaN becomes 0, as in ref::Activation)
    assert np.isinf(ref).any() and np.isfinite(ref).any()
    dx, df, db, dr, do = (ctx.upload(a) for a in (x, f, bias, r, np.zeros_like(ref)))
    options = dict(f32_gather=2, f32_bn=64, f32_splits=splits) if splits else {}
    _with_options(ctx, lambda: ctx.conv2d_f32_residual(dx, df, db, dr, do, N, C, HW, HW, O, 3, 3, (1, 1), (1, 1), (1, 1),
                                                       (HW, HW), 1), **options)
    got = ctx.download(do, ref.shape, np.float32)
    assert np.array_equal(np.isinf(got), np.isinf(ref)) and np.array_equal(np.isnan(got), np.isnan(ref))
    finite = np.isfinite(ref)
    assert np.abs(got[finite] - ref[finite]).max() <= 1e-4
    for b in (dx, df, db, dr, do):
        b.free()


@pytest.mark.parametrize("shape", [(1, 1000, 2048), (3, 77, 1023), (40, 130, 516)])
def test_gemv_f32_on_tensor_cores(ctx, orc, gather, shape):
    batch, rows, K = shape
    rng = np.random.Generator(np.random.PCG64(rows))
    w = rng.standard_normal((rows, K)).astype(np.float32)
    x = rng.standard_normal((batch, K)).astype(np.float32)
    bias = rng.standard_normal(rows).astype(np.float32)
    dw, dx, db, do = ctx.upload(w), ctx.upload(x), ctx.upload(bias), ctx.alloc(batch * rows * 4)
    ctx.gemv_f32(dw, dx, db, do, batch, rows, K)
    ref = orc.gemv_f32(w, x, bias, batch, rows, K, False, True).reshape(batch, rows)
    assert rel_err(ctx.download(do, ref.shape, np.float32), ref, 1e-4, "gemv_f32 on tensor cores") <= 5e-5
    for b in (dw, dx, db, do):
        b.free()


@pytest.mark.parametrize("k", [3, 5])
@pytest.mark.parametrize("stride", [1, 2])
@pytest.mark.parametrize("shape", [(1, 3, 7, 9, 1), (2, 300, 33, 31, 1), (3, 5, 20, 65, 2), (4, 130, 57, 112, 1),
                                   (8, 96, 56, 56, 1)])
def test_dwconv_f32_rows(ctx, orc, k, stride, shape):
    """Runs of one and two rows, ragged last runs, narrow maps, a channel multiplier; 3x3 on rows of whole words takes the
    kernel of test_dwconv_f32_whole_words.  The longer runs: test_dwconv_f32_long_runs."""
    N, C, H, W, mult = shape
    rng = np.random.Generator(np.random.PCG64(C + k))
    x = rng.standard_normal((N, C, H, W)).astype(np.float32)
    f = rng.standard_normal((mult, C, k, k)).astype(np.float32)
    bias = rng.standard_normal(C * mult).astype(np.float32)
    ho, wo, ph, pw = orc.calc_padding_and_output_size(H, W, k, k, (1, 1), (stride, stride), 1)
    ref = orc.dwconv_f32(x, f, bias, (stride, stride), (1, 1), (ph >> 1, pw >> 1), (ho, wo), 1)
    dx, df, db, do = ctx.upload(x), ctx.upload(f), ctx.upload(bias), ctx.alloc(ref.nbytes)
    ctx.dwconv_f32(dx, df, db, do, N, C, H, W, mult, k, k, (stride, stride), (1, 1), (ph >> 1, pw >> 1), (ho, wo), 1)
    assert rel_err(ctx.download(do, ref.shape, np.float32), ref, 1e-5, "dwconv_f32") <= 1e-5
    for b in (dx, df, db, do):
        b.free()


@pytest.mark.parametrize("stride,shape", [
    # one word per row, a multiplier, ragged runs of 2, 4 and 8 rows
    (1, (1, 1, 5, 4, 1)), (2, (1, 1, 5, 4, 1)), (1, (2, 3, 7, 8, 2)), (2, (2, 3, 7, 8, 2)), (1, (4, 64, 57, 112, 1)),
    (2, (9, 64, 111, 108, 1)), (2, (25, 64, 113, 112, 1)), (1, (7, 64, 113, 112, 1)), (1, (13, 64, 115, 112, 1))])
def test_dwconv_f32_whole_words(ctx, orc, stride, shape):
    N, C, H, W, mult = shape
    rng = np.random.Generator(np.random.PCG64(N + W))
    x = rng.standard_normal((N, C, H, W)).astype(np.float32)
    f = rng.standard_normal((mult, C, 3, 3)).astype(np.float32)
    bias = rng.standard_normal(C * mult).astype(np.float32)
    ho, wo, ph, pw = orc.calc_padding_and_output_size(H, W, 3, 3, (1, 1), (stride, stride), 1)
    ref = orc.dwconv_f32(x, f, bias, (stride, stride), (1, 1), (ph >> 1, pw >> 1), (ho, wo), 1)
    dx, df, db, do = ctx.upload(x), ctx.upload(f), ctx.upload(bias), ctx.alloc(ref.nbytes)
    ctx.dwconv_f32(dx, df, db, do, N, C, H, W, mult, 3, 3, (stride, stride), (1, 1), (ph >> 1, pw >> 1), (ho, wo), 1)
    assert rel_err(ctx.download(do, ref.shape, np.float32), ref, 1e-5, "dwconv_f32") <= 1e-5
    for b in (dx, df, db, do):
        b.free()


@pytest.mark.parametrize("k,stride,shape", [
    # rows that are no whole words, as many values per SM as make runs of 2, 4 and 8 rows (2, 4, 8 times 1024), ragged last runs
    (3, 1, (2, 40, 75, 75)), (3, 1, (4, 64, 57, 57)), (3, 1, (3, 64, 89, 91)), (3, 2, (6, 64, 59, 57)), (3, 2, (5, 64, 87, 91)),
    (3, 2, (8, 64, 101, 99)), (5, 1, (3, 64, 89, 91)), (5, 2, (8, 64, 101, 99)), (5, 1, (4, 64, 57, 56)), (5, 2, (3, 64, 89, 88))])
def test_dwconv_f32_long_runs(ctx, orc, k, stride, shape):
    N, C, H, W = shape
    rng = np.random.Generator(np.random.PCG64(C + W))
    x = rng.standard_normal((N, C, H, W)).astype(np.float32)
    f = rng.standard_normal((1, C, k, k)).astype(np.float32)
    bias = rng.standard_normal(C).astype(np.float32)
    ho, wo, ph, pw = orc.calc_padding_and_output_size(H, W, k, k, (1, 1), (stride, stride), 1)
    values = N * C * ho * wo / (1024 * 148)
    assert values >= 2  # (runs of 2 from there, of 4 from 4, of 8 from 8)
    ref = orc.dwconv_f32(x, f, bias, (stride, stride), (1, 1), (ph >> 1, pw >> 1), (ho, wo), 1)
    dx, df, db, do = ctx.upload(x), ctx.upload(f), ctx.upload(bias), ctx.alloc(ref.nbytes)
    ctx.dwconv_f32(dx, df, db, do, N, C, H, W, 1, k, k, (stride, stride), (1, 1), (ph >> 1, pw >> 1), (ho, wo), 1)
    assert rel_err(ctx.download(do, ref.shape, np.float32), ref, 1e-5, "dwconv_f32") <= 1e-5
    for b in (dx, df, db, do):
        b.free()


def test_dwconv_f32(ctx, orc, kats):
    k = kats["dwconv_f32_2x2_valid"]  # SimpleValidTest, depthwise_conv2d_test.cc:26-84
    x = np.transpose(np.array(k["input"], np.float32).reshape(1, 3, 3, 2), (0, 3, 1, 2)).copy()
    f = np.array(k["filter"], np.float32).reshape(1, 2, 2, 2)
    bias = np.array(k["bias"], np.float32)
    dx, df, db, do = ctx.upload(x), ctx.upload(f), ctx.upload(bias), ctx.alloc(8 * 4)
    ctx.dwconv_f32(dx, df, db, do, 1, 2, 3, 3, 1, 2, 2, (1, 1), (1, 1), (0, 0), (2, 2))
    got = np.transpose(ctx.download(do, (1, 2, 2, 2), np.float32), (0, 2, 3, 1))
    np.testing.assert_allclose(got.ravel(), np.array(k["expected"], np.float32), rtol=1e-5)
    rng = np.random.Generator(np.random.PCG64(1))
    x = rng.standard_normal((2, 12, 17, 15)).astype(np.float32)
    f = rng.standard_normal((2, 12, 3, 3)).astype(np.float32)
    bias = rng.standard_normal(24).astype(np.float32)
    ref = orc.dwconv_f32(x, f, bias, (2, 2), (1, 1), (0, 0), (9, 8), 1)
    dx, df, db, do = ctx.upload(x), ctx.upload(f), ctx.upload(bias), ctx.alloc(ref.nbytes)
    ctx.dwconv_f32(dx, df, db, do, 2, 12, 17, 15, 2, 3, 3, (2, 2), (1, 1), (0, 0), (9, 8), 1)
    assert rel_err(ctx.download(do, ref.shape, np.float32), ref, 1e-4, "dwconv_f32") <= 1e-4


def test_winograd_config1_full_size(ctx, orc):
    """Input [32,64,56,56], filter [64,64,3,3], SAME (the full configuration): every image against the oracle's direct convolution (threaded, a few seconds), and one
    image of the batch-32 call against the same image run alone (the batch entries are independent)."""
    N, C, H, W, O = 32, 64, 56, 56, 64
    rng = np.random.Generator(np.random.PCG64(0))
    x = rng.random((N, C, H, W), dtype=np.float32)
    f = (rng.standard_normal((O, C, 3, 3)) * np.sqrt(2.0 / (9 * C))).astype(np.float32)
    bias = (rng.standard_normal(O) * 0.01).astype(np.float32)
    dx, df, db = ctx.upload(x), ctx.upload(f), ctx.upload(bias)
    do = ctx.alloc(N * O * H * W * 4)
    ctx.winograd_f32(dx, df, db, do, N, C, H, W, O, (1, 1), (H, W))
    got = ctx.download(do, (N, O, H, W), np.float32)
    ref = orc.conv2d_f32(x, f, bias, (1, 1), (1, 1), (1, 1), (H, W), 0, 0.0, 0.0)  # all 32 images
    assert rel_err(got, ref, 1e-3, "winograd_config1_vs_direct") <= 1e-3
    d1, o1 = ctx.upload(x[17:18]), ctx.alloc(O * H * W * 4)
    ctx.winograd_f32(d1, df, db, o1, 1, C, H, W, O, (1, 1), (H, W))
    alone = ctx.download(o1, (1, O, H, W), np.float32)
    assert np.array_equal(alone[0], got[17])


@pytest.mark.parametrize("case", [
    # N, C, H, W, O, KH, KW, stride, dilation, padding, activation
    (3, 3, 64, 64, 64, 7, 7, 2, 1, "SAME", 1),     # stem shape: K = 147 (filter rows repacked), 1024 positions
    (2, 64, 30, 30, 48, 1, 1, 2, 1, "SAME", 0),    # 1x1 stride 2: 225 positions -> images merged
    (5, 96, 7, 7, 40, 1, 1, 1, 1, "VALID", 1),     # 1x1 stride 1 with 49 positions -> images merged
    (2, 32, 20, 24, 24, 3, 3, 2, 1, "SAME", 6),    # 3x3 stride 2: 120 positions -> merged
    (2, 16, 40, 40, 32, 3, 3, 1, 2, "SAME", 2),    # dilated 3x3, 1600 positions per image
    (1, 8, 33, 47, 16, 5, 3, 1, 1, "FULL", 0),     # ragged everything
])
@pytest.mark.parametrize("budget_mb", [1024, 1])
def test_conv2d_f32_column_route(ctx, orc, case, budget_mb):
    """General convolutions large enough for the im2col + tensor-core GEMM route, with the
    column matrix in one piece and split into chunks of images (1 MiB budget)."""
    N, C, H, W, O, KH, KW, st, dil, padding, act = case
    x, f, bias = _conv_inputs((N, C, H, W), (O, C, KH, KW), H * 5 + C)
    x = x * 2 - 1
    Ho, Wo, ph, pw = orc.calc_padding_and_output_size(H, W, KH, KW, (dil, dil), (st, st), PAD[padding])
    ref = orc.conv2d_f32(x, f, bias, (st, st), (dil, dil), (ph >> 1, pw >> 1), (Ho, Wo), act, 0.5, 0.1)
    dx, df, db, do = ctx.upload(x), ctx.upload(f), ctx.upload(bias), ctx.alloc(ref.nbytes)
    ctx.set_option("col_budget_mb", budget_mb)
    before = ctx.launches_tensor_core
    try:
        ctx.conv2d_f32(dx, df, db, do, N, C, H, W, O, KH, KW, (st, st), (dil, dil), (ph >> 1, pw >> 1),
                       (Ho, Wo), act, 0.5, 0.1)
    finally:
        ctx.set_option("col_budget_mb", 1024)
    assert ctx.launches_tensor_core > before, "tensor-core GEMM did not run"
    assert rel_err(ctx.download(do, ref.shape, np.float32), ref, 1e-4, "conv2d_f32_column_route") <= 1e-4
    for b in (dx, df, db, do):
        b.free()


@pytest.mark.parametrize("case", [
    # N, C, H, W, kernel, stride, dilation, padding
    (2, 5, 17, 19, 3, 2, 1, "SAME"),      # ResNet's 3x3 stride-2 max pool
    (1, 3, 8, 8, 2, 2, 1, "VALID"),
    (2, 16, 7, 7, 7, 1, 1, "VALID"),      # global pooling
    (1, 4, 13, 11, 3, 1, 2, "SAME"),      # dilated
    (2, 3, 10, 10, 5, 3, 1, "FULL"),      # windows that overlap the border by more than half
    (2, 6, 16, 24, 3, 2, 1, "SAME"),      # rows of a multiple of 4: four outputs per thread, 128-bit accesses
    (1, 3, 20, 20, 3, 2, 1, "VALID"),     # ... with an output width that is not a multiple of 4
    (2, 4, 112, 112, 3, 2, 1, "SAME"),    # ResNet's pooling layer at full size
])
@pytest.mark.parametrize("ptype", [1, 2])
def test_pooling_f32(ctx, orc, case, ptype):
    N, C, H, W, k, st, dil, padding = case
    rng = np.random.Generator(np.random.PCG64(H + ptype))
    x = rng.standard_normal((N, C, H, W)).astype(np.float32)
    Ho, Wo, ph, pw = orc.calc_padding_and_output_size(H, W, k, k, (dil, dil), (st, st), PAD[padding])
    ref = orc.pooling_f32(x, (k, k), (st, st), (dil, dil), (ph >> 1, pw >> 1), (Ho, Wo), ptype)
    dx, do = ctx.upload(x), ctx.alloc(ref.nbytes)
    ctx.pooling_f32(dx, do, N, C, H, W, (k, k), (st, st), (dil, dil), (ph >> 1, pw >> 1), (Ho, Wo), ptype)
    got = ctx.download(do, ref.shape, np.float32)
    if ptype == 2:
        assert np.array_equal(got, ref)          # a maximum has no rounding
    else:
        assert rel_err(got, ref, 1e-6, "pooling_f32") <= 1e-6
    dx.free(); do.free()


def test_pooling_f32_reference_literals(ctx):
    """PoolingOpTest.MAX_VALID / AVG_VALID (test/ccunit/mace/ops/pooling_test.cc:27-61, 301-336)."""
    x = np.ascontiguousarray(np.arange(32, dtype=np.float32).reshape(1, 2, 4, 4))
    dx, do = ctx.upload(x), ctx.alloc(8 * 4)
    ctx.pooling_f32(dx, do, 1, 2, 4, 4, (2, 2), (2, 2), (1, 1), (0, 0), (2, 2), 2)
    assert ctx.download(do, (8,), np.float32).tolist() == [5, 7, 13, 15, 21, 23, 29, 31]
    ctx.pooling_f32(dx, do, 1, 2, 4, 4, (2, 2), (2, 2), (1, 1), (0, 0), (2, 2), 1)
    assert ctx.download(do, (8,), np.float32).tolist() == [2.5, 4.5, 10.5, 12.5, 18.5, 20.5, 26.5, 28.5]


@pytest.mark.parametrize("size", [1, 6, 1000, 4099, 1 << 20])
def test_eltwise_f32(ctx, orc, size):
    """Same-shape and tensor-scalar forms; the results are single IEEE operations (or two
    products and a sum), so they must be bit-identical to the CPU's."""
    rng = np.random.Generator(np.random.PCG64(size))
    a = rng.standard_normal(size).astype(np.float32)
    b = (rng.standard_normal(size) + 2.5).astype(np.float32)
    da, db, do = ctx.upload(a), ctx.upload(b), ctx.alloc(size * 4)
    for type_ in (0, 1, 2, 3, 4, 5, 6, 7, 8):
        for swapped in (False, True):
            ctx.eltwise_f32(da, db, do, size, type_, swapped=swapped)
            assert np.array_equal(ctx.download(do, (size,), np.float32),
                                  orc.eltwise_f32(a, b, type_, swapped=swapped)), (type_, swapped)
            ctx.eltwise_f32(da, None, do, size, type_, swapped=swapped, scalar=0.75)
            assert np.array_equal(ctx.download(do, (size,), np.float32),
                                  orc.eltwise_f32(a, None, type_, swapped=swapped, scalar=0.75)), type_
    for swapped in (False, True):
        ctx.eltwise_f32(da, db, do, size, 0, coeff=(0.3, -1.7), swapped=swapped)
        assert np.array_equal(ctx.download(do, (size,), np.float32),
                              orc.eltwise_f32(a, b, 0, coeff=(0.3, -1.7), swapped=swapped))
    ctx.eltwise_f32(da, None, do, size, 12, coeff=(-0.5, 0.25))
    assert np.array_equal(ctx.download(do, (size,), np.float32), orc.eltwise_f32(a, None, 12, coeff=(-0.5, 0.25)))
    import mace_b200
    with pytest.raises(mace_b200.MaceB200Error):
        ctx.eltwise_f32(da, db, do, size, 9)           # POW is not built
    with pytest.raises(mace_b200.MaceB200Error):
        ctx.eltwise_f32(da, None, do, size, 12, coeff=(1.0, 0.0))   # Clip needs min < max
    for buf in (da, db, do):
        buf.free()


@pytest.mark.parametrize("act", [0, 1, 2, 6])
def test_activation_f32(ctx, orc, act):
    rng = np.random.Generator(np.random.PCG64(act))
    x = (rng.standard_normal(100003) * 3).astype(np.float32)
    dx, do = ctx.upload(x), ctx.alloc(x.nbytes)
    ctx.activation_f32(dx, do, x.size, act, 2.0, 0.1)
    assert rel_err(ctx.download(do, x.shape, np.float32), orc.activation_f32(x, act, 2.0, 0.1), 1e-7, "activation") <= 1e-7
    ctx.activation_f32(dx, dx, x.size, act, 2.0, 0.1)   # in place
    assert rel_err(ctx.download(dx, x.shape, np.float32), orc.activation_f32(x, act, 2.0, 0.1), 1e-7, "activation") <= 1e-7
    dx.free(); do.free()


@pytest.mark.parametrize("shape", [(2, 4, 1), (3, 1001, 1), (64, 1000, 1), (2, 21, 35), (1, 3, 1000)])
@pytest.mark.parametrize("use_log", [False, True])
def test_softmax_f32(ctx, orc, shape, use_log):
    outer, classes, inner = shape
    rng = np.random.Generator(np.random.PCG64(classes))
    x = (rng.standard_normal(shape) * 4).astype(np.float32)
    if shape == (2, 4, 1):
        x = np.array([1, 1, 1, 1, 1, 2, 3, 4], np.float32).reshape(shape)  # softmax_test.cc:37-38
    dx, do = ctx.upload(x), ctx.alloc(x.nbytes)
    ctx.softmax_f32(dx, do, outer, classes, inner, use_log)
    got = ctx.download(do, shape, np.float32)
    ref = orc.softmax_f32(x, outer, classes, inner, use_log).reshape(shape)
    # the reference's own softmax tests compare at 1e-5 (softmax_test.cc:96); expf on the
    # device and std::exp on the host differ by a few ulps
    assert np.abs(got - ref).max() <= (1e-4 if use_log else 1e-5)
    dx.free(); do.free()


@pytest.mark.parametrize("case", [
    # N, C, H, W, O, KH, stride, activation
    (3, 64, 16, 16, 160, 1, 1, 1),     # 1x1 stride 1, 256 pixels: sum + ReLU in the GEMM's epilogue, ragged N tile
    (2, 32, 12, 11, 48, 1, 1, 6),      # 132 pixels (a multiple of 4), LEAKYRELU
    (4, 40, 7, 7, 72, 1, 1, 1),        # 49 pixels: images merged, then one in-place sum + ReLU pass
    (2, 16, 14, 14, 24, 3, 1, 2),      # 3x3: convolution, then the in-place pass
    (1, 8, 9, 9, 8, 1, 2, 0),          # tiny: direct kernel, then the in-place pass
])
def test_conv2d_f32_residual(ctx, orc, case):
    """out = act((conv + bias) + residual) equals Conv2D (no activation), Eltwise SUM and
    Activation run one after the other."""
    N, C, H, W, O, k, st, act = case
    x, f, bias = _conv_inputs((N, C, H, W), (O, C, k, k), H * 7 + O)
    x = x * 2 - 1
    Ho, Wo, ph, pw = orc.calc_padding_and_output_size(H, W, k, k, (1, 1), (st, st), PAD["SAME"])
    rng = np.random.Generator(np.random.PCG64(O))
    res = rng.standard_normal((N, O, Ho, Wo)).astype(np.float32)
    conv = orc.conv2d_f32(x, f, bias, (st, st), (1, 1), (ph >> 1, pw >> 1), (Ho, Wo), 0)
    ref = orc.activation_f32(orc.eltwise_f32(conv, res, 0), act, 0.5, 0.1)
    dx, df, db, dr, do = ctx.upload(x), ctx.upload(f), ctx.upload(bias), ctx.upload(res), ctx.alloc(ref.nbytes)
    ctx.conv2d_f32_residual(dx, df, db, dr, do, N, C, H, W, O, k, k, (st, st), (1, 1), (ph >> 1, pw >> 1),
                            (Ho, Wo), act, 0.5, 0.1)
    assert rel_err(ctx.download(do, ref.shape, np.float32), ref, 1e-4, "conv2d_f32_residual") <= 1e-4
    for b in (dx, df, db, dr, do):
        b.free()



def test_zz_report_measured_errors():
    """Prints the worst measured errors of this module's comparisons (pytest -s shows them):
    the element-wise ratio |got - ref| / (abs_err + rel_err * |ref|) and the range-normalised
    error."""
    for label, (ratio, rng_err) in sorted(WORST.items()):
        print("%-32s element-wise ratio %.4f   range-normalised %.3e" % (label, ratio, rng_err))
    assert all(r <= 1.0 for r, _ in WORST.values())
