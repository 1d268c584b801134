"""The fp32 GEMM on pairs of halves (gemm_f32_pairs.cu) against float64, with bounds derived from its arithmetic, at the edges of
its tiles, and where its split of a value into two halves does not reach."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import mace_b200
    c = mace_b200.Context(0)
    yield c
    c.close()


def _bound(A, B):
    """hi + lo of a value is within 2^-22 of it; the accumulator is cut off by at most 2^-23 of what it holds after each of three MMAs
    per 16 of the depth."""
    A, B = np.abs(A), np.abs(B)
    K = A.shape[-1]
    return (A @ B) * (2.0 ** -21 + (3 * K / 16 + 4) * 2.0 ** -23) + 1e-37


def _matmul(ctx, A, B, pairs=2):
    batch, M, K = A.shape
    N = B.shape[2]
    dA, dB, dC = ctx.upload(A), ctx.upload(B), ctx.upload(np.full((batch, M, N), 7, np.float32))
    ctx.set_option("f32_gather", 1)
    ctx.set_option("f32_pairs", pairs)
    ctx.gemm_f32(dA, dB, dC, batch, M, N, K)
    for name in ("f32_gather", "f32_pairs"):
        ctx.set_option(name, 0)
    got = ctx.download(dC, (batch, M, N), np.float32)
    for b in (dA, dB, dC):
        b.free()
    return got


@pytest.mark.parametrize("shape", [
    # batch, M (channels), N (pixels), K: narrow and wide column tiles, depths of one to many steps with odd halves of the last one,
    # more tiles than SMs, results that TMA does not store (fewer than 16 rows)
    (1, 16, 128, 4), (1, 64, 132, 16), (2, 65, 32, 20), (3, 7, 260, 48), (1, 128, 256, 32), (2, 200, 100, 64), (5, 33, 1000, 260),
    (30, 130, 640, 36), (1, 1000, 40, 1028), (9, 64, 3000, 100)])
def test_gemm_f32_pairs(ctx, shape):
    batch, M, N, K = shape
    rng = np.random.Generator(np.random.PCG64(M))
    A = rng.standard_normal((batch, M, K)).astype(np.float32)
    B = rng.standard_normal((batch, K, N)).astype(np.float32)
    before = ctx.launches_tensor_core, ctx.launches
    got = _matmul(ctx, A, B)
    assert (ctx.launches_tensor_core, ctx.launches) == (before[0] + 1, before[1] + 2)
    A, B = A.astype(np.float64), B.astype(np.float64)
    assert (np.abs(got - A @ B) <= _bound(A, B)).all()


@pytest.mark.parametrize("shape", [(2, 32, 144, 64), (3, 100, 576, 130), (1, 20, 196, 8), (2, 260, 784, 256)])
@pytest.mark.parametrize("act", [0, 1, 2, 6])
@pytest.mark.parametrize("residual", [False, True])
def test_conv1x1_f32_pairs(ctx, shape, act, residual):
    """Bias, residual sum and activation of a 1x1 convolution (the residual lands where the result leaves from)."""
    N, C, HW, O = shape
    rng = np.random.Generator(np.random.PCG64(O))
    x = rng.standard_normal((N, C, HW)).astype(np.float32)
    f = (rng.standard_normal((O, C)) * 0.2).astype(np.float32)
    bias = rng.standard_normal(O).astype(np.float32) if act != 1 else None
    r = rng.standard_normal((N, O, HW)).astype(np.float32)
    dx, df, dr, do = ctx.upload(x), ctx.upload(f), ctx.upload(r), ctx.upload(np.zeros((N, O, HW), np.float32))
    db = ctx.upload(bias) if bias is not None else None
    side = (HW // 4, 4)
    for name, value in (("f32_gather", 1), ("f32_pairs", 2)):
        ctx.set_option(name, value)
    if residual:
        ctx.conv2d_f32_residual(dx, df, db, dr, do, N, C, *side, O, 1, 1, (1, 1), (1, 1), (0, 0), side, act, 0.6, 0.25)
    else:
        ctx.conv2d_f32(dx, df, db, do, N, C, *side, O, 1, 1, (1, 1), (1, 1), (0, 0), side, act, 0.6, 0.25)
    for name in ("f32_gather", "f32_pairs"):
        ctx.set_option(name, 0)
    got = ctx.download(do, (N, O, HW), np.float32)
    x, f = x.astype(np.float64), np.broadcast_to(f.astype(np.float64), (N, O, C))
    ref = f @ x + (bias.astype(np.float64)[None, :, None] if bias is not None else 0) + (r if residual else 0)
    size = np.abs(ref)
    ref = {0: ref, 1: np.maximum(ref, 0), 2: np.clip(ref, 0, np.float32(0.6)), 6: np.where(ref > 0, ref, ref * 0.25)}[act]
    assert (np.abs(got - ref) <= _bound(f, x) + 2.0 ** -22 * (size + 1)).all()
    for b in (dx, df, dr, do) + ((db,) if db else ()):
        b.free()


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("where", ["pairs", "gather", "neither"])
def test_conv1x1_f32_residual_in_place(where, captured):
    """A residual that is the output itself: nothing is read where a result already stands."""
    import mace_b200
    ctx = mace_b200.Context(0)
    L = mace_b200.lib()
    N, C, HW, O = 2, 132, 144, 48
    rng = np.random.Generator(np.random.PCG64(O))
    x = rng.standard_normal((N, C, HW)).astype(np.float32)
    f = rng.standard_normal((O, C)).astype(np.float32)
    r = rng.standard_normal((N, O, HW)).astype(np.float32)
    x[:, 96:, ::3] *= np.float32(2.0 ** 20)
    x[1, 50, 9], f[21, 100] = np.inf, -np.inf
    dx, df, do, dr = ctx.upload(x), ctx.upload(f), ctx.upload(r), ctx.upload(r)
    for name, value in {"pairs": {"f32_gather": 1, "f32_pairs": 2}, "gather": {"f32_gather": 2}, "neither": {"tensor_cores": 0}}[where].items():
        ctx.set_option(name, value)

    def call(out):
        ctx.conv2d_f32_residual(dx, df, None, out, out, N, C, 36, 4, O, 1, 1, (1, 1), (1, 1), (0, 0), (36, 4))

    if captured:
        call(dr)
        g = ctypes.c_void_p()
        ctx._check(L.mb_graph_begin(ctx.h))
        call(do)
        ctx._check(L.mb_graph_end(ctx.h, ctypes.byref(g)))
        ctx._check(L.mb_graph_launch(ctx.h, g))
    else:
        call(do)
    got = ctx.download(do, (N, O, HW), np.float32)
    if captured:
        ctx._check(L.mb_graph_destroy(ctx.h, g))
    ctx.close()
    x, f = x.astype(np.float64), np.broadcast_to(f.astype(np.float64), (N, O, C))
    with np.errstate(all="ignore"):
        ref = f @ x + r
        finite = np.isfinite(ref)
    x, f = np.where(np.isfinite(x), x, 0), np.where(np.isfinite(f), f, 0)
    assert finite.mean() > 0.9 and np.array_equal(np.isfinite(got), finite)
    # (tf32 pairs: 22 bits, an accumulator cut off after each of twelve MMAs per 32 of k; fp32 FMAs: a rounding for each of k)
    bound = (np.abs(f) @ np.abs(x)) * (2.0 ** -20 + (12 * C / 32 + C + 4) * 2.0 ** -23) + 1e-6
    assert (np.abs(got[finite] - ref[finite]) <= bound[finite]).all()


@pytest.mark.parametrize("M", [40, 150])
@pytest.mark.parametrize("what", ["zeros", "late", "tiny", "huge", "steep", "inf", "nan", "inf_row"])
def test_gemm_f32_pairs_beyond_the_split(ctx, M, what):
    """Rows and columns of zeros, scales that a later step exceeds, values that halves do not hold: FMAs take over."""
    batch, N, K = 2, 300, 132
    rng = np.random.Generator(np.random.PCG64(M))
    A = rng.standard_normal((batch, M, K)).astype(np.float32)
    B = rng.standard_normal((batch, K, N)).astype(np.float32)
    if what == "zeros":
        A[:, 3], B[:, :, 7], B[0, :100], B[1, :40, 128:] = 0, 0, 0, 0
    elif what == "late":
        B[:, 96:, ::3] *= np.float32(2.0 ** 18)
    elif what == "tiny":
        A *= np.float32(1e-25)
        B *= np.float32(1e-3)
    elif what == "huge":
        A *= np.float32(1e25)
        B *= np.float32(1e-22)
    elif what == "steep":
        A *= np.float32(10.0) ** rng.integers(-9, 9, (1, M, 1)).astype(np.float32)
        B *= np.float32(10.0) ** rng.integers(-9, 9, (1, 1, N)).astype(np.float32)
    elif what == "inf":
        B[1, 50, 9] = np.inf
    elif what == "nan":
        B[0, 131, 299] = np.nan
    elif what == "inf_row":
        A[0, 5, 0] = -np.inf
    got = _matmul(ctx, A, B)
    with np.errstate(all="ignore"):
        A, B = A.astype(np.float64), B.astype(np.float64)
        ref = np.einsum("bmk,bkn->bmn", A, B)
        assert np.array_equal(np.isnan(got), np.isnan(ref))
        assert np.array_equal(got[np.isinf(ref)], ref[np.isinf(ref)])
        finite = np.isfinite(ref)
        A, B = np.where(np.isfinite(A), A, 0), np.where(np.isfinite(B), B, 0)
        # (worked out again, a sum of K products rounds K times)
        bound = _bound(A, B) + (np.abs(A) @ np.abs(B)) * K * 2.0 ** -24
        assert (np.abs(got - ref)[finite] <= bound[finite]).all()


@pytest.mark.parametrize("spread", [2.0 ** 8, 2.0 ** 12])
@pytest.mark.parametrize("M", [40, 150])
def test_gemm_f32_pairs_spread(ctx, M, spread):
    """Small values that meet large ones of the other operand keep their bits."""
    rng = np.random.Generator(np.random.PCG64(M))
    A = rng.standard_normal((2, M, 260)).astype(np.float32)
    B = rng.standard_normal((2, 260, 300)).astype(np.float32)
    plain, exact = _matmul(ctx, A, B), A.astype(np.float64) @ B.astype(np.float64)
    A[:, :, ::7] *= np.float32(1 / spread)
    B[:, ::7] *= np.float32(spread)
    got = _matmul(ctx, A, B)
    assert (np.abs(got - exact) <= _bound(A, B)).all()
    assert np.linalg.norm(got - exact) <= 1.05 * np.linalg.norm(plain - exact)


def _within_reach(x):
    return np.copysign(np.clip(np.abs(x), 2.0 ** -5, 4), x).astype(np.float32)


@pytest.mark.parametrize("shape,power", [((30, 40, 1280, 132), -14), ((30, 130, 1280, 132), -14), ((30, 130, 1280, 132), -18),
                                         ((38000, 8, 132, 36), -14)])
def test_gemm_f32_pairs_grows(ctx, shape, power):
    """Rows of X whose first step is far smaller than the later ones, for which the weights make up, in some of a CTA's tiles (up to
    514 of them, the last of which share marks with the first): the same results, bit for bit, and so none of them is worked out
    again by FMAs."""
    batch, M, N, K = shape
    rng = np.random.Generator(np.random.PCG64(M))
    A = _within_reach(rng.standard_normal((batch, M, K), dtype=np.float32))
    B = _within_reach(rng.standard_normal((batch, K, N), dtype=np.float32))
    plain = _matmul(ctx, A, B)
    for b in (0, 3, 10, 17, 18, batch - 1):
        A[b, :, :32] *= np.float32(2.0) ** -power
        B[b, :32] *= np.float32(2.0) ** power
    B[1, K // 2, 5] = B[-1, K - 1, N - 1] = np.inf
    got = _matmul(ctx, A, B)
    assert not np.isfinite(got[1, :, 5]).any() and not np.isfinite(got[-1, :, N - 1]).any()
    plain[1, :, 5], plain[-1, :, N - 1] = got[1, :, 5], got[-1, :, N - 1]
    assert np.array_equal(got, plain, equal_nan=True)


@pytest.mark.parametrize("act", [0, 6])
@pytest.mark.parametrize("residual", [False, True])
@pytest.mark.parametrize("O", [40, 130])
def test_conv1x1_f32_pairs_grows(ctx, O, residual, act):
    """... with the residual, which is read once more."""
    N, C, HW = 70, 68, 400
    rng = np.random.Generator(np.random.PCG64(O))
    x, f = _within_reach(rng.standard_normal((N, C, HW))), _within_reach(rng.standard_normal((O, C)))
    bias = rng.standard_normal(O).astype(np.float32)
    r = rng.standard_normal((N, O, HW)).astype(np.float32)
    got = []
    for grown in (False, True):
        if grown:
            x[:, :32] *= np.float32(2.0 ** -14)
            f[:, :32] *= np.float32(2.0 ** 14)
        dx, df, db, dr, do = (ctx.upload(v) for v in (x, f, bias, r, np.zeros((N, O, HW), np.float32)))
        for name, value in (("f32_gather", 1), ("f32_pairs", 2)):
            ctx.set_option(name, value)
        if residual:
            ctx.conv2d_f32_residual(dx, df, db, dr, do, N, C, HW // 4, 4, O, 1, 1, (1, 1), (1, 1), (0, 0), (HW // 4, 4), act, 0.6, 0.25)
        else:
            ctx.conv2d_f32(dx, df, db, do, N, C, HW // 4, 4, O, 1, 1, (1, 1), (1, 1), (0, 0), (HW // 4, 4), act, 0.6, 0.25)
        for name in ("f32_gather", "f32_pairs"):
            ctx.set_option(name, 0)
        got.append(ctx.download(do, (N, O, HW), np.float32))
        for b in (dx, df, db, dr, do):
            b.free()
    assert np.array_equal(*got)


@pytest.mark.parametrize("M", [40, 150])
@pytest.mark.parametrize("columns", [(0,), (5, 22), (20, 100), (259,)])
def test_gemm_f32_pairs_outliers(ctx, M, columns):
    """Columns of X 1e8 times larger than the others, which meet zeros or weights as much smaller: the others keep their bits."""
    rng = np.random.Generator(np.random.PCG64(M))
    A = rng.standard_normal((2, M, 260)).astype(np.float32)
    B = rng.standard_normal((2, 260, 300)).astype(np.float32)
    plain, exact = _matmul(ctx, A, B), A.astype(np.float64) @ B.astype(np.float64)
    plain = np.linalg.norm(plain - exact) / np.linalg.norm(exact)
    B[:, columns] *= np.float32(1e8)
    A[:, :, columns] *= np.float32(1e-8)
    A[:, ::2, columns] = 0
    exact = A.astype(np.float64) @ B.astype(np.float64)
    got = _matmul(ctx, A, B)
    assert np.linalg.norm(got - exact) / np.linalg.norm(exact) <= 1.2 * plain


@pytest.mark.parametrize("powers", [(-100, 0), (0, -100), (-70, -40), (60, -110), (-110, 60), (90, -60)])
@pytest.mark.parametrize("M", [40, 150])
def test_gemm_f32_pairs_scales(ctx, M, powers):
    """Results are those of operands of ordinary size, bit for bit: nothing is worked out again because a row is small or large."""
    rng = np.random.Generator(np.random.PCG64(M))
    A = rng.standard_normal((2, M, 100)).astype(np.float32)
    B = rng.standard_normal((2, 100, 300)).astype(np.float32)
    plain = _matmul(ctx, A, B)
    a, b = (np.float32(2.0) ** p for p in powers)
    A[:, ::3] *= a
    B[:, :, 5:200] *= b
    plain[:, ::3] *= a
    plain[:, :, 5:200] *= b
    assert np.array_equal(_matmul(ctx, A, B), plain)


def test_gemm_f32_pairs_choice(ctx):
    """By rule for a product of many steps, with an error no larger than the other kernel's."""
    rng = np.random.Generator(np.random.PCG64(0))
    A = rng.standard_normal((1, 256, 512)).astype(np.float32)
    B = rng.standard_normal((1, 512, 128 * 600)).astype(np.float32)
    exact = A[0].astype(np.float64) @ B[0].astype(np.float64)
    err = [np.linalg.norm(_matmul(ctx, A, B, pairs)[0] - exact) for pairs in (0, 1, 2)]
    assert err[0] == err[2] < err[1]
