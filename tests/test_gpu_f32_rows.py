"""The fp32 GEMM of operands that both have their depth contiguous (gemm_f32_rows.cu) against float64, with bounds derived from its
arithmetic, at the edges of its tiles, and where its split of a value into two halves does not reach."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import mace_b200
    c = mace_b200.Context(0)
    yield c
    c.close()


def _matmul(ctx, A, B, rows=2, bn=0):
    """A [batch, M, K] times B [batch, N, K] transposed."""
    batch, M, K = A.shape
    N = B.shape[1]
    dA, dB, dC = ctx.upload(A), ctx.upload(B), ctx.upload(np.full((batch, M, N), 7, np.float32))
    ctx.set_option("f32_rows", rows)
    ctx.set_option("f32_bn", bn)
    ctx.gemm_f32(dA, dB, dC, batch, M, N, K, b_col_major=True)
    ctx.set_option("f32_rows", 0)
    ctx.set_option("f32_bn", 0)
    got = ctx.download(dC, (batch, M, N), np.float32)
    for b in (dA, dB, dC):
        b.free()
    return got


def _bound(A, B):
    """hi + lo of a value is within 2^-22 of it; an accumulator holds at most three steps (six MMAs of large products, each cut off by
    at most 2^-23 of it), and the sums of the runs round once each."""
    A, B = np.abs(A), np.swapaxes(np.abs(B), -1, -2)
    K = A.shape[-1]
    return (A @ B) * (2.0 ** -21 + (6 + K / 32 + 4) * 2.0 ** -23) + 1e-37


@pytest.mark.parametrize("bn", [64, 128])
@pytest.mark.parametrize("shape", [
    # batch, M, N, K: single rows, ragged tiles on either side, depths of one step with a tail to many runs, more tiles than SMs
    (1, 1, 1, 4), (1, 128, 64, 32), (2, 129, 65, 68), (3, 40, 130, 100), (1, 64, 300, 1000), (5, 257, 200, 20), (30, 130, 390, 384),
    (1, 1, 1000, 512), (2, 700, 3, 36)])
def test_gemm_f32_rows(ctx, shape, bn):
    batch, M, N, K = shape
    rng = np.random.Generator(np.random.PCG64(M))
    A = rng.standard_normal((batch, M, K)).astype(np.float32)
    B = rng.standard_normal((batch, N, K)).astype(np.float32)
    before = ctx.launches_tensor_core
    got = _matmul(ctx, A, B, bn=bn)
    assert ctx.launches_tensor_core == before + 1
    A, B = A.astype(np.float64), B.astype(np.float64)
    assert (np.abs(got - A @ np.swapaxes(B, 1, 2)) <= _bound(A, B)).all()


@pytest.mark.parametrize("bn", [64, 128])
@pytest.mark.parametrize("what", ["zeros", "late", "tiny", "huge", "steep", "inf", "nan", "inf_row"])
def test_gemm_f32_rows_beyond_the_split(ctx, bn, what):
    """Rows of zeros, scales that a later step exceeds, values that halves do not hold: FMAs take over."""
    batch, M, N, K = 2, 150, 140, 132
    rng = np.random.Generator(np.random.PCG64(bn))
    A = rng.standard_normal((batch, M, K)).astype(np.float32)
    B = rng.standard_normal((batch, N, K)).astype(np.float32)
    if what == "zeros":
        A[:, 3], B[:, 7], B[0, :, :100], A[1, :, :40] = 0, 0, 0, 0
    elif what == "late":
        B[:, ::3, 96:] *= np.float32(2.0 ** 18)
    elif what == "tiny":
        A *= np.float32(1e-25)
        B *= np.float32(1e-3)
    elif what == "huge":
        A *= np.float32(1e25)
        B *= np.float32(1e-22)
    elif what == "steep":
        A *= np.float32(10.0) ** rng.integers(-9, 9, (1, M, 1)).astype(np.float32)
        B *= np.float32(10.0) ** rng.integers(-9, 9, (1, N, 1)).astype(np.float32)
    elif what == "inf":
        B[1, 9, 50] = np.inf
    elif what == "nan":
        B[0, 139, 131] = np.nan
    elif what == "inf_row":
        A[0, 5, 0] = -np.inf
    got = _matmul(ctx, A, B, bn=bn)
    with np.errstate(all="ignore"):
        A, B = A.astype(np.float64), B.astype(np.float64)
        ref = np.einsum("bmk,bnk->bmn", A, B)
        assert np.array_equal(np.isnan(got), np.isnan(ref))
        assert np.array_equal(got[np.isinf(ref)], ref[np.isinf(ref)])
        finite = np.isfinite(ref)
        A, B = np.where(np.isfinite(A), A, 0), np.where(np.isfinite(B), B, 0)
        # (worked out again, a sum of K products rounds K times)
        bound = _bound(A, B) + (np.abs(A) @ np.swapaxes(np.abs(B), 1, 2)) * K * 2.0 ** -24
        assert (np.abs(got - ref)[finite] <= bound[finite]).all()


@pytest.mark.parametrize("spread", [2.0 ** 10, 2.0 ** 20])
@pytest.mark.parametrize("bn", [64, 128])
def test_gemm_f32_rows_spread(ctx, bn, spread):
    """Small values that meet large ones of the other operand keep their bits."""
    rng = np.random.Generator(np.random.PCG64(bn))
    A = rng.standard_normal((2, 150, 420)).astype(np.float32)
    B = rng.standard_normal((2, 140, 420)).astype(np.float32)
    plain, exact = _matmul(ctx, A, B, bn=bn), A.astype(np.float64) @ np.swapaxes(B, 1, 2).astype(np.float64)
    A[:, :, ::7] *= np.float32(1 / spread)
    B[:, :, ::7] *= np.float32(spread)
    got = _matmul(ctx, A, B, bn=bn)
    assert (np.abs(got - exact) <= _bound(A, B)).all()
    assert np.linalg.norm(got - exact) <= 1.05 * np.linalg.norm(plain - exact)


@pytest.mark.parametrize("powers", [(-100, 0), (0, -100), (-70, -40), (60, -110), (-110, 60), (90, -60)])
@pytest.mark.parametrize("bn", [64, 128])
def test_gemm_f32_rows_scales(ctx, bn, powers):
    """Results are those of operands of ordinary size, bit for bit: nothing is worked out again because a row is small or large."""
    rng = np.random.Generator(np.random.PCG64(bn))
    A = rng.standard_normal((2, 150, 100)).astype(np.float32)
    B = rng.standard_normal((2, 140, 100)).astype(np.float32)
    plain = _matmul(ctx, A, B, bn=bn)
    a, b = (np.float32(2.0) ** p for p in powers)
    A[:, ::3] *= a
    B[:, 5:100] *= b
    plain[:, ::3] *= a
    plain[:, :, 5:100] *= b
    assert np.array_equal(_matmul(ctx, A, B, bn=bn), plain)


@pytest.mark.parametrize("power", [-40, -16, 16, 40])
@pytest.mark.parametrize("K", [164, 420])
@pytest.mark.parametrize("bn", [64, 128])
def test_gemm_f32_rows_steps(ctx, bn, K, power):
    """Steps of another size than the first, in which the other operand makes up for it: the same results, bit for bit, and so none
    of them is worked out again."""
    rng = np.random.Generator(np.random.PCG64(bn))
    A = rng.standard_normal((2, 150, K)).astype(np.float32)
    B = rng.standard_normal((2, 140, K)).astype(np.float32)
    plain = _matmul(ctx, A, B, bn=bn)
    for k0, k1 in ((32, 64), (96, 164)) if K < 384 else ((96, 192), (288, 420)):  # (runs of one step and of three)
        A[:, :, k0:k1] *= np.float32(2.0) ** power
        B[:, :, k0:k1] *= np.float32(2.0) ** -power
    assert np.array_equal(_matmul(ctx, A, B, bn=bn), plain)


@pytest.mark.parametrize("shape", [(9, 300, 200, 352), (1, 1024, 1024, 1024)])
def test_gemm_f32_rows_choice(ctx, shape):
    """By rule, with an error no larger than that of the kernel that fetches its own operands."""
    batch, M, N, K = shape
    rng = np.random.Generator(np.random.PCG64(K))
    A = rng.standard_normal((batch, M, K)).astype(np.float32)
    B = rng.standard_normal((batch, N, K)).astype(np.float32)
    exact = A.astype(np.float64) @ np.swapaxes(B, 1, 2).astype(np.float64)
    err = [np.linalg.norm(_matmul(ctx, A, B, rows) - exact) for rows in (0, 1, 2)]
    assert err[0] == err[2] < err[1]


@pytest.mark.parametrize("c_col,a_batched,b_batched", [(0, 0, 1), (0, 1, 0), (1, 1, 1), (1, 0, 1), (1, 1, 0), (0, 0, 0)])
def test_gemm_f32_rows_order_and_broadcast(ctx, c_col, a_batched, b_batched):
    """The result by rows or by columns, an operand shared by the batch."""
    batch, M, N, K = 3, 140, 200, 100
    rng = np.random.Generator(np.random.PCG64(c_col))
    A = rng.standard_normal((batch if a_batched else 1, M, K)).astype(np.float32)
    B = rng.standard_normal((batch if b_batched else 1, N, K)).astype(np.float32)
    dA, dB, dC = ctx.upload(A), ctx.upload(B), ctx.upload(np.full((batch, M, N), 7, np.float32))
    ctx.set_option("f32_rows", 2)
    ctx.gemm_f32(dA, dB, dC, batch, M, N, K, b_col_major=True, c_col_major=bool(c_col), a_batched=bool(a_batched),
                 b_batched=bool(b_batched))
    ctx.set_option("f32_rows", 0)
    got = ctx.download(dC, (batch, N, M) if c_col else (batch, M, N), np.float32)
    for b in (dA, dB, dC):
        b.free()
    if c_col:
        got = got.swapaxes(1, 2)
    A, B = np.broadcast_to(A, (batch, M, K)).astype(np.float64), np.broadcast_to(B, (batch, N, K)).astype(np.float64)
    assert (np.abs(got - A @ np.swapaxes(B, 1, 2)) <= _bound(A, B)).all()
