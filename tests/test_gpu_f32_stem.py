"""The fp32 convolution of a few input channels with a stride of two columns (conv_f32_stem.cu) against float64, with bounds derived
from its arithmetic, at the edges of its strips and tiles, and where its split of a value into two halves does not reach."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import mace_b200
    c = mace_b200.Context(0)
    yield c
    c.close()


def _conv(ctx, x, f, bias, sh, pad, out_hw, stem=2, act=0):
    N, C, H, W = x.shape
    O, _, KH, KW = f.shape
    dx, df, db = ctx.upload(x), ctx.upload(f), ctx.upload(bias)
    out = ctx.upload(np.full((N, O) + out_hw, 7, np.float32))
    ctx.set_option("f32_stem", stem)
    ctx.conv2d_f32(dx, df, db, out, N, C, H, W, O, KH, KW, (sh, 2), (1, 1), pad, out_hw, act=act)
    ctx.set_option("f32_stem", 0)
    got = ctx.download(out, (N, O) + out_hw, np.float32)
    for b in (dx, df, db, out):
        b.free()
    return got


def _exact(x, f, sh, pad, out_hw):
    """The convolution in float64, padded as far as the output reaches."""
    KH, KW = f.shape[2:]
    bottom = max((out_hw[0] - 1) * sh + KH - pad[0] - x.shape[2], 0)
    right = max((out_hw[1] - 1) * 2 + KW - pad[1] - x.shape[3], 0)
    x = torch.nn.functional.pad(torch.from_numpy(x.astype(np.float64)), (pad[1], right, pad[0], bottom))
    return torch.nn.functional.conv2d(x, torch.from_numpy(f.astype(np.float64)), stride=(sh, 2)).numpy()[:, :, :out_hw[0], :out_hw[1]]


def _bound(x, f, bias, sh, pad, out_hw, ref):
    """hi + lo of a value is within 2^-22 of it; an accumulator holds at most six MMAs per filter row, each of which cuts off at most
    2^-23 of it; the bias and the sum of the two accumulators round once."""
    size = _exact(np.abs(x), np.abs(f), sh, pad, out_hw)
    return size * (2.0 ** -21 + (6 * f.shape[2] + 2) * 2.0 ** -23) + (np.abs(ref) + np.abs(bias)[None, :, None, None]) * 2.0 ** -23 + 1e-37


@pytest.mark.parametrize("shape", [
    # N, C, H, W, O, KH, KW, sh, pad, (Ho, Wo)
    (1, 3, 224, 224, 64, 7, 7, 2, (3, 3), (112, 112)), (2, 3, 33, 38, 64, 7, 7, 2, (3, 3), (17, 19)),
    (1, 1, 9, 466, 5, 5, 5, 1, (2, 2), (9, 233)), (3, 4, 20, 232, 33, 7, 7, 2, (2, 2), (10, 116)),
    (1, 4, 31, 234, 64, 7, 5, 3, (0, 1), (9, 117)), (2, 2, 17, 16, 32, 8, 8, 1, (4, 4), (18, 8)), (1, 3, 2, 2, 1, 1, 1, 1, (0, 0), (2, 1)),
    (2, 3, 40, 58, 64, 3, 3, 2, (1, 1), (20, 29)), (160, 1, 6, 60, 17, 5, 7, 2, (2, 3), (3, 30)), (1, 3, 12, 20, 8, 7, 7, 2, (9, 10), (12, 16))])
def test_conv_f32_stem(ctx, shape):
    N, C, H, W, O, KH, KW, sh, pad, out_hw = shape
    rng = np.random.Generator(np.random.PCG64(H * W))
    x = rng.standard_normal((N, C, H, W)).astype(np.float32)
    f = rng.standard_normal((O, C, KH, KW)).astype(np.float32)
    bias = rng.standard_normal(O).astype(np.float32)
    before = ctx.launches_tensor_core
    got = _conv(ctx, x, f, bias, sh, pad, out_hw)
    assert ctx.launches_tensor_core == before + 1
    ref = _exact(x, f, sh, pad, out_hw) + bias[None, :, None, None]
    bound = _bound(x, f, bias, sh, pad, out_hw, ref)
    assert (np.abs(got - ref) <= bound).all()
    relu = _conv(ctx, x, f, bias, sh, pad, out_hw, act=1)
    assert (np.abs(relu - np.maximum(ref, 0)) <= bound).all()


@pytest.mark.parametrize("what", ["zeros", "zero_strip", "outlier", "tiny", "huge", "steep", "inf", "nan"])
def test_conv_f32_stem_beyond_the_split(ctx, what):
    """Strips of zeros, values far above their strip's others, values that halves do not hold: FMAs take over."""
    N, C, H, W, O, KH, KW, sh, pad, out_hw = 2, 3, 60, 60, 40, 7, 7, 2, (3, 3), (30, 30)
    rng = np.random.Generator(np.random.PCG64(5))
    x = rng.standard_normal((N, C, H, W)).astype(np.float32)
    f = rng.standard_normal((O, C, KH, KW)).astype(np.float32)
    bias = rng.standard_normal(O).astype(np.float32)
    if what == "zeros":
        x[0], f[3] = 0, 0
    elif what == "zero_strip":
        x[:, :, :40] = 0
    elif what == "outlier":
        x[1, 2, 30, 31] = 1e9
    elif what == "tiny":
        x *= np.float32(1e-25)
        f *= np.float32(1e-3)
    elif what == "huge":
        x *= np.float32(1e25)
        f *= np.float32(1e-22)
    elif what == "steep":
        x *= np.float32(10.0) ** rng.integers(-9, 9, (N, 1, H, 1)).astype(np.float32)
        f *= np.float32(10.0) ** rng.integers(-9, 9, (O, 1, 1, 1)).astype(np.float32)
    elif what == "inf":
        x[0, 1, 20, 20] = np.inf
    elif what == "nan":
        x[1, 0, 59, 59] = np.nan
    got = _conv(ctx, x, f, bias, sh, pad, out_hw)
    with np.errstate(all="ignore"):
        ref = _exact(x, f, sh, pad, out_hw) + bias[None, :, None, None]
        assert np.array_equal(np.isnan(got), np.isnan(ref))
        assert np.array_equal(got[np.isinf(ref)], ref[np.isinf(ref)])
        finite = np.isfinite(ref)
        x = np.where(np.isfinite(x), x, 0)
        # (worked out again, a sum of K products rounds K times)
        bound = _bound(x, f, bias, sh, pad, out_hw, np.where(finite, ref, 0)) + \
            _exact(np.abs(x), np.abs(f), sh, pad, out_hw) * C * KH * KW * 2.0 ** -24
        assert (np.abs(got - ref)[finite] <= bound[finite]).all()
        if what == "outlier":  # (results without it in their sum keep their bits)
            far = np.ones(out_hw, bool)
            far[13:19, 13:19] = False
            rest = x.copy()
            rest[1, 2, 30, 31] = 0
            tight = _bound(rest, f, bias, sh, pad, out_hw, ref)
            assert (np.abs(got - ref) <= tight)[:, :, far].all()


@pytest.mark.parametrize("spread", [2.0 ** 10, 2.0 ** 20])
def test_conv_f32_stem_spread(ctx, spread):
    """Small values that meet large weights keep their bits, and so do dark regions beside bright ones."""
    rng = np.random.Generator(np.random.PCG64(6))
    x = rng.standard_normal((2, 3, 60, 60)).astype(np.float32)
    f = rng.standard_normal((40, 3, 7, 7)).astype(np.float32)
    args = (np.zeros(40, np.float32), 2, (3, 3), (30, 30))

    def error(x, f, part):
        got, exact = _conv(ctx, x, f, *args), _exact(x, f, *args[1:])
        assert (np.abs(got - exact) <= _bound(x, f, *args, exact)).all()
        return np.linalg.norm((got - exact)[part]) / np.linalg.norm(exact[part])

    plain, all_of_it = error(x, f, np.s_[:, :, :, :18]), error(x, f, np.s_[:])
    dim = x.copy()
    dim[:, :, :, :40] *= np.float32(1 / spread)
    assert error(dim, f, np.s_[:, :, :, :18]) <= 1.05 * plain
    x[:, 1] *= np.float32(1 / spread)
    f[:, 1] *= np.float32(spread)
    assert error(x, f, np.s_[:]) <= 1.05 * all_of_it


def test_conv_f32_stem_beside_an_outlier(ctx):
    """One value up to 1e6 times larger than its strip's others, which is held with them: they keep their bits, and so do its results."""
    rng = np.random.Generator(np.random.PCG64(8))
    x = rng.standard_normal((1, 3, 60, 60)).astype(np.float32)
    f = rng.standard_normal((40, 3, 7, 7)).astype(np.float32)
    args = (np.zeros(40, np.float32), 2, (3, 3), (30, 30))
    far = np.ones((30, 30), bool)
    far[12:18, 12:18] = False
    plain, exact = _conv(ctx, x, f, *args), _exact(x, f, *args[1:])
    error = np.linalg.norm((plain - exact)[:, :, far]) / np.linalg.norm(exact[:, :, far])
    for value in (3e4, 1e6):
        x[0, 1, 30, 30] = value
        got, exact = _conv(ctx, x, f, *args), _exact(x, f, *args[1:])
        assert (np.abs(got - exact) <= _bound(x, f, *args, exact)).all()
        assert np.linalg.norm((got - exact)[:, :, far]) / np.linalg.norm(exact[:, :, far]) <= 1.05 * error


@pytest.mark.parametrize("powers", [(-100, 0), (0, -100), (-70, -40), (60, -110), (-110, 60), (90, -60)])
def test_conv_f32_stem_scales(ctx, powers):
    """Results are those of operands of ordinary size, bit for bit: nothing is worked out again because a row is small or large."""
    rng = np.random.Generator(np.random.PCG64(6))
    x = rng.standard_normal((2, 3, 60, 60)).astype(np.float32)
    f = rng.standard_normal((40, 3, 7, 7)).astype(np.float32)
    args = (np.zeros(40, np.float32), 2, (3, 3), (30, 30))
    plain = _conv(ctx, x, f, *args)
    a, b = (np.float32(2.0) ** p for p in powers)
    f[::3] *= a
    plain[:, ::3] *= a
    assert np.array_equal(_conv(ctx, x * b, f, *args), plain * b)


def test_conv_f32_stem_choice(ctx):
    """By rule: large ones, with an error no larger than that of the kernel that fetches its own operands."""
    rng = np.random.Generator(np.random.PCG64(9))
    x = rng.standard_normal((32, 3, 224, 224)).astype(np.float32)
    f = rng.standard_normal((64, 3, 7, 7)).astype(np.float32)
    bias = rng.standard_normal(64).astype(np.float32)
    args = (f, bias, 2, (3, 3), (112, 112))
    got, other = _conv(ctx, x, *args, stem=0), _conv(ctx, x, *args, stem=1)
    assert np.array_equal(got, _conv(ctx, x, *args, stem=2)) and not np.array_equal(got, other)
    exact = _exact(x[:2], f, 2, (3, 3), (112, 112)) + bias[None, :, None, None]
    assert np.linalg.norm(got[:2] - exact) < np.linalg.norm(other[:2] - exact)
    small = (f[:, :, :3, :3].copy(), bias, 2, (1, 1), (112, 112))  # too shallow
    assert np.array_equal(_conv(ctx, x[:4], *small, stem=0), _conv(ctx, x[:4], *small, stem=1))


@pytest.mark.parametrize("geometry", [((1, 1), (3, 3), 30, 1), ((2, 2), (3, 3), 31, 1), ((2, 2), (3, 3), 30, 2), ((2, 4), (3, 3), 30, 1)])
def test_conv_f32_stem_refuses(ctx, geometry):
    """Other strides and dilations and odd widths go where they went."""
    strides, pad, W, dil = geometry
    rng = np.random.Generator(np.random.PCG64(2))
    x = rng.standard_normal((2, 3, 30, W)).astype(np.float32)
    f = rng.standard_normal((8, 3, 7, 7)).astype(np.float32)
    Ho, Wo = (30 + 6 - 6 * dil - 1) // strides[0] + 1, (W + 6 - 6 * dil - 1) // strides[1] + 1
    got = []
    dx, df = ctx.upload(x), ctx.upload(f)
    for stem in (1, 2):
        out = ctx.upload(np.zeros((2, 8, Ho, Wo), np.float32))
        ctx.set_option("f32_stem", stem)
        ctx.conv2d_f32(dx, df, None, out, 2, 3, 30, W, 8, 7, 7, strides, (dil, dil), pad, (Ho, Wo))
        ctx.set_option("f32_stem", 0)
        got.append(ctx.download(out, (2, 8, Ho, Wo), np.float32))
        out.free()
    for b in (dx, df):
        b.free()
    assert np.array_equal(got[0], got[1])


def test_conv_f32_stem_in_two_contexts(ctx):
    """A call that needs little shared memory, in a context of its own, takes none from a larger one's next call."""
    import mace_b200
    rng = np.random.Generator(np.random.PCG64(1))
    large, small = [(rng.standard_normal((1, c, 16, 16)).astype(np.float32), rng.standard_normal((64, c, k, k)).astype(np.float32), k)
                    for c, k in ((3, 7), (3, 1))]
    bias = np.zeros(64, np.float32)

    def run(c, x, f, k):
        return _conv(c, x, f, bias, 2 if k > 1 else 1, (k // 2, k // 2), (8, 8) if k > 1 else (16, 8))
    first = run(ctx, *large)
    other = mace_b200.Context(0)
    run(other, *small)
    other.close()
    assert np.array_equal(run(ctx, *large), first)
