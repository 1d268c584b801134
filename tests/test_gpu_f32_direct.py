"""The direct stride-1 fp32 convolution on the tensor cores (conv_f32_direct.cu) against float64, with bounds derived from its
arithmetic, at the edges of its tiles, and where its split of a value into two halves does not reach."""
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


def _windows(a, KH, KW):
    ph, pw = KH // 2, KW // 2
    padded = np.pad(a, ((0, 0), (0, 0), (ph, ph), (pw, pw)))
    return np.lib.stride_tricks.sliding_window_view(padded, (KH, KW), axis=(2, 3))


def _exact(x, f):
    return np.einsum("nchwij,ocij->nohw", _windows(x, *f.shape[2:]), f, optimize=True)


def _bound(x, f):
    """hi + lo of a value is within 2^-22 of it, and the accumulator is cut off by at most 2^-23 of what it holds after each of its
    MMAs (18 of large products between two hand-overs with the default runs here, a rounding for each hand-over)."""
    ax, af = np.abs(x), np.abs(f)
    K = f[0].size
    terms = _exact(ax, af)
    cut = min(K, 32 * f.shape[2] * f.shape[3]) / 16 + K / 32 + 4
    return terms * (2.0 ** -21 + cut * 2.0 ** -23) + 1e-37


def _run(ctx, x, f, bias, act=0, max_limit=0.0, coef=0.0, direct=2):
    N, C, H, W = x.shape
    O, _, KH, KW = f.shape
    dx, df, do = ctx.upload(x), ctx.upload(f), ctx.upload(np.full((N, O, H, W), 7, np.float32))
    db = ctx.upload(bias) if bias is not None else None
    ctx.set_option("f32_direct", direct)
    ctx.conv2d_f32(dx, df, db, do, N, C, H, W, O, KH, KW, (1, 1), (1, 1), (KH // 2, KW // 2), (H, W), act, max_limit, coef)
    ctx.set_option("f32_direct", 0)
    got = ctx.download(do, (N, O, H, W), np.float32)
    for b in (dx, df, do) + ((db,) if db else ()):
        b.free()
    return got


@pytest.mark.parametrize("case", [
    # N, C, H, W, O, KH, KW: a pixel, one channel, a block of channels and one more or less, tiles that span images, two and three
    # column tiles, rows that take the input warps two and three passes, more tiles than SMs, filters of other sizes
    (1, 1, 1, 1, 1, 3, 3), (1, 31, 5, 3, 2, 3, 3), (3, 32, 7, 7, 64, 3, 3), (2, 33, 9, 13, 65, 3, 3), (1, 96, 12, 10, 129, 3, 3),
    (1, 40, 3, 130, 20, 3, 3), (1, 8, 4, 200, 70, 3, 3), (40, 70, 23, 21, 30, 3, 3), (30, 65, 31, 17, 90, 3, 3),
    (2, 20, 11, 9, 66, 5, 5), (1, 34, 6, 14, 10, 7, 3), (1, 16, 16, 9, 33, 1, 5), (2, 100, 10, 10, 40, 1, 1)])
@pytest.mark.parametrize("act", [0, 1, 2, 6])
def test_direct_conv2d_f32(ctx, case, act):
    N, C, H, W, O, KH, KW = case
    rng = np.random.Generator(np.random.PCG64(C + O))
    x = rng.standard_normal((N, C, H, W)).astype(np.float32)
    f = (rng.standard_normal((O, C, KH, KW)) * 0.1).astype(np.float32)
    bias = rng.standard_normal(O).astype(np.float32) if act != 2 else None
    before = ctx.launches_tensor_core
    got = _run(ctx, x, f, bias, act, 0.75, 0.2)
    assert ctx.launches_tensor_core == before + 1
    x, f = x.astype(np.float64), f.astype(np.float64)
    ref = _exact(x, f) + (bias.astype(np.float64)[None, :, None, None] if bias is not None else 0.0)
    ref = {0: ref, 1: np.maximum(ref, 0), 2: np.clip(ref, 0, 0.75), 6: np.where(ref > 0, ref, ref * 0.2)}[act]
    assert (np.abs(got - ref) <= _bound(x, f) + 2.0 ** -22 * np.abs(ref)).all()


@pytest.mark.parametrize("O", [20, 100])
@pytest.mark.parametrize("what", ["zeros", "late", "tiny", "huge", "outlier", "inf", "nan", "inf_weight", "zero_weights", "steep"])
def test_direct_conv2d_f32_beyond_the_split(ctx, O, what):
    """Tiles and channels of zeros, scales that a later block of channels exceeds, values that halves do not hold."""
    N, C, HW = 3, 70, 15
    rng = np.random.Generator(np.random.PCG64(O))
    x = rng.standard_normal((N, C, HW, HW)).astype(np.float32)
    f = (rng.standard_normal((O, C, 3, 3)) * 0.1).astype(np.float32)
    if what == "zeros":
        x[:, :40], x[1] = 0, 0
    elif what == "late":
        x[:, 64:] *= np.float32(2.0 ** 16)
    elif what == "tiny":
        x *= np.float32(1e-25)
    elif what == "huge":
        x *= np.float32(1e30)
    elif what == "outlier":
        x[0, 3, 7, 7] = 1e12
    elif what == "inf":
        x[0, 3, 7, 7] = np.inf
    elif what == "nan":
        x[2, 69, 0, 0] = np.nan
    elif what == "inf_weight":
        f[5, 2, 1, 1] = -np.inf
    elif what == "zero_weights":
        f[:, :33], f[7] = 0, 0
    elif what == "steep":
        f *= np.float32(10.0) ** rng.integers(-12, 12, (O, 1, 1, 1)).astype(np.float32)
    got = _run(ctx, x, f, None)
    with np.errstate(all="ignore"):
        x, f = x.astype(np.float64), f.astype(np.float64)
        # (padding is left out: a weight that is infinite meets no zero there)
        w = _windows(x, 3, 3)
        inside = _windows(np.ones_like(x), 3, 3) > 0
        ref = np.stack([np.where(inside, w * f[o][None, :, None, None], 0).sum(axis=(1, 4, 5)) for o in range(O)], axis=1)
        assert np.array_equal(np.isnan(got), np.isnan(ref))
        finite = np.isfinite(ref)
        assert np.array_equal(got[~finite & ~np.isnan(ref)], ref[~finite & ~np.isnan(ref)])
        xs, fs = np.where(np.isfinite(x), x, 0), np.where(np.isfinite(f), f, 0)
        # (worked out again, a sum of K products rounds K times)
        bound = _bound(xs, fs) + _exact(np.abs(xs), np.abs(fs)) * f[0].size * 2.0 ** -24
        assert (np.abs(got - ref)[finite] <= bound[finite]).all()


@pytest.mark.parametrize("spread", [2.0 ** 10, 2.0 ** 20])
@pytest.mark.parametrize("O", [20, 100])
def test_direct_conv2d_f32_spread(ctx, O, spread):
    """Small values that meet large weights keep their bits, and so do dark regions beside bright ones."""
    rng = np.random.Generator(np.random.PCG64(O))
    x = rng.standard_normal((2, 70, 15, 15)).astype(np.float32)
    f = (rng.standard_normal((O, 70, 3, 3)) * 0.1).astype(np.float32)
    def error(x, f, part):
        got, exact = _run(ctx, x, f, None), _exact(x.astype(np.float64), f.astype(np.float64))
        assert (np.abs(got - exact) <= _bound(x, f)).all()
        return np.linalg.norm((got - exact)[part]) / np.linalg.norm(exact[part])

    for dim, dark in ((np.s_[:, :, :8], np.s_[:, :, :7]), (np.s_[:, :, :, 8:], np.s_[:, :, :, 9:])):
        plain, y = error(x, f, dark), x.copy()
        y[dim] *= np.float32(1 / spread)
        assert error(y, f, dark) <= 1.05 * plain
    plain = error(x, f, np.s_[:])
    x[:, ::7] *= np.float32(1 / spread)
    f[:, ::7] *= np.float32(spread)
    assert error(x, f, np.s_[:]) <= 1.05 * plain


@pytest.mark.parametrize("O", [20, 100])
def test_direct_conv2d_f32_beside_an_outlier(ctx, O):
    """One value up to 1e6 times larger than its tile's others, which is held with them: they keep their bits, and so do its results."""
    rng = np.random.Generator(np.random.PCG64(O))
    x = rng.standard_normal((1, 70, 15, 15)).astype(np.float32)
    f = (rng.standard_normal((O, 70, 3, 3)) * 0.1).astype(np.float32)
    far = np.ones((15, 15), bool)
    far[6:9, 4:7] = False
    plain, exact = _run(ctx, x, f, None), _exact(x.astype(np.float64), f.astype(np.float64))
    error = np.linalg.norm((plain - exact)[:, :, far]) / np.linalg.norm(exact[:, :, far])
    for value in (3e4, 1e6):
        x[0, 40, 7, 5] = value
        got, exact = _run(ctx, x, f, None), _exact(x.astype(np.float64), f.astype(np.float64))
        assert (np.abs(got - exact) <= _bound(x, f)).all()
        assert np.linalg.norm((got - exact)[:, :, far]) / np.linalg.norm(exact[:, :, far]) <= 1.05 * error


@pytest.mark.parametrize("powers", [(-100, 0), (0, -100), (-70, -40), (60, -110), (-110, 60), (90, -60)])
@pytest.mark.parametrize("O", [20, 100])
def test_direct_conv2d_f32_scales(ctx, O, powers):
    """Results are those of operands of ordinary size, bit for bit: nothing is worked out again because a row is small or large."""
    rng = np.random.Generator(np.random.PCG64(O))
    x = rng.standard_normal((2, 40, 12, 12)).astype(np.float32)
    f = (rng.standard_normal((O, 40, 3, 3)) * 0.1).astype(np.float32)
    plain = _run(ctx, x, f, None)
    a, b = (np.float32(2.0) ** p for p in powers)
    f[::3] *= a
    plain[:, ::3] *= a
    assert np.array_equal(_run(ctx, x * b, f, None), plain * b)


@pytest.mark.parametrize("power", [-16, -8, 8, 16])
@pytest.mark.parametrize("KH", [3, 5])
@pytest.mark.parametrize("O", [20, 100])
def test_direct_conv2d_f32_blocks(ctx, O, KH, power):
    """Blocks of channels of another size than the first, for which the weights make up: the same results, bit for bit, and so none of
    them is worked out again."""
    rng = np.random.Generator(np.random.PCG64(O))
    x = rng.standard_normal((2, 100, 12, 70)).astype(np.float32)
    f = (rng.standard_normal((O, 100, KH, 3)) * 0.1).astype(np.float32)
    f = np.sign(f) * np.clip(np.abs(f), 2.0 ** -7, 0.5)  # (all of them within reach of both halves)
    plain = _run(ctx, x, f, None)
    for c0, c1 in ((32, 64), (96, 100)):
        x[:, c0:c1] *= np.float32(2.0) ** power
        f[:, c0:c1] *= np.float32(2.0) ** -power
    assert np.array_equal(_run(ctx, x, f, None), plain)


def test_direct_conv2d_f32_choice(ctx):
    """By rule: a batch of 3x3 and 5x5 layers, and no smaller an accuracy there than the other kernels have."""
    rng = np.random.Generator(np.random.PCG64(0))
    N, C, HW, O = 16, 64, 28, 64
    for k in (3, 5):
        x = rng.standard_normal((N, C, HW, HW)).astype(np.float32)
        f = (rng.standard_normal((O, C, k, k)) * np.sqrt(2.0 / (k * k * C))).astype(np.float32)
        exact = _exact(x.astype(np.float64), f.astype(np.float64))
        err = [np.linalg.norm(_run(ctx, x, f, None, direct=d) - exact) / np.linalg.norm(exact) for d in (0, 1, 2)]
        assert err[0] <= 1.02 * err[1] and err[2] <= err[1]


def test_direct_conv2d_f32_inside_a_capture(ctx):
    """A graph keeps the block of its split filter although later calls need a larger one."""
    import mace_b200
    c = mace_b200.Context(0)
    rng = np.random.Generator(np.random.PCG64(1))
    x = rng.standard_normal((2, 32, 12, 12)).astype(np.float32)
    f = rng.standard_normal((64, 32, 3, 3)).astype(np.float32)
    exact = _exact(x.astype(np.float64), f.astype(np.float64))
    dx, df, do = c.upload(x), c.upload(f), c.alloc(exact.size * 4)

    def call():
        c.conv2d_f32(dx, df, None, do, 2, 32, 12, 12, 64, 3, 3, (1, 1), (1, 1), (1, 1), (12, 12))

    def check():
        assert np.abs(c.download(do, exact.shape, np.float32) - exact).max() <= 1e-4 * np.abs(exact).max()

    L = mace_b200.lib()
    c.set_option("f32_direct", 2)
    graphs = []
    for _ in range(2):
        c._check(L.mb_graph_begin(c.h))
        call()
        graphs.append(ctypes.c_void_p())
        c._check(L.mb_graph_end(c.h, ctypes.byref(graphs[-1])))
        call()
        check()
    big = c.upload(rng.standard_normal((256, 512, 3, 3)).astype(np.float32))
    bx, bo = c.upload(rng.standard_normal((1, 512, 8, 8)).astype(np.float32)), c.alloc(256 * 64 * 4)
    c.conv2d_f32(bx, big, None, bo, 1, 512, 8, 8, 256, 3, 3, (1, 1), (1, 1), (1, 1), (8, 8))
    c.sync()
    for g in graphs:
        c._check(L.mb_memset(c.h, do.ptr, 0, do.nbytes))
        c._check(L.mb_graph_launch(c.h, g))
        check()
        c._check(L.mb_graph_destroy(c.h, g))
    c.close()


def test_direct_conv2d_f32_first_inside_a_capture():
    """The same bits whether or not calls before the recording left room for the split filters."""
    import mace_b200
    c = mace_b200.Context(0)
    L = mace_b200.lib()
    rng = np.random.Generator(np.random.PCG64(2))
    layers = []
    for C, O in ((32, 64), (256, 256)):  # (the second one's block is a larger one)
        x, f = rng.standard_normal((2, C, 12, 12)).astype(np.float32), rng.standard_normal((O, C, 3, 3)).astype(np.float32)
        layers.append((c.upload(x), c.upload(f), c.alloc(2 * O * 144 * 4), C, O))

    def calls():
        for x, f, out, C, O in layers:
            c.conv2d_f32(x, f, None, out, 2, C, 12, 12, O, 3, 3, (1, 1), (1, 1), (1, 1), (12, 12))

    def results():
        got = [c.download(out, (2, O, 144), np.float32) for _, _, out, _, O in layers]
        for layer in layers:
            c._check(L.mb_memset(c.h, layer[2].ptr, 0, layer[2].nbytes))
        return got

    c.set_option("f32_direct", 2)
    c._check(L.mb_graph_begin(c.h))
    calls()
    g = ctypes.c_void_p()
    c._check(L.mb_graph_end(c.h, ctypes.byref(g)))
    c._check(L.mb_graph_launch(c.h, g))
    recorded = results()
    calls()
    for a, b in zip(recorded, results()):
        assert np.array_equal(a, b)
    c._check(L.mb_graph_launch(c.h, g))
    for a, b in zip(recorded, results()):
        assert np.array_equal(a, b)
    c._check(L.mb_graph_destroy(c.h, g))
    c.close()


@pytest.mark.parametrize("O", [64, 128])
def test_direct_conv2d_f32_in_two_contexts(ctx, O):
    """A call that needs little shared memory, in a context of its own, takes none from a larger one's next call."""
    import mace_b200
    rng = np.random.Generator(np.random.PCG64(1))
    large, small = [(rng.standard_normal((1, c, hw, hw)).astype(np.float32), rng.standard_normal((O, c, 3, 3)).astype(np.float32))
                    for c, hw in ((256, 56), (16, 8))]
    first = _run(ctx, *large, None)
    other = mace_b200.Context(0)
    _run(other, *small, None)
    other.close()
    assert np.array_equal(_run(ctx, *large, None), first)
