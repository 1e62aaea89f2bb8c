"""MakeThumbs' sums on the GPU (aln_decimate_batch): the parallel form of
MeanStd's sequential FP64 sums, bit for bit against the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import alignment_projects_gb300 as aln
    c = aln.Context(0)
    yield c
    c.close()


def _image(kind, h, w, rng):
    if kind == "u8":
        return rng.integers(0, 256, (h, w)).astype(np.uint8)
    if kind == "u16":
        return rng.integers(0, 65536, (h, w)).astype(np.uint16)
    if kind == "f32+":       # non-negative, full significands: ties in the sum of squares
        return rng.random((h, w)).astype(np.float32)
    if kind == "f64+":
        return rng.random((h, w)) * 10.0 ** rng.integers(-12, 6, (h, w))
    if kind == "f32-":       # signed: the first rows positive, then both signs
        x = rng.standard_normal((h, w)).astype(np.float32)
        x[: h // 2] = np.abs(x[: h // 2])
        return x
    x = rng.integers(0, 256, (h, w)).astype(np.uint8)   # "late": zeros, then values
    x[: h - 2] = 0
    return x


@pytest.mark.parametrize("kind,h,w,lbin", [
    ("u8", 1, 1, 1), ("u8", 3, 2, 1), ("u8", 64, 64, 1), ("u8", 64, 65, 1),
    ("u8", 512, 700, 8), ("u8", 523, 701, 8), ("u8", 333, 444, 3), ("u8", 900, 1200, 1),
    ("u8", 518, 1030, 4), ("u16", 900, 1200, 1), ("u16", 517, 700, 4), ("f32+", 300, 411, 1),
    ("f32+", 517, 701, 8), ("f64+", 200, 303, 1), ("f32-", 301, 399, 1), ("late", 97, 130, 1),
    ("late", 97, 130, 5)])
def test_sequential_sums_bitwise(ctx, orc, kind, h, w, lbin):
    img = _image(kind, h, w, np.random.default_rng(h * 1000 + w + lbin))
    yy, xx = np.mgrid[0:h, 0:w]
    pts = np.stack([xx.ravel(), yy.ravel()], 1).astype(np.float64)
    xy, v = orc.decimate_normalize(pts, img.ravel().astype(np.float64), w, h, lbin)
    vals, pres, _ = ctx.decimate([img], lbin)[0]
    ys, xs = np.nonzero(pres)
    assert np.array_equal(np.stack([xs, ys], 1), xy.astype(np.int64))
    assert np.array_equal(vals[ys, xs], v, equal_nan=True)   # bit for bit


@pytest.mark.parametrize("value", [1e308, 1e154])   # the sum, the sum of squares overflows
@pytest.mark.parametrize("at", [300, 4094, 4700])   # in a chunk, over its end, in the next one
def test_sums_that_overflow(ctx, orc, value, at):
    """A running sum that reaches infinity stays there, as one thread's would."""
    h, w = 90, 101
    img = np.random.default_rng(at).random(h * w) + 0.5
    img[at:at + 4] = value
    img[at + 700:at + 704] = value
    img = img.reshape(h, w)
    yy, xx = np.mgrid[0:h, 0:w]
    pts = np.stack([xx.ravel(), yy.ravel()], 1).astype(np.float64)
    with np.errstate(all="ignore"):
        _, v = orc.decimate_normalize(pts, img.ravel(), w, h, 1)
    vals, pres, _ = ctx.decimate([img], 1)[0]
    assert pres.all()
    assert np.array_equal(vals.ravel(), v, equal_nan=True)


@pytest.mark.parametrize("n", [1, 16])
@pytest.mark.parametrize("kind", ["u8", "f64+", "f32-", "late"])
@pytest.mark.parametrize("h,w,lbin", [(2, 1, 1), (8, 8, 1), (16, 16, 1), (16, 17, 1), (32, 32, 16),
                                      (40, 36, 3)])
def test_small_thumbnails(ctx, orc, kind, h, w, lbin, n):
    """Up to 256 bins the sums are made where the bins are normalised: bit for
    bit, alone and beside a larger image, whose sums have a kernel of their own."""
    rng = np.random.default_rng(h * w)
    imgs = [_image(kind, h, w, rng) for _ in range(n)] + [_image(kind, 40, 50, rng)]
    yy, xx = np.mgrid[0:h, 0:w]
    pts = np.stack([xx.ravel(), yy.ravel()], 1).astype(np.float64)
    alone, beside = ctx.decimate(imgs[:n], lbin), ctx.decimate(imgs, lbin)
    for img, (vals, pres, sd), (vals2, pres2, sd2) in zip(imgs, alone, beside):
        with np.errstate(all="ignore"):
            xy, v = orc.decimate_normalize(pts, img.ravel().astype(np.float64), w, h, lbin)
        ys, xs = np.nonzero(pres)
        assert np.array_equal(np.stack([xs, ys], 1), xy.astype(np.int64))
        assert np.array_equal(vals[ys, xs], v, equal_nan=True)
        assert np.array_equal(vals, vals2, equal_nan=True) and np.array_equal(pres, pres2)
        assert sd == sd2


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("at", [3, 5000])   # among the first bins, in a later chunk
def test_sums_of_infinities(ctx, orc, value, at):
    h, w = 90, 101
    img = np.random.default_rng(at).random(h * w).astype(np.float32)
    img[at] = value
    img = img.reshape(h, w)
    yy, xx = np.mgrid[0:h, 0:w]
    pts = np.stack([xx.ravel(), yy.ravel()], 1).astype(np.float64)
    with np.errstate(all="ignore"):
        _, v = orc.decimate_normalize(pts, img.ravel().astype(np.float64), w, h, 1)
    vals, pres, _ = ctx.decimate([img], 1)[0]
    assert pres.all() and np.array_equal(vals.ravel(), v, equal_nan=True)
