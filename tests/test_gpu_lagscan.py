"""The lag scan's tables and legality (k3_satp, k2_sat2w, k2_lagscan).

uint8 pairs whose overlaps fit take packed tables, the same pixels as uint16
take 64-bit pairs; both hold exact integers, so the two calls give the same
numbers bit for bit.  A LegalRgn rule tabulated by the caller is looked up per
lag, the typed rule becomes a range of box widths per lag row: the same again.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import alignment_projects_gb300 as aln
    c = aln.Context(0)
    c.set_tuning(False)   # one column plan for both pixel types
    yield c
    c.close()


def _pair(rng, w, h, extreme=False, zeros=0.0):
    big = rng.integers(0, 256, (h + 8, w + 8))
    if extreme:
        big = np.where(big < 128, 0, 255)
    big[rng.random(big.shape) < zeros] = 0
    a = big[4:4 + h, 4:4 + w]
    ty, tx = (int(v) for v in rng.integers(-3, 4, 2))
    b = big[4 + ty:4 + ty + h, 4 + tx:4 + tx + w]
    return a.astype(np.uint8), b.astype(np.uint8)


def _view(t, col, pitch):
    """The same raster on the device inside a wider one, at column col."""
    import torch
    host = torch.from_numpy(t)
    big = torch.zeros((t.shape[0], pitch), dtype=host.dtype, device="cuda")
    big[:, col:col + t.shape[1]] = host.cuda()
    return big[:, col:col + t.shape[1]]


@pytest.mark.parametrize("w,h,radius,cnt", [
    (8, 9, 4096, 0), (17, 40, 4096, 0), (63, 65, 20, 0), (64, 64, 4096, 1), (65, 130, 4096, 1),
    (127, 500, 30, 0), (235, 700, 64, 0), (129, 33, 4096, 1), (700, 130, 64, 1),
    (300, 301, 4096, 0)])
def test_packed_tables_equal_wide_ones(ctx, w, h, radius, cnt):
    import alignment_projects_gb300 as aln
    rng = np.random.default_rng(w * 1000 + h)
    jobs = []
    for k in range(4):
        a, b = _pair(rng, w, h, extreme=k == 1, zeros=0.3 if cnt else 0.0)
        lg = aln.legal(aln.RGN_MIN, min(5, w), min(5, h), 0,
                       aln.CNT_GT if cnt else aln.CNT_NONE, w * h // 10)
        col, pitch = (0, w) if k < 2 else (k - 1, w + 5 + k)   # odd starts and strides
        jobs.append([dict(a=_view(x, col, pitch), b=_view(y, col, pitch), radius=radius, legal=lg)
                     for x, y in ((a, b), (a.astype(np.uint16), b.astype(np.uint16)))])
    got8 = ctx.corr_patches_batch([j[0] for j in jobs])
    got16 = ctx.corr_patches_batch([j[1] for j in jobs])
    assert got8 == got16
    assert any(g["status"] == aln.ALN_OK for g in got8)


@pytest.mark.parametrize("w,h", [(1448, 1448), (1449, 1448)])
def test_packing_limit(ctx, w, h):
    """Overlaps just below 2^21 pixels (packed) and just above (not)."""
    rng = np.random.default_rng(w)
    a, b = _pair(rng, w, h, extreme=True)
    one = dict(radius=6)
    got = [ctx.corr_patches_batch([dict(a=x, b=y, **one)])[0]
           for x, y in ((a, b), (a.astype(np.uint16), b.astype(np.uint16)))]
    # 16-bit overlaps from 2^20 pixels take the FP64 formula for r
    assert abs(got[0]["r"] - got[1]["r"]) < 1e-6
    assert (got[0]["peak_x"], got[0]["peak_y"]) == (got[1]["peak_x"], got[1]["peak_y"])
    white = np.full((h, w), 255, np.uint8)
    white[::7, ::5] = 0
    g = ctx.corr_patches_batch([dict(a=white, b=white, **one)])[0]
    # every lag of the pattern's period (5, 7) matches exactly
    assert (g["peak_x"] % 5, g["peak_y"] % 7) == (0, 0) and abs(g["r"] - 1) < 1e-5


def _rule(kind, sx, sy, a, b, area):
    import alignment_projects_gb300 as aln
    if kind == aln.RGN_MIN:
        return (sx >= a) & (sy >= b) & (sx * sy > area)
    if kind == aln.RGN_SECTION:
        return (sx * sy > area) & ((sx >= a) | (sy > b))
    return (sx == a) & (sy == b)


@pytest.mark.parametrize("w,h", [(60, 90), (110, 70)])   # as is, and solved transposed
@pytest.mark.parametrize("kind,a,b,area", [
    (1, 20, 30, 0), (1, 0, 0, 1500), (1, 55, 61, 3000), (1, 7, 9, -5), (1, 10, 10, 1 << 40),
    (2, 30, 45, 1200), (2, 0, 80, 2000), (2, 200, 200, 0), (2, 52, 0, 900), (3, 47, 66, 0),
    (3, 500, 1, 0)])
def test_typed_rule_equals_its_table(ctx, w, h, kind, a, b, area):
    import alignment_projects_gb300 as aln
    rng = np.random.default_rng(w + a + b)
    sx, sy = np.meshgrid(np.arange(1, w + 1), np.arange(1, h + 1))
    table = _rule(kind, sx, sy, a, b, area).astype(np.uint8)
    A, B = _pair(rng, w, h)
    for dt in (np.uint8, np.uint16, np.float32):
        x, y = A.astype(dt), B.astype(dt)
        got = ctx.corr_patches_batch([
            dict(a=x, b=y, radius=40, legal=aln.legal(kind, a, b, area)),
            dict(a=x, b=y, radius=40, legal=aln.legal(table=table))])
        assert got[0] == got[1], dt
        imgs = ctx.corr_images_batch([
            dict(kind=aln.CORR_R, a=x, b=y, legal=aln.legal(kind, a, b, area)),
            dict(kind=aln.CORR_R, a=x, b=y, legal=aln.legal(table=table))])
        assert imgs[0] == imgs[1], dt


@pytest.mark.parametrize("data", ["normal", "f32", "offset", "tiny", "flat", "u8", "u16", "mixed"])
@pytest.mark.parametrize("rule", ["none", "min", "counts", "oval", "mincor", "mincor-none"])
def test_corr_images_r_bound(ctx, orc, data, rule):
    """CorrImagesR's scan looks closer only where an FP32 bound of R reaches the
    best R found: the oracle's peak for images that make the bound tight, loose
    or useless, under each kind of rule."""
    import oracle as O
    from test_gpu_images import aln_legal, check
    rng = np.random.default_rng(len(data) * 100 + len(rule))
    big = rng.standard_normal((70, 66))
    for _ in range(2):   # some structure: neighbours alike
        big = (big + np.roll(big, 1, 0) + np.roll(big, 1, 1)) / 1.7
    a, b = big[5:47, 6:45], big[9:61, 3:58]
    b = b + 0.2 * rng.standard_normal(b.shape)
    if data == "offset":
        a, b = 3000.0 + a, 3000.0 + b
    elif data == "tiny":
        a, b = 1e-9 * a, 1e-9 * b
    elif data == "flat":
        a, b = np.where(a < 1.5, 0.0, a), np.where(b < 1.0, 0.0, b)
    elif data in ("u8", "u16", "mixed"):
        top = 255 if data != "u16" else 4095
        a, b = (np.clip(np.rint((v + 4) * top / 8), 0, top) for v in (a, b))
        a = a.astype(np.uint16 if data == "u16" else np.uint8)
        b = b.astype({"u8": np.uint8, "u16": np.uint16, "mixed": np.float32}[data])
    if data in ("f32", "flat"):
        a, b = a.astype(np.float32), b.astype(np.float32)
    n = 400 if rule == "counts" else 0
    lg = O.legal(*((O.RGN_MIN, 12, 12, 300) if rule != "none" else (0, 0, 0, 0)),
                 1 if rule == "counts" else 0, n)
    mincor = 0.05 if rule == "mincor" else 1.5 if rule == "mincor-none" else 0.0
    disc = (3, -4, 17, 9) if rule == "oval" else (0, 0, -1, -1)
    g = ctx.corr_images(1, a, b, aln_legal(lg), mincor, 0.75, *disc)
    pts = [np.stack([v.ravel() for v in np.mgrid[0:m.shape[0], 0:m.shape[1]][::-1]], 1)
           .astype(np.float64) for m in (a, b)]
    o = orc.corr_images(1, pts[0], a.ravel().astype(np.float64), pts[1],
                        b.ravel().astype(np.float64), lg, mincor, 0.75, *disc)
    check(g, o, 1, (data, rule))


@pytest.mark.parametrize("kinds", ["u8 u8", "u16 u16", "u8 u16", "f32 f32", "f64 f64", "u8 f32"])
@pytest.mark.parametrize("away,sd", [(60, 0.4), (100, 0.5), (120, 0.8)])
def test_corr_images_r_flat_overlaps(ctx, kinds, away, sd):
    """Images whose searched overlaps are nearly flat and far from the image's
    mean, where FP32 gives R to 1e-3 only: the scan's peak is the largest
    of the values that the same call gives lag by lag (a box rule that one lag of
    the oval meets; the correlation is the same numbers), alone and in a batch."""
    import alignment_projects_gb300 as aln
    rng = np.random.default_rng(away)
    h, w, rx, ry = 48, 1024, 128, 10
    cx = w // 2 + rx   # lags that overlap a's dark left half with b's dark right half
    lags = [(x, y) for y in range(-ry, ry + 1) for x in range(cx - rx, cx + rx + 1)
            if (x - cx) ** 2 + (rx / ry) ** 2 * y * y <= rx * rx]
    for _ in range(3):
        job = {}
        for name, dt, dark in zip("ab", kinds.split(), (0, w // 2)):
            scale = 16 if dt == "u16" else 1
            v = np.full((h, w), 128.0 + away)
            v[:, dark:dark + w // 2] -= 2 * away
            v = np.rint((v + sd * rng.standard_normal((h, w))) * scale)
            job[name] = _view(np.clip(v, 0, 255 * scale).astype(
                dict(u8=np.uint8, u16=np.uint16, f32=np.float32, f64=np.float64)[dt]), 0, w)
        job.update(kind=aln.CORR_R, ox=cx, oy=0, rx=rx, ry=ry,
                   legal=aln.legal(aln.RGN_MIN, 8, 8, 0))
        each = ctx.corr_images_batch([
            dict(job, ox=x, oy=y, rx=1, ry=1,
                 legal=aln.legal(aln.RGN_EXACT, w - x, h - abs(y), 0)) for x, y in lags])
        assert all(e["status"] == aln.ALN_OK and (e["peak_x"], e["peak_y"]) == q
                   for e, q in zip(each, lags))
        best = max(range(len(lags)), key=lambda k: each[k]["r"])
        for g in ctx.corr_images_batch([job]) + ctx.corr_images_batch([job] * 40):
            assert (g["r"], (g["peak_x"], g["peak_y"])) == (each[best]["r"], lags[best])


@pytest.mark.parametrize("dtype", [np.uint8, np.uint16, np.float32])
def test_far_disc_centre(ctx, orc, dtype):
    """A disc around a point 40000 px off whose edge crosses the lags: the
    oracle's peak, for CorrPatches' circle and CorrImages' oval."""
    import oracle as O
    from test_gpu_corr import assert_parity
    from test_gpu_images import aln_legal, check
    rng = np.random.default_rng(8)
    a, b = _pair(rng, 60, 70)
    b[::5, ::3] //= 2   # (equal images: R = 1, which CorrImages takes as 0)
    a, b = a.astype(dtype), b.astype(dtype)
    lg = O.legal(O.RGN_MIN, 20, 20, 0)
    pa, pb = (O.image_to_points(t) for t in (a, b))
    for ox, oy in ((43000, 0), (-43000, 0), (0, 43000), (5, -43000)):
        rad = 43000 + 12
        g = ctx.corr_patches_batch([dict(a=a, b=b, ox=ox, oy=oy, radius=rad,
                                         legal=aln_legal(lg))])[0]
        assert_parity(g, orc.corr_patches(*pa, *pb, ox, oy, rad, lg), f"disc {ox} {oy}")
        for kind in (1, 2):
            g = ctx.corr_images(kind, a, b, aln_legal(lg), 0.0, 0.75, ox, oy, rad, rad)
            o = orc.corr_images(kind, *pa, *pb, lg, 0.0, 0.75, ox, oy, rad, rad)
            check(g, o, kind, f"oval {kind} {ox} {oy}")


@pytest.mark.parametrize("w,h", [(33, 5), (127, 31), (128, 32), (129, 33), (131, 64), (512, 30),
                                 (513, 97), (640, 36), (1030, 203)])
@pytest.mark.parametrize("col", [0, 1, 2])
def test_transposed_solve(ctx, w, h, col):
    """A wide pair is solved on its transposed images: the same as the pair
    handed over transposed, at tile edges, odd sizes, starts and strides."""
    rng = np.random.default_rng(w + h + col)
    a, b = _pair(rng, w, h)
    wide = dict(a=_view(a, col, w + 3 * col), b=_view(b, col, w + 3 * col), radius=20)
    tall = dict(a=np.ascontiguousarray(a.T), b=np.ascontiguousarray(b.T), radius=20)
    g, t = ctx.corr_patches_batch([wide, tall])
    assert (g["r"], g["dx"], g["dy"], g["peak_x"], g["peak_y"]) == \
        (t["r"], t["dy"], t["dx"], t["peak_y"], t["peak_x"])


@pytest.mark.parametrize("dtype", ["u8", "u16"])
@pytest.mark.parametrize("w,h", [(90, 300), (300, 90)])
def test_overlapped_launches(ctx, w, h, dtype):
    """Alone, a pair's kernels are launched ahead of the end of the one before
    them; a batch's grids of many waves wait.  The same numbers bit for bit."""
    rng = np.random.default_rng(w)
    dt = np.uint8 if dtype == "u8" else np.uint16
    kinds = [dict(zip("ab", (_view(t.astype(dt), 0, w) for t in _pair(rng, w, h))), radius=20)
             for _ in range(8)]
    alone = [ctx.corr_patches_batch([k])[0] for k in kinds]
    batch = ctx.corr_patches_batch([kinds[i % 8] for i in range(1600)])
    assert batch == [alone[i % 8] for i in range(1600)]


@pytest.mark.parametrize("dtype", [np.uint8, np.uint16, np.float32, np.float64])
@pytest.mark.parametrize("kind", [1, 2])   # CORR_R, CORR_S
def test_overlapped_image_launches(ctx, dtype, kind):
    """The same for CorrImages' kernels, with and without a count rule and a
    mincor."""
    import alignment_projects_gb300 as aln
    rng = np.random.default_rng(kind)
    jobs = []
    for k in range(8):
        a, b = _pair(rng, 70, 60, zeros=0.2)
        b[::4, ::3] //= 2
        jobs.append(dict(kind=kind, a=_view(a.astype(dtype), 0, 70), b=_view(b.astype(dtype), 0, 70),
                         mincor=0.05 * (k // 4),
                         legal=aln.legal(aln.RGN_MIN, 20, 20, 0, aln.CNT_GT if k % 2 else 0, 300)))
    alone = [ctx.corr_images_batch([j])[0] for j in jobs]
    assert all(g["status"] == aln.ALN_OK for g in alone)
    batch = ctx.corr_images_batch([jobs[i % 8] for i in range(1600)])
    assert batch == [alone[i % 8] for i in range(1600)]


@pytest.mark.parametrize("dtype", [np.uint8, np.uint16, np.float32])
@pytest.mark.parametrize("images", [False, True])
def test_long_scans_alone_and_batched(ctx, dtype, images):
    """A pair over all lags, whose scan waits for its lag image or is launched
    ahead by how many blocks there are: the same numbers alone and in a batch."""
    import alignment_projects_gb300 as aln
    rng = np.random.default_rng(7)
    job = dict(zip("ab", (_view(t.astype(dtype), 0, 400) for t in _pair(rng, 400, 430))),
               legal=aln.legal(aln.RGN_MIN, 40, 40, 0), **(dict(kind=1) if images else {}))
    call = ctx.corr_images_batch if images else ctx.corr_patches_batch
    alone = call([job])
    for n in (3, 9):
        assert call([job] * n) == alone * n


@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_images_with_infinities(ctx, orc, dtype, value):
    """A pixel that is no number spoils every lag: R is 0 at all of them, as the
    oracle has it, and S and CorrPatches find no peak."""
    import oracle as O
    from test_gpu_images import aln_legal, check
    a, b = (t.astype(dtype) for t in _pair(np.random.default_rng(4), 50, 41))
    a[20, 30] = value
    lg = O.legal(O.RGN_MIN, 10, 10, 0)
    pa, pb = (O.image_to_points(t) for t in (a, b))
    with np.errstate(all="ignore"):
        o = orc.corr_images(1, *pa, *pb, lg)
    job = dict(a=a, b=b, legal=aln_legal(lg))
    for g in ctx.corr_images_batch([dict(job, kind=1)] * 3):
        check(g, o, 1, (dtype, value))
    none = ctx.corr_images_batch([dict(job, kind=2)]) + ctx.corr_patches_batch([job])
    assert all(g["status"] == 1 and g["r"] == 0 for g in none)
