"""The matcher's work as its users have it done: the cases that timings of this
framework refer to.

Each case is a dict of plain values; its "path" names the public entry point
it goes through:

  pair      one CorrPatches call per pair (aln_corr_patches)
  strips    a batch of montage overlap strips (aln_corr_patches_batch)
  uneven    a batch of 16-bit patches of mixed sizes (the same call)
  window    a batch of square patches over every lag (the same call)
  images    a batch of CorrImagesR / CorrImagesS calls (aln_corr_images_batch)
  fft       FFT_2D and IFT_2D on host arrays (Context.fft_2d, Context.ift_2d)
  thumbs    MakeThumbs' binning and normalisation (Context.decimate)
  sweep     CThmScan on thumbnail pairs (aln_thm_search_batch): the correlator
            at one angle, a coarse scan, or the whole search
  approx    ApproximateMatch on tile pairs (Context.approx_match_batch)

The correlators transform in FP32 and hand their numbers over in C doubles; a
match table keeps them as FP32, and so do the outputs here.  FFT_2D and the
thumbnails come as the call returns them.

Inputs are synthetic EM-like images: noise with a 1/f^1.5 power spectrum, dark
membrane ellipses painted over it, sensor noise on every exposure.
"""
import ctypes as C
import math

import numpy as np
import torch

import alignment_projects_gb300 as aln
from alignment_projects_gb300.native import (AlnImage, AlnImageJob, AlnPair, AlnResult,
                                             AlnThmParams, AlnThmResult, AlnThumbs)

DEV = "cuda"
JITTER = 40           # stage error of a montage tile, px
STRIP_RADIUS = 64     # the disc searched around the expected offset
DECOYS = 0.02         # overlaps whose tiles do not show the same tissue

RESULT = np.dtype([("r", "f8"), ("dx", "f8"), ("dy", "f8"), ("status", "i4"), ("px", "i4"),
                   ("py", "i4"), ("nx", "i4"), ("ny", "i4")], align=True)
THM = np.dtype([("A", "f8"), ("X", "f8"), ("Y", "f8"), ("R", "f8"), ("T", "f8", 6),
                ("err", "i4"), ("ncalls", "i4")], align=True)


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

def listed():
    return [
        # one left-right overlap of two 2048^2 tiles, one call: what an
        # interactive re-match or a caller that was not batched waits for
        {"name": "strip_pair", "path": "pair", "w": 235, "h": 2048, "dtype": "u8"},
        # a whole section's neighbour overlaps in one submission, tiles on the device
        {"name": "strips_section", "path": "strips", "n": 4096, "long": 2048, "host": False},
        # the same from page-locked host memory, as a tile reader leaves it
        {"name": "strips_host", "path": "strips", "n": 512, "long": 2048, "host": True},
        # regions of any shape between layers: 16-bit, ragged, nearly every grid
        {"name": "uneven_batch", "path": "uneven", "n": 3000, "smin": 64, "smax": 1024},
        # full search of small tiles, no prior offset: the whole lag image
        {"name": "window_512", "path": "window", "n": 48, "side": 512},
        # CorrImagesR on normalised rasters with a count rule (in-section overlap)
        {"name": "images_r", "path": "images", "kind": "R", "n": 24, "w1": 300, "h1": 421,
         "w2": 339, "h2": 400, "dtype": "f64", "oval": 0},
        # the FFT pair on its own, there and back, host arrays as in the reference
        {"name": "fft_1024", "path": "fft", "nx": 1024, "ny": 1024},
        # thumbnails of eight 2048^2 tiles at the pipeline's factor of 8
        {"name": "thumbs_8", "path": "thumbs", "n": 8, "w": 2048, "h": 2048, "bin": 8,
         "dtype": "u8"},
        # one correlator call of the sweep: one pair at one angle
        {"name": "sweep_angle", "path": "sweep", "mode": "angle", "n": 1, "side": 256},
        # the coarse scan of many cross-layer pairs
        {"name": "sweep_scan", "path": "sweep", "mode": "scan", "n": 48, "side": 256},
        # the whole search: coarse scan, fine scan and peak hunt
        {"name": "sweep_search", "path": "sweep", "mode": "search", "n": 24, "side": 256},
        # the chain the pipeline runs per tile pair, from the host's tiles
        {"name": "approx_match", "path": "approx", "n": 3, "tile": 1024, "dec": 4},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["pair", "strips", "strips", "uneven", "window", "images", "images", "fft",
                       "thumbs", "sweep", "sweep", "sweep", "approx"])
    if path == "pair":
        long_side, w = _log(rng, 512, 2048), rng.randint(64, 307)
        w, h = (w, long_side) if rng.random() < 0.5 else (long_side, w)
        return {"path": path, "w": w, "h": h, "dtype": rng.choice(["u8", "u8", "u16"])}
    if path == "strips":
        host = rng.random() < 0.4
        return {"path": path, "n": _log(rng, 8, 512 if host else 3000),
                "long": rng.choice([1024, 1700, 2048, 2048]), "host": host}
    if path == "uneven":
        smin = _log(rng, 48, 200)
        return {"path": path, "n": _log(rng, 50, 2500), "smin": smin,
                "smax": rng.randint(2 * smin, 1024)}
    if path == "window":
        side = _log(rng, 48, 700)
        return {"path": path, "n": _log(rng, 1, max(2, min(400, 14000000 // (side * side)))),
                "side": side}
    if path == "images":
        w1, h1 = rng.randint(96, 500), rng.randint(96, 500)
        w2, h2 = rng.randint(96, 500), rng.randint(96, 500)
        return {"path": path, "kind": rng.choice(["R", "S"]), "n": _log(rng, 1, 40), "w1": w1,
                "h1": h1, "w2": w2, "h2": h2, "dtype": rng.choice(["u8", "f32", "f64"]),
                "oval": rng.choice([0, 0, 60])}
    if path == "fft":
        return {"path": path, "nx": 2 ** rng.randint(7, 11), "ny": 2 ** rng.randint(7, 11)}
    if path == "thumbs":
        k = rng.choice([4, 8, 8, 5, 1])   # 1: the normalisation alone, as the last stage has it
        lo, hi = (300, 1000) if k == 1 else (700, 2100)
        return {"path": path, "n": _log(rng, 1, 8), "w": rng.randint(lo, hi),
                "h": rng.randint(lo, hi), "bin": k,
                "dtype": rng.choice(["u8", "u8", "u16", "f32"])}
    if path == "sweep":
        mode = rng.choice(["angle", "scan", "scan", "search"])
        return {"path": path, "mode": mode, "side": rng.randint(100, 260),
                "n": _log(rng, 1, 40) if mode != "search" else rng.randint(12, 20)}
    return {"path": path, "n": rng.randint(1, 3), "tile": rng.choice([512, 720, 1024]),
            "dec": rng.choice([4, 4, 8])}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _gen(seed, *more):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(np.random.SeedSequence([int(seed), *more]).generate_state(1)[0]))
    return g


def _field(g, h, w, mean=128.0, std=30.0):
    """An EM-like field: FP32, mean and std given, ellipses at mean - 3 std."""
    f = torch.fft.rfft2(torch.randn((h, w), generator=g, device=DEV))
    fy = torch.fft.fftfreq(h, device=DEV)[:, None]
    fx = torch.fft.rfftfreq(w, device=DEV)[None, :]
    k = fx * fx + fy * fy
    k[0, 0] = 1.0
    amp = k.pow(-0.375)
    amp[0, 0] = 0.0
    img = torch.fft.irfft2(f * amp, s=(h, w))
    img = (img - img.mean()) / img.std() * std + mean
    n = max(1, int(round(200.0 * h * w / 2048.0 ** 2)))
    u = torch.rand((n, 5), generator=g, device=DEV)
    r = torch.arange(-21, 22, device=DEV)
    for s in range(0, n, 1024):
        cx, cy = u[s:s + 1024, 0, None, None] * w, u[s:s + 1024, 1, None, None] * h
        a, b = 4 + 16 * u[s:s + 1024, 2, None, None], 4 + 16 * u[s:s + 1024, 3, None, None]
        c, sn = (t(u[s:s + 1024, 4, None, None] * math.pi) for t in (torch.cos, torch.sin))
        y, x = cy.floor() + r[:, None], cx.floor() + r[None, :]
        dx, dy = (x - cx).expand(-1, 43, 43), (y - cy).expand(-1, 43, 43)
        x, y = x.expand(-1, 43, 43), y.expand(-1, 43, 43)
        m = ((c * dx + sn * dy) / a) ** 2 + ((c * dy - sn * dx) / b) ** 2 <= 1
        m &= (x >= 0) & (x < w) & (y >= 0) & (y < h)
        img[y[m].long(), x[m].long()] = mean - 3 * std
    return img


def _shot(f, g, noise, top):
    """One exposure of a field, as whole numbers 0..top in an int32 tensor."""
    return (f + noise * torch.randn(f.shape, generator=g, device=DEV)).round().clamp(
        0, top).to(torch.int32)


def _cast(x, dtype):
    if dtype == "u8":
        return x.to(torch.uint8)
    if dtype == "u16":
        return x.to(torch.uint16)
    return x.to(torch.float32 if dtype == "f32" else torch.float64)


def _two_shots(seed, h, w, top=255, mean=128.0, std=30.0, noise=8.0):
    g = _gen(seed, h, w)
    f = _field(g, h, w, mean, std)
    return _shot(f, g, noise, top), _shot(f, g, noise, top)


def _crop(im, y, x, h, w):
    return im[y:y + h, x:x + w].contiguous()


def _overlap(rng, A, B, h, w, jit, decoy):
    """Rasters of the same tissue (or not, a decoy) cut from two exposures,
    the second displaced by up to jit px."""
    H, W = A.shape
    y, x = int(rng.integers(jit, H - h - jit + 1)), int(rng.integers(jit, W - w - jit + 1))
    ty, tx = (int(v) for v in rng.integers(-jit, jit + 1, 2))
    if decoy:
        yb, xb = int(rng.integers(0, H - h + 1)), int(rng.integers(0, W - w + 1))
    else:
        yb, xb = y + ty, x + tx
    return _crop(A, y, x, h, w), _crop(B, yb, xb, h, w)


def _pair_input(case, seed):
    w, h = case["w"], case["h"]
    top, mean, std = (4095, 2048.0, 480.0) if case["dtype"] == "u16" else (255, 128.0, 30.0)
    A, B = _two_shots(seed, h + 2 * JITTER + 8, w + 2 * JITTER + 8, top, mean, std, std / 4)
    rng = np.random.default_rng([seed, 1])
    return [tuple(_cast(t, case["dtype"])
                  for t in _overlap(rng, A, B, h, w, min(JITTER, w // 4, h // 4), False))]


def _strips_input(case, seed):
    """n neighbour overlaps: 8-15 % of the tile wide, half of them left-right."""
    n, long_side = case["n"], case["long"]
    side = 8192 if n > 256 else long_side + 2 * JITTER + 512
    A, B = (t.to(torch.uint8) for t in _two_shots(seed, side, side))
    rng = np.random.default_rng([seed, 2])
    out = []
    for _ in range(n):
        w = int(rng.integers(long_side * 8 // 100 + 1, long_side * 15 // 100 + 1))
        h, w = (long_side, w) if rng.random() < 0.5 else (w, long_side)
        out.append(_overlap(rng, A, B, h, w, JITTER, rng.random() < DECOYS))
    if case["host"]:   # one page-locked block, rows back to back, as a reader fills it
        block = torch.empty(sum(a.numel() + b.numel() for a, b in out), dtype=torch.uint8,
                            pin_memory=True)
        at, host = 0, []
        for pair in out:
            views = []
            for t in pair:
                v = block[at:at + t.numel()].view(t.shape)
                v.copy_(t, non_blocking=True)
                views.append(v)
                at += t.numel()
            host.append(tuple(views))
        torch.cuda.synchronize()
        out = host
    return out


def _uneven_input(case, seed):
    A, B = _two_shots(seed, 4096, 4096, 4095, 2048.0, 480.0, 30.0)
    A, B = A.to(torch.int16), B.to(torch.int16)   # values 0..4095: the same bits as uint16
    rng = np.random.default_rng([seed, 3])
    out = []
    for _ in range(case["n"]):
        s = int(round(math.exp(rng.uniform(math.log(case["smin"]), math.log(case["smax"])))))
        short = max(8, int(round(s / rng.uniform(1.0, 4.0))))
        w, h = (s, short) if rng.random() < 0.5 else (short, s)
        a, b = _overlap(rng, A, B, h, w, max(1, short // 4), False)
        out.append((a.view(torch.uint16), b.view(torch.uint16)))
    return out


def _window_input(case, seed):
    n, s = case["n"], case["side"]
    jit = max(2, s // 8)
    side = max(1024, s + 2 * jit + 64)
    A, B = (t.to(torch.uint8) for t in _two_shots(seed, side, side))
    rng = np.random.default_rng([seed, 4])
    return [_overlap(rng, A, B, s, s, jit, False) for _ in range(n)]


def _images_input(case, seed):
    H, W = max(case["h1"], case["h2"]) + 100, max(case["w1"], case["w2"]) + 100
    rng = np.random.default_rng([seed, 5])
    out = []
    big = [_two_shots(seed + 7919 * k, H + 200, W + 200) for k in range(2)]
    for k in range(case["n"]):
        A, B = big[k % 2]
        y, x = int(rng.integers(20, 200)), int(rng.integers(20, 200))
        ty, tx = (int(v) for v in rng.integers(-20, 21, 2))
        a = _crop(A, y, x, case["h1"], case["w1"])
        b = _crop(B, y + ty, x + tx, case["h2"], case["w2"])
        if case["dtype"] in ("f32", "f64"):   # normalised, as the callers pass them
            a, b = ((t.double() - t.double().mean()) / t.double().std() for t in (a, b))
        out.append((_cast(a, case["dtype"]), _cast(b, case["dtype"])))
    return out


def _fft_input(case, seed):
    return _field(_gen(seed, 6), case["ny"], case["nx"], 0.0, 1.0).double().cpu().numpy()


def _thumbs_input(case, seed):
    out = []
    top, mean, std = (4095, 2048.0, 480.0) if case["dtype"] == "u16" else (255, 128.0, 30.0)
    g = _gen(seed, 7)
    big = _field(g, case["h"] + 64, case["w"] + 64, mean, std)
    for k in range(case["n"]):
        f = big[7 * k:7 * k + case["h"], 5 * k:5 * k + case["w"]]
        x = _cast(_shot(f, g, std / 4, top), case["dtype"])
        out.append(x.cpu().numpy())
    return out


def _bilinear(f, x, y):
    x0 = x.floor().long().clamp(0, f.shape[1] - 2)
    y0 = y.floor().long().clamp(0, f.shape[0] - 2)
    ax, ay = x - x0, y - y0
    return ((1 - ax) * (1 - ay) * f[y0, x0] + ax * (1 - ay) * f[y0, x0 + 1]
            + (1 - ax) * ay * f[y0 + 1, x0] + ax * ay * f[y0 + 1, x0 + 1])


def _turned(f, side, at, deg, shift):
    """side x side samples of f around (at + side / 2), turned by deg and shifted."""
    k = torch.arange(side, device=DEV, dtype=torch.float32) - side / 2.0
    yy, xx = torch.meshgrid(k, k, indexing="ij")
    c, s = math.cos(math.radians(deg)), math.sin(math.radians(deg))
    return _bilinear(f, c * xx - s * yy + side / 2.0 + shift[0] + at[1],
                     s * xx + c * yy + side / 2.0 + shift[1] + at[0])


def _sweep_input(case, seed):
    """Thumbnail pairs across two layers: turned by up to 10 degrees, shifted,
    another gain, normalised as MakeThumbs leaves them (FP64, host)."""
    n, s = case["n"], case["side"]
    pad = s // 4 + 16
    rng = np.random.default_rng([seed, 8])
    g = _gen(seed, 8, s)
    out, f = [], None
    for k in range(n):
        if k % 4 == 0:
            # an 8-fold box average keeps the field's low frequencies
            f = _field(g, 2 * s + 2 * pad, 2 * s + 2 * pad, 0.0, 1.0)
        at = [pad + int(v) for v in rng.integers(0, s, 2)]
        deg, shift = float(rng.uniform(-9.5, 9.5)), rng.uniform(-4, 4, 2)
        a = f[at[0]:at[0] + s, at[1]:at[1] + s]
        b = float(rng.uniform(0.9, 1.1)) * _turned(f, s, at, deg, shift)
        pair = []
        for t in (a, b):
            t = (t + 0.05 * torch.randn((s, s), generator=g, device=DEV)).double()
            pair.append(((t - t.mean()) / t.std()).cpu().numpy())
        out.append(tuple(pair))
    return out


def _approx_input(case, seed):
    t = case["tile"]
    rng = np.random.default_rng([seed, 9])
    g = _gen(seed, 9, t)
    pad = t // 2
    out = []
    for _ in range(case["n"]):
        f = _field(g, t + 2 * pad, t + 2 * pad)
        deg = float(rng.uniform(-4, 4))
        s = np.array([t * 0.18, t * 0.06]) * rng.choice([-1.0, 1.0], 2)
        a = f[pad:pad + t, pad:pad + t]
        b = float(rng.uniform(0.9, 1.1)) * _turned(f, t, (pad, pad), deg, s)
        a, b = (_shot(v, g, 6.0, 255).to(torch.uint8).cpu().numpy() for v in (a, b))
        tab = -s + rng.uniform(-6, 6, 2)
        out.append((a, b, (float(tab[0]), float(tab[1]))))
    return out


INPUT = {"pair": _pair_input, "strips": _strips_input, "uneven": _uneven_input,
         "window": _window_input, "images": _images_input, "fft": _fft_input,
         "thumbs": _thumbs_input, "sweep": _sweep_input, "approx": _approx_input}

# the legality rules the callers of each path pass (kind, a, b, area[, count])


def _rule(case, a):
    h, w = a.shape
    if case["path"] in ("pair", "strips"):
        # InSectionOverlap: a long side of at least three quarters of the tile
        return aln.RGN_SECTION, int(0.73 * max(h, w)), int(0.73 * max(h, w)), 15000
    if case["path"] == "uneven":
        return aln.RGN_MIN, 8, 8, 0
    return aln.RGN_MIN, min(32, w // 4), min(32, h // 4), 0


def _radius(case, a):
    if case["path"] in ("pair", "strips"):
        return STRIP_RADIUS
    return max(1, min(a.shape) // 2) if case["path"] == "uneven" else 4096


def _req_area(side):
    return side * side // 20


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------

_CTX = None


def _ctx():
    """A program keeps one context: a stream and its workspaces."""
    global _CTX
    if _CTX is None:
        _CTX = aln.Context(0)
    return _CTX


_DT = {torch.uint8: aln.U8, torch.uint16: aln.U16, torch.float32: aln.F32,
       torch.float64: aln.F64}


def _image(t):
    return AlnImage(t.data_ptr(), _DT[t.dtype], t.shape[1], t.shape[0], t.stride(0), 0, 0,
                    1 if t.is_cuda else 0)


def prepare(case, seed):
    path = case["path"]
    st = {"case": case, "path": path, "ctx": _ctx(), "in": INPUT[path](case, seed)}
    if path == "pair":
        a = st["in"][0][0]
        st["legal"] = aln.legal(*_rule(case, a))
    elif path in ("strips", "uneven", "window"):
        arr = (AlnPair * len(st["in"]))()
        rules = {}
        for k, (a, b) in enumerate(st["in"]):
            rule = _rule(case, a)
            if rule not in rules:
                rules[rule] = aln.legal(*rule)
            p = arr[k]
            p.a, p.b, p.radius, p.legal = _image(a), _image(b), _radius(case, a), rules[rule]
        st["jobs"], st["out"] = arr, (AlnResult * len(arr))()
    elif path == "images":
        arr = (AlnImageJob * len(st["in"]))()
        for k, (a, b) in enumerate(st["in"]):
            j = arr[k]
            j.a, j.b = _image(a), _image(b)
            j.kind = aln.CORR_R if case["kind"] == "R" else aln.CORR_S
            area = min(a.numel(), b.numel()) // 20
            j.legal = aln.legal(*_rule(case, a)[:3], area, aln.CNT_GT, area // 2)
            j.nbmaxht = 0.75
            j.rx = j.ry = case["oval"] if case["oval"] else -1
        st["jobs"], st["out"] = arr, (AlnResult * len(arr))()
    elif path == "sweep":
        arr = (AlnThumbs * case["n"])()
        for k, (a, b) in enumerate(st["in"]):
            t = arr[k]
            t.a, t.a_mask = a.ctypes.data, None
            t.a_h, t.a_w = a.shape
            t.a_stride = t.a_w
            t.b = AlnImage(b.ctypes.data, aln.F64, b.shape[1], b.shape[0], b.shape[1], 0, 0, 0)
            t.req_area, t.olap1d = _req_area(case["side"]), 0
        P = AlnThmParams()
        P.rthresh, P.nbmaxht, P.constxy, P.pretweak, P.usecorrr = 0.3, 0.75, 1, 0, 1
        P.rx = P.ry = -1
        P.tdfm[0] = P.tdfm[4] = 1.0
        st["jobs"], st["params"], st["out"] = arr, P, (AlnThmResult * len(arr))()
        st["mode"] = {"angle": (aln.THM_RFROMANGLE, 1.5), "scan": (aln.THM_SCAN_MAXR, 0.0),
                      "search": (aln.THM_DENOVO, 0.0)}[case["mode"]]
    return st


def _table(recs, dtype, floats, ints):
    """The result records of one call as a match table keeps them."""
    v = np.frombuffer(recs, dtype)
    out = {k: v[k].astype(np.float32) for k in floats}
    out.update({k: v[k].copy() for k in ints})
    return out


def run(st):
    path, ctx = st["path"], st["ctx"]
    L = aln.lib()
    if path == "pair":
        a, b = st["in"][0]
        o = ctx.corr_patches(a, b, 0, 0, STRIP_RADIUS, st["legal"])
        return {"px": o["peak_x"], "py": o["peak_y"], "status": o["status"],
                "r": np.float32(o["r"]), "dx": np.float32(o["dx"]), "dy": np.float32(o["dy"])}
    if path in ("strips", "uneven", "window", "images"):
        call = L.aln_corr_images_batch if path == "images" else L.aln_corr_patches_batch
        ctx._check(call(ctx.h, len(st["jobs"]), st["jobs"], st["out"]))
        return _table(st["out"], RESULT, ("r", "dx", "dy"), ("status", "px", "py"))
    if path == "fft":
        x = st["in"]
        F = ctx.fft_2d(x)
        return {"spectrum": F, "back": ctx.ift_2d(F, x.shape[1])}
    if path == "thumbs":
        return [{"v": v, "m": m, "sd": sd} for v, m, sd in ctx.decimate(st["in"], st["case"]["bin"])]
    if path == "sweep":
        mode, ang0 = st["mode"]
        ctx._check(L.aln_thm_search_batch(ctx.h, len(st["jobs"]), st["jobs"],
                                          C.byref(st["params"]), mode, ang0, 10.0, 0.5,
                                          st["out"]))
        return _table(st["out"], THM, ("A", "X", "Y", "R", "T"), ("err", "ncalls"))
    res = ctx.approx_match_batch(st["in"], thmdec=st["case"]["dec"], olap2d=40000)
    out = {k: np.array([r[k] for r in res], np.float32) for k in ("A", "X", "Y", "R", "T")}
    out.update({k: np.array([r[k] for r in res], np.int32) for k in ("status", "err", "crop")})
    return out


# ---------------------------------------------------------------------------
# the work no implementation can do without
# ---------------------------------------------------------------------------

_SIZE = {"u8": 1, "u16": 2, "f32": 4, "f64": 8}


def _fast_len(n):
    """The least length >= n of the form 2^a 3^b 5^c."""
    best = 1 << (n - 1).bit_length()
    p5 = 1
    while p5 < best:
        p3 = p5
        while p3 < best:
            k = p3
            while k < n:
                k *= 2
            best = min(best, k)
            p3 *= 3
        p5 *= 5
    return best


def _corr_flops(w1, h1, w2, h2, lags_x, lags_y):
    """Two real transforms and one inverse on the smallest alias-free grid for
    the lags that are asked for, the product, and r per lag."""
    nx = _fast_len(max(w1, w2, min(w1 + w2 - 1, max(w1, w2) + lags_x // 2)))
    ny = _fast_len(max(h1, h2, min(h1 + h2 - 1, max(h1, h2) + lags_y // 2)))
    n = nx * ny
    return 3 * 2.5 * n * math.log2(n) + 3 * n + 30 * lags_x * lags_y


def _sizes(case):
    """(w1, h1, w2, h2, radius or None, pairs of that size): exact or the mean."""
    path = case["path"]
    if path == "pair":
        return [(case["w"], case["h"], case["w"], case["h"], STRIP_RADIUS, 1)]
    if path == "strips":
        w = case["long"] * 0.115
        return [(w, case["long"], w, case["long"], STRIP_RADIUS, case["n"])]
    if path == "uneven":
        lo, hi, m = math.log(case["smin"]), math.log(case["smax"]), 16
        out = []
        for k in range(m):
            s = math.exp(lo + (hi - lo) * (k + 0.5) / m)
            short = s * math.log(4.0) / 3.0
            out.append((short, s, short, s, short / 2, case["n"] / m))
        return out
    if path == "window":
        s = case["side"]
        return [(s, s, s, s, None, case["n"])]
    return [(case["w1"], case["h1"], case["w2"], case["h2"], None, case["n"])]


def work(case):
    path = case["path"]
    if path in ("pair", "strips", "uneven", "window", "images"):
        e = _SIZE[case.get("dtype", "u16" if path == "uneven" else "u8")]
        nbytes = flops = 0.0
        for w1, h1, w2, h2, rad, n in _sizes(case):
            w1, h1, w2, h2 = (int(v) for v in (w1, h1, w2, h2))
            lx = w1 + w2 - 1 if rad is None else min(w1 + w2 - 1, int(2 * rad) + 1)
            ly = h1 + h2 - 1 if rad is None else min(h1 + h2 - 1, int(2 * rad) + 1)
            nbytes += n * ((w1 * h1 + w2 * h2) * e + 24)
            flops += n * _corr_flops(w1, h1, w2, h2, lx, ly)
        return {"bytes": nbytes, "flops": flops}
    if path == "fft":
        n = case["nx"] * case["ny"]
        return {"bytes": 32.0 * n, "flops": 2 * 2.5 * n * math.log2(n)}
    if path == "thumbs":
        n = case["n"] * case["w"] * case["h"]
        return {"bytes": n * _SIZE[case["dtype"]] + 9.0 * n / case["bin"] ** 2, "flops": 2.0 * n}
    if path == "sweep":
        s, calls = case["side"], {"angle": 1, "scan": 55, "search": 139}[case["mode"]]
        r = int(s * 1.15)
        n = 1 << (s + r - 2).bit_length()
        # b's transform once, per call the turned a, its transform and one inverse
        one = 2 * 2.5 * n * n * math.log2(n * n) + 12 * n * n + 20 * r * r
        return {"bytes": case["n"] * 16.0 * s * s,
                "flops": case["n"] * (calls * one + 2.5 * n * n * math.log2(n * n))}
    t, d = case["tile"], case["dec"]
    s = int(t * 0.9 / d)
    thumbs = work({"path": "sweep", "mode": "search", "n": case["n"], "side": s})
    full = work({"path": "sweep", "mode": "angle", "n": case["n"], "side": int(t * 0.9)})
    return {"bytes": 2.0 * case["n"] * t * t, "flops": thumbs["flops"] + full["flops"]}


# ---------------------------------------------------------------------------
# the same numbers in 64 bits, plain torch and numpy
# ---------------------------------------------------------------------------

def _sat(v):
    """Summed-area table with a zero row and column in front."""
    return torch.nn.functional.pad(v.cumsum(0).cumsum(1), (1, 0, 1, 0))


def _box(t, y0, y1, x0, x1):
    """Sums over rows [y0, y1) and columns [x0, x1) for all combinations."""
    return t[y1][:, x1] - t[y0][:, x1] - t[y1][:, x0] + t[y0][:, x0]


class _Lags:
    """Correlation of two rasters over a window of lags, FP64."""

    def __init__(self, a, b, xlo, xhi, ylo, yhi):
        self.a, self.b = a, b
        self.h1, self.w1 = a.shape
        self.h2, self.w2 = b.shape
        self.x = torch.arange(xlo, xhi + 1, device=DEV)
        self.y = torch.arange(ylo, yhi + 1, device=DEV)
        # the overlap of the two boxes at each lag, in b's and in a's frame
        self.bx0, self.bx1 = self.x.clamp(min=0), (self.x + self.w1).clamp(max=self.w2)
        self.by0, self.by1 = self.y.clamp(min=0), (self.y + self.h1).clamp(max=self.h2)
        self.ax0, self.ax1 = self.bx0 - self.x, self.bx1 - self.x
        self.ay0, self.ay1 = self.by0 - self.y, self.by1 - self.y
        self.olw, self.olh = (self.bx1 - self.bx0)[None, :], (self.by1 - self.by0)[:, None]

    def of_a(self, v):
        return _box(_sat(v), self.ay0, self.ay1, self.ax0, self.ax1)

    def of_b(self, v):
        return _box(_sat(v), self.by0, self.by1, self.bx0, self.bx1)

    def sums(self):
        """sum over the overlap of a(p) b(p + lag), on an alias-free grid."""
        nx = _fast_len(max(self.w1, self.w2, self.w2 - int(self.x[0]), int(self.x[-1]) + self.w1))
        ny = _fast_len(max(self.h1, self.h2, self.h2 - int(self.y[0]), int(self.y[-1]) + self.h1))
        nx += nx & 1
        F = torch.fft.rfft2(self.b, s=(ny, nx)) * torch.fft.rfft2(self.a, s=(ny, nx)).conj()
        return torch.fft.irfft2(F, s=(ny, nx))[self.y % ny][:, self.x % nx]

    def r(self):
        ma, mb = self.a.mean().round(), self.b.mean().round()
        n = (self.olw * self.olh).double()
        save = self.a, self.b
        self.a, self.b = save[0] - ma, save[1] - mb
        c = self.sums()
        s1, s2 = self.of_a(self.a), self.of_b(self.b)
        d1 = n * self.of_a(self.a * self.a) - s1 * s1
        d2 = n * self.of_b(self.b * self.b) - s2 * s2
        self.a, self.b = save
        d = d1 * d2
        return torch.where(d < n * n * 1e-9, 0.0, (n * c - s1 * s2) / d.clamp_min(1e-300).sqrt())

    def legal(self, rule, cnt=None):
        kind, p, q, area = rule
        big = self.olw * self.olh > area
        ok = (big & (self.olw >= p) & (self.olh >= q)) if kind == aln.RGN_MIN else \
            (big & ((self.olw >= p) | (self.olh > q)))
        if cnt is not None:
            ok &= (self.of_a((self.a != 0).double()) > cnt) & (self.of_b((self.b != 0).double()) > cnt)
        return ok


def _parab(lo, mid, hi):
    t = (lo - hi) / (2 * (lo + hi - 2 * mid))
    return t if abs(t) <= 8 else 0.0


def _patches(a, b, radius, rule):
    """CorrPatches: the disc around lag 0, r's maximum, refined for positive lags."""
    a, b = a.to(DEV).double(), b.to(DEV).double()
    (h1, w1), (h2, w2) = a.shape, b.shape
    g = _Lags(a, b, max(1 - w1, -radius), min(w2 - 1, radius), max(1 - h1, -radius),
              min(h2 - 1, radius))
    disc = g.x[None, :] ** 2 + g.y[:, None] ** 2 <= radius * radius
    r = torch.where(g.legal(rule) & disc, g.r(), 0.0)
    key = torch.where(g.legal(rule) & disc, r, -1e30)
    k = int(key.argmax())
    j, i = divmod(k, r.shape[1])
    x, y = int(g.x[i]), int(g.y[j])
    near = torch.nn.functional.pad(r, (1, 1, 1, 1))[j:j + 3, i:i + 3].tolist()
    mid = near[1][1]
    fx, fy = float(x), float(y)
    if x >= 1 and near[1][0] and near[1][2]:
        fx += _parab(near[1][0], mid, near[1][2])
    if y >= 1 and near[0][1] and near[2][1]:
        fy += _parab(near[0][1], mid, near[2][1])
    return mid, fx, fy


def _key_peak(g, key, ok):
    """The best legal lag of a whole lag image, refined where neighbours are positive."""
    k = int(torch.where(ok, key, -1e30).argmax())
    j, i = divmod(k, key.shape[1])
    near = torch.nn.functional.pad(key, (1, 1, 1, 1))[j:j + 3, i:i + 3].tolist()
    mid, fx, fy = near[1][1], float(g.x[i]), float(g.y[j])
    if 0 < i < key.shape[1] - 1 and near[1][0] > 0 and near[1][2] > 0:
        fx += _parab(near[1][0], mid, near[1][2])
    if 0 < j < key.shape[0] - 1 and near[0][1] > 0 and near[2][1] > 0:
        fy += _parab(near[0][1], mid, near[2][1])
    return mid, fx, fy


def _whitened(a, b, spec_b=None):
    """S: the inverse of P / sqrt|P| on the power-of-two frame, over every lag."""
    (h1, w1), (h2, w2) = a.shape, b.shape
    nx, ny = (1 << (m + n - 2).bit_length() for m, n in ((w1, w2), (h1, h2)))
    P = (torch.fft.rfft2(b, s=(ny, nx)) if spec_b is None else spec_b(ny, nx)) * \
        torch.fft.rfft2(a, s=(ny, nx)).conj()
    m = P.abs()
    P = torch.where(m > 1e-10, P / m.clamp_min(1e-300).sqrt(), P)
    S = torch.fft.irfft2(P, s=(ny, nx))
    y = torch.arange(1 - h1, h2, device=DEV) % ny
    x = torch.arange(1 - w1, w2, device=DEV) % nx
    return S[y][:, x]


def _images(a, b, kind, rule, cnt, oval=0, spec_b=None):
    (h1, w1), (h2, w2) = a.shape, b.shape
    g = _Lags(a, b, 1 - w1, w2 - 1, 1 - h1, h2 - 1)
    ok = g.legal(rule, cnt)
    if oval:
        ok = ok & (g.x[None, :] ** 2 + g.y[:, None] ** 2 <= oval * oval)
    if kind == "R":
        key = g.r()
        key = torch.where((key > -1) & (key < 1), key, 0.0)
        return _key_peak(g, key, ok)
    key = _whitened(a, b, spec_b)
    top, fx, fy = _key_peak(g, key, ok)
    return float(10 * (top - key.mean()) / (key.std() * math.sqrt(key.numel()))), fx, fy


def _splat(a, deg):
    """a's grid points turned about the origin, spread bilinearly over their box."""
    s = a.shape[0]
    t = deg * 3.14159265358 / 180.0   # the reference's value of pi
    k = torch.arange(s, device=DEV, dtype=torch.float64)
    yy, xx = torch.meshgrid(k, k, indexing="ij")
    x = xx * math.cos(t) - yy * math.sin(t)
    y = xx * math.sin(t) + yy * math.cos(t)
    x0, y0 = math.floor(float(x.min())), math.floor(float(y.min()))
    w, h = math.ceil(float(x.max())) - x0 + 1, math.ceil(float(y.max())) - y0 + 1
    x, y = (x - x0).reshape(-1), (y - y0).reshape(-1)
    i, j = x.floor().long(), y.floor().long()
    fx, fy = x - i, y - j
    out = torch.zeros(h * w, device=DEV, dtype=torch.float64)
    v = a.reshape(-1)
    for di, wx in ((0, 1 - fx), (1, fx)):
        for dj, wy in ((0, 1 - fy), (1, fy)):
            at = (j + dj).clamp(max=h - 1) * w + (i + di).clamp(max=w - 1)
            out.index_put_((at,), v * wx * wy, accumulate=True)
    return out.view(h, w), x0, y0


def _at_angles(a, b, angles):
    """(A, X, Y, R) of the sweep's correlator at the first best of these angles."""
    a, b = (torch.from_numpy(t).to(DEV) for t in (a, b))
    area = _req_area(a.shape[0])
    keep = {}

    def spec(ny, nx):
        if (ny, nx) not in keep:
            keep[ny, nx] = torch.fft.rfft2(b, s=(ny, nx))
        return keep[ny, nx]

    best = None
    for deg in angles:
        turned, x0, y0 = _splat(a, deg)
        r, fx, fy = _images(turned, b, "S", (aln.RGN_MIN, 0, 0, area), area, 0, spec)
        if best is None or r > best[3]:
            best = (deg, fx - x0, fy - y0, r)
    return best


def _scan_angles(center, half, step):
    """A coarse scan's angles: the centre, a finer fan around it, then the range."""
    out, wide, fine = [center], 2.0 * step, step / 3.0
    a = center - wide
    while a <= center + wide:
        out.append(a)
        a += fine
    a = center - half
    while a <= center + half:
        out.append(a)
        a += step
    return out


def exact(case, seed):
    path = case["path"]
    if path == "approx" or path == "sweep" and case["mode"] == "search":
        # the search halves brackets on differences in R's last digits: its
        # angle has no value of its own in 64 bits
        return None
    data = INPUT[path](case, seed)
    none = {"status": None, "px": None, "py": None}
    if path == "pair":
        a, b = data[0]
        r, x, y = _patches(a, b, _radius(case, a), _rule(case, a))
        return {**none, **{k: np.float64(v) for k, v in (("r", r), ("dx", x), ("dy", y))}}
    if path in ("strips", "uneven", "window"):
        got = np.array([_patches(a, b, _radius(case, a), _rule(case, a)) for a, b in data])
        return {**none, "r": got[:, 0], "dx": got[:, 1], "dy": got[:, 2]}
    if path == "images":
        got = []
        for a, b in data:
            area = min(a.numel(), b.numel()) // 20
            got.append(_images(a.double(), b.double(), case["kind"],
                               (*_rule(case, a)[:3], area), area // 2, case["oval"]))
        got = np.array(got)
        return {**none, "r": got[:, 0], "dx": got[:, 1], "dy": got[:, 2]}
    if path == "fft":
        F = np.fft.rfft2(data)
        return {"spectrum": F, "back": np.fft.irfft2(F, s=data.shape) * data.size}
    if path == "thumbs":
        out = []
        for x in data:
            h, w = x.shape
            k = case["bin"]
            ys, xs = np.arange(0, h, k), np.arange(0, w, k)
            s = np.add.reduceat(np.add.reduceat(x.astype(np.float64), ys, 0), xs, 1)
            v = s / np.outer(np.diff(np.append(ys, h)), np.diff(np.append(xs, w)))
            sd = v.std(ddof=1)
            out.append({"v": (v - v.mean()) / sd, "m": None, "sd": float(sd)})
        return out
    angles = [1.5] if case["mode"] == "angle" else _scan_angles(0.0, 10.0, 0.5)
    got = np.array([_at_angles(a, b, angles) for a, b in data])
    return {"A": got[:, 0], "X": got[:, 1], "Y": got[:, 2], "R": got[:, 3], "T": None,
            "err": None, "ncalls": None}
