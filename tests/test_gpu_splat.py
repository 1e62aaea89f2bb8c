"""The rotate-and-splat of the sweep (k_splat) under transforms far from a
rotation, against the oracle: points spread over more pixels than a step of
three, offsets that leave the short fixed-point form, masks, odd grids; and a
batch whose jobs share one thumbnail b against the jobs alone."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = {
    "turn": (1, 0, 0, 1), "half turn": (-1, 0, 0, -1), "shrink": (0.21, 0, 0, 0.33),
    "grow": (7.5, 0, 0, 5.25), "huge": (130.0, 0, 0, 118.0), "shear": (1, 1.7, 0, 1),
    "nearly flat": (1, 0.985, 0.985, 1), "mirror": (1, 0.2, 0.3, -1)}


@pytest.fixture(scope="module")
def ctx():
    import alignment_projects_gb300 as aln
    c = aln.Context(0)
    yield c
    c.close()


def _points(rng, w, h, masked):
    yy, xx = np.mgrid[0:h, 0:w]
    keep = rng.random((h, w)) < 0.8 if masked else np.ones((h, w), bool)
    return np.stack([xx[keep], yy[keep]], 1).astype(np.float64), rng.standard_normal(keep.sum())


def _spread(pts, v, t, deg):
    """The points moved by R(deg) t, spread bilinearly: what b is made of."""
    c, s = math.cos(math.radians(deg)), math.sin(math.radians(deg))
    m = np.array([[c, -s], [s, c]]) @ np.array(t, np.float64).reshape(2, 2)
    q = pts @ m.T
    q -= np.floor(q.min(0))
    i = np.floor(q).astype(int)
    f = q - i
    out = np.zeros(i.max(0)[::-1] + 2)
    for dx in (0, 1):
        for dy in (0, 1):
            wgt = (f[:, 0] if dx else 1 - f[:, 0]) * (f[:, 1] if dy else 1 - f[:, 1])
            np.add.at(out, (i[:, 1] + dy, i[:, 0] + dx), v * wgt)
    return out


@pytest.mark.parametrize("shape", sorted(SHAPES))
@pytest.mark.parametrize("masked", [False, True])
def test_splat_under_any_transform(ctx, orc, shape, masked):
    import alignment_projects_gb300 as aln
    rng = np.random.default_rng(len(shape) + masked)
    t = SHAPES[shape]
    w, h = (9, 11) if shape == "huge" else (41, 38)
    pts, v = _points(rng, w, h, masked)
    deg = 3.7
    b = _spread(pts, v, t, deg)
    b = b + 0.01 * rng.standard_normal(b.shape)
    yy, xx = np.mgrid[0:b.shape[0], 0:b.shape[1]]
    pb, vb = np.stack([xx.ravel(), yy.ravel()], 1).astype(np.float64), b.ravel()
    td = (t[0], t[1], 0, t[2], t[3], 0)
    g = ctx.thm_search_batch([aln.thumbs_from_points(pts, v, pb, vb, 20)],
                             mode=aln.THM_RFROMANGLE, ang0=deg, tdfm=td)[0]
    o = orc.thm_search(pts, v, pb, vb, 20, mode=1, ang0=deg, tdfm=td)
    assert abs(g["R"] - o["R"]) <= 1e-4 * abs(o["R"])
    assert abs(g["X"] - o["X"]) <= 0.01 and abs(g["Y"] - o["Y"]) <= 0.01


def test_shared_b_equals_alone(ctx):
    """A scan's jobs read one count table of b; each angle alone makes its own."""
    import alignment_projects_gb300 as aln
    rng = np.random.default_rng(5)
    thumbs = []
    for n in (40, 57):
        pts, v = _points(rng, n, n - 3, True)
        pb, vb = _points(rng, n + 5, n, True)
        thumbs.append(aln.thumbs_from_points(pts, v, pb, vb, 400))
    scan = ctx.thm_search_batch(thumbs, mode=aln.THM_SCAN_MAXR, ang0=0.0, hfang=3.0, step=0.5)
    for k, s in enumerate(scan):
        alone = ctx.thm_search_batch([thumbs[k]], mode=aln.THM_RFROMANGLE, ang0=s["A"])[0]
        assert (alone["R"], alone["X"], alone["Y"]) == (s["R"], s["X"], s["Y"])
