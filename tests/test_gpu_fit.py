"""The quad fit's size classes (csrc/at_kernels.cu) against the oracle on
square outlines whose clusters lie at the classes' edges (up to 1024, 6144,
13312 points, and above, where the sort works in global memory). Corners are
compared as bits: the fit's sums are the reference's, in its order."""
import numpy as np
import pytest

import apriltags_fast_b200 as AT
from oracle import oracle as O
from tests import helpers as H

pytestmark = pytest.mark.gpu


def _squares(w, h, sides, tilt, seed):
    """Filled dark squares, the k-th at its own place, edges at `tilt` rows
    per column, on a light noisy ground."""
    rng = np.random.default_rng(seed)
    img = np.full((h, w), 200.0)
    yy, xx = np.mgrid[0:h, 0:w]
    x0 = 8
    for s in sides:
        u, v = xx - x0 + tilt * (yy - 8), yy - 8 - tilt * (xx - x0)
        img[(u >= tilt * s) & (u < s + tilt * s) & (v >= 0) & (v < s)] = 40
        x0 += int(s * (1 + 2 * tilt)) + 12
    return np.clip(img + rng.normal(0, 2, img.shape), 0, 255).astype(np.uint8)


CASES = {
    "small": (1000, 300, (120, 127, 128, 129, 136), 0.0),
    "large": (1700, 900, (767, 768), 0.0),
    "large-tilted": (1750, 800, (700, 640), 0.03),
    "huge": (2500, 1720, (769, 1664), 0.0),
    "huge-tilted": (2000, 1800, (1500,), 0.05),
    "global": (3900, 2900, (1665, 2100), 0.0),
    "global-tilted": (3000, 2700, (2400,), 0.04),
}


@pytest.mark.parametrize("name", CASES)
def test_quads_of_large_clusters(name):
    img = _squares(*CASES[name], seed=3)
    det = AT.Detector(["tag36h11"], 2, quad_decimate=1.0)
    got = [d.key() for d in det.detect(img)]
    r = O.detect(img, [H.oracle_family("tag36h11")], [2], O.default_params(quad_decimate=1.0), order=O.ORDER_CANON)
    sizes = np.diff(r.cstart)
    quads = det.diag("quads")
    assert len(quads) == len(r.quads) > 0
    ref = np.array([q[0] for q in r.quads], np.float32)
    assert np.array_equal(quads["p"].view(np.uint32), ref.view(np.uint32))
    assert got == r.dets
    lo, hi = {"small": (900, 1100), "large": (5000, 6144), "huge": (6145, 13312), "global": (13313, 65535)}[
        name.split("-")[0]]
    fitted = sizes[[q[2] for q in r.quads]]
    assert ((fitted >= lo) & (fitted <= hi)).any()


def _same(img, **params):
    det = AT.Detector(["tag36h11"], 2, quad_decimate=1.0, **params)
    got = [d.key() for d in det.detect(img)]
    r = O.detect(img, [H.oracle_family("tag36h11")], [2], O.default_params(quad_decimate=1.0, **params),
                 order=O.ORDER_CANON)
    quads = det.diag("quads")
    assert len(quads) == len(r.quads)
    ref = np.array([q[0] for q in r.quads], np.float32).reshape(-1, 4, 2)
    assert np.array_equal(quads["p"].view(np.uint32), ref.view(np.uint32))
    assert got == r.dets
    return r


@pytest.mark.parametrize("rows", [33, 36])
def test_few_and_many_mid_clusters(rows):
    """Clusters of 257-512 points: a block each up to 1184, a warp each above."""
    img = np.full((rows * 50 + 16, rows * 50 + 16), 200)
    for y in range(rows):
        for x in range(rows):
            s = 33 + (7 * x + 3 * y) % 10
            img[8 + 50 * y : 8 + 50 * y + s, 8 + 50 * x : 8 + 50 * x + s] = 40
    r = _same(img.astype(np.uint8))
    sizes = np.diff(r.cstart)
    mid = ((sizes > 256) & (sizes <= 512)).sum()
    assert len(r.quads) > 900 and (mid <= 1184 if rows == 33 else mid > 1184)


def _share(pts, buckets):
    """Points in a point's bucket on average, by the points' own slopes."""
    x, y = (pts & 0xFFFF).astype(np.float32), (pts >> 16 & 0xFFFF).astype(np.float32)
    dx = x - np.float32((float(x.min()) + float(x.max())) * 0.5 + 0.05118)
    dy = y - np.float32((float(y.min()) + float(y.max())) * 0.5 - 0.028581)
    turn = (np.arctan2(dy, dx) / (np.pi / 2)) % 4
    t = np.tan((turn % 1) * (np.pi / 2))
    n = np.bincount((np.floor(turn) + 1 - 1 / (1 + t)).__mul__(buckets // 4).astype(int))
    return (n.astype(float) ** 2).sum() / len(pts)


@pytest.mark.parametrize("h,w,buckets", [(1, 62, 256), (2, 124, 256), (3, 250, 1024), (4, 250, 1024), (8, 1500, 2048),
                                         (20, 1500, 2048), (24, 3200, 4096), (30, 3900, 4096)])
def test_uneven_angles(h, w, buckets):
    """Bars so long that most points share a few angles: the sort falls back
    from buckets to the one it replaced, in every class."""
    img = np.full((h + 60, w + 80), 200.0)
    img[30 : 30 + h, 40 : 40 + w] = 20
    img += np.random.default_rng(1).normal(0, 0.4, img.shape)
    r = _same(np.clip(img, 0, 255).astype(np.uint8))
    assert max(_share(r.pts[a:b], buckets) for a, b in zip(r.cstart[:-1], r.cstart[1:])) > 17


@pytest.mark.parametrize("side,pitch,lo,hi", [(100, 112, 513, 1024), (146, 160, 1025, 6144)])
def test_clusters_with_and_without_a_quad_in_turn(side, pitch, lo, hi):
    """More clusters of a block class than it has blocks, squares beside discs
    and bars: each cluster is judged by its own best four corners."""
    nx, ny = 4100 // pitch, 3000 // pitch
    img = np.full((ny * pitch + 16, nx * pitch + 16), 200.0)
    yy, xx = np.mgrid[0:side, 0:side] - (side - 1) / 2
    discs = yy**2 + xx**2 <= side**2 / 4, abs(yy) + 0.9 * abs(xx - yy) < side / 2, np.ones((side, side), bool)
    rng = np.random.default_rng(8)
    for k, s in enumerate(rng.integers(0, 4, nx * ny)):
        y, x = 8 + pitch * (k // nx), 8 + pitch * (k % nx)
        img[y : y + side, x : x + side][discs[min(s, 2)]] = 40
    r = _same(np.clip(img + rng.normal(0, 2, img.shape), 0, 255).astype(np.uint8))
    sizes = np.diff(r.cstart)
    n = ((sizes >= lo) & (sizes <= hi)).sum()
    quads = ((sizes >= lo) & (sizes <= hi))[[q[2] for q in r.quads]].sum()
    print(n, quads)
    assert n > 148 * (4 if hi == 1024 else 2) and 0.2 * n < quads < 0.8 * n
