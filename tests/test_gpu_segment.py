"""Runs, components and points from the row masks (csrc/at_segment.cu,
csrc/at_cluster.cu) against the oracle at the widths and heights where words
(32 columns) and bands (8, 4 and 2 rows; one above 8192 columns) begin and
end, on images of random blobs: the labels of all pixels, the points and the
clusters are equal."""
import numpy as np
import pytest

import apriltags_fast_b200 as AT
from oracle import oracle as O
from tests import helpers as H
from tests.test_gpu_parity import oracle_pixel_labels

pytestmark = pytest.mark.gpu


def _blobs(w, h, cell, seed):
    """Random cells of cell x cell pixels, dark, light or flat, with noise."""
    rng = np.random.default_rng(seed)
    g = rng.choice([30, 220, 220, 30, 125], size=(h // cell + 1, w // cell + 1))
    img = np.kron(g, np.ones((cell, cell), int))[:h, :w]
    return np.clip(img + rng.normal(0, 3, (h, w)), 0, 255).astype(np.uint8)


def _check(imgs, min_px, dec=1.0):
    det = AT.Detector(["tag36h11"], 2, quad_decimate=dec, min_cluster_pixels=min_px)
    fams = [H.oracle_family("tag36h11")]
    prm = O.default_params(quad_decimate=dec, min_cluster_pixels=min_px)
    for img in imgs:
        det.detect(img)
        r = O.detect(img, fams, [2], prm, order=O.ORDER_CANON)
        assert np.array_equal(det.diag("threshold"), r.thresh)
        assert np.array_equal(det.diag("labels"), oracle_pixel_labels(r, min_px))
        assert np.array_equal(det.diag("points"), r.pts)
        assert np.array_equal(det.diag("clusters"), r.cstart[:-1])


@pytest.mark.parametrize("w,h", [(31, 40), (32, 33), (33, 16), (34, 17), (64, 8), (65, 9), (97, 47), (1023, 24),
                                 (1025, 23), (2048, 17), (2049, 18), (4097, 11), (4161, 12)])
def test_word_and_band_edges(w, h):
    _check([_blobs(w, h, cell, 7 * w + cell) for cell in (1, 2, 3, 5)], 24)


@pytest.mark.parametrize("min_px", [2, 5, 200])
def test_component_gate(min_px):
    _check([_blobs(203, 99, 1, 5), _blobs(203, 99, 3, 6)], min_px)


@pytest.mark.parametrize("w", [8200, 16390])
def test_wide_frames(w):
    """Bands of one row (with and without unions in shared memory): labels
    of blank frames (detected as empty) and of a frame with one edge, which
    is wider than the order of same-id detections allows and so refused; at
    a higher decimation the quad image is narrow again."""
    det = AT.Detector(["tag36h11"], 2, quad_decimate=1.0)
    fams = [H.oracle_family("tag36h11")]
    blank = np.full((64, w), 90, np.uint8)
    edge = blank[:40].copy()
    edge[8:32, w // 2:] = 250
    for img, refused in ((blank, False), (edge, True)):
        if refused:
            with pytest.raises(RuntimeError, match="too wide"):
                det.detect(img)
        else:
            assert det.detect(img) == [] and det.nquads == 0
        r = O.detect(img, fams, [2], O.default_params(quad_decimate=1.0), order=O.ORDER_CANON)
        assert np.array_equal(det.diag("labels"), oracle_pixel_labels(r, 24))
    _check([_blobs(w, 48, 7, w)], 24, 3.0 if w < 12000 else 4.0)


@pytest.mark.parametrize("w", [512, 700, 1024, 1025, 2080])
@pytest.mark.parametrize("tooth", [1, 2])
def test_dense_points(w, tooth):
    """Two combs in one another: up to two points a pixel, so that 1024
    columns hold more than a warp lists at a time, of one pair of labels."""
    img = np.where(np.arange(w) // tooth % 2, 30, 220).astype(np.uint8)[None].repeat(40, 0)
    img[:8], img[32:] = 220, 30
    _check([img], 24)
    r = O.detect(img, [H.oracle_family("tag36h11")], [2], O.default_params(quad_decimate=1.0), order=O.ORDER_CANON)
    per_row = len(r.pts) / 24  # the rows of the teeth
    assert per_row > (1.9 if tooth == 1 else 0.95) * w, per_row


@pytest.mark.parametrize("w", [300, 1025])
def test_rows_above_a_limit(w):
    """Rows with more points (over two a pixel, below the teeth of a comb) or
    more pairs of labels (stripes) than the scan has room for, beside a frame
    without: the sorting path takes every point of the batch."""
    teeth = np.where(np.arange(w) % 2, 30, 220).astype(np.uint8)[None].repeat(40, 0)
    comb = teeth.copy()
    comb[:8], comb[32:] = 220, 30
    stripes = np.where(np.arange(w) // 2 % 2, 30, 220).astype(np.uint8)[None].repeat(40, 0)
    _check([comb, stripes, _blobs(w, 40, 3, w)], 24)
    det = AT.Detector(["tag36h11"], 2, quad_decimate=1.0)
    imgs = [_blobs(w, 40, 3, w), comb, stripes]
    pts = [O.detect(i, [H.oracle_family("tag36h11")], [2], O.default_params(quad_decimate=1.0), order=O.ORDER_CANON).pts
           for i in imgs]
    det.detect_batch(imgs)
    assert np.array_equal(det.diag("points"), np.concatenate(pts))


@pytest.mark.parametrize("n", [1, 63, 64, 129, 1022, 1023, 1024, 2049, 4094, 4095, 4096])
def test_cluster_counts(n):
    """n clusters or one more (in one block up to 1024, gathered in one up to
    4096, by several kernels above), n quads: alone, and in a batch."""
    img = np.full((65 * 15 + 8, 65 * 15 + 8), 210, np.uint8)
    for k in range(n):
        y, x = 4 + 15 * (k // 65), 4 + 15 * (k % 65)
        img[y : y + 9, x : x + 9 + k % 2] = 40
    _check([img], 24)
    fams = [H.oracle_family("tag36h11")]
    prm = O.default_params(quad_decimate=1.0)
    imgs = [_blobs(97, 60, 5, 1), img, _blobs(97, 60, 5, 2)]
    ref = [O.detect(i, fams, [2], prm, order=O.ORDER_CANON) for i in imgs]
    assert len(ref[1].cstart) - 1 in (n, n + 1) and len(ref[1].quads) == n
    det = AT.Detector(["tag36h11"], 2, quad_decimate=1.0)
    got = det.detect_batch(imgs)
    assert np.array_equal(det.diag("points"), np.concatenate([r.pts for r in ref]))
    quads = det.diag("quads")
    want = np.array([q[0] for r in ref for q in r.quads], np.float32)
    assert np.array_equal(quads["p"].view(np.uint32), want.view(np.uint32))
    assert np.array_equal(quads["frame"], np.repeat([0, 1, 2], [len(r.quads) for r in ref]))
    assert [[d.key() for d in f] for f in got] == [r.dets for r in ref]


def _strips(n, h):
    """n strips side by side, light and dark in turn, with a slow ramp (no
    contrast) between them but at both ends, where they touch; dots too small
    for components keep each strip's contrast. So each pair of neighbours has
    few points, first and last row far apart."""
    w, gap, end = 12, 44, 16
    lv = [(134, 122) if k % 2 == 0 else (122, 134) for k in range(n)]
    img = np.zeros((h, n * (w + gap) + 24))
    for x in range(img.shape[1]):
        k, r = divmod(x - w, w + gap)
        a, b = lv[k % 2]
        img[:, x] = a + (b - a) * max(r - w, 0) / gap
    for k in range(n):
        x0 = w + k * (w + gap)
        for y in range(4, h - 4, 8):
            img[y : y + 3, x0 + 4 : x0 + 7] = lv[k][1]
        if k + 1 == n:
            break
        x0 += w
        m = x0 + gap // 2
        for y0 in (0, h - end):
            img[y0 : y0 + end, x0:m], img[y0 : y0 + end, m : x0 + gap] = lv[k]
            for x in range(x0 + 2, x0 + gap - 3, 8):
                if abs(x + 1 - m) >= 6:
                    for y in range(y0 + 4, y0 + end - 3, 8):
                        img[y : y + 3, x : x + 3] = lv[k][x < m]
    return np.round(img).astype(np.uint8)


@pytest.mark.parametrize("frames,n,h", [(1, 20, 1200), (15, 72, 500)])
def test_pairs_that_span_many_rows(frames, n, h):
    """The rows that the pairs span outnumber the row tables' first room
    (points + 64 a pair + 4096), with few pairs (one block orders them) and
    more than 1024: the batch runs again with more room, and later calls
    have it."""
    img = _strips(n, h)
    r = O.detect(img, [H.oracle_family("tag36h11")], [2], O.default_params(quad_decimate=1.0), order=O.ORDER_CANON)
    y = (r.pts >> np.uint64(16) & np.uint64(0xFFFF)).astype(int) // 2
    spans = sum(y[a:b].max() - y[a:b].min() + 1 for a, b in zip(r.cstart[:-1], r.cstart[1:]))
    pairs = len(r.cstart) - 1
    assert frames * spans > frames * (len(r.pts) + 64 * pairs) + 4096
    assert (frames * pairs > 1024) == (frames > 1)
    det = AT.Detector(["tag36h11"], 2, quad_decimate=1.0)
    launches = []
    for rep in range(2):
        before = int(det.diag("sizes")[5])
        got = det.detect_batch([img] * frames)
        launches.append(int(det.diag("sizes")[5]) - before)
        assert np.array_equal(det.diag("points"), np.tile(r.pts, frames))
        at = np.arange(frames)[:, None] * len(r.pts) + r.cstart[:-1].astype(int)
        assert np.array_equal(det.diag("clusters").astype(int), at.ravel())
        assert [[d.key() for d in f] for f in got] == [r.dets] * frames
        assert det.last_batch_nquads == [len(r.quads)] * frames
    assert launches[0] > launches[1] > 0


@pytest.mark.parametrize("w", [131104, 425984, 425985])
def test_very_wide_blank_frames(w):
    """Rows whose words alone fill the shared memory of a band."""
    det = AT.Detector(["tag36h11"], 2, quad_decimate=1.0)
    blank = np.full((12, w), 90, np.uint8)
    if w > 425984:
        with pytest.raises(RuntimeError, match="too wide"):
            det.detect(blank)
        return
    assert det.detect(blank) == [] and det.nquads == 0
    assert (det.diag("labels") == 0xFFFFFFFF).all()
