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
