"""The roots that order same-id detections (csrc/at_order.cu), found from the
last union back, against the oracle's sequential union by size: noisy
backgrounds that are targets themselves, odd sizes, shapes whose sets meet
late or in long chains, and links of the last column. Whole numbers: equal."""
import numpy as np
import pytest

import apriltags_fast_b200 as AT
from apriltags_fast_b200 import synth
from oracle import oracle as O
from tests import helpers as H

pytestmark = pytest.mark.gpu
CHECKED = []  # a (width, decimation) per root compared


def _frame(w, h, noise, pattern, seed):
    """Eight tags of two codes (ids repeat) beside a pattern that
    touches the background: teeth joined late ("comb"), teeth that join one
    after another ("stairs"), a white last column beside rows of dashes
    ("edge")."""
    cfg = synth.Config(w, h, families=("tag25h9",), ntags=(8, 8), side=(36, 60), noise=noise)
    codes, *rest = synth.builtin_table("tag25h9")
    img = synth.make_frame(cfg, seed, {"tag25h9": (codes[:2], *rest)})[0]
    if pattern == "comb":
        img[4:h - 8, 4:w // 5:8] = 250
        img[h - 8:h - 4, 4:w // 5] = 250
    elif pattern == "stairs":
        for k, x in enumerate(range(4, w // 4, 8)):
            img[4 + 4 * (k % 7):h // 3 + 6 * k, x:x + 4] = 250
            img[min(h - 5, h // 3 + 6 * k):min(h - 1, h // 3 + 6 * k + 4), max(0, x - 8):x + 4] = 250
    elif pattern == "edge":
        img[:, w - 2:] = 250
        img[::6, w - 40:w - 2] = 250
        img[1::6, w - 40:w - 2] = 250
        img[3::6, w - 4:w - 2] = 10
        img[4::6, w - 4:w - 2] = 10
    return img


@pytest.mark.parametrize("dec", [2.0, 1.0, 1.5])
@pytest.mark.parametrize("w,h,noise,pattern", [(640, 480, 3.0, ""), (1293, 727, 6.0, ""), (640, 480, 0.0, "comb"),
                                               (801, 602, 5.0, "stairs"), (640, 480, 4.0, "edge"),
                                               (1923, 411, 9.0, "comb")])
def test_roots_equal_the_oracle(w, h, noise, pattern, dec):
    det = AT.Detector(["tag25h9"], 2, quad_decimate=dec)
    fams = [H.oracle_family("tag25h9")]
    for seed in range(3):
        img = _frame(w, h, noise, pattern, 50 + seed)
        got = [d.key() for d in det.detect(img)]
        r = O.detect(img, fams, [2], O.default_params(quad_decimate=dec), order=O.ORDER_REF)
        assert got == r.dets, seed
        for label, root in det.diag("order_roots"):
            assert r.label[label] == label and r.ref_root[label] == root, (seed, int(label))
            CHECKED.append((w, dec))


def test_roots_were_checked():
    """Ids that repeat are up to the drawn codes and what is detected: over
    all frames above, many targets, and some at each decimation."""
    assert len(CHECKED) >= 100 and len({dec for _, dec in CHECKED}) == 3
