"""GPU JPEG decode (csrc/at_jpeg.cu) through its C ABI against the CPU
oracle (oracle/at_jpeg.c, pinned to the reference's common/pjpeg.c by
tests/test_jpeg_oracle.py) and, where it is built, the reference's own
decoder (oracle/_ref). Pixels and error codes must be equal byte for byte.
A gray frame is component 0 cropped to the image (pjpeg_to_u8_baseline);
where the reference would read outside its planes there (no scan of
component 0, or a plane smaller than the image) the GPU decoder refuses
the image with an error code instead."""
import numpy as np
import pytest

import apriltags_fast_b200 as AT
from apriltags_fast_b200 import synth
from oracle import oracle as O
from tests import helpers as H
from tests import jpeg_cases as J
from tests.jpeg_cases import bad_files, encode_matrix

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dec():
    d = AT.JpegDecoder()
    yield d
    d.close()


def expected_gray(buf, flags):
    """(error or 'refused', frame) as the oracle decodes the file."""
    e, w, h, p = O.jpeg_decode(buf, flags)
    if e:
        return e, None
    if not p or p[0].shape[0] < h or p[0].shape[1] < w:
        return "refused", None
    return 0, O.gray_of(w, h, p)


def check_batch(dec, cases, device=False, pad=0):
    by_flags = {}
    for name, buf, flags, *_ in cases:
        by_flags.setdefault(flags, []).append((name, buf))
    for flags, items in by_flags.items():
        bufs = [b for _, b in items]
        if device:
            frames, errs = dec.decode_device(bufs, flags, pad)
            frames = [f.cpu().numpy() if f is not None else None for f in frames]
        else:
            frames, errs = dec.decode(bufs, flags)
        for (name, buf), f, e in zip(items, frames, errs):
            xe, xf = expected_gray(buf, flags)
            if xe == "refused":
                assert e != 0, name
                continue
            assert e == xe, (name, e, xe)
            if xe == 0:
                assert f.shape == xf.shape and (f == xf).all(), name


def frames_1080p():
    out = []
    cfg = synth.Config(1920, 1080)
    for seed, q in ((0, 75), (1, 90), (2, 95)):
        img = synth.make_frame(cfg, seed)
        img = img[0] if isinstance(img, tuple) else img
        out.append((f"1080p q{q}", O.jpeg_encode(img, q), 0))
        rgb = np.stack([img, np.roll(img, 3, 1), 255 - img], -1)
        out.append((f"1080p 4:2:0 q{q}", O.jpeg_encode(rgb, q, (2, 2), 0, O.JPEG_OPTIMIZE), 0))
    out.append(("1080p restart 8", O.jpeg_encode(img, 85, (1, 1), 8), 0))
    return out


def test_matrix_to_host_frames(dec):
    check_batch(dec, encode_matrix(small=False))


def test_bad_and_truncated_files(dec):
    check_batch(dec, bad_files())


def test_device_frames_with_padded_rows(dec):
    check_batch(dec, encode_matrix(small=True), device=True, pad=13)


def test_1080p_frames_one_batch(dec):
    cases = frames_1080p()
    check_batch(dec, cases, device=True)
    st = dec.last_stats()
    assert st["substreams"] > 1000 and st["entropy_bytes"] > 500_000


@pytest.mark.parametrize("bits", [64, 256, 2048, 65536])
def test_substream_size_does_not_change_pixels(bits):
    d = AT.JpegDecoder(sub_bits=bits)
    try:
        check_batch(d, frames_1080p()[:2] + encode_matrix(small=True)[::7])
    finally:
        d.close()


def test_pjpeg_dropin_planes_and_rgb():
    """pjpeg_create_from_buffer gives the reference's planes (every
    component, padding columns zero) and pjpeg_to_u8x3_baseline its RGB."""
    ref = O.ref_lib() is not None
    for name, buf, flags in encode_matrix(small=True)[::3] + [frames_1080p()[1]]:
        a = AT.pjpeg_decode(buf, flags)
        b = O.jpeg_decode(buf, flags)
        assert a[:3] == b[:3] and len(a[3]) == len(b[3]), name
        for x, y in zip(a[3], b[3]):
            assert x.shape == y.shape and (x == y).all(), name
        if ref:
            r = O.ref_jpeg_rgb(buf, flags)
            g = AT.pjpeg_rgb(buf, flags)
            assert (r is None) == (g is None), name
            if r is not None:
                assert (r == g).all(), name


def test_detect_on_a_decoded_jpeg(dec):
    """Camera frame as JPEG -> GPU decode into device memory -> detector on
    that device frame: the detections of the reference's pixels."""
    cfg = synth.Config(1920, 1080)
    img = synth.make_frame(cfg, 4)
    img = img[0] if isinstance(img, tuple) else img
    buf = O.jpeg_encode(img, 92)
    frames, errs = dec.decode_device([buf])
    assert errs == [0]
    e, w, h, p = O.jpeg_decode(buf)
    host = O.gray_of(w, h, p)
    det = AT.Detector()
    assert det.add_family("tag36h11", 2)
    got = [d.key() for d in det.detect(frames[0])]
    want = O.detect(host, [H.oracle_family("tag36h11")], [2], O.default_params(), order=O.ORDER_REF).dets
    assert got == want and len(got) >= 3


def _flip_entropy(buf, rng, nflips):
    """Random bytes of the entropy-coded data changed, none of them an FF,
    next to an FF, or made into one (the markers stay where they were)."""
    b = bytearray(buf)
    sos = buf.find(b"\xff\xda")
    lo = sos + 2 + (buf[sos + 2] << 8 | buf[sos + 3])
    hi = len(buf) - 2
    done = 0
    while done < nflips:
        i = int(rng.integers(lo + 1, hi - 1))
        if 0xFF in (b[i - 1], b[i], b[i + 1]):
            continue
        v = int(rng.integers(0, 255))  # never 0xFF
        if v == b[i]:
            continue
        b[i] = v
        done += 1
    return bytes(b)


def test_damaged_entropy_data_equals_the_oracle(dec):
    """Damaged scans decode as the oracle decodes them (codes that match
    nothing, runs past the last coefficient, decodes that stop moving),
    gray, 4:2:0 with restart markers, and 4:4:4, with no fault."""
    rng = np.random.default_rng(42)
    cfg = synth.Config(640, 480)
    img = synth.make_frame(cfg, 9)[0]
    rgb = np.stack([img, np.roll(img, 5, 0), 255 - img], -1)
    bases = [O.jpeg_encode(img, 90), O.jpeg_encode(rgb, 80, (2, 2), 6), O.jpeg_encode(rgb, 95, (1, 1))]
    cases = []
    for k, base in enumerate(bases):
        for n in (1, 3, 8, 40):
            for rep in range(3):
                cases.append((f"base{k} flips{n} #{rep}", _flip_entropy(base, rng, n), 0))
    check_batch(dec, cases)
    check_batch(dec, cases[::5], device=True, pad=3)


@pytest.mark.parametrize("counts", [{2: 2, 10: 160}, {2: 3, 9: 60, 12: 99}, {3: 6, 16: 156}, {2: 1, 8: 100, 11: 61},
                                    {1: 1, 13: 161}])
@pytest.mark.parametrize("color", [False, True])
def test_code_lengths(counts, color):
    """AC tables with other code lengths put into a file (its data then
    decodes to other pixels; with restart intervals, to an error): codes of up
    to 9 bits, longer ones under few and under more than 64 prefixes, windows
    without a code. Pixels and error codes as the oracle's."""
    g = J._gray(120, 168, 11)
    buf = bytearray(O.jpeg_encode(J._rgb(120, 168, 12), 95, (2, 2), 5) if color else O.jpeg_encode(g, 95))
    want, at = bytes(counts.get(i, 0) for i in range(1, 17)), 0
    assert sum(want) == 162
    while (at := buf.find(b"\xff\xc4", at)) >= 0:  # each DHT segment: AC tables of 162 symbols
        o, end = at + 4, at + 2 + int.from_bytes(buf[at + 2:at + 4], "big")
        while o < end:
            n = sum(buf[o + 1:o + 17])
            if buf[o] >> 4 == 1 and n == 162:
                buf[o + 1:o + 17] = want
            o += 17 + n
        at = end
    e, w, h, planes = O.jpeg_decode(bytes(buf))
    dec = AT.JpegDecoder()
    frames, errs = dec.decode([bytes(buf)])
    dec.close()
    assert errs == [e]
    if e == 0:
        assert np.array_equal(frames[0], O.gray_of(w, h, planes))


@pytest.mark.parametrize("sel", [0x20, 0x30])
def test_scans_that_take_ac_tables_for_dc(dec, sel):
    """Scan headers that name table 2 or 3 for DC codes (and, for a gray file
    without AC table 1, the missing table's error), beside ordinary files."""
    cases = []
    for k, (rst, fl) in enumerate([(0, 0), (0, O.JPEG_OPTIMIZE), (0, O.JPEG_OPTIMIZE)]):
        plain = O.jpeg_encode(J._rgb(101, 150, 20 + k), 90, (2, 2) if k < 2 else (1, 1), rst, fl)
        cases += [(f"plain {k}", plain, 0), (f"color {k}", J.dc_selector(plain, sel), 0)]
    cases.append(("gray", J.dc_selector(O.jpeg_encode(J._gray(101, 150, 30), 85), sel), 0))
    check_batch(dec, cases)
    check_batch(dec, cases, device=True)


def test_device_frames_wait_for_the_work_on_their_memory(dec):
    """Frames decoded into memory that torch has just got back, while work
    queued on its stream still reads what was there: that work is done first."""
    import torch

    bufs = [O.jpeg_encode(J._gray(480, 640, k), 90) for k in (1, 2)]
    for stream in (torch.cuda.current_stream(), torch.cuda.Stream()):
        with torch.cuda.stream(stream):
            (frame,), _ = dec.decode_device(bufs[:1])
            want, copy, ptr = frame.cpu(), torch.empty_like(frame), frame.data_ptr()
            torch.cuda._sleep(100_000_000)  # cycles: some 50 ms
            copy.copy_(frame)
            del frame
            (again,), _ = dec.decode_device(bufs[1:])
            assert again.data_ptr() == ptr
            assert torch.equal(copy.cpu(), want)
            assert np.array_equal(again.cpu().numpy(), expected_gray(bufs[1], 0)[1])
            del again, copy


def test_a_job_whose_tables_pass_2_22_entries(dec):
    """Files of many scans with tables of their own: alone, and after one
    another in a call, so that a later file's tables lie high."""
    cases = [(f"{n} scans", J.many_tables(n, n), 0) for n in (1, 132, 2)]
    check_batch(dec, cases[1:2])
    check_batch(dec, cases)
    check_batch(dec, cases, device=True)
