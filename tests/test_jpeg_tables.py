"""The JPEG decoder's Huffman tables on the CPU: tests/jpeg_tables.cu built
for the host around csrc/at_jpeg.cu."""
import os
import shutil
import subprocess

import pytest

import oracle.oracle as O
from tests import jpeg_cases as J

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    if shutil.which("nvcc") is None:
        pytest.skip("no nvcc")
    out = str(tmp_path_factory.mktemp("tables") / "jpeg_tables")
    subprocess.check_call(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O1", "-std=c++17", "-I",
                           os.path.join(ROOT, "include"), "-o", out, os.path.join(ROOT, "tests", "jpeg_tables.cu")])
    return out


def _run(*cmd):
    p = subprocess.run(cmd, capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stdout[-2000:]


def test_second_levels_of_any_number_of_tables(exe):
    """A job's tables all decode right, also those whose second levels lie
    above 2^22 entries, and those for which no room is left."""
    _run(exe, "places")


def test_equal_tables_of_a_job_are_kept_once(exe, tmp_path):
    paths = []
    for k in range(2):
        paths.append(str(tmp_path / f"{k}.jpg"))
        open(paths[-1], "wb").write(O.jpeg_encode(J._gray(64, 64, 3 + 40 * k), 95, (1, 1), 0, O.JPEG_OPTIMIZE))
    _run(exe, "shared", *paths)


@pytest.mark.parametrize("sel", [0x00, 0x20, 0x30])
def test_a_scan_that_takes_ac_tables_for_dc(exe, tmp_path, sel):
    """A scan header may name table 2 or 3 for DC codes: the AC tables 0 and 1,
    as DC codes (common/pjpeg.c indexes one array of four)."""
    p = str(tmp_path / "a.jpg")
    open(p, "wb").write(J.dc_selector(O.jpeg_encode(J._rgb(64, 64, 5), 90, (2, 2), 0, O.JPEG_OPTIMIZE), sel))
    _run(exe, "scans", p)


def test_a_file_whose_tables_pass_2_22_entries(exe, tmp_path):
    """132 scans of four tables with 64 second levels each."""
    p = str(tmp_path / "a.jpg")
    buf = J.many_tables(132, 5)
    assert O.jpeg_decode(buf)[0] == 0
    open(p, "wb").write(buf)
    _run(exe, "scans", p)
