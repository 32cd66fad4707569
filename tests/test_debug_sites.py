"""The bounds checks of the debug library cover what its documentation names.

Each checked kind of access has a site number; the ring stage checks spectra (101, 102, 105),
pixels of both streams (103, 104), shared-memory slots (106), twiddles and belt factors (107), chirp
spectra (108) and chirp factors (110), the Legendre kernels their tables, rows and sums (2xx).
"""

from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "jht_b200" / "csrc"


def _source(name: str) -> str:
    return re.sub(r"//[^\n]*", "", (CSRC / name).read_text())


@pytest.mark.parametrize("name,sites", [
    ("ringfft.cu", {101, 102, 103, 104, 105, 106, 107, 108, 110}),
    ("legendre.cu", {201, 202, 203, 204}),
    ("legendre_batch.cu", {206, 207, 208, 209}),
    ("tc_synth.cu", {301}),
    ("tc_adjoint.cu", {401, 402}),
    ("vecops.cu", {501}),
])
def test_sites(name, sites):
    found = {int(m) for m in re.findall(r",\s*(\d{3})\)", _source(name))}
    assert sites <= found, sorted(sites - found)


def test_ring_stage_tables_and_streams_are_checked():
    src = _source("ringfft.cu")
    # twiddles of the FFT passes as well as the belt's factors
    assert len(re.findall(r"JHTB_IN\([^;]*?, 107\)", src)) >= 2
    # both pixel streams, in and out
    for site in (103, 104):
        assert {m for m in re.findall(rf"JHTB_IN\(s\.(off[XY]) \+ j, [^;]*?, {site}\)", src)} == {"offX", "offY"}
    # no table entry of the chirps is read past its check
    for table in ("bh", "ctab"):
        assert all(f"a.{table}_len" in line for line in src.splitlines() if re.search(rf"__ldg\(&a\.{table}\[", line))
