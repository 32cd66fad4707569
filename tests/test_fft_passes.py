"""The FFT kernel's passes restated in NumPy: radix choice, index arithmetic and output order.

Decimation in frequency: pass p works on blocks of m R elements, butterfly j of a block takes the
elements j + q m, transforms them and multiplies result q by e^{-2 pi i j q / (m R)}; the last
pass's butterflies run in the order of their outputs.  Swept over every 2,3,5-smooth length up to the
shared-memory limit, with the kernel's own reciprocals in place of divisions.
"""

from __future__ import annotations

import re
from pathlib import Path

import numpy as np

from jht_b200 import _fft

SRC = (Path(__file__).resolve().parents[1] / "jht_b200" / "csrc" / "fft.cu").read_text()
RADICES = [int(r) for r in re.search(r"for \(int r : \{([\d, ]+)\}\)", SRC).group(1).split(",")]
MAX_PASS = int(re.search(r"kFftMaxPass = (\d+)", SRC).group(1))


def _pick(n):
    """The fewest passes, among these the smallest sum, the first found in the search's order."""
    best = [MAX_PASS + 1, 1 << 30, None]

    def search(n, cap, cur):
        if n == 1:
            if (len(cur), sum(cur)) < (best[0], best[1]):
                best[:] = [len(cur), sum(cur), list(cur)]
            return
        if len(cur) >= best[0] or len(cur) >= MAX_PASS:
            return
        for r in RADICES:
            if r <= cap and n % r == 0:
                search(n // r, r, cur + [r])

    search(n, 10, [])
    return best[2] if n > 1 else [1]


def _inv(d):
    return ((1 << 31) + d - 1) // d


def _div(a, inv):
    """f_div: the high word of 2 a times ceil(2^31 / d)."""
    return (2 * a * inv) >> 32


def _model(x):
    n, radices = x.size, _pick(x.size)
    m = [n // int(np.prod(radices[: p + 1])) for p in range(len(radices))]
    roots, buf = _fft._roots_host(n), x.copy()
    for p, R in enumerate(radices):
        b = np.arange(n // R, dtype=np.int64)
        last = p == len(radices) - 1
        if last:
            j, base, r = 0 * b, 0 * b, b
            for i in range(p):
                t = _div(r, _inv(radices[i]))
                base, r = base + (r - t * radices[i]) * m[i], t
            mp = 1
        else:
            mp = m[p]
            g = _div(b, _inv(mp)) if p else 0 * b
            j = b - g * mp
            base = g * mp * R + j
        at = base[None, :] + np.arange(R)[:, None] * mp
        assert np.array_equal(np.sort(at.ravel()), np.arange(n))  # every element once
        dft = np.exp(-2j * np.pi * np.outer(np.arange(R), np.arange(R)) / R)
        v = dft @ buf[at]
        if last:
            out = np.empty(n, complex)
            out[b[None, :] + np.arange(R)[:, None] * (n // R)] = v
            return out
        step = np.arange(R)[:, None] * (j * (n // (mp * R)))[None, :]
        assert step.max() < n
        buf = buf.copy()
        buf[at] = v * roots[step]


def test_reciprocals_divide_exactly():
    a = np.arange(1 << 14, dtype=np.int64)
    for d in range(1, _fft.SM_MAX + 1):
        assert _inv(d) < 1 << 32
        np.testing.assert_array_equal(_div(a, _inv(d)), a // d)


def test_passes_compose_to_the_dft_for_every_length():
    rng = np.random.default_rng(3)
    lengths = [n for n in range(1, _fft.SM_MAX + 1) if _fft._smooth(n)]
    for n in lengths:
        assert int(np.prod(_pick(n))) == n
        x = rng.standard_normal(n) + 1j * rng.standard_normal(n)
        ref = np.fft.fft(x)
        assert np.abs(_model(x) - ref).max() <= 1e-12 * max(1.0, np.abs(ref).max()), n
