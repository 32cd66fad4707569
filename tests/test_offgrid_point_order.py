"""The library's point order is 32 bits wide: no longer point set reaches it in one call.

Point sets above that size run on meta tensors (shapes without memory), with the library call
replaced by a record of what it was given.
"""

from __future__ import annotations

from types import SimpleNamespace

import pytest

torch = pytest.importorskip("torch")

from jht_b200 import offgrid  # noqa: E402

LIMIT = 2**31


@pytest.mark.parametrize("deriv", [False, True])
@pytest.mark.parametrize("tiles", [100, 1 << 12])  # grouped by the library, and by torch (too many tiles)
@pytest.mark.parametrize("npts", [LIMIT - 1024, LIMIT, 3 * LIMIT + 5])
def test_interpolation_orders_fit_32_bits(npts, tiles, deriv, monkeypatch):
    calls = []

    def raw(g, grid, theta, phi, deriv, order):
        assert theta.numel() == phi.numel()
        if order is None:  # too few points to be worth an order
            assert theta.numel() < offgrid._SORT_MIN_POINTS
        else:
            assert order.dtype == torch.int32 and order.numel() == theta.numel()
        calls.append(theta.numel())
        out = torch.empty(theta.numel(), dtype=torch.complex128, device="meta")
        return (out, out, out) if deriv else (out, None, None)

    def grouped(g, theta, phi, vals=None):
        return SimpleNamespace(theta=theta, phi=phi, order=torch.empty(theta.numel(), dtype=torch.int32, device="meta"))

    grouped.takes = offgrid._Grouped.takes
    monkeypatch.setattr(offgrid, "_interp_raw", raw)
    monkeypatch.setattr(offgrid, "_Grouped", grouped)
    g = SimpleNamespace(nk=1 << 17, nm=1 << 17, tiles_k=tiles, tiles_m=tiles)
    theta, phi = torch.empty((2, npts), dtype=torch.float64, device="meta")
    outs = offgrid._interp(g, None, theta, phi, deriv)
    assert sum(calls) == npts and max(calls) < LIMIT
    assert [o if o is None else o.numel() for o in outs] == [npts] + [npts if deriv else None] * 2
