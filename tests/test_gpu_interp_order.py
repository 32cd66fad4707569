"""Interpolation through a point order, values and both derivatives.

A point's sums do not depend on its place: grouped by the library, ordered by torch (grids with
too many tiles) and taken part by part, every point has the bits it has in input order.
"""

from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU hosts
    pytest.skip("no CUDA device", allow_module_level=True)

from jht_b200 import offgrid  # noqa: E402


@pytest.mark.parametrize("deriv", [False, True])
@pytest.mark.parametrize("eps", [1e-4, 1e-10])
@pytest.mark.parametrize("npts", [1 << 16, 150003])
def test_orders_keep_every_point(npts, eps, deriv, monkeypatch):
    g = offgrid._geometry(50, 0, eps, torch.cuda.current_device())
    gen = torch.Generator(device="cuda").manual_seed(npts)
    grid = torch.randn(g.nk, g.nm, dtype=torch.complex128, device="cuda", generator=gen)
    theta, phi = 21.0 * torch.rand(2, npts, dtype=torch.float64, device="cuda", generator=gen) - 7.0
    ref = offgrid._interp_raw(g, grid, theta, phi, deriv, None)
    assert offgrid._Grouped.takes(g, npts)
    runs = [offgrid._interp(g, grid, theta, phi, deriv)]
    with monkeypatch.context() as m:
        m.setattr(offgrid, "_GROUP_MAX_TILES", 0)
        runs.append(offgrid._interp(g, grid, theta, phi, deriv))
    with monkeypatch.context() as m:
        m.setattr(offgrid, "_ORDER_MAX", 70000)
        m.setattr(offgrid, "_ORDER_PART", 66000)
        runs.append(offgrid._interp(g, grid, theta, phi, deriv))
    for out in runs:
        for a, b in zip(out, ref):
            assert (a is None and b is None) or torch.equal(a, b)
