"""Tiled spread (jhtb_nufft_spread_tiles): which points are summed on chip, and those that are not.

A tile's sum reaches the grid as one addition per cell.  Points whose contributions are each
below half an ulp of the grid's values therefore show in the result only if they were summed before:
that tells the two paths apart.  The on-chip sum is exact to far below that ulp, so a cell may be off
by its one rounding, 2^-53 at values in [1, 2).

The direct path is compared with NumPy: a cell is a sum of products of three FP64 values, as in
the untiled spread, so the bound is the same 2e-13 of the largest sum of the terms' sizes.
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU hosts
    pytest.skip("no CUDA device", allow_module_level=True)

from jht_b200 import _lib  # noqa: E402

TWO_PI = 2 * np.pi


def _weights(coord, n, W, beta):
    u = coord * n / TWO_PI
    f = np.ceil(u - 0.5 * W)
    z = (u[:, None] - (f[:, None] + np.arange(W))) * (2.0 / W)
    w = np.where(z * z < 1, np.exp(beta * (np.sqrt(np.clip(1 - z * z, 0, None)) - 1)), 0.0)
    return (f[:, None].astype(np.int64) + np.arange(W)) % n, w


def _reference(th, ph, v, nk, nm, W, beta):
    ik, wk = _weights(th, nk, W, beta)
    im, wm = _weights(ph, nm, W, beta)
    out = np.zeros((nk, nm), complex)
    np.add.at(out, (ik[:, :, None], im[:, None, :]), wk[:, :, None] * wm[:, None, :] * v[:, None, None])
    return out


def _spread(th, ph, v, nk, nm, W, beta, grid, group):
    """Points grouped by the library, or (group False) all in one segment of tile 0."""
    cu, n, lib, s = dict(device="cuda"), th.size, _lib.load_library(), _lib.stream_ptr()
    t, p, vv = (torch.as_tensor(x, **cu) for x in (th, ph, v))
    tk, tm = nk // 32 + 2, nm // 32 + 2
    if group:
        nseg = tk * tm + n // 1024
        ts, ps, vs = torch.empty_like(t), torch.empty_like(p), torch.empty_like(vv)
        work = torch.empty(16 * tk * tm + 8192 + 2 * n, dtype=torch.int32, **cu)
        order, count = torch.empty(n, dtype=torch.int32, **cu), torch.empty(nseg, dtype=torch.int32, **cu)
        start, tile = torch.empty((2, nseg), dtype=torch.int64, **cu)
        _lib.check(lib.jhtb_nufft_group_points(
            t.data_ptr(), p.data_ptr(), vv.data_ptr(), n, nk, nm, tk, tm, work.data_ptr(), order.data_ptr(),
            ts.data_ptr(), ps.data_ptr(), vs.data_ptr(), count.data_ptr(), start.data_ptr(), tile.data_ptr(), s), "group")
        t, p, vv = ts, ps, vs
    else:
        nseg, count = 1, torch.full((1,), n, dtype=torch.int32, **cu)
        start, tile = torch.zeros((2, 1), dtype=torch.int64, **cu)
    g = torch.as_tensor(grid, **cu)
    _lib.check(lib.jhtb_nufft_spread_tiles(vv.data_ptr(), t.data_ptr(), p.data_ptr(), n, nseg, start.data_ptr(),
                                           count.data_ptr(), tile.data_ptr(), tm, nk, nm, W, beta, g.data_ptr(), s), "spread")
    return g.cpu().numpy()


@pytest.mark.parametrize("W", [6, 14, 16])
@pytest.mark.parametrize("periods", [(0, 0), (0, -1), (-1, 0), (1, -3), (2, 1)])
@pytest.mark.parametrize("nk,nm", [(864, 810), (40, 64)])
def test_points_of_any_period_are_summed_on_chip(nk, nm, periods, W):
    rng = np.random.default_rng(W)
    n, beta = 64, 2.3 * W
    # about the middle of tile (0, 1), a tenth of a cell apart
    th = (16 + rng.uniform(-0.05, 0.05, n)) * TWO_PI / nk + periods[0] * TWO_PI
    ph = (32 + 16 + rng.uniform(-0.05, 0.05, n)) * TWO_PI / nm + periods[1] * TWO_PI
    v = np.full(n, 0.4 * 2.0**-53 * (1 + 1j))  # alone, none of them moves a cell that holds 1
    got = _spread(th, ph, v, nk, nm, W, beta, np.full((nk, nm), 1 + 1j), True)
    ref = _reference(th, ph, v, nk, nm, W, beta)
    assert ref.real.max() > 15 * 2.0**-53
    for part in (np.real, np.imag):
        assert np.abs((part(got) - 1.0) - part(ref)).max() <= 1.01 * 2.0**-53


@pytest.mark.parametrize("W", [6, 8, 10, 14, 16])
@pytest.mark.parametrize("nk,nm", [(81, 96), (40, 33)])
def test_points_of_other_tiles(nk, nm, W):
    rng = np.random.default_rng(nk + W)
    n, beta = 300, 2.3 * W
    th, ph = rng.uniform(-7, 14, n), rng.uniform(-7, 14, n)
    v = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    got = _spread(th, ph, v, nk, nm, W, beta, np.zeros((nk, nm), complex), False)
    size = _reference(th, ph, np.abs(v), nk, nm, W, beta).real.max()
    assert np.abs(got - _reference(th, ph, v, nk, nm, W, beta)).max() <= 2e-13 * size


@pytest.mark.parametrize("W", [6, 14, 16])
@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_values_that_are_not_finite_stay_in_their_window(bad, W):
    """The cells of such a point's window are not finite; every other cell has its ordinary sum."""
    rng = np.random.default_rng(W)
    nk, nm, n, beta = 128, 160, 200, 2.3 * W
    # all of one tile, so that they share the products of a round
    th = rng.uniform(33, 63, n) * TWO_PI / nk
    ph = rng.uniform(65, 95, n) * TWO_PI / nm
    v = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    one = np.zeros(n, bool)
    one[7] = True
    got = _spread(th, ph, np.where(one, complex(bad, 1.0), v), nk, nm, W, beta, np.zeros((nk, nm), complex), True)
    hit = _reference(th[one], ph[one], np.ones(1), nk, nm, W, beta) != 0
    assert not np.isfinite(got.real[hit]).any()
    ref = _reference(th[~one], ph[~one], v[~one], nk, nm, W, beta)
    size = _reference(th, ph, np.abs(v), nk, nm, W, beta).real.max()
    assert np.abs(got - ref)[~hit].max() <= 2e-13 * size
