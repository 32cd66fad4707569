"""jhtb_nufft_group_points: a counting sort of the points by grid tile.  Whole numbers, so the
result is exact: every point once, its coordinates and value beside its place, segments of at
most 1024 points that cover the places once and hold points of one tile.  Points outside one
period, on the tile edges, at infinity and NaN, all in one tile, and counts about a segment's
and a warp's size."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU hosts
    pytest.skip("no CUDA device", allow_module_level=True)

from jht_b200 import _lib  # noqa: E402


@pytest.mark.parametrize("nk,nm", [(20, 33), (864, 810), (4320, 2000)])
@pytest.mark.parametrize("npts,crowded", [(1, False), (31, False), (1025, True), (5000, True), (70001, False)])
def test_group_points(nk, nm, npts, crowded):
    rng = np.random.default_rng(npts + nk)
    th, ph = rng.uniform(-7, 14, npts), rng.uniform(-7, 14, npts)
    if crowded:
        th[:], ph[:] = 1.0, 2.0
    else:
        th[: npts // 3] = np.round(th[: npts // 3] * nk / (64 * np.pi)) * (64 * np.pi) / nk  # tile edges
    if npts > 20:
        th[5], ph[7], th[9], ph[11] = np.inf, np.nan, -0.0, 2 * np.pi
    v = rng.standard_normal(npts) + 1j * rng.standard_normal(npts)
    tk, tm = nk // 32 + 2, nm // 32 + 2
    nseg = tk * tm + npts // 1024
    cu = dict(device="cuda")
    t, p, vv = (torch.as_tensor(x, **cu) for x in (th, ph, v))
    ts, ps, vs = torch.empty_like(t), torch.empty_like(p), torch.empty_like(vv)
    work = torch.empty(16 * tk * tm + 8192 + 2 * npts, dtype=torch.int32, **cu)
    order = torch.empty(npts, dtype=torch.int32, **cu)
    count = torch.empty(nseg, dtype=torch.int32, **cu)
    start, tile = torch.empty(nseg, dtype=torch.int64, **cu), torch.empty(nseg, dtype=torch.int64, **cu)
    _lib.check(_lib.load_library().jhtb_nufft_group_points(
        t.data_ptr(), p.data_ptr(), vv.data_ptr(), npts, nk, nm, tk, tm, work.data_ptr(), order.data_ptr(),
        ts.data_ptr(), ps.data_ptr(), vs.data_ptr(), count.data_ptr(), start.data_ptr(), tile.data_ptr(),
        _lib.stream_ptr()), "group")
    o = order.cpu().numpy()
    assert np.array_equal(np.sort(o), np.arange(npts))
    for got, ref in ((ts, th), (ps, ph), (vs, v)):
        np.testing.assert_array_equal(got.cpu().numpy(), ref[o])
    c, s, k = count.cpu().numpy(), start.cpu().numpy(), tile.cpu().numpy()
    used = int((c > 0).sum())
    assert (c[:used] > 0).all() and (c[used:] == 0).all() and c.max() <= 1024
    assert np.array_equal(s[:used], np.cumsum(c[:used]) - c[:used]) and c.sum() == npts
    assert (np.diff(k[:used]) >= 0).all() and k[:used].min() >= 0 and k[:used].max() < tk * tm
    # each point lies in its segment's tile, to rounding at the edges
    seg = np.repeat(k[:used], c[:used])
    for x, n, tt in ((th[o], nk, seg // tm), (ph[o], nm, seg % tm)):
        ok = np.isfinite(x)
        u = np.mod(x[ok], 2 * np.pi) * n / (2 * np.pi)
        d = np.minimum(np.abs(u - 32 * tt[ok] - 16), np.abs(n - np.abs(u - 32 * tt[ok] - 16)))
        assert (d <= 16 + 1e-6).all()
