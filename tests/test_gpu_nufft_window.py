"""The window sums at the points (jhtb_nufft_interp) and their transpose (jhtb_nufft_spread)
against the same sums in NumPy, for every window width, point counts that leave lanes of a warp
without a point, grids smaller than a window (cells wrap more than once) and points whose window
crosses the grid's edges.

Each output is a sum of at most W^2 products of FP64 values; W^2 eps = 6e-14 of the sum of the
terms' sizes for W = 16, doubled for the weights' own rounding (the derivative's division and
square root near the window's edge add a few more): 2e-13 of the largest such sum.
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU hosts
    pytest.skip("no CUDA device", allow_module_level=True)

from jht_b200 import _lib  # noqa: E402

TOL = 2e-13


def _weights(coord, n, W, beta):
    u = coord * n / (2 * np.pi)
    f = np.ceil(u - 0.5 * W)
    t = u[:, None] - (f[:, None] + np.arange(W))
    z = t * (2.0 / W)
    r = np.sqrt(np.clip(1 - z * z, 0, None))
    w = np.where(z * z < 1, np.exp(beta * (r - 1)), 0.0)
    with np.errstate(divide="ignore", invalid="ignore"):
        dw = np.where(z * z < 1, -w * beta * z * (2.0 / W) / r, 0.0) * (n / (2 * np.pi))
    return (f[:, None].astype(np.int64) + np.arange(W)) % n, w, dw


@pytest.mark.parametrize("W", [6, 8, 10, 14, 16])
@pytest.mark.parametrize("nk,nm,npts", [(5, 7, 1), (40, 33, 2), (64, 50, 31), (81, 96, 517)])
def test_window_sums(W, nk, nm, npts):
    rng = np.random.default_rng(W * 1000 + npts)
    beta = 2.3 * W
    th, ph = rng.uniform(-7.0, 14.0, npts), rng.uniform(-7.0, 14.0, npts)
    th[0], ph[0] = 0.0, 2 * np.pi
    grid = rng.standard_normal((nk, nm)) + 1j * rng.standard_normal((nk, nm))
    v = rng.standard_normal(npts) + 1j * rng.standard_normal(npts)
    ik, wk, dk = _weights(th, nk, W, beta)
    im, wm, dm = _weights(ph, nm, W, beta)
    cells = grid[ik[:, :, None], im[:, None, :]]

    lib = _lib.load_library()
    tg, tt, tp, tv = (torch.as_tensor(x, device="cuda") for x in (grid, th, ph, v))
    outs = [torch.empty(npts, dtype=torch.complex128, device="cuda") for _ in range(4)]
    s = _lib.stream_ptr()
    args = (tg.data_ptr(), nk, nm, W, beta, tt.data_ptr(), tp.data_ptr(), npts)
    _lib.check(lib.jhtb_nufft_interp(*args, outs[0].data_ptr(), outs[1].data_ptr(), outs[2].data_ptr(), s), "interp")
    _lib.check(lib.jhtb_nufft_interp(*args, outs[3].data_ptr(), None, None, s), "interp")
    for out, (a, b) in zip(outs, ((wk, wm), (dk, wm), (wk, dm), (wk, wm))):
        ref = np.einsum("jab,ja,jb->j", cells, a, b)
        size = np.einsum("jab,ja,jb->j", np.abs(cells), np.abs(a), np.abs(b)).max()
        assert np.abs(out.cpu().numpy() - ref).max() <= TOL * size

    got = torch.zeros((nk, nm), dtype=torch.complex128, device="cuda")
    _lib.check(lib.jhtb_nufft_spread(tv.data_ptr(), tt.data_ptr(), tp.data_ptr(), npts, nk, nm, W, beta,
                                     got.data_ptr(), s), "spread")
    ref, size = np.zeros((nk, nm), complex), np.zeros((nk, nm))
    ww = wk[:, :, None] * wm[:, None, :]
    np.add.at(ref, (ik[:, :, None], im[:, None, :]), ww * v[:, None, None])
    np.add.at(size, (ik[:, :, None], im[:, None, :]), ww * np.abs(v)[:, None, None])
    assert np.abs(got.cpu().numpy() - ref).max() <= TOL * size.max()
