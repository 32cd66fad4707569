"""The FFT kernel with several transforms per CTA, against NumPy.

Batches large enough for 2, 4 and 8 neighbouring transforms per CTA (the launch takes as many as
leave every SM two CTAs and fit their shared memory), with a last group that is not full, and the
four-step composition of a grid whose two calls run that way.  The off-grid torus grid at lengths
that take 2 and 4 is compared with the composition of batched FFTs.  Bounds as for single transforms:
1e-13 of the largest value per transform, 6e-13 between two chains of three.
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU hosts
    pytest.skip("no CUDA device", allow_module_level=True)

from jht_b200 import _fft, offgrid  # noqa: E402


@pytest.mark.parametrize("n,columns", [(2, 4001), (9, 2371), (60, 2403), (243, 2375), (800, 2373), (1000, 1189),
                                       (1620, 1187), (2160, 597), (5000, 594), (12288, 30), (17280, 21)])
@pytest.mark.parametrize("sign", [-1, 1])
def test_columns_match_numpy(n, columns, sign):
    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, columns)) + 1j * rng.standard_normal((n, columns))
    got = _fft.fft(torch.as_tensor(x, device="cuda"), 0, sign).cpu().numpy()
    ref = np.fft.fft(x, axis=0) if sign < 0 else np.fft.ifft(x, axis=0) * n
    assert np.abs(got - ref).max() <= 1e-13 * np.abs(ref).max()


@pytest.mark.parametrize("spin", [0, 2])
@pytest.mark.parametrize("lmax", [640, 1100, 1700])
def test_torus_grid_matches_composition(lmax, spin, monkeypatch):
    g = offgrid._geometry(lmax, spin, 1e-10, torch.cuda.current_device())
    assert g.one_call
    gen = torch.Generator(device="cuda").manual_seed(lmax + spin)

    def white(*shape):
        return torch.randn(*shape, dtype=torch.complex128, device="cuda", generator=gen)

    F, grid = white(g.ncomp, g.ns, lmax + 1), white(g.nk, g.nm)
    got = offgrid._torus_grid(g, F), offgrid._torus_grid_adjoint(g, grid)
    monkeypatch.setattr(g, "one_call", False)
    ref = offgrid._torus_grid(g, F), offgrid._torus_grid_adjoint(g, grid)
    for a, b in zip(got, ref):
        assert (a - b).abs().max() <= 6e-13 * b.abs().max()
