"""The off-grid transforms' torus grid in one library call (jhtb_torus_grid and its adjoint)
against the composition of batched FFTs and tensor operations that longer lengths use.

White ring coefficients and grids; the lengths cover one to five passes, grids without and with
padding and the smallest lmax.  Each side is three transforms of at most 1e-13 of the largest
value (the FFT's own bound), so the two differ by at most 6e-13 of it.
"""

from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU hosts
    pytest.skip("no CUDA device", allow_module_level=True)

from jht_b200 import offgrid  # noqa: E402

TOL = 6e-13


@pytest.mark.parametrize("spin", [0, 2])
@pytest.mark.parametrize("lmax", [2, 5, 24, 121, 200, 511])
def test_one_call_matches_composition(lmax, spin, monkeypatch):
    g = offgrid._geometry(lmax, spin, 1e-10, torch.cuda.current_device())
    assert g.one_call
    rng = torch.Generator(device="cuda").manual_seed(lmax + spin)

    def white(*shape):
        return torch.randn(*shape, dtype=torch.complex128, device="cuda", generator=rng)

    F, grid = white(g.ncomp, g.ns, lmax + 1), white(g.nk, g.nm)
    got = offgrid._torus_grid(g, F), offgrid._torus_grid_adjoint(g, grid)
    monkeypatch.setattr(g, "one_call", False)
    ref = offgrid._torus_grid(g, F), offgrid._torus_grid_adjoint(g, grid)
    for a, b in zip(got, ref):
        assert a.shape == b.shape
        assert (a - b).abs().max() <= TOL * b.abs().max()
