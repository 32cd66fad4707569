"""The batched FP64 Legendre kernels (legendre_batch.cu) against the one-map kernels, at sizes that reach them.

A batch goes to them from 148 x 16 (map, order, synthesis tile) items on, in groups of 8 (spin 0) or 4
(spin 2) maps, at most one of half that width, and at most one single map; every case here is
checked to lie above that line.  The batches leave each kind of remainder, the grids one partial tile
up to several blocks of 256 rings, and the ring set runs the Legendre entry points, whose spin-0
rows are not paired.

Both paths add the same FP64 values in another order.  A sum has at most 650 terms of either sign;
its rounding is a few 1e-15 of a map's largest value, the bound 1e-13 of it.
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU hosts
    pytest.skip("no CUDA device", allow_module_level=True)

import jht_b200 as jhtb  # noqa: E402
from jht_b200 import _lib  # noqa: E402

TOL = 1e-13
MIN_ITEMS = 148 * 16


def _items(half_rings, lmax, spin, B):
    return B * (lmax + 1) * -(-half_rings // (64 if spin else 128))


def _alm(gen, B, lmax, spin):
    nc, K = (1 if spin == 0 else 2), jhtb.alm_size(lmax)
    ell = torch.as_tensor(np.concatenate([np.arange(m, lmax + 1) for m in range(lmax + 1)]), device="cuda")
    a = torch.randn(B, nc, K, dtype=torch.complex128, device="cuda", generator=gen) / (ell + 1.0)
    a[..., : lmax + 1] = a[..., : lmax + 1].real.to(a.dtype)
    a[..., ell < spin] = 0
    return a * 10.0 ** torch.linspace(-2, 2, B, dtype=torch.float64, device="cuda")[:, None, None]


def _close(got, ref):
    for g, r in zip(got, ref):
        assert float((g - r).abs().max()) <= TOL * float(r.abs().max())


@pytest.mark.parametrize("spin,B", [(0, 2), (0, 3), (0, 4), (0, 5), (0, 9), (0, 10), (0, 12), (2, 2), (2, 3), (2, 5), (2, 6)])
@pytest.mark.parametrize("nside,lmax", [(300, 641), (520, 500)])
def test_groups_match_single_maps(nside, lmax, spin, B):
    assert _items(2 * nside, lmax, spin, B) >= MIN_ITEMS
    _compare(nside, lmax, spin, B)


@pytest.mark.parametrize("spin,B", [(0, 4), (0, 7), (2, 4), (2, 10)])
def test_one_partial_tile(spin, B):
    nside, lmax = 16, 620
    assert _items(2 * nside, lmax, spin, B) >= MIN_ITEMS
    _compare(nside, lmax, spin, B)


def _compare(nside, lmax, spin, B):
    gen = torch.Generator(device="cuda").manual_seed(nside + B)
    a = _alm(gen, B, lmax, spin)
    v = torch.randn(B, a.shape[1], 12 * nside**2, dtype=torch.float64, device="cuda", generator=gen)
    pick = (lambda t: t[:, 0]) if spin == 0 else (lambda t: t)
    one = (lambda t: t[0]) if spin == 0 else (lambda t: t)
    _close(jhtb.synthesis_batch(pick(a), nside, lmax, spin), [jhtb.synthesis(one(x), nside, lmax, spin) for x in a])
    _close(jhtb.adjoint_synthesis_batch(pick(v), nside, lmax, spin),
           [jhtb.adjoint_synthesis(one(x), nside, lmax, spin) for x in v])


@pytest.mark.parametrize("spin,B", [(0, 5), (0, 11), (2, 3), (2, 6)])
@pytest.mark.parametrize("nr", [145, 601])
def test_groups_on_a_ring_set(nr, spin, B):
    lmax, half = 500, (nr + 1) // 2
    assert _items(half, lmax, spin, B) >= MIN_ITEMS
    x = np.cos(np.arange(nr) * np.pi / (nr - 1))[:half]
    x[-1] = 0.0
    gen = torch.Generator(device="cuda").manual_seed(nr + B)
    a = _alm(gen, B, lmax, spin)
    V = torch.randn(B, a.shape[1], nr, lmax + 1, dtype=torch.complex128, device="cuda", generator=gen)
    plan = _lib.Plan(0, lmax, spin, "fp64", max_batch=B, rings=(nr, x))

    def both(al, rows, nb):
        F, b = torch.empty_like(rows), torch.empty_like(al)
        _lib.check(plan.lib.jhtb_legendre_synthesis(plan.handle, al.data_ptr(), F.data_ptr(), nb, _lib.stream_ptr()), "synthesis")
        _lib.check(plan.lib.jhtb_legendre_adjoint(plan.handle, rows.data_ptr(), b.data_ptr(), nb, _lib.stream_ptr()), "adjoint")
        return F, b

    F, b = both(a, V, B)
    for q in range(B):
        F1, b1 = both(a[q : q + 1].contiguous(), V[q : q + 1].contiguous(), 1)
        _close(F[q : q + 1], F1)
        _close(b[q : q + 1], b1)
    torch.cuda.synchronize()
    plan.close()
