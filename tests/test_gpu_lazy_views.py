"""Lazily conjugated and negated tensors (``a.conj()``, ``a.conj().imag``) as inputs.

torch keeps the conjugation or the sign as a bit of the view, and ``data_ptr()`` shows the values
without it.  Every entry point that hands memory to the library has to give the same bits for such
a view as for the tensor with the bit carried out (the same values through the same kernels).
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU hosts
    pytest.skip("no CUDA device", allow_module_level=True)

import jht_b200 as jhtb  # noqa: E402
from jht_b200 import distributed, masked  # noqa: E402

NSIDE, LMAX = 8, 12
NPIX, K = 12 * NSIDE**2, jhtb.alm_size(LMAX)


def _conj(gen, *shape):
    t = torch.randn(*shape, dtype=torch.complex128, device="cuda", generator=gen).conj()
    assert t.is_conj() and t.is_contiguous()
    return t


def _neg(gen, *shape):
    """A contiguous real tensor with the negation bit."""
    t = torch._neg_view(torch.randn(*shape, dtype=torch.float64, device="cuda", generator=gen))
    assert t.is_neg() and t.is_contiguous()
    return t


def _plain(t):
    return t.resolve_conj().resolve_neg()


@pytest.fixture
def gen():
    return torch.Generator(device="cuda").manual_seed(11)


@pytest.mark.parametrize("spin", [0, 2])
def test_transforms(spin, gen):
    nc = () if spin == 0 else (2,)
    for B in ((), (3,)):
        f, g = (jhtb.synthesis_batch, jhtb.adjoint_synthesis_batch) if B else (jhtb.synthesis, jhtb.adjoint_synthesis)
        a, v = _conj(gen, *B, *nc, K), _neg(gen, *B, *nc, NPIX)
        assert torch.equal(f(a, NSIDE, LMAX, spin), f(_plain(a), NSIDE, LMAX, spin))
        assert torch.equal(g(v, NSIDE, LMAX, spin), g(_plain(v), NSIDE, LMAX, spin))
    assert torch.equal(jhtb.analysis(v[0], NSIDE, LMAX, spin), jhtb.analysis(_plain(v[0]), NSIDE, LMAX, spin))


@pytest.mark.parametrize("spin", [0, 2])
def test_sharded_transform(spin, gen):
    nc = 1 if spin == 0 else 2
    t = distributed.ShardedTransform(NSIDE, LMAX, spin)
    a, v = _conj(gen, 1, nc, K), _neg(gen, 1, nc, NPIX)
    assert torch.equal(t.synthesis(a), t.synthesis(_plain(a)))
    assert torch.equal(t.adjoint_synthesis(v), t.adjoint_synthesis(_plain(v)))
    torch.cuda.synchronize()
    t.close()


@pytest.mark.parametrize("spin", [0, 2])
def test_dof_layouts(spin, gen):
    nc = 1 if spin == 0 else 2
    a, x = _conj(gen, 3, nc, K), _neg(gen, 3, jhtb.n_dof(LMAX, spin))
    assert torch.equal(masked._real_batch(a, LMAX, spin), masked._real_batch(_plain(a), LMAX, spin))
    assert torch.equal(masked._alm_batch(x, LMAX, spin), masked._alm_batch(_plain(x), LMAX, spin))


def test_warm_starts(gen):
    """x0 of the solvers: without a step the answer is the start itself."""
    m, mask = torch.randn(2, NPIX, dtype=torch.float64, device="cuda", generator=gen), np.ones(NPIX)
    x0 = _conj(gen, 2, K)
    args = dict(max_iter=0, x0=x0)
    plain = dict(args, x0=_plain(x0))
    assert torch.equal(jhtb.deconvolve_batch(m, mask, NSIDE, LMAX, **args), jhtb.deconvolve_batch(m, mask, NSIDE, LMAX, **plain))
    cl = np.ones(LMAX + 1)
    assert torch.equal(masked.wiener_batch(m, cl, NSIDE, LMAX, mask=mask, **args),
                       masked.wiener_batch(m, cl, NSIDE, LMAX, mask=mask, **plain))


@pytest.mark.parametrize("spin", [0, 2])
def test_offgrid(spin, gen):
    nc = () if spin == 0 else (2,)
    loc = _neg(gen, 1, 2)  # one point: its two coordinates are contiguous as they lie
    a, f = _conj(gen, *nc, K), _neg(gen, *nc, 1)

    def both(alm, field, at):
        return (jhtb.synthesis_general(alm, at, spin=spin, lmax=LMAX),
                jhtb.adjoint_synthesis_general(field, at, spin=spin, lmax=LMAX))

    for got, ref in zip(both(a, f, loc), both(_plain(a), _plain(f), _plain(loc))):
        assert torch.equal(got, ref)

