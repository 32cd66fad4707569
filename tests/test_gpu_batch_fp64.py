"""The batched FP64 Legendre kernels (legendre_batch.cu) against the one-map kernels.

Batches that leave full, half-filled and single-map groups, at resolutions with one partial
tile up to several blocks of 256 rings (the last one ragged), through the public batched
calls, on a plan restricted to a ring range, and through the Legendre entry points of a
ring-set plan.  Both paths add the same FP64 values in another order: with at most 650 terms
of either sign per sum the results differ by a few 1e-15 of a map's largest value; the bound
is 1e-13 of it.
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


def _inputs(nside, lmax, spin, B, seed):
    rng = np.random.default_rng(seed)
    K = (lmax + 1) * (lmax + 2) // 2
    nc = 1 if spin == 0 else 2
    ell = np.concatenate([np.arange(m, lmax + 1) for m in range(lmax + 1)])
    amp = 10.0 ** rng.uniform(-2, 2, B)[:, None, None]
    a = amp * (rng.standard_normal((B, nc, K)) + 1j * rng.standard_normal((B, nc, K))) / (ell + 1.0)
    a[..., : lmax + 1] = a[..., : lmax + 1].real
    a[..., ell < spin] = 0
    v = amp * rng.standard_normal((B, nc, 12 * nside * nside))
    return torch.as_tensor(a, device="cuda"), torch.as_tensor(v, device="cuda")


def _close(got, ref):
    for g, r in zip(got, ref):
        assert float((g - r).abs().max()) <= TOL * float(r.abs().max())


@pytest.mark.parametrize("spin", [0, 2])
@pytest.mark.parametrize("nside,lmax,B", [(1, 4, 2), (8, 12, 5), (33, 65, 4), (64, 128, 3), (130, 300, 8), (300, 641, 6),
                                          (256, 512, 9), (16, 200, 17)])
def test_batch_matches_one_map(nside, lmax, B, spin):
    a, v = _inputs(nside, lmax, spin, B, nside + B)
    pick = (lambda t: t[:, 0]) if spin == 0 else (lambda t: t)
    one = (lambda t: t[0]) if spin == 0 else (lambda t: t)
    got = jhtb.synthesis_batch(pick(a), nside, lmax, spin)
    _close(got, [jhtb.synthesis(one(x), nside, lmax, spin) for x in a])
    got = jhtb.adjoint_synthesis_batch(pick(v), nside, lmax, spin)
    _close(got, [jhtb.adjoint_synthesis(one(x), nside, lmax, spin) for x in v])


@pytest.mark.parametrize("spin", [0, 2])
def test_batch_on_a_ring_range(spin):
    nside, lmax, B = 400, 90, 6
    a, v = _inputs(nside, lmax, spin, B, 3)
    full = jhtb.adjoint_synthesis_batch(v[:, 0] if spin == 0 else v, nside, lmax, spin).reshape(B, -1)
    plan = _lib.Plan(nside, lmax, spin, "fp64", max_batch=B)
    total = torch.zeros_like(a)
    for t0, t1 in ((0, 256), (256, 512), (512, 800)):
        plan.set_ring_range(t0, t1)
        out = torch.empty_like(a)
        _lib.check(plan.lib.jhtb_adjoint_synthesis(plan.handle, v.data_ptr(), out.data_ptr(), B, _lib.stream_ptr()), "adjoint")
        total += out
    torch.cuda.synchronize()
    plan.close()
    _close(total.reshape(B, -1), full)


@pytest.mark.parametrize("spin", [0, 2])
def test_batch_on_a_ring_set(spin):
    lmax, B, nr = 70, 5, 145
    x = np.cos(np.arange(nr) * np.pi / (nr - 1))[: (nr + 1) // 2]
    x[-1] = 0.0
    a, _ = _inputs(1, lmax, spin, B, 4)
    nc = a.shape[1]
    plan = _lib.Plan(0, lmax, spin, "fp64", max_batch=B, rings=(nr, x))
    rng = np.random.default_rng(5)
    V = torch.as_tensor(rng.standard_normal((B, nc, nr, lmax + 1)) + 1j * rng.standard_normal((B, nc, nr, lmax + 1)), device="cuda")

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
