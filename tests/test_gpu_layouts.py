"""The one-launch coefficient layouts (vecops.cu) against the torch operations they replace.

Copies, exact doublings and one scaling by sqrt 2 per value: the vectors and the gradients must
be the same bits as the torch path's, the coefficients (a division by sqrt 2, which torch carries
out as a complex one) within two ulp.
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU hosts
    pytest.skip("no CUDA device", allow_module_level=True)

import jht_b200 as jhtb  # noqa: E402
from jht_b200 import masked  # noqa: E402


@pytest.mark.parametrize("spin", [0, 2])
@pytest.mark.parametrize("lmax,B", [(0, 1), (1, 2), (2, 3), (3, 1), (65, 5)])
def test_dof_layouts(lmax, B, spin):
    g = torch.Generator(device="cuda").manual_seed(lmax + spin)
    nc, K = (1 if spin == 0 else 2), jhtb.alm_size(lmax)
    a = torch.randn((B, nc, K), dtype=torch.complex128, device="cuda", generator=g)
    x = torch.randn((B, jhtb.n_dof(lmax, spin)), dtype=torch.float64, device="cuda", generator=g)
    assert torch.equal(masked._real_batch(a, lmax, spin), masked._real_batch(a.requires_grad_(True), lmax, spin))
    got, ref = masked._alm_batch(x, lmax, spin), masked._alm_batch(x.requires_grad_(True), lmax, spin)
    assert torch.all((got - ref).abs() <= 2 * 2.3e-16 * ref.abs())


@pytest.mark.parametrize("spin", [0, 2])
@pytest.mark.parametrize("nside,lmax", [(1, 2), (16, 33), (64, 96)])
def test_gradient_is_that_of_the_differentiable_path(nside, lmax, spin):
    rng = np.random.default_rng(lmax)
    K = jhtb.alm_size(lmax)
    shape, npix = ((K,), (12 * nside**2,)) if spin == 0 else ((2, K), (2, 12 * nside**2))
    a = torch.as_tensor(rng.standard_normal(shape) + 1j * rng.standard_normal(shape), device="cuda").requires_grad_(True)
    v = torch.as_tensor(rng.standard_normal(npix), device="cuda")
    plain, = torch.autograd.grad(jhtb.synthesis(a, nside, lmax, spin), a, v)
    graph, = torch.autograd.grad(jhtb.synthesis(a, nside, lmax, spin), a, v, create_graph=True)
    assert torch.equal(plain, graph.detach())
