"""The tuning knob leg_ctas limits the CTAs of every FP64 Legendre kernel, and only them.

The launched grids are read from a trace of the calls; the results are the same bits at every
setting (the same items, each summed by one CTA in the same order).
"""

from __future__ import annotations

import json

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU hosts
    pytest.skip("no CUDA device", allow_module_level=True)

from torch.profiler import ProfilerActivity, profile  # noqa: E402

import jht_b200 as jhtb  # noqa: E402
from jht_b200 import _lib  # noqa: E402


def _pair(plan, a, v):
    m, b = torch.empty_like(v), torch.empty_like(a)
    s, nb = _lib.stream_ptr(), a.shape[0]
    _lib.check(plan.lib.jhtb_synthesis(plan.handle, a.data_ptr(), m.data_ptr(), nb, s), "synthesis")
    _lib.check(plan.lib.jhtb_adjoint_synthesis(plan.handle, v.data_ptr(), b.data_ptr(), nb, s), "adjoint")
    torch.cuda.synchronize()
    return m, b


def _legendre_grids(call, path):
    with profile(activities=[ProfilerActivity.CUDA, ProfilerActivity.CPU]) as p:
        call()
    p.export_chrome_trace(str(path))
    kernels = [e for e in json.loads(path.read_text())["traceEvents"] if e.get("cat") == "kernel"]
    if not kernels:
        pytest.skip("no kernel trace on this machine")
    return [e["args"]["grid"][0] for e in kernels if any(k in e["name"] for k in (
        "synth0_kernel", "synth2_kernel", "synth_batch_kernel", "adj0_kernel", "adj2_kernel", "adj_batch_kernel"))]


@pytest.mark.parametrize("spin", [0, 2])
@pytest.mark.parametrize("nside,lmax,B", [(32, 96, 1), (130, 300, 1), (256, 512, 11), (400, 800, 1)])
def test_leg_ctas_limits_the_grids(nside, lmax, B, spin, tmp_path):
    nc, nsm = (1 if spin == 0 else 2), torch.cuda.get_device_properties(0).multi_processor_count
    gen = torch.Generator(device="cuda").manual_seed(nside)
    a = torch.randn(B, nc, jhtb.alm_size(lmax), dtype=torch.complex128, device="cuda", generator=gen)
    v = torch.randn(B, nc, 12 * nside**2, dtype=torch.float64, device="cuda", generator=gen)
    plan = _lib.Plan(nside, lmax, spin, "fp64", max_batch=B)
    ref = _pair(plan, a, v)
    for c in (1, 2):
        plan.set_tuning(leg_ctas=c)
        out = []
        grids = _legendre_grids(lambda: out.extend(_pair(plan, a, v)), tmp_path / f"trace{c}.json")
        assert len(grids) >= 2 and max(grids) <= c * nsm
        assert torch.equal(out[0], ref[0]) and torch.equal(out[1], ref[1])
    plan.close()
