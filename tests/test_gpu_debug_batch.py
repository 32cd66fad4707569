"""The bounds-checked debug library on FP64 batches large enough for the batched Legendre kernels.

Full, half-filled and single-map groups of both spins, with a ragged last tile: no failed access,
and the release library's results on the same inputs (the same operations, so to 1e-14 of the largest
value, which only leaves room for the compiler's choice of fused operations).
"""

from __future__ import annotations

import json
import os
import subprocess
import sys
import textwrap
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU hosts
    pytest.skip("no CUDA device", allow_module_level=True)

import jht_b200 as jhtb  # noqa: E402
from jht_b200 import _lib  # noqa: E402

ROOT = Path(__file__).resolve().parents[1]
MIN_ITEMS = 148 * 16  # (map, order, synthesis tile) items from which the batched kernels run

# (nside, lmax, spin, batch)
CASES = [(256, 511, 0, 13), (256, 511, 0, 3), (130, 300, 2, 7), (300, 641, 0, 2), (300, 641, 2, 2)]

CHILD = textwrap.dedent("""
    import json, sys
    sys.path.insert(0, {tests!r})
    import test_gpu_debug_batch as T
    import numpy as np
    out = {{}}
    for i, case in enumerate(T.CASES):
        m, b = T.transforms(*case)
        np.save({tmp!r} + f"/m{{i}}.npy", m)
        np.save({tmp!r} + f"/b{{i}}.npy", b)
        out[i] = T._lib.debug_bounds()
    print("RECORD " + json.dumps(out))
""")


def transforms(nside, lmax, spin, nb):
    gen = torch.Generator(device="cuda").manual_seed(nside + nb)
    shape = (nb, jhtb.alm_size(lmax)) if spin == 0 else (nb, 2, jhtb.alm_size(lmax))
    a = torch.randn(*shape, dtype=torch.complex128, device="cuda", generator=gen)
    v = torch.randn(*shape[:-1], 12 * nside**2, dtype=torch.float64, device="cuda", generator=gen)
    m, b = jhtb.synthesis_batch(a, nside, lmax, spin), jhtb.adjoint_synthesis_batch(v, nside, lmax, spin)
    return m.cpu().numpy(), b.cpu().numpy()


def test_cases_reach_the_batched_kernels():
    for nside, lmax, spin, nb in CASES:
        tile = 64 if spin else 128  # rings of a synthesis tile
        assert nb * (lmax + 1) * -(-2 * nside // tile) >= MIN_ITEMS


def test_no_failed_access_and_the_release_results(tmp_path):
    code = CHILD.format(tests=str(ROOT / "tests"), tmp=str(tmp_path))
    env = dict(os.environ, JHTB_LIBRARY=str(_lib.DEBUG_LIB_PATH), PYTHONPATH=str(ROOT))
    res = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=600)
    assert res.returncode == 0, res.stderr[-3000:]
    line = [ln for ln in res.stdout.splitlines() if ln.startswith("RECORD ")][-1]
    for key, rec in json.loads(line[len("RECORD "):]).items():
        assert rec["count"] == 0, (CASES[int(key)], rec)
    for i, case in enumerate(CASES):
        for got, name in zip(transforms(*case), "mb"):
            ref = np.load(tmp_path / f"{name}{i}.npy")
            assert np.abs(got - ref).max() <= 1e-14 * np.abs(ref).max(), (case, name)
