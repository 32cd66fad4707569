"""What lanes of a warp hand one another through shared memory is ordered by a barrier.

A vote or a shuffle makes lanes meet but orders no memory accesses, so between a lane's write and
another lane's read there has to be a ``__syncwarp`` (or a block barrier).  Which order a chip happens
to keep cannot be seen from results, so the source is checked: in the interpolation kernel every
lane writes the window start of its own point and the lanes of a point read those of another.
"""

from __future__ import annotations

import re
from pathlib import Path

SRC = Path(__file__).resolve().parents[1] / "jht_b200" / "csrc" / "nufft.cu"


def _body(source: str, kernel: str) -> str:
    """Text of a kernel from its name to the closing brace, without comments."""
    source = re.sub(r"//[^\n]*", "", source)
    at = source.index("{", source.index(kernel + "("))
    depth = 0
    for i in range(at, len(source)):
        depth += {"{": 1, "}": -1}.get(source[i], 0)
        if depth == 0:
            return source[at : i + 1]
    raise AssertionError(f"{kernel}: unbalanced braces")


def test_interpolation_reads_window_starts_after_a_barrier():
    body = _body(SRC.read_text(), "interp_kernel")
    for name in ("su", "sf", "sbase"):
        write = body.index(f"{name}[warp][lane] =")
        read = body.index(f"{name}[warp][i]")
        assert write < read
        assert re.search(r"__sync(warp|threads)\(", body[write:read]), f"{name}: read without a barrier after the write"
        # and the next batch's write waits for this batch's reads: the loop starts with a barrier
        assert re.search(r"__syncwarp\(", body[body.index("for (long long bi"): write])
