"""The azimuthal stage's transforms (ringfft.cu) at the edges of their classes.

On the CPU: the FFT's pass structure and shared-memory layout, restated in NumPy, must give
the DFT for every length the kernels are built for, with every position inside the buffer and
written by its reader; the chirp-z pieces must give a ring's DFT with the kernel's factor
columns.  On the GPU: the stage against NumPy's FFTs at resolutions whose ring lengths
straddle the class limits (plain sums up to 128 points; chirp lengths 64 / 65, 128 /
129, ..., 2048 / 2049; power-of-two belts in one and two pieces; band limits below and far
above the ring lengths).
"""

from __future__ import annotations

import numpy as np
import pytest

from oracle import jht_oracle as O


class Fft:
    """Index arithmetic of ringfft.cu's Fft<LOGP>."""

    def __init__(self, lg):
        self.lg, self.P, self.TP, self.NP = lg, 1 << lg, (1 << lg) // 16, (lg + 3) // 4
        self.RL = 1 << (lg - 4 * (self.NP - 1))
        self.PAD = 5 if lg == 10 else 3 if lg == 9 else 1
        self.LEN = self.P + 16 * self.PAD + (self.P // 16 if lg == 13 else 0)

    def pidx(self, i):
        return i + self.PAD * (i >> (self.lg - 4)) + (2 * (i >> 5) if self.lg == 13 else 0)

    def rev(self, c):
        if self.NP <= 2:
            return c
        if self.NP == 3:
            return ((c & 15) << 4) | (c >> 4)
        return ((c & 15) << 8) | (((c >> 4) & 15) << 4) | (c >> 8)

    def raw(self, p, t, q):
        if p == self.NP - 1:
            return self.rev(t + self.TP * (q // self.RL)) * self.RL + q % self.RL
        bl = self.lg - 4 * p
        sl = bl - 4
        return ((t >> sl) << bl) + (t & ((1 << sl) - 1)) + (q << sl)

    def grid(self, p):
        t, q = np.meshgrid(np.arange(self.TP), np.arange(16), indexing="ij")
        f = np.vectorize(lambda a, b: self.raw(p, a, b))
        return f(t, q)

    def twiddle(self, p, sign):
        bl = self.lg - 4 * p
        j = np.arange(self.TP)[:, None] & ((1 << (bl - 4)) - 1)
        return np.exp(sign * 2j * np.pi * j * np.arange(16)[None, :] / (1 << bl))

    def radix(self, v, R, sign):
        w = np.exp(sign * 2j * np.pi * np.outer(np.arange(R), np.arange(R)) / R)
        return (v.reshape(self.TP, 16 // R, R) @ w.T).reshape(self.TP, 16)

    def forward(self, x):
        buf = np.full(self.LEN, np.nan, complex)
        v = x[self.grid(0)]
        for p in range(self.NP):
            last = p == self.NP - 1
            v = self.radix(v, self.RL if last else 16, +1)
            if not last:
                buf[self.pidx(self.grid(p))] = v * self.twiddle(p, +1)
                v = buf[self.pidx(self.grid(p + 1))]
        return v

    def out_index(self):
        t, q = np.meshgrid(np.arange(self.TP), np.arange(16), indexing="ij")
        return t + self.TP * (q // self.RL) + (self.P // self.RL) * (q % self.RL)

    def backward(self, v):
        buf = np.full(self.LEN, np.nan, complex)
        for p in range(self.NP - 1, -1, -1):
            last = p == self.NP - 1
            if not last:
                v = v * self.twiddle(p, -1)
            v = self.radix(v, self.RL if last else 16, -1)
            if p:
                buf[self.pidx(self.grid(p))] = v
                v = buf[self.pidx(self.grid(p - 1))]
        x = np.empty(self.P, complex)
        x[self.grid(0)] = v
        return x


@pytest.mark.parametrize("lg", range(7, 14))
def test_fft_passes_and_layout(lg):
    f = Fft(lg)
    rng = np.random.default_rng(lg)
    x = rng.standard_normal(f.P) + 1j * rng.standard_normal(f.P)
    for p in range(f.NP):
        g = f.pidx(f.grid(p))
        assert g.min() >= 0 and g.max() < f.LEN and np.unique(g).size == f.P
    X = np.empty(f.P, complex)
    v = f.forward(x)
    X[f.out_index()] = v
    ref = np.fft.ifft(x) * f.P
    assert np.max(np.abs(X - ref)) <= 1e-13 * np.max(np.abs(ref)) * lg
    assert np.max(np.abs(f.backward(v) / f.P - x)) <= 1e-13 * lg


@pytest.mark.parametrize("i", [33, 64, 65, 100, 257, 1024])
@pytest.mark.parametrize("shifted", [False, True])
def test_chirp_pieces(i, shifted):
    """Piece s of a ring of N = 4 i points: synthesis pixels 4 j + s, and W'[4 k + s] of the adjoint."""
    N, lg = 4 * i, 7
    while (1 << lg) < 2 * i - 1:
        lg += 1
    P = 1 << lg
    rng = np.random.default_rng(i)
    D = rng.standard_normal(N) + 1j * rng.standard_normal(N)
    k = np.arange(i)
    cis = lambda a: np.exp(1j * np.pi * (a % (2 * N)) / N)  # noqa: E731
    n = np.minimum(np.arange(P), P - np.arange(P))
    b = np.where(n < i, np.conj(np.exp(1j * np.pi * (n.astype(np.int64) ** 2 % (2 * i)) / i)), 0)
    B = np.fft.ifft(b)  # the e^{+} transform divided by P
    conv = lambda a: np.fft.fft(np.fft.ifft(np.pad(a, (0, P - i))) * P * B)[:i]  # noqa: E731
    out, W = np.empty(N, complex), np.empty(N, complex)
    for s in range(4):
        q = D.reshape(4, i) * (np.exp(1j * np.pi * np.arange(4) / 4)[:, None] if shifted else 1)
        a = (1j ** (s * np.arange(4)))[:, None] * q
        col = (1 + 2 * s) * k + 4 * k * k if shifted else 2 * s * k + 4 * k * k
        out[s::4] = conv(a.sum(0) * cis(col)) * cis(4 * k * k)
        a = (1j ** (s * np.arange(4)))[:, None] * np.conj(D.reshape(4, i))
        last = 4 * k * k + 4 * k + s if shifted else 4 * k * k
        W[s::4] = np.conj(conv(a.sum(0) * cis(2 * s * k + 4 * k * k)) * cis(last))
    ph = np.exp(1j * np.pi * np.arange(N) / N) if shifted else 1
    ref, refW = np.fft.ifft(D * ph) * N, np.fft.fft(D) * np.conj(ph)
    assert np.max(np.abs(out - ref)) <= 1e-12 * np.max(np.abs(ref))
    assert np.max(np.abs(W - refW)) <= 1e-12 * np.max(np.abs(refW))


# The stage alone: the library's own ring spectra (the Legendre stage through the C ABI, whose
# rounding is not under test) transformed by NumPy.  Bound: an FFT of at most 3 x 13 radix-2
# levels and five factors, about four FP64 roundings each, stays below 200 x 1.1e-16 = 2.2e-14
# of the largest value; 1e-13 leaves room for the differences of the sums over degrees.
TOL = 1e-13


@pytest.mark.gpu
@pytest.mark.parametrize("spin", [0, 2])
@pytest.mark.parametrize("nside,lmax", [(1, 4), (3, 300), (32, 40), (33, 65), (64, 300), (66, 12), (130, 64), (130, 600),
                                        (256, 1100), (258, 20), (514, 9), (1026, 10), (1024, 5), (2048, 6), (2050, 6)])
def test_ring_classes(nside, lmax, spin):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import jht_b200 as jhtb
    from jht_b200 import _lib

    rng = np.random.default_rng(nside + lmax)
    ell, m = O.lm_of_index(lmax)
    nc = 1 if spin == 0 else 2
    a = rng.standard_normal((nc, ell.size)) + 1j * rng.standard_normal((nc, ell.size))
    a = np.where(m == 0, a.real, a) / (ell + 1.0)
    if spin:
        a[:, ell < 2] = 0
    v = rng.standard_normal((nc, 12 * nside * nside))
    geo = O.Rings(nside)
    mm = np.arange(lmax + 1)[:, None]
    ph = np.exp(1j * np.pi * (mm % (2 * geo.nring)) / geo.nring)
    ph[:, geo.phi0 == 0.0] = 1.0
    plan = _lib.get_plan(nside, lmax, spin)
    ta = torch.as_tensor(a, device="cuda")
    F = torch.empty((nc, plan.nrings, lmax + 1), dtype=torch.complex128, device="cuda")
    _lib.check(plan.lib.jhtb_legendre_synthesis(plan.handle, ta.data_ptr(), F.data_ptr(), 1, _lib.stream_ptr()), "synthesis")
    G = [f.T * ph for f in F.cpu().numpy()]
    ref = O.rings_synth(geo, G[0], G[-1], lmax)
    ref = np.stack([ref.real, ref.imag])[:nc]
    got = jhtb.synthesis(ta.reshape(nc, -1) if spin else ta[0], nside, lmax, spin).cpu().numpy().reshape(nc, -1)
    assert np.max(np.abs(got - ref)) <= TOL * np.max(np.abs(ref))

    Wp, Wm = O.rings_adjoint(geo, v[0] + 1j * v[1] if spin else v[0].astype(complex), lmax)
    V = torch.as_tensor(np.ascontiguousarray(np.stack([(w * ph.conj()).T for w in (Wp, Wm)[:nc]])), device="cuda")
    b = torch.empty((nc, ell.size), dtype=torch.complex128, device="cuda")
    _lib.check(plan.lib.jhtb_legendre_adjoint(plan.handle, V.data_ptr(), b.data_ptr(), 1, _lib.stream_ptr()), "adjoint")
    ref = b.cpu().numpy()
    got = jhtb.adjoint_synthesis(v if spin else v[0], nside, lmax, spin).cpu().numpy().reshape(nc, -1)
    assert np.max(np.abs(got - ref)) <= TOL * np.max(np.abs(ref))
