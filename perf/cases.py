"""Timed cases of the framework: what its users have it do, over the range of sizes they use.

A HEALPix transform library is called in three ways: many small calls inside a fit or a test
(nside 8 to 64, where launches and latency count), ordinary map-making and power-spectrum
work (nside 128 to 1024, one map or a batch of simulations, forward and backward), and the
full-resolution transforms (nside 2048, lmax 4096).  Beside these stand the iterated
solvers (Jacobi analysis, the masked CG), the batched split-BF16 transforms, and the
off-grid transforms at arbitrary points.  lmax runs from nside / 2 to 3 nside - 1; nside is
a power of two in most work, any whole number is allowed.

`exact` restates every case in plain torch in 64 bits (its own recursions, torch.fft for the
rings, a direct sum for the off-grid points), except where that takes longer than a user
of this file wants to wait.
"""

from __future__ import annotations

import math

import numpy as np
import torch

import jht_b200 as jht


# ---------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------
def listed():
    return [
        # the smallest call: one low-resolution map, bound by launches and host work
        {"name": "synth_n16_l24_s0", "kind": "synthesis", "nside": 16, "lmax": 24, "spin": 0, "batch": 1, "precision": "fp64"},
        # a small polarised map back to coefficients, as a fit evaluates it
        {"name": "adjoint_n64_l96_s2", "kind": "adjoint", "nside": 64, "lmax": 96, "spin": 2, "batch": 1, "precision": "fp64"},
        # one gradient step of a small polarised model: forward and backward through autograd
        {"name": "grad_n128_l256_s2", "kind": "grad", "nside": 128, "lmax": 256, "spin": 2, "batch": 1, "precision": "fp64"},
        # a resolution that is no power of two and an odd band limit above 2 nside: ragged tiles, every ring a chirp-z
        {"name": "pair_n300_l641_s0", "kind": "pair", "nside": 300, "lmax": 641, "spin": 0, "batch": 1, "precision": "fp64"},
        # a batch of polarised simulations in FP64, both directions
        {"name": "pair_b8_n256_l512_s2", "kind": "pair", "nside": 256, "lmax": 512, "spin": 2, "batch": 8, "precision": "fp64"},
        # the iterated estimate of one temperature map's coefficients: seven transforms and the residuals
        {"name": "analysis_n1024_l2048_s0", "kind": "analysis", "nside": 1024, "lmax": 2048, "spin": 0, "batch": 1, "precision": "fp64", "niter": 3},
        # the full-resolution polarised transform and its gradient: the benchmark's step
        {"name": "grad_n2048_l4096_s2", "kind": "grad", "nside": 2048, "lmax": 4096, "spin": 2, "batch": 1, "precision": "fp64"},
        # Monte-Carlo batches on the tensor cores, many small maps and fewer large polarised ones
        {"name": "pair_b64_n512_l1024_s0_bf16x3", "kind": "pair", "nside": 512, "lmax": 1024, "spin": 0, "batch": 64, "precision": "bf16x3"},
        {"name": "pair_b16_n1024_l2048_s2_bf16x3", "kind": "pair", "nside": 1024, "lmax": 2048, "spin": 2, "batch": 16, "precision": "bf16x3"},
        # a cut-sky deconvolution of four maps, eight CG steps
        {"name": "cg_b4_n256_l512_s0", "kind": "cg", "nside": 256, "lmax": 512, "spin": 0, "batch": 4, "precision": "fp64", "niter": 8},
        # off-grid evaluation and its transpose: a catalogue's worth of points, and a map's worth
        {"name": "offgrid_l200_p20000_s0", "kind": "offgrid", "lmax": 200, "spin": 0, "points": 20000},
        {"name": "offgrid_l1024_p3M_s2", "kind": "offgrid", "lmax": 1024, "spin": 2, "points": 3000000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["synthesis", "adjoint", "grad", "pair", "pair", "analysis", "cg", "offgrid"])
    spin = rng.choice([0, 2])
    if kind == "offgrid":
        return {"kind": kind, "lmax": _log_int(rng, 60, 1024), "spin": spin, "points": _log_int(rng, 1000, 3000000)}
    top = 256 if kind == "cg" else 1024
    # maps at a power of two, or at any other resolution
    nside = 2 ** rng.randint(3, int(math.log2(top))) if rng.random() < 0.6 else _log_int(rng, 8, top)
    lmax = min(2048, max(4, rng.randint(nside // 2, 3 * nside - 1)))
    case = {"kind": kind, "nside": nside, "lmax": lmax, "spin": spin, "batch": 1, "precision": "fp64"}
    if kind in ("pair", "cg") and nside <= 512:
        case["batch"] = rng.randint(1, 16)
    if kind == "pair" and 64 <= nside <= 512 and rng.random() < 0.4:
        case["precision"], case["batch"] = "bf16x3", rng.randint(2, 32)
    if kind in ("analysis", "cg"):
        case["niter"] = rng.randint(1, 4) if kind == "analysis" else rng.randint(3, 8)
    return case


# ---------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------
_DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _ells(lmax):
    """(l, m) of every packed coefficient, on the device."""
    l, m = torch.meshgrid(torch.arange(lmax + 1, device=_DEV), torch.arange(lmax + 1, device=_DEV), indexing="xy")
    keep = l >= m  # row m, column l: the packed order
    return l[keep], m[keep]


def _alm(gen, batch, lmax, spin):
    """Coefficients with an amplitude falling as 1 / (l + 10), real at m = 0, zero below the spin."""
    nc = 1 if spin == 0 else 2
    l, m = _ells(lmax)
    a = torch.randn((batch, nc, l.numel()), dtype=torch.complex128, device=_DEV, generator=gen)
    a = torch.where(m == 0, a.real.to(torch.complex128), a) / (l + 10.0)
    return torch.where(l < abs(spin), torch.zeros_like(a), a)


def _z(nside):
    """cos(theta) of the rings, north to south."""
    i = torch.arange(1, 2 * nside + 1, device=_DEV, dtype=torch.float64)
    z = torch.where(i < nside, 1.0 - i * i / (3.0 * nside * nside), 4.0 / 3.0 - 2.0 * i / (3.0 * nside))
    return z, torch.cat([z, -z[:-1].flip(0)])


def _ring_sizes(nside):
    r = torch.arange(1, 4 * nside, device=_DEV)
    return 4 * torch.minimum(torch.minimum(r, 4 * nside - r), torch.full_like(r, nside))


def _maps(gen, batch, nside, spin):
    """Noise on a smooth large-scale signal."""
    nc = 1 if spin == 0 else 2
    v = torch.randn((batch, nc, 12 * nside * nside), dtype=torch.float64, device=_DEV, generator=gen)
    z = torch.repeat_interleave(_z(nside)[1], _ring_sizes(nside))
    return v + torch.cos(3.0 * z) + 0.5 * z


def _points(gen, n):
    """(theta, phi) uniform on the sphere."""
    u = torch.rand((n, 2), dtype=torch.float64, device=_DEV, generator=gen)
    return torch.stack([torch.arccos(1.0 - 2.0 * u[:, 0]), 2.0 * math.pi * u[:, 1]], dim=1)


def _mask(nside):
    """A galactic cut: pixels with |cos theta| < 0.34 removed."""
    z = torch.repeat_interleave(_z(nside)[1], _ring_sizes(nside))
    return (z.abs() >= 0.34).to(torch.float64)


def prepare(case, seed):
    gen = torch.Generator(device=_DEV)
    gen.manual_seed(1000003 * int(seed) + 17)
    kind, spin = case["kind"], case["spin"]
    state = {"case": case}
    if kind == "offgrid":
        state["alm"] = _alm(gen, 1, case["lmax"], spin)[0]
        state["loc"] = _points(gen, case["points"])
        state["field"] = torch.randn((1 if spin == 0 else 2, case["points"]), dtype=torch.float64, device=_DEV, generator=gen)
        return state
    nside, lmax, b = case["nside"], case["lmax"], case["batch"]
    amp = torch.ones((b, 1, 1), dtype=torch.float64, device=_DEV)
    if b > 1:  # maps of one batch differ in amplitude
        amp = 10.0 ** (2.0 * torch.rand((b, 1, 1), dtype=torch.float64, device=_DEV, generator=gen) - 1.0)
    if kind in ("synthesis", "grad", "pair"):
        state["alm"] = amp * _alm(gen, b, lmax, spin)
    if kind in ("adjoint", "grad", "pair", "analysis", "cg"):
        state["maps"] = amp * _maps(gen, b, nside, spin)
    if kind == "cg":
        state["mask"] = _mask(nside)
    return state


# ---------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------
def _one(t, spin):
    """The public shape of one map's tensors (spin 0 has no component axis)."""
    return t[0, 0] if spin == 0 else t[0]


def run(state):
    case = state["case"]
    kind, lmax, spin = case["kind"], case["lmax"], case["spin"]
    if kind == "offgrid":
        a = state["alm"][0] if spin == 0 else state["alm"]
        f = state["field"][0] if spin == 0 else state["field"]
        return (jht.synthesis_general(a, state["loc"], spin=spin, lmax=lmax),
                jht.adjoint_synthesis_general(f, state["loc"], spin=spin, lmax=lmax))
    nside, precision = case["nside"], case["precision"]
    if kind == "synthesis":
        return jht.synthesis(_one(state["alm"], spin), nside, lmax, spin)
    if kind == "adjoint":
        return jht.adjoint_synthesis(_one(state["maps"], spin), nside, lmax, spin)
    if kind == "grad":
        a = _one(state["alm"], spin).detach().requires_grad_(True)
        m = jht.synthesis(a, nside, lmax, spin)
        m.backward(_one(state["maps"], spin))
        return m.detach(), a.grad
    if kind == "pair":
        a, v = state["alm"], state["maps"]
        if spin == 0:
            a, v = a[:, 0], v[:, 0]
        return (jht.synthesis_batch(a, nside, lmax, spin, precision=precision),
                jht.adjoint_synthesis_batch(v, nside, lmax, spin, precision=precision))
    if kind == "analysis":
        return jht.analysis(_one(state["maps"], spin), nside, lmax, spin, niter=case["niter"])
    v = state["maps"][:, 0] if spin == 0 else state["maps"]
    return jht.deconvolve_batch(v, state["mask"], nside, lmax, spin, max_iter=case["niter"])


def _transforms(case):
    """How many S or S^T one pass runs per map."""
    return {"synthesis": 1, "adjoint": 1, "grad": 2, "pair": 2, "analysis": 1 + 2 * case.get("niter", 0),
            "cg": 1 + 2 * case.get("niter", 0)}[case["kind"]]


def work(case):
    nc = 1 if case["spin"] == 0 else 2
    lmax = case["lmax"]
    k = (lmax + 1) * (lmax + 2) // 2
    per = 8 if nc == 1 else 24  # the recursion and the sums of one (l, m, ring pair)
    if case["kind"] == "offgrid":
        p = case["points"]
        nt, w = 2 * (lmax + 1), 14
        grid = (2 * nt) * (2 * (2 * lmax + 1))
        return {"bytes": 2 * 16 * nc * k + 2 * 8 * (nc + 2) * p,
                "flops": 2 * (per * k * ((lmax + 1) // 2) + 5 * grid * math.log2(grid) + 4 * w * w * p)}
    nside, b = case["nside"], case["batch"]
    npix = 12 * nside * nside
    n = _transforms(case)
    io = {"synthesis": (1, 1), "adjoint": (1, 1), "grad": (2, 2), "pair": (2, 2), "analysis": (1, 1), "cg": (1, 1)}[case["kind"]]
    return {"bytes": b * nc * (io[0] * 16 * k + io[1] * 8 * npix),
            "flops": b * n * (per * k * 2 * nside + nc * 2.5 * npix * math.log2(4 * nside))}


# ---------------------------------------------------------------------------------------
# the same in plain torch, 64 bits
# ---------------------------------------------------------------------------------------
def _columns(x, lmax, spin):
    """Yields (l, rows): rows[h][m, ring] for m <= l, the orthonormal spin-weighted functions
    of degree l at cos(theta) = x (h = 0: +spin, h = 1: -spin), by the three-term recursion
    in l on values mant * 2^(512 e); what is still scaled is far below rounding and given as 0."""
    M, dev = lmax + 1, x.device
    m = torch.arange(M, device=dev, dtype=torch.float64)[:, None]
    lmin = torch.clamp(m, min=float(abs(spin)))
    states = []
    for s in ((0,) if spin == 0 else (spin, -spin)):
        if spin == 0:
            lg = 0.5 * (torch.lgamma(2 * m + 2) - 2 * m * math.log(2.0) - 2 * torch.lgamma(m + 1) - math.log(4 * math.pi))
            lg = lg + torch.where(m > 0, m * 0.5 * torch.log((1 - x) * (1 + x)), torch.zeros_like(x))
            sign = 1.0 - 2.0 * (m % 2)
        else:  # d^{lmin}_{-m, s}: a single term
            k0 = torch.clamp(-m - s, min=0.0)
            pc, ps = 2 * lmin - 2 * k0 - m - s, 2 * k0 + m + s
            lg = 0.5 * (torch.lgamma(lmin - m + 1) + torch.lgamma(lmin + m + 1) + torch.lgamma(lmin + s + 1) + torch.lgamma(lmin - s + 1))
            lg = lg - torch.lgamma(k0 + 1) - torch.lgamma(lmin - m - k0 + 1) - torch.lgamma(lmin - s - k0 + 1) - torch.lgamma(k0 + m + s + 1)
            lg = lg + 0.5 * torch.log((2 * lmin + 1) / (4 * math.pi))
            for p, h in ((pc, (1 + x) / 2), (ps, (1 - x) / 2)):
                lg = lg + torch.where(p > 0, p * 0.5 * torch.log(h), torch.zeros_like(x))
            sign = (1.0 - 2.0 * (k0 % 2)) * (1.0 - 2.0 * (m % 2))
        lg = torch.clamp(lg / math.log(2.0), min=-1e7)
        e = torch.clamp(torch.floor((lg + 256) / 512), max=0.0)
        states.append([sign * torch.exp2(lg - 512 * e), torch.zeros_like(lg), e, s])
    for l in range(abs(spin), lmax + 1):
        n = l + 1
        rows = []
        for st in states:
            u, prev, e, s = st
            if l > abs(spin):  # every order that has started moves one degree; order l starts now
                o = n - 1
                mo, j = m[:o], float(l)
                c1 = torch.sqrt((j * j - mo * mo) * (j * j - s * s) / (j * j * (4 * j * j - 1)))
                i = j - 1
                c0 = torch.sqrt(torch.clamp((i * i - mo * mo) * (i * i - s * s) / (max(i * i, 1.0) * (4 * i * i - 1)), min=0.0)) if i > 0 else torch.zeros_like(mo)
                add = s * mo / (i * (i + 1)) if s else 0.0
                new = ((x + add) * u[:o] - c0 * prev[:o]) / c1
                prev[:o] = u[:o]
                u[:o] = new
                if l % 8 == 0:
                    big = (e[:o] < 0) & (u[:o].abs() > 2.0 ** 256)
                    f = torch.exp2(-512.0 * big.to(torch.float64))
                    u[:o] *= f
                    prev[:o] *= f
                    e[:o] += big
            rows.append(torch.where(e[:n] < 0, 0.0, u[:n]))
        yield l, rows


def _col(lmax, l):
    """Packed places of (l, m) for m = 0..l."""
    m = torch.arange(l + 1, device=_DEV)
    return m * (2 * lmax + 1 - m) // 2 + l


def _rings_of(a, x, lmax, spin, mirror):
    """(B, nc, K) -> F[channel] (B, M, ring): the sums over l at x, and with `mirror` at -x."""
    B, M, T = a.shape[0], lmax + 1, x.numel()
    nc = 1 if spin == 0 else 2
    F = torch.zeros((2 if mirror else 1, nc, B, M, T), dtype=torch.complex128, device=a.device)
    for l, rows in _columns(x, lmax, spin):
        al = a[:, :, _col(lmax, l)][..., None]
        par = (1.0 - 2.0 * ((torch.arange(l + 1, device=a.device) + l) % 2))[:, None]
        if spin == 0:
            v = al[:, 0] * rows[0]
            F[0, 0, :, : l + 1] += v
            if mirror:
                F[1, 0, :, : l + 1] += par * v
        else:
            cp, cm = -(al[:, 0] + 1j * al[:, 1]), -(al[:, 0] - 1j * al[:, 1])
            F[0, 0, :, : l + 1] += cp * rows[0]
            F[0, 1, :, : l + 1] += cm * rows[1]
            if mirror:
                F[1, 0, :, : l + 1] += cp * (par * rows[1])
                F[1, 1, :, : l + 1] += cm * (par * rows[0])
    return F


def _alm_of(V, x, lmax, spin, mirror):
    """The transpose: V (side, channel, B, M, ring) -> (p, m) sums (nc, B, K)."""
    nc, B = V.shape[1], V.shape[2]
    out = torch.zeros((nc, B, (lmax + 1) * (lmax + 2) // 2), dtype=torch.complex128, device=x.device)
    for l, rows in _columns(x, lmax, spin):
        par = (1.0 - 2.0 * ((torch.arange(l + 1, device=x.device) + l) % 2))[:, None]
        for c in range(nc):
            s = (V[0, c, :, : l + 1] * rows[c]).sum(-1)
            if mirror:
                s = s + (V[1, c, :, : l + 1] * (par * rows[nc - 1 - c])).sum(-1)
            out[c][:, _col(lmax, l)] = s
    return out


def _ring_groups(nside):
    """(ring numbers, their length, first azimuth, first pixels) for rings alike."""
    n = _ring_sizes(nside).cpu().numpy()
    start = np.concatenate([[0], np.cumsum(n)[:-1]])
    r = np.arange(1, 4 * nside)
    belt = (r >= nside) & (r <= 3 * nside)
    shifted = ~belt | ((r - nside) % 2 == 0)
    groups = [(np.array([i - 1, 4 * nside - 1 - i]), 4 * i, True) for i in range(1, nside)]
    groups += [(np.nonzero(belt & (shifted == s))[0], 4 * nside, bool(s)) for s in (True, False)]
    return [(g, N, math.pi / N if s else 0.0, start[g]) for g, N, s in groups if len(g)]


def _synthesis(a, nside, lmax, spin):
    """(B, nc, K) -> (B, nc, Npix)."""
    B, T = a.shape[0], 2 * nside
    if spin == 0:
        a = torch.cat([a[..., : lmax + 1].real.to(a.dtype), a[..., lmax + 1:]], dim=-1)
    F = _rings_of(a, _z(nside)[0], lmax, spin, True)
    F = torch.cat([F[0], F[1][..., : T - 1].flip(-1)], dim=-1)  # (nc, B, M, rings)
    out = torch.empty((B, 1 if spin == 0 else 2, 12 * nside * nside), dtype=torch.float64, device=a.device)
    m = torch.arange(lmax + 1, device=a.device)
    for g, N, phi0, start in _ring_groups(nside):
        ph = torch.exp(1j * (m.double() * phi0))[:, None]
        gi = torch.as_tensor(g, device=a.device)
        D = torch.zeros((B, N, len(g)), dtype=torch.complex128, device=a.device)
        D.index_add_(1, m % N, F[0][..., gi] * ph)
        D.index_add_(1, (-m[1:]) % N, (F[-1][..., gi] * ph)[:, 1:].conj())
        v = torch.fft.ifft(D, dim=1) * N
        pix = (torch.as_tensor(start, device=a.device)[None, :] + torch.arange(N, device=a.device)[:, None])
        out[:, 0, pix] = v.real
        if spin:
            out[:, 1, pix] = v.imag
    return out


def _adjoint(v, nside, lmax, spin):
    """(B, nc, Npix) -> (B, nc, K)."""
    B, T, M = v.shape[0], 2 * nside, lmax + 1
    nc = 1 if spin == 0 else 2
    V = torch.empty((nc, B, M, 4 * nside - 1), dtype=torch.complex128, device=v.device)
    m = torch.arange(M, device=v.device)
    for g, N, phi0, start in _ring_groups(nside):
        ph = torch.exp(-1j * (m.double() * phi0))[:, None]
        gi = torch.as_tensor(g, device=v.device)
        pix = (torch.as_tensor(start, device=v.device)[None, :] + torch.arange(N, device=v.device)[:, None])
        w = torch.fft.fft(torch.complex(v[:, 0, pix], v[:, 1, pix] if spin else torch.zeros_like(v[:, 0, pix])), dim=1)
        V[0][..., gi] = w[:, m % N] * ph
        if spin:
            V[1][..., gi] = w[:, (-m) % N].conj() * ph
    south = torch.zeros((nc, B, M, T), dtype=torch.complex128, device=v.device)
    south[..., : T - 1] = V[..., T:].flip(-1)
    s = _alm_of(torch.stack([V[..., :T], south]), _z(nside)[0], lmax, spin, True)
    if spin == 0:
        return s[0][:, None]
    return torch.stack([0.5 * (-s[0] - s[1]), 0.5j * (s[0] - s[1])], dim=1)


def _pixel_weights(nside):
    """4 pi / Npix (1 + w_ring), w the least-norm correction that integrates even degrees to 2 nside."""
    z, n = _z(nside)[0].cpu().numpy(), _ring_sizes(nside).cpu().numpy()[: 2 * nside].astype(float)
    mult = np.full(2 * nside, 2.0)
    mult[-1] = 1.0
    A = ((mult * n)[:, None] * np.polynomial.legendre.legvander(z, 2 * nside)[:, ::2]).T
    rhs = -A.sum(axis=1)
    rhs[0] += 12 * nside * nside
    w = torch.as_tensor(np.linalg.lstsq(A, rhs, rcond=None)[0], device=_DEV)
    w = torch.cat([w, w[:-1].flip(0)])
    return 4 * math.pi / (12 * nside * nside) * (1 + torch.repeat_interleave(w, _ring_sizes(nside)))


def _deconvolved(v, mask, nside, lmax, spin, steps):
    """CG on S^T (mask W) S a = S^T (mask W) m in the metric (2 - delta_m0), tolerance 1e-8."""
    w = mask * _pixel_weights(nside)
    l, m = _ells(lmax)
    g = torch.where(m == 0, 1.0, 2.0) * (l >= abs(spin))

    def dot(p, q):
        return (g * (p.conj() * q).real).sum((1, 2), keepdim=True)

    def low(a):
        a = torch.where(m == 0, a.real.to(a.dtype), a)
        return torch.where(l < abs(spin), torch.zeros_like(a), a)

    r = low(_adjoint(w * v, nside, lmax, spin))
    a, p, gam = torch.zeros_like(r), r, dot(r, r)
    stop = 1e-16 * gam
    for _ in range(steps):
        q = low(_adjoint(w * _synthesis(p, nside, lmax, spin), nside, lmax, spin))
        on = gam > stop
        alpha = torch.where(on, gam / dot(p, q), 0.0)
        a, r = a + alpha * p, r - alpha * q
        new = dot(r, r)
        p = torch.where(on, r + new / gam * p, p)
        gam = torch.where(on, new, gam)
    return a


def exact(case, seed):
    kind, lmax, spin = case["kind"], case["lmax"], case["spin"]
    if kind == "offgrid":
        if lmax * lmax * case["points"] > 3e9:
            return None
        s = prepare(case, seed)
        theta, phi = s["loc"][:, 0], s["loc"][:, 1]
        ph = torch.exp(1j * torch.arange(lmax + 1, device=_DEV)[:, None] * phi)
        a, f = s["alm"][None], s["field"]
        if spin == 0:
            a = torch.cat([a[..., : lmax + 1].real.to(a.dtype), a[..., lmax + 1:]], dim=-1)
        F = _rings_of(a, torch.cos(theta), lmax, spin, False)[0][:, 0]
        z = (F[0] * ph).sum(0) + (F[-1] * ph)[1:].conj().sum(0)
        fc = f[0].to(torch.complex128) if spin == 0 else torch.complex(f[0], f[1])
        V = torch.stack([fc * ph.conj()] + ([fc.conj() * ph.conj()] if spin else []))[None, :, None]
        b = _alm_of(V, torch.cos(theta), lmax, spin, False)[:, 0]
        if spin == 0:
            return z.real, b[0]
        b[1][: lmax + 1] = 0  # at m = 0 the one channel carries the whole sum
        b = torch.stack([-b[0] - b[1], 1j * (b[0] - b[1])])
        b[:, lmax + 1:] *= 0.5
        return torch.stack([z.real, z.imag]), b
    nside, b = case["nside"], case["batch"]
    nc = 1 if spin == 0 else 2
    if (lmax + 1) ** 2 * nside * nc * b * _transforms(case) > 6e11 or (lmax + 1) * nside * b * nc > 6e8:
        return None
    s = prepare(case, seed)
    out = (lambda t: t[:, 0]) if spin == 0 else (lambda t: t)
    if kind in ("synthesis", "grad"):
        m = _one(_synthesis(s["alm"], nside, lmax, spin), spin)
        if kind == "synthesis":
            return m
        g = _adjoint(s["maps"], nside, lmax, spin)[0]
        order = _ells(lmax)[1]
        if spin == 0:
            return m, torch.where(order == 0, 1.0, 2.0) * g[0]
        e, bb = g[0, : lmax + 1].real.clone(), g[1, : lmax + 1].real.clone()
        g = 2.0 * g
        g[0, : lmax + 1], g[1, : lmax + 1] = torch.complex(e, bb), torch.complex(bb, -e)
        return m, g
    if kind == "adjoint":
        return _one(_adjoint(s["maps"], nside, lmax, spin), spin)
    if kind == "pair":
        return out(_synthesis(s["alm"], nside, lmax, spin)), out(_adjoint(s["maps"], nside, lmax, spin))
    if kind == "analysis":
        w = _pixel_weights(nside)
        a = _adjoint(w * s["maps"], nside, lmax, spin)
        for _ in range(case["niter"]):
            a = a + _adjoint(w * (s["maps"] - _synthesis(a, nside, lmax, spin)), nside, lmax, spin)
        return _one(a, spin)
    return out(_deconvolved(s["maps"], s["mask"], nside, lmax, spin, case["niter"]))
