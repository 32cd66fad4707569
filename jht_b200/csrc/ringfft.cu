// Azimuthal stage: per-ring phase shift, m -> k fold and length-N DFT (sm_100a).
//
// jht (healpix.py:280-355) groups rings by length and emits one FFT per distinct
// length, with scatter-adds for the m -> k fold.  Here a transform takes two rows of ring
// spectra, P and M, to two real pixel streams x, y (and back):
//   synthesis  D[k] = sum_{m = k mod N} P_m e^{i m phi0} + sum_{m>=1, -m = k mod N} conj(M_m e^{i m phi0})
//              x[j] + i y[j] = sum_k D[k] e^{+2 pi i jk/N}
//   adjoint    W[k] = sum_j (x[j] + i y[j]) e^{-2 pi i jk/N}
//              P_m = W[m mod N] e^{-i m phi0},  M_m = conj(W[-m mod N]) e^{-i m phi0}
// Spin 2: P and M are the +2 and -2 channels of one ring, x = Q and y = U.  Spin 0: one
// complex transform serves a northern ring and its southern mirror (same length and
// azimuth): the rows hold P = F_north + i F_south and M = F_north - i F_south (the Legendre
// kernels write and read that form), x is the northern ring and y the southern one, so the
// stage runs half the transforms of one real ring each.
//
// On the HEALPix grid phi0 is 0 or pi / N and N = 4 i (healpix.py:107-140), so every factor is
// e^{i pi a / N} for an integer a.  A ring runs as pieces, one transform per output residue
// class (decimation in frequency on the input):
//   direct   N a power of two (the belt at a power-of-two nside): Q = N / 4096 pieces (1 up
//            to 4096 points) of one FFT each;
//   chirp    every other ring: four pieces of length i, each a chirp-z transform
//            (_azimuth.py:150-191) of P >= 2 i - 1 points: FFT, chirp spectrum, inverse FFT;
//   small    N <= 128: a plain sum over k with the ring's 2 N roots of unity in shared memory.
// An FFT keeps 16 points per thread in registers: radix-16 passes (one smaller last pass),
// decimation in frequency forward and its transpose backward, so that neither needs a
// reordering pass and the chirp spectrum is applied in registers between the two; a pass
// writes back where it read, so an exchange costs one barrier.
#include <cuda_runtime.h>

#include <algorithm>

#include "jhtb_internal.cuh"

namespace jhtb {
namespace {

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ double2 cmulc(double2 a, double2 b) {  // a conj(b)
    return make_double2(fma(a.x, b.x, a.y * b.y), fma(a.y, b.x, -a.x * b.y));
}
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 conjd(double2 a) { return make_double2(a.x, -a.y); }
__device__ __forceinline__ double2 zero2() { return make_double2(0.0, 0.0); }

// The synthesis reads each ring's spectrum once: past the L1, which so keeps the FFT passes'
// twiddles and the chirp factors (64 maps at nside 512: 2.05 -> 1.93 ms).  Pixels and tables gain
// nothing from it: four lanes share a pixel's sector, and neighbouring rings their tables.
__device__ __forceinline__ double2 ld_stream(const double2 *p) {
    double2 v;
    asm("ld.global.L1::no_allocate.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
    return v;
}

// e^{i pi a / N}, a taken modulo 2 N and folded to the first octant in integers, so the one
// rounding of the argument is that of a value <= 1/4.
__device__ __forceinline__ double2 cis_pi(long long a, int N) {
    const int n2 = 2 * N;
    int r = (int)(a % n2);
    if (r < 0) r += n2;
    const bool neg = r > N;  // lower half plane
    if (neg) r = n2 - r;
    const bool flip = 2 * r > N;  // second quadrant
    if (flip) r = N - r;
    const bool swap = 4 * r > N;  // second octant: pi/2 - angle = pi (N - 2 r) / (2 N)
    double s, c;
    if (swap) sincospi((double)(N - 2 * r) / (double)n2, &c, &s);
    else sincospi((double)r / (double)N, &s, &c);
    return make_double2(flip ? -c : c, neg ? -s : s);
}

// ---------------------------------------------------------------------------------
// register FFTs
// ---------------------------------------------------------------------------------
// cos and sin of k pi / 8, k < 8 (the 16th roots of unity)
__host__ __device__ constexpr double cos16(int k) {
    return k == 0 ? 1.0 : k == 1 ? 0.9238795325112867 : k == 2 ? 0.7071067811865476 : k == 3 ? 0.3826834323650898
         : k == 4 ? 0.0 : k == 5 ? -0.3826834323650898 : k == 6 ? -0.7071067811865476 : -0.9238795325112867;
}
__host__ __device__ constexpr double sin16(int k) { return cos16(k <= 4 ? 4 - k : k - 4); }
__host__ __device__ constexpr int brev_ct(int i, int bits) {
    int r = 0;
    for (int b = 0; b < bits; ++b) r |= ((i >> b) & 1) << (bits - 1 - b);
    return r;
}
__host__ __device__ constexpr int ilog2_ct(int n) { return n <= 1 ? 0 : 1 + ilog2_ct(n / 2); }

// R-point DFT of v[O .. O + R) in registers (R <= 16), natural order in and out: radix-2 DIT
// after a bit reversal, all indices and roots fixed at compile time.  DIR = -1:
// e^{-2 pi i jk/R}; +1: e^{+...}.  HALF: the upper half of the inputs is zero, so the first
// stage copies.
template <int R, int O, int DIR, int LEN, int I, int K>
__device__ __forceinline__ void rf_bfly(double2 (&v)[16]) {
    constexpr int h = LEN / 2, ROOT = K * (16 / LEN);  // e^{DIR 2 pi i ROOT / 16}
    const double2 a = v[O + I + K];
    double2 b = v[O + I + K + h];
    if constexpr (ROOT == 4) b = DIR > 0 ? make_double2(-b.y, b.x) : make_double2(b.y, -b.x);
    else if constexpr (ROOT == 2) {  // (1 + i DIR) / sqrt 2
        constexpr double c = 0.7071067811865476;
        b = DIR > 0 ? make_double2(c * (b.x - b.y), c * (b.x + b.y)) : make_double2(c * (b.x + b.y), c * (b.y - b.x));
    } else if constexpr (ROOT == 6) {
        constexpr double c = 0.7071067811865476;
        b = DIR > 0 ? make_double2(-c * (b.x + b.y), c * (b.x - b.y)) : make_double2(c * (b.y - b.x), -c * (b.x + b.y));
    } else if constexpr (ROOT != 0) b = cmul(b, make_double2(cos16(ROOT), DIR * sin16(ROOT)));
    v[O + I + K] = cadd(a, b);
    v[O + I + K + h] = csub(a, b);
}
template <int R, int O, int DIR, int LEN, int IDX>
__device__ __forceinline__ void rf_stage(double2 (&v)[16]) {
    if constexpr (IDX < R / 2) {
        constexpr int h = LEN / 2;
        rf_bfly<R, O, DIR, LEN, (IDX / h) * LEN, IDX % h>(v);
        rf_stage<R, O, DIR, LEN, IDX + 1>(v);
    }
}
template <int R, int O, int DIR, int LEN>
__device__ __forceinline__ void rf_stages(double2 (&v)[16]) {
    if constexpr (LEN <= R) {
        rf_stage<R, O, DIR, LEN, 0>(v);
        rf_stages<R, O, DIR, LEN * 2>(v);
    }
}
template <int R, int O, int I>
__device__ __forceinline__ void rf_bitrev(double2 (&v)[16]) {
    if constexpr (I < R) {
        constexpr int J = brev_ct(I, ilog2_ct(R));
        if constexpr (J > I) {
            const double2 t = v[O + I];
            v[O + I] = v[O + J];
            v[O + J] = t;
        }
        rf_bitrev<R, O, I + 1>(v);
    }
}
template <int R, int DIR, bool HALF, int O = 0>
__device__ __forceinline__ void reg_fft(double2 (&v)[16]) {  // every group of R points of v
    if constexpr (O < 16) {
        rf_bitrev<R, O, 0>(v);
        if constexpr (HALF) {
#pragma unroll
            for (int q = 0; q < R; q += 2) v[O + q + 1] = v[O + q];
            rf_stages<R, O, DIR, 4>(v);
        } else {
            rf_stages<R, O, DIR, 2>(v);
        }
        reg_fft<R, DIR, HALF, O + R>(v);
    }
}

// ---------------------------------------------------------------------------------
// FFT of P = 2^LOGP points by TP = P / 16 threads (thread t), 16 points each in registers
// ---------------------------------------------------------------------------------
template <int LOGP>
struct Fft {
    static constexpr int P = 1 << LOGP, TP = P / 16, NP = (LOGP + 3) / 4;
    static constexpr int RLAST = 1 << (LOGP - 4 * (NP - 1));  // radix of the last pass
    // shared-memory layout: pads after every P / 16 points (and every 32 at 8192) spread the
    // strided accesses of the passes over the 16-byte bank groups
    static constexpr int PAD = LOGP == 10 ? 5 : (LOGP == 9 ? 3 : 1);
    static __device__ __forceinline__ int pidx(int i) {
        int r = i + PAD * (i >> (LOGP - 4));
        if (LOGP == 13) r += 2 * (i >> 5);
        return r;
    }
    static constexpr int LEN = P + 16 * PAD + (LOGP == 13 ? P / 16 : 0);

    // the output digits (k1 least significant) of butterfly c of the last pass -> its block
    static __device__ __forceinline__ int rev(int c) {
        if (NP <= 2) return c;
        if (NP == 3) return ((c & 15) << 4) | (c >> 4);
        return ((c & 15) << 8) | (((c >> 4) & 15) << 4) | (c >> 8);
    }
    // position of point q of this thread in pass PASS
    template <int PASS>
    static __device__ __forceinline__ int pos(int t, int q) {
        constexpr int BLOG = LOGP - 4 * PASS;
        if constexpr (PASS == NP - 1) {
            return pidx((rev(t + TP * (q / RLAST)) * RLAST) + q % RLAST);
        } else {
            constexpr int SLOG = BLOG - 4;
            return pidx(((t >> SLOG) << BLOG) + (t & ((1 << SLOG) - 1)) + (q << SLOG));
        }
    }
    // multiply point q of pass PASS by e^{+-2 pi i j q / B}, B the pass's block: four table
    // entries and products of at most three of them
    template <int PASS, bool PLUS>
    static __device__ __forceinline__ void twiddle(double2 (&v)[16], int t, const double2 *__restrict__ tw) {
        constexpr int BLOG = LOGP - 4 * PASS, SLOG = BLOG - 4;
        const int at = tw_offset(BLOG) + 4 * (t & ((1 << SLOG) - 1));
        if (!JHTB_IN(at + 3, kTwLen, 107)) return;
        const double2 *T = tw + at;  // e^{-2 pi i j {1, 4, 8, 12} / B}
        const double2 w1 = __ldg(&T[0]);
        const double2 w2 = cmul(w1, w1), w3 = cmul(w2, w1);
        v[1] = PLUS ? cmulc(v[1], w1) : cmul(v[1], w1);
        v[2] = PLUS ? cmulc(v[2], w2) : cmul(v[2], w2);
        v[3] = PLUS ? cmulc(v[3], w3) : cmul(v[3], w3);
#pragma unroll
        for (int a = 4; a < 16; a += 4) {
            const double2 wa = __ldg(&T[a / 4]);
            v[a] = PLUS ? cmulc(v[a], wa) : cmul(v[a], wa);
            const double2 u1 = cmul(wa, w1), u2 = cmul(wa, w2), u3 = cmul(wa, w3);
            v[a + 1] = PLUS ? cmulc(v[a + 1], u1) : cmul(v[a + 1], u1);
            v[a + 2] = PLUS ? cmulc(v[a + 2], u2) : cmul(v[a + 2], u2);
            v[a + 3] = PLUS ? cmulc(v[a + 3], u3) : cmul(v[a + 3], u3);
        }
    }
    template <int PASS>
    static __device__ __forceinline__ void put(const double2 (&v)[16], double2 *buf, int t) {
#pragma unroll
        for (int q = 0; q < 16; ++q)
            if (JHTB_IN(pos<PASS>(t, q), LEN, 106)) buf[pos<PASS>(t, q)] = v[q];
    }
    template <int PASS>
    static __device__ __forceinline__ void get(double2 (&v)[16], const double2 *buf, int t) {
#pragma unroll
        for (int q = 0; q < 16; ++q) v[q] = JHTB_IN(pos<PASS>(t, q), LEN, 106) ? buf[pos<PASS>(t, q)] : zero2();
    }
    // forward, e^{+}: v[q] = x[t + TP q] in, v[g RLAST + q] = X[out_index(t, g RLAST + q)] out.
    // The buffer must be free on entry; `on` is false for idle threads, which only meet the barriers.
    template <int PASS, bool HALF>
    static __device__ __forceinline__ void forward_from(double2 (&v)[16], double2 *buf, int t, bool on,
                                                        const double2 *__restrict__ tw) {
        if constexpr (PASS == NP - 1) {
            if (on) reg_fft<RLAST, 1, HALF>(v);
        } else {
            if (on) {
                reg_fft<16, 1, HALF>(v);
                twiddle<PASS, true>(v, t, tw);
                put<PASS>(v, buf, t);
            }
            __syncthreads();
            if (on) get<PASS + 1>(v, buf, t);
            forward_from<PASS + 1, false>(v, buf, t, on, tw);
        }
    }
    template <bool HALF>
    static __device__ __forceinline__ void forward(double2 (&v)[16], double2 *buf, int t, bool on,
                                                   const double2 *__restrict__ tw) {
        forward_from<0, HALF>(v, buf, t, on, tw);
    }
    static __device__ __forceinline__ int out_index(int t, int q) { return t + TP * (q / RLAST) + (P / RLAST) * (q % RLAST); }
    // the transpose with e^{-}: takes forward's output layout back to v[q] = x[t + TP q] (times P)
    template <int PASS>
    static __device__ __forceinline__ void backward_from(double2 (&v)[16], double2 *buf, int t, bool on,
                                                         const double2 *__restrict__ tw) {
        if (on) {
            if constexpr (PASS == NP - 1) reg_fft<RLAST, -1, false>(v);
            else {
                twiddle<PASS, false>(v, t, tw);
                reg_fft<16, -1, false>(v);
            }
        }
        if constexpr (PASS > 0) {
            if (on) put<PASS>(v, buf, t);
            __syncthreads();
            if (on) get<PASS - 1>(v, buf, t);
            backward_from<PASS - 1>(v, buf, t, on, tw);
        }
    }
    static __device__ __forceinline__ void backward(double2 (&v)[16], double2 *buf, int t, bool on,
                                                    const double2 *__restrict__ tw) {
        backward_from<NP - 1>(v, buf, t, on, tw);
    }
};

// ---------------------------------------------------------------------------------
// the fold
// ---------------------------------------------------------------------------------
// D[k] without its ring phase: with m = k + jN in the first sum and m = jN - k in the second,
// e^{i m phi0} = (-1)^j e^{+-i pi k / N} when phi0 = pi / N, so
// D[k] = e^{i pi k / N} [sum_j (-1)^j P_{k+jN} + sum_j (-1)^j conj(M_{jN-k})];
// `shifted` selects the (-1)^j signs, the caller applies e^{i pi k / N}.  Aliases
// j = part, part + parts, ... only (the caller sums the parts in a fixed order).
__device__ __forceinline__ double2 fold_sum(const double2 *__restrict__ Pr, const double2 *__restrict__ Mr, int k,
                                            int N, int lmax, bool shifted, int part = 0, int parts = 1) {
    double2 d = zero2();
    const double flip = (shifted && (parts & 1)) ? -1.0 : 1.0;  // sign change per step of `parts` aliases
    double sg = (shifted && (part & 1)) ? -1.0 : 1.0;
    const int step = parts * N;
#pragma unroll 4
    for (int m = k + part * N; m <= lmax; m += step) {
        const double2 f = JHTB_IN(m, lmax + 1, 101) ? ld_stream(Pr + m) : zero2();
        d.x = fma(sg, f.x, d.x);
        d.y = fma(sg, f.y, d.y);
        sg *= flip;
    }
    // m = jN - k, j >= 1: alias j = 1 + part, 1 + part + parts, ...
    sg = (shifted && ((1 + part) & 1)) ? -1.0 : 1.0;
#pragma unroll 4
    for (int m = (1 + part) * N - k; m <= lmax; m += step) {
        const double2 f = JHTB_IN(m, lmax + 1, 102) ? ld_stream(Mr + m) : zero2();
        d.x = fma(sg, f.x, d.x);
        d.y = fma(-sg, f.y, d.y);
        sg *= flip;
    }
    return d;
}

// The same for a ring longer than lmax: at most one term per sum, no loop, so that a caller's
// unrolled loads are all issued before the first is used.
__device__ __forceinline__ double2 fold_one(const double2 *__restrict__ Pr, const double2 *__restrict__ Mr, int k,
                                            int N, int lmax, bool shifted) {
    const double2 p = (k <= lmax && JHTB_IN(k, lmax + 1, 101)) ? ld_stream(Pr + k) : zero2();
    const double2 q = (k >= 1 && N - k <= lmax && JHTB_IN(N - k, lmax + 1, 102)) ? ld_stream(Mr + (N - k)) : zero2();
    const double sg = shifted ? -1.0 : 1.0;
    return make_double2(fma(sg, q.x, p.x), fma(-sg, q.y, p.y));
}

// e^{i pi k / 4}, k mod 8
__device__ __forceinline__ double2 root8(int k) {
    constexpr double h = 0.70710678118654752440;
    const int q = k & 7;
    const double c = (q & 3) == 0 ? 1.0 : ((q & 3) == 2 ? 0.0 : h), s = (q & 3) == 0 ? 0.0 : ((q & 3) == 2 ? 1.0 : h);
    // q = 0: (1,0) 1: (h,h) 2: (0,1) 3: (-h,h) 4: (-1,0) ...
    const double cx = (q & 3) == 3 ? -h : c;
    return q & 4 ? make_double2(-cx, -s) : make_double2(cx, s);
}

// ---------------------------------------------------------------------------------
// what one CTA works on, shared by both directions
// ---------------------------------------------------------------------------------
struct RingArgs {
    const RingUnit *units;
    const RingDesc *rings;
    int lmax, M, nrows, spin;  // nrows: rows per channel
    long long npix;
    const double2 *tw;     // twiddles of the FFT passes (tw_offset)
    const double2 *bh;     // chirp spectra
    const double2 *ctab;   // per chirp length i: kRingCols columns of i factors
    long long bh_len, ctab_len;
    const double2 *belt;   // e^{i pi a / Nb}, a < 2 Nb, of the power-of-two belt
    int belt_n;            // Nb
};

// the two rows and the two pixel streams of a transform
struct Streams {
    size_t rowP, rowM;      // element offsets of m = 0
    long long offX, offY;   // pixel offsets; offY < 0: no second stream
};
__device__ __forceinline__ Streams streams_of(const RingArgs &a, int r, const RingDesc &rd) {
    Streams s;
    s.rowP = (size_t)r * a.M;
    s.offX = rd.start;
    if (a.spin) {
        s.rowM = (size_t)(a.nrows + r) * a.M;
        s.offY = a.npix + rd.start;
    } else {
        s.rowM = (size_t)(a.nrows - 1 - r) * a.M;
        s.offY = rd.mirror;
    }
    return s;
}

// shared-memory slots of one ring's staged points: [class s mod 4][k] with the classes two
// bank groups apart
__device__ __forceinline__ int class_stride(int i) { return ((i + 5) & ~7) + 2; }  // >= i, = 2 mod 8

// ring phase factor of a power-of-two ring: e^{i pi a / N} from the belt's table
__device__ __forceinline__ double2 belt_phase(const RingArgs &a, int e, int N) {
    const int i = (e & (2 * N - 1)) * (a.belt_n / N);
    return JHTB_IN(i, 2 * a.belt_n, 107) ? __ldg(&a.belt[i]) : zero2();
}

// A point W'[k] = W[k] e^{-i pi k / N} (shifted) of a spectrum to every order it appears in:
// P_{k+aN} = (-1)^a W'[k] and M_{aN-k} = (-1)^a conj(W'[k]) (a >= 1, and a = 0 for k = 0), the
// signs for shifted rings only.
__device__ __forceinline__ void scatter_orders(double2 *Pr, double2 *Mr, bool store_m, double2 w, int k, int N, int lmax,
                                               bool shifted) {
    double sg = 1.0;
    const double flip = shifted ? -1.0 : 1.0;
    for (int m = k; m <= lmax; m += N) {
        if (JHTB_IN(m, lmax + 1, 105)) Pr[m] = make_double2(sg * w.x, sg * w.y);
        sg *= flip;
    }
    if (!store_m) return;
    sg = k ? flip : 1.0;
    for (int m = k ? N - k : 0; m <= lmax; m += N) {
        if (JHTB_IN(m, lmax + 1, 105)) Mr[m] = make_double2(sg * w.x, -sg * w.y);
        sg *= flip;
    }
}

// Every order of a ring from its staged spectrum W'(k), in order of m by all `nt` threads.
template <typename Get>
__device__ __forceinline__ void gather_orders(double2 *Pr, double2 *Mr, bool store_m, int N, int lmax, bool shifted,
                                              int tid, int nt, Get W) {
    const unsigned magic = (unsigned)((0x100000000ull + N - 1) / N);  // m / N = umulhi(m, magic) for m N < 2^32
    for (int m = tid; m <= lmax; m += nt) {
        const int a = (int)__umulhi((unsigned)m, magic), k = m - a * N;
        const bool odd = shifted && (a & 1);
        double2 p = W(k);
        if (odd) p = make_double2(-p.x, -p.y);
        if (JHTB_IN(m, lmax + 1, 105)) Pr[m] = p;
        if (!store_m) continue;
        double2 q = conjd(W(k ? N - k : 0));
        if (shifted && (odd != (k != 0))) q = make_double2(-q.x, -q.y);
        if (JHTB_IN(m, lmax + 1, 105)) Mr[m] = q;
    }
}

// a staged point in a unit's `len` slots of shared memory
__device__ __forceinline__ double2 staged(const double2 *buf, int i, int len) { return JHTB_IN(i, len, 106) ? buf[i] : zero2(); }
__device__ __forceinline__ void stage(double2 *buf, int i, int len, double2 v) {
    if (JHTB_IN(i, len, 106)) buf[i] = v;
}
// factor k of a chirp length's column that starts at table entry `col`
__device__ __forceinline__ double2 chirp_factor(const RingArgs &a, long long col, int k) {
    return JHTB_IN(col + k, a.ctab_len, 110) ? __ldg(&a.ctab[col + k]) : zero2();
}

__device__ __forceinline__ double2 load_pixel(const double *map, const Streams &s, long long npix, int nstream, int j) {
    const double x = JHTB_IN(s.offX + j, npix * nstream, 103) ? map[s.offX + j] : 0.0;
    const double y = s.offY >= 0 && JHTB_IN(s.offY + j, npix * nstream, 103) ? map[s.offY + j] : 0.0;
    return make_double2(x, y);
}
__device__ __forceinline__ void store_pixel(double *map, const Streams &s, long long npix, int nstream, int j, double2 v) {
    if (JHTB_IN(s.offX + j, npix * nstream, 104)) map[s.offX + j] = v.x;
    if (s.offY >= 0 && JHTB_IN(s.offY + j, npix * nstream, 104)) map[s.offY + j] = v.y;
}

// ---------------------------------------------------------------------------------
// direct: power-of-two pieces of 2^LOGP points
// ---------------------------------------------------------------------------------
template <int LOGP, bool ADJ>
__device__ __forceinline__ void direct_unit(const RingArgs &a, const RingUnit &u, const double2 *F, double2 *V,
                                            const double *in, double *out, double2 *buf) {
    using X = Fft<LOGP>;
    const int g = threadIdx.x / X::TP, t = threadIdx.x % X::TP;  // ring of the unit, thread of its FFT
    const bool on = g < u.n;
    const int r = u.ring + (on ? g : 0), s = u.piece;
    const RingDesc rd = a.rings[r];
    const Streams st = streams_of(a, r, rd);
    const int N = rd.N, Q = N >> LOGP, nstream = a.spin ? 2 : 1;
    const bool sh = rd.shifted;
    const double2 *tw = a.tw;
    double2 v[16];
    if (on) {
        if constexpr (!ADJ) {
            const double2 *Pr = F + st.rowP, *Mr = F + st.rowM;
            const int c = (sh ? 1 : 0) + 2 * s;  // term k carries e^{i pi c k / N} (ring phase and piece twiddle)
            // e^{i pi c (k1 + P k2) / N} = e^{i pi c k1 / N} e^{i pi c k2 / Q}
            if (N > a.lmax) {
#pragma unroll
                for (int q = 0; q < 16; ++q) v[q] = fold_one(Pr, Mr, t + X::TP * q, N, a.lmax, sh);
                for (int k2 = 1; k2 < Q; ++k2) {
                    const double2 w = root8((4 / Q) * c * k2);
#pragma unroll
                    for (int q0 = 0; q0 < 16; q0 += 4) {
                        double2 d[4];
#pragma unroll
                        for (int q = 0; q < 4; ++q) d[q] = fold_one(Pr, Mr, t + X::TP * (q0 + q) + X::P * k2, N, a.lmax, sh);
#pragma unroll
                        for (int q = 0; q < 4; ++q) v[q0 + q] = cadd(v[q0 + q], cmul(d[q], w));
                    }
                }
            } else {  // aliased rings (lmax >= N) go through this thread's own buffer slots: one copy of the loop
                double2 *fb = buf + g * X::LEN;
#pragma unroll 1
                for (int q = 0; q < 16; ++q) {
                    const int k1 = t + X::TP * q;
                    double2 d = fold_sum(Pr, Mr, k1, N, a.lmax, sh);
#pragma unroll 1
                    for (int k2 = 1; k2 < Q; ++k2)
                        d = cadd(d, cmul(fold_sum(Pr, Mr, k1 + X::P * k2, N, a.lmax, sh), root8((4 / Q) * c * k2)));
                    stage(fb, X::template pos<0>(t, q), X::LEN, d);
                }
#pragma unroll
                for (int q = 0; q < 16; ++q) v[q] = staged(fb, X::template pos<0>(t, q), X::LEN);
            }
            if (c) {
#pragma unroll
                for (int q = 0; q < 16; ++q) v[q] = cmul(v[q], belt_phase(a, c * (t + X::TP * q), N));
            }
        } else {  // the transform of the conjugate: sum_j conj(v_j) e^{+2 pi i j (Q k + s) / N} = conj(W[Q k + s])
#pragma unroll
            for (int q = 0; q < 16; ++q) v[q] = conjd(load_pixel(in, st, a.npix, nstream, t + X::TP * q));
            for (int j2 = 1; j2 < Q; ++j2) {
                const double2 w = root8((8 / Q) * s * j2);
#pragma unroll
                for (int q = 0; q < 16; ++q)
                    v[q] = cadd(v[q], cmul(conjd(load_pixel(in, st, a.npix, nstream, t + X::TP * q + X::P * j2)), w));
            }
            if (s) {
#pragma unroll
                for (int q = 0; q < 16; ++q) v[q] = cmul(v[q], belt_phase(a, 2 * s * (t + X::TP * q), N));
            }
        }
    }
    X::template forward<false>(v, buf + g * X::LEN, t, on, tw);
    if (!on) return;
    if constexpr (!ADJ) {
#pragma unroll
        for (int q = 0; q < 16; ++q) store_pixel(out, st, a.npix, nstream, Q * X::out_index(t, q) + s, v[q]);
    } else {
        double2 *Pr = V + st.rowP, *Mr = V + st.rowM;
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            const int k = Q * X::out_index(t, q) + s;
            const double2 w = conjd(sh ? cmul(v[q], belt_phase(a, k, N)) : v[q]);
            scatter_orders(Pr, Mr, st.rowM != st.rowP, w, k, N, a.lmax, sh);
        }
    }
}

// ---------------------------------------------------------------------------------
// chirp: rings of N = 4 i points as four chirp-z transforms of length i
// ---------------------------------------------------------------------------------
// PPC pieces of 2^LOGP points of one ring per group of PPC * TP threads.  With
// D[k1 + i k2] the (phased) input, piece s transforms
//   a_s[k1] = in_s[k1] sum_{k2 < 4} i^{s k2} D[k1 + i k2],
// in_s the table column that joins the piece twiddle, the ring phase and the chirp; the
// result y[j] gets its last chirp factor from another column (kRingCols in the header).
// Where a CTA holds all four pieces (i <= 512) the ring's points are staged in shared memory
// on the way in and out, so that global accesses run in order; with two pieces on the way in
// only; with one they are read from global memory (through L2) by every piece.
template <int LOGP, int PPC, bool ADJ>
__device__ __forceinline__ void chirp_unit(const RingArgs &a, const RingUnit &u, const double2 *F, double2 *V,
                                           const double *in, double *out, double2 *buf) {
    using X = Fft<LOGP>;
    constexpr int GT = X::TP * PPC;  // threads of one ring
    const int g = threadIdx.x / GT, tg = threadIdx.x % GT;
    const int s = u.piece + tg / X::TP, t = tg % X::TP;
    const bool on = g < u.n;
    const int r = u.ring + (on ? g : 0);
    const RingDesc rd = a.rings[r];
    const Streams st = streams_of(a, r, rd);
    const int N = rd.N, i = N >> 2, nstream = a.spin ? 2 : 1;
    const bool sh = rd.shifted;
    constexpr int RB = PPC * X::LEN;  // slots of one ring
    double2 *rb = buf + g * PPC * X::LEN;  // this ring's part of the buffer
    const double2 *Pr = F + st.rowP, *Mr = F + st.rowM;
    // e^{i pi k2 / 4}: the part of the ring phase that depends on the quarter
    auto quarter = [&](double2 d, int k2) {
        if (ADJ || !sh) return d;
        return k2 == 0 ? d : cmul(d, root8(k2));
    };
    const int cs = class_stride(i);
    if (PPC >= 2) {  // stage the ring's points, quarter after quarter
        if (on) {
            constexpr int U = 4;
            if (!ADJ && N <= a.lmax) {
#pragma unroll 1
                for (int k = tg; k < N; k += GT)
                    stage(rb, k, RB, quarter(fold_sum(Pr, Mr, k, N, a.lmax, sh), (k >= i) + (k >= 2 * i) + (k >= 3 * i)));
            } else for (int k0 = tg; k0 < N; k0 += U * GT) {
                double2 d[U];
                if (ADJ) {
#pragma unroll
                    for (int e = 0; e < U; ++e)
                        d[e] = k0 + e * GT < N ? conjd(load_pixel(in, st, a.npix, nstream, k0 + e * GT)) : zero2();
                } else {
#pragma unroll
                    for (int e = 0; e < U; ++e)
                        d[e] = k0 + e * GT < N ? fold_one(Pr, Mr, k0 + e * GT, N, a.lmax, sh) : zero2();
                }
#pragma unroll
                for (int e = 0; e < U; ++e) {
                    const int k = k0 + e * GT;
                    if (k < N) stage(rb, k, RB, quarter(d[e], (k >= i) + (k >= 2 * i) + (k >= 3 * i)));
                }
            }
        }
        __syncthreads();
    }
    double2 v[16];
    const long long win = rd.ctab_off + (ADJ ? (long long)(kColAdjIn + s) : (long long)((sh ? kColSynth : kColAdjIn) + s)) * i;
    double2 *fb = rb + (tg / X::TP) * X::LEN;
    if (on) {
        const bool odd = s & 1;
        const double sn = s & 2 ? -1.0 : 1.0;
        // sum_{k2} i^{s k2} d[k2] = (d0 +- d2) + i^s (d1 +- d3)
        auto combine = [&](const double2 (&d)[4]) {
            const double2 e = odd ? csub(d[0], d[2]) : cadd(d[0], d[2]);
            const double2 o = odd ? csub(d[1], d[3]) : cadd(d[1], d[3]);
            return cadd(e, odd ? make_double2(-sn * o.y, sn * o.x) : make_double2(sn * o.x, sn * o.y));
        };
        if (PPC == 1 && !ADJ && N <= a.lmax) {  // aliased: through this thread's own buffer slots, one copy of the loop
#pragma unroll 1
            for (int q = 0; q < 8; ++q) {
                const int k1 = t + X::TP * q;
                if (k1 >= i) continue;
                double2 d[4];
#pragma unroll 1
                for (int k2 = 0; k2 < 4; ++k2) {
                    const double2 f = quarter(fold_sum(Pr, Mr, k1 + i * k2, N, a.lmax, sh), k2);
                    if (k2 == 3) d[3] = f;
                    else if (k2 == 2) d[2] = f;
                    else if (k2 == 1) d[1] = f;
                    else d[0] = f;
                }
                stage(fb, X::template pos<0>(t, q), X::LEN, combine(d));
            }
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int k1 = t + X::TP * q;
            if (k1 < i) {
                double2 x;
                if (PPC == 1 && !ADJ && N <= a.lmax) {
                    x = staged(fb, X::template pos<0>(t, q), X::LEN);
                } else {
                    double2 d[4];
#pragma unroll
                    for (int k2 = 0; k2 < 4; ++k2) {
                        const int k = k1 + i * k2;
                        if (PPC >= 2) d[k2] = staged(rb, k, RB);
                        else if (ADJ) d[k2] = conjd(load_pixel(in, st, a.npix, nstream, k));
                        else d[k2] = quarter(fold_one(Pr, Mr, k, N, a.lmax, sh), k2);
                    }
                    x = combine(d);
                }
                v[q] = cmul(x, chirp_factor(a, win, k1));
            } else {
                v[q] = zero2();
            }
        }
    }
    if (PPC >= 2) __syncthreads();  // the staged points are read: the buffer is free
    X::template forward<true>(v, fb, t, on, a.tw);
    if (on) {
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            const long long b = rd.bh_off + X::out_index(t, q);
            v[q] = cmul(v[q], JHTB_IN(b, a.bh_len, 108) ? __ldg(&a.bh[b]) : zero2());
        }
    }
    X::backward(v, fb, t, on, a.tw);
    // y[j] times the last chirp factor: pixel 4 j + s, or conj -> W'[4 j + s]
    const long long wout = rd.ctab_off + (ADJ ? (long long)(sh ? kColAdjOut + s : kColAdjIn) : (long long)kColAdjIn) * i;
    if (PPC == 4) {
        __syncthreads();  // every thread has read its last points
        if (on) {
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int j = t + X::TP * q;
                if (j < i) {
                    const double2 w = cmul(v[q], chirp_factor(a, wout, j));
                    stage(rb, s * cs + j, RB, ADJ ? conjd(w) : w);
                }
            }
        }
        __syncthreads();
        if (!on) return;
        if (!ADJ) {
            for (int j = tg; j < N; j += GT) store_pixel(out, st, a.npix, nstream, j, staged(rb, (j & 3) * cs + (j >> 2), RB));
        } else {
            gather_orders(V + st.rowP, V + st.rowM, st.rowM != st.rowP, N, a.lmax, sh, tg, GT,
                          [&](int k) { return staged(rb, (k & 3) * cs + (k >> 2), RB); });
        }
        return;
    }
    if (!on) return;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int j = t + X::TP * q;
        if (j >= i) continue;
        const double2 w = cmul(v[q], chirp_factor(a, wout, j));
        if (!ADJ) store_pixel(out, st, a.npix, nstream, 4 * j + s, w);
        else scatter_orders(V + st.rowP, V + st.rowM, st.rowM != st.rowP, conjd(w), 4 * j + s, N, a.lmax, sh);
    }
}

// ---------------------------------------------------------------------------------
// small: N <= kSmallRing points, one ring per CTA, a plain sum over k
// ---------------------------------------------------------------------------------
template <bool ADJ>
__device__ __forceinline__ void small_unit(const RingArgs &a, const RingUnit &u, const double2 *F, double2 *V,
                                           const double *in, double *out, double2 *buf) {
    constexpr int NT = kRingThreads;
    const int r = u.ring;
    const RingDesc rd = a.rings[r];
    const Streams st = streams_of(a, r, rd);
    const int N = rd.N, n2 = 2 * N, nstream = a.spin ? 2 : 1;
    const bool sh = rd.shifted;
    double2 *root = buf, *D = buf + 2 * kSmallRing, *part = D + kSmallRing;  // part: NT slots
    if ((int)threadIdx.x < n2) root[threadIdx.x] = cis_pi(threadIdx.x, N);
    const int parts = NT / N;  // >= 2
    const int k = threadIdx.x % N, p = threadIdx.x / N;
    if (ADJ) {
        if (p == 0) D[k] = load_pixel(in, st, a.npix, nstream, k);
        __syncthreads();
    } else {
        // the aliases of each k split over the ring's parts, summed in a fixed order
        if (p < parts) part[threadIdx.x] = fold_sum(F + st.rowP, F + st.rowM, k, N, a.lmax, sh, p, parts);
        __syncthreads();
        if (p == 0) {
            double2 d = part[k];
            for (int q = 1; q < parts; ++q) d = cadd(d, part[q * N + k]);
            D[k] = d;
        }
        __syncthreads();
    }
    // output k (pixel j or spectrum index): sum over e = p, p + parts, ... of D[e] times the root
    // of index (2 k + sh) e mod 2 N (synthesis, phase e^{i pi e / N} of a shifted ring included) or
    // -2 k e (adjoint)
    if (p < parts) {
        double2 acc = zero2();
        const int step1 = ADJ ? (n2 - 2 * k) % n2 : (2 * k + (sh ? 1 : 0)) % n2;
        int idx = (int)((long long)step1 * p % n2);
        const int step = (int)((long long)step1 * parts % n2);
        for (int e = p; e < N; e += parts) {
            const double2 d = staged(D, e, kSmallRing), w = staged(root, idx, 2 * kSmallRing);
            acc.x = fma(d.x, w.x, fma(-d.y, w.y, acc.x));
            acc.y = fma(d.x, w.y, fma(d.y, w.x, acc.y));
            idx += step;
            if (idx >= n2) idx -= n2;
        }
        part[threadIdx.x] = acc;
    }
    __syncthreads();
    if (p == 0) {
        double2 d = part[k];
        for (int q = 1; q < parts; ++q) d = cadd(d, part[q * N + k]);
        if (!ADJ) store_pixel(out, st, a.npix, nstream, k, d);
        else D[k] = sh ? cmulc(d, root[k]) : d;  // W'[k]
    }
    if (!ADJ) return;
    __syncthreads();
    gather_orders(V + st.rowP, V + st.rowM, st.rowM != st.rowP, N, a.lmax, sh, threadIdx.x, NT, [&](int q) { return staged(D, q, kSmallRing); });
}

template <bool ADJ>
__device__ __forceinline__ void ring_unit(const RingArgs &a, const RingUnit &u, const double2 *F, double2 *V,
                                          const double *in, double *out, double2 *buf) {
    switch (u.cls) {
        case kClsDirect + 8: direct_unit<8, ADJ>(a, u, F, V, in, out, buf); break;
        case kClsDirect + 9: direct_unit<9, ADJ>(a, u, F, V, in, out, buf); break;
        case kClsDirect + 10: direct_unit<10, ADJ>(a, u, F, V, in, out, buf); break;
        case kClsDirect + 11: direct_unit<11, ADJ>(a, u, F, V, in, out, buf); break;
        case kClsDirect + 12: direct_unit<12, ADJ>(a, u, F, V, in, out, buf); break;
        case kClsChirp + 7: chirp_unit<7, 4, ADJ>(a, u, F, V, in, out, buf); break;
        case kClsChirp + 8: chirp_unit<8, 4, ADJ>(a, u, F, V, in, out, buf); break;
        case kClsChirp + 9: chirp_unit<9, 4, ADJ>(a, u, F, V, in, out, buf); break;
        case kClsChirp + 10: chirp_unit<10, 4, ADJ>(a, u, F, V, in, out, buf); break;
        case kClsChirp + 11: chirp_unit<11, 2, ADJ>(a, u, F, V, in, out, buf); break;
        case kClsChirp + 12: chirp_unit<12, 1, ADJ>(a, u, F, V, in, out, buf); break;
        default: small_unit<ADJ>(a, u, F, V, in, out, buf); break;
    }
}

// One CTA per work unit and map, every class in one launch.  256 threads with up to 128
// registers (16 complex points and their twiddles) and 74 KB of shared memory, two CTAs per SM.
// Bound by instruction issue and L2 latency, not by HBM: the spectra and pixels of one spin-2
// map at nside 1024 / lmax 2048 (0.47 GB) take 0.07 ms at 6.65 TB/s.  An earlier form (radix-16
// passes of one generic length, a twiddle of two table entries per point, a sincospi per chirp
// factor, every spin-0 ring by itself) issued 4000 instructions per thread for 16 points.
// Measured, synthesis + adjoint, earlier -> this form: nside 1024 / lmax 2048, spin 2, one map
// 0.62 + 0.58 -> 0.32 + 0.32 ms; nside 512 / lmax 1024, spin 0, 64 maps 9.42 + 9.48 -> 2.15 + 2.27 ms
// (4.3x, of which 2x is the pairing); nside 2048 / lmax 4096, spin 2, 2.58 + 2.09 -> 1.39 + 1.20 ms.
__global__ void __launch_bounds__(kRingThreads, 2) ring_synth_kernel(RingArgs a, const double2 *__restrict__ F,
                                                                     double *__restrict__ maps, size_t fmap,
                                                                     long long pmap) {
    extern __shared__ double2 buf[];
    const RingUnit u = a.units[blockIdx.x];
    ring_unit<false>(a, u, F + blockIdx.y * fmap, nullptr, nullptr, maps + blockIdx.y * pmap, buf);
}
__global__ void __launch_bounds__(kRingThreads, 2) ring_adjoint_kernel(RingArgs a, const double *__restrict__ maps,
                                                                       double2 *__restrict__ V, size_t fmap,
                                                                       long long pmap) {
    extern __shared__ double2 buf[];
    const RingUnit u = a.units[blockIdx.x];
    ring_unit<true>(a, u, V + blockIdx.y * fmap, V + blockIdx.y * fmap, maps + blockIdx.y * pmap, nullptr, buf);
}
// Chirp-z transforms of 8192 points (rings above 8192 points that are no power of two, nside >
// 2048): 512 threads and 139 KB of shared memory.
template <bool ADJ>
__global__ void __launch_bounds__(512, 1) ring_long_kernel(RingArgs a, const double2 *__restrict__ F, double2 *__restrict__ V,
                                                           const double *__restrict__ in, double *__restrict__ out,
                                                           size_t fmap, long long pmap) {
    extern __shared__ double2 buf[];
    const RingUnit u = a.units[blockIdx.x];
    chirp_unit<13, 1, ADJ>(a, u, ADJ ? nullptr : F + blockIdx.y * fmap, ADJ ? V + blockIdx.y * fmap : nullptr,
                           ADJ ? in + blockIdx.y * pmap : nullptr, ADJ ? nullptr : out + blockIdx.y * pmap, buf);
}

// ---------------------------------------------------------------------------------
// tables (plan creation)
// ---------------------------------------------------------------------------------
// The factor columns of one chirp length i (N = 4 i), every entry e^{i pi a / N}:
//   kColAdjIn + s    a = 2 s k + 4 k^2             (s = 0: the chirp itself)
//   kColSynth + s    a = (1 + 2 s) k + 4 k^2
//   kColAdjOut + s   a = 4 k^2 + 4 k + s
__global__ void ring_table_kernel(const int *__restrict__ lens, const long long *__restrict__ offs, double2 *__restrict__ tab) {
    const int i = lens[blockIdx.x];
    double2 *out = tab + offs[blockIdx.x];
    const int s = blockIdx.y & 3, what = blockIdx.y >> 2;
    for (int k = threadIdx.x; k < i; k += blockDim.x) {
        const long long kk = 4LL * k * k;
        const long long e = what == 0 ? 2LL * s * k + kk : what == 1 ? (1 + 2LL * s) * k + kk : kk + 4LL * k + s;
        out[(size_t)blockIdx.y * i + k] = cis_pi(e, 4 * i);
    }
}
static_assert(kColAdjIn == 0 && kColSynth == 4 && kColAdjOut == 8 && kRingCols == 12, "column order of ring_table_kernel");

// e^{i pi a / N}, a < 2 N
__global__ void belt_table_kernel(int N, double2 *__restrict__ tab) {
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a < 2 * N) tab[a] = cis_pi(a, N);
}

// Chirp spectrum of length i at P = 2^LOGP points: the transform of conj(w(n)) on |n| < i,
// w(n) = e^{i pi n^2 / i}, divided by P.  One CTA per length of this P.
template <int LOGP>
__global__ void __launch_bounds__(Fft<LOGP>::TP < 32 ? 32 : Fft<LOGP>::TP) chirp_spectrum_kernel(
    const int *__restrict__ lens, const long long *__restrict__ offs, const double2 *__restrict__ tw, double2 *__restrict__ bh) {
    using X = Fft<LOGP>;
    extern __shared__ double2 buf[];
    const int i = lens[blockIdx.x], t = threadIdx.x;
    const bool on = t < X::TP;
    double2 v[16];
    if (on) {
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            const int p = t + X::TP * q;
            const int n = p < i ? p : X::P - p;  // w(-n) = w(n)
            v[q] = (p < i || n < i) ? conjd(cis_pi((long long)n * n, i)) : zero2();
        }
    }
    X::template forward<false>(v, buf, t, on, tw);
    if (!on) return;
    double2 *out = bh + offs[blockIdx.x];
    const double inv = 1.0 / (double)X::P;
#pragma unroll
    for (int q = 0; q < 16; ++q) out[X::out_index(t, q)] = make_double2(v[q].x * inv, v[q].y * inv);
}

template <typename K>
int ensure_smem(K kernel, int bytes) {
    JHTB_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    return JHTB_OK;
}

RingArgs make_args(const Plan &p) {
    RingArgs a{};
    a.rings = p.d_rings;
    a.lmax = p.lmax;
    a.M = p.M;
    a.nrows = p.nrings;
    a.spin = p.spin;
    a.npix = p.npix;
    a.tw = p.d_tw;
    a.bh = p.d_bh;
    a.ctab = p.d_ctab;
    a.bh_len = p.bh_len;
    a.ctab_len = p.ctab_len;
    a.belt = p.d_belt;
    a.belt_n = p.belt_n;
    return a;
}

// shared memory of the unit kernels: the largest layout of the classes (chirp 128-point pieces)
template <int LOGP>
constexpr int class_slots(int transforms) { return transforms * Fft<LOGP>::LEN; }
constexpr int kRingSlots = std::max({class_slots<12>(1), class_slots<11>(2), class_slots<10>(4), class_slots<9>(8),
                                     class_slots<8>(16), class_slots<7>(32), 3 * kSmallRing + kRingThreads});
constexpr int kRingSmem = kRingSlots * (int)sizeof(double2);
constexpr int kLongSmem = Fft<13>::LEN * (int)sizeof(double2);

template <int LOGP>
int launch_spectrum(const int *lens, const long long *offs, int n, const double2 *tw, double2 *bh, cudaStream_t s) {
    using X = Fft<LOGP>;
    if (n <= 0) return JHTB_OK;
    const int smem = X::LEN * (int)sizeof(double2);
    int rc;
    if ((rc = ensure_smem(chirp_spectrum_kernel<LOGP>, smem))) return rc;
    chirp_spectrum_kernel<LOGP><<<n, X::TP < 32 ? 32 : X::TP, smem, s>>>(lens, offs, tw, bh);
    JHTB_CUDA_TRY(cudaGetLastError());
    return JHTB_OK;
}

}  // namespace

JHTB_DEBUG_ACCESSOR(ringfft)

int launch_ring_synth(const Plan &p, const double2 *F, double *maps, int nb, cudaStream_t s) {
    if (nb <= 0) return JHTB_OK;
    RingArgs a = make_args(p);
    const size_t fmap = (size_t)p.ncomp * p.nrings * p.M;
    const long long pmap = (long long)p.ncomp * p.npix;
    if (p.nunit_long > 0) {
        a.units = p.d_ring_units + p.nunit;
        ring_long_kernel<false><<<dim3(p.nunit_long, nb), 512, kLongSmem, s>>>(a, F, nullptr, nullptr, maps, fmap, pmap);
        JHTB_CUDA_TRY(cudaGetLastError());
    }
    if (p.nunit > 0) {
        a.units = p.d_ring_units;
        ring_synth_kernel<<<dim3(p.nunit, nb), kRingThreads, kRingSmem, s>>>(a, F, maps, fmap, pmap);
        JHTB_CUDA_TRY(cudaGetLastError());
    }
    return JHTB_OK;
}

int launch_ring_adjoint(const Plan &p, const double *maps, double2 *V, int nb, cudaStream_t s) {
    if (nb <= 0) return JHTB_OK;
    RingArgs a = make_args(p);
    const size_t fmap = (size_t)p.ncomp * p.nrings * p.M;
    const long long pmap = (long long)p.ncomp * p.npix;
    if (p.nunit_long > 0) {
        a.units = p.d_ring_units + p.nunit;
        ring_long_kernel<true><<<dim3(p.nunit_long, nb), 512, kLongSmem, s>>>(a, nullptr, V, maps, nullptr, fmap, pmap);
        JHTB_CUDA_TRY(cudaGetLastError());
    }
    if (p.nunit > 0) {
        a.units = p.d_ring_units;
        ring_adjoint_kernel<<<dim3(p.nunit, nb), kRingThreads, kRingSmem, s>>>(a, maps, V, fmap, pmap);
        JHTB_CUDA_TRY(cudaGetLastError());
    }
    return JHTB_OK;
}

int launch_ring_tables(const Plan &p, const int *lens, const long long *ctab_offs, const long long *bh_offs,
                       const int (&count)[14], cudaStream_t s) {
    int rc;
    // the kernels' shared-memory limits, once per plan (on its device) instead of at each launch
    if ((rc = ensure_smem(ring_synth_kernel, kRingSmem)) || (rc = ensure_smem(ring_adjoint_kernel, kRingSmem)) ||
        (rc = ensure_smem(ring_long_kernel<false>, kLongSmem)) || (rc = ensure_smem(ring_long_kernel<true>, kLongSmem)))
        return rc;
    if (p.belt_n > 0) {
        belt_table_kernel<<<(2 * p.belt_n + 255) / 256, 256, 0, s>>>(p.belt_n, p.d_belt);
        JHTB_CUDA_TRY(cudaGetLastError());
    }
    int n = 0;
    for (int c : count) n += c;
    if (n <= 0) return JHTB_OK;
    ring_table_kernel<<<dim3(n, kRingCols), 128, 0, s>>>(lens, ctab_offs, p.d_ctab);
    JHTB_CUDA_TRY(cudaGetLastError());
    // the lengths are sorted by their P: count[log2 P] of each
    int o = 0;
#define JHTB_SPECTRUM(L)                                                                                   \
    if ((rc = launch_spectrum<L>(lens + o, bh_offs + o, count[L], p.d_tw, p.d_bh, s))) return rc; \
    o += count[L];
    JHTB_SPECTRUM(7)
    JHTB_SPECTRUM(8)
    JHTB_SPECTRUM(9)
    JHTB_SPECTRUM(10)
    JHTB_SPECTRUM(11)
    JHTB_SPECTRUM(12)
    JHTB_SPECTRUM(13)
#undef JHTB_SPECTRUM
    return JHTB_OK;
}

}  // namespace jhtb
