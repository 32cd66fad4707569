// Complex FP64 FFTs of 2,3,5-smooth lengths (sm_100a): the off-grid transforms' theta FFT and
// the FFTs of the oversampled torus grid (jht _nufft.py:164-191 runs them as jnp.fft inside
// XLA).
//
// A CTA runs C neighbouring transforms (C > 1 where a transform's elements lie apart, so that
// the lanes of a warp read and write whole sectors) as decimation-in-frequency passes of radix
// 2 to 10, the fewest passes the length allows.  The first pass reads its butterflies from
// global memory and the last writes its outputs there in natural order; only the passes
// between go through shared memory, in place, one 16-byte pad per 256 bytes.  The roots come
// from the caller's table of the n-th roots of unity, two or three per butterfly with their
// products in between (without a table, from a sincospi of an exactly reduced rational
// argument).  Lengths up to kFftSmMax run in one CTA; the host composes longer ones from two
// batched calls (four-step).
//
// What a pass reads and writes is a functor.  FftStrided is the general batched call:
// batch index b = outer * inner_count + t reads in[o * in_dist_outer + t * in_dist_inner +
// i * in_stride] for i < n and writes out[...] likewise with the out strides, so row, column
// and four-step transforms of a row-major array are all one call.  The off-grid path's six
// transforms have their own, which take over the zero padding, centring, deconvolution and
// mirrored rings around them: the padded modes are neither stored nor read, and nothing is
// copied between the transforms (lmax 1024: 1374 -> 535 us from ring coefficients to the grid;
// lmax 200: 234 -> 42 us).
//
// Bound: memory.  The column transforms of a 4320 x 4320 grid move 0.6 GB.  One CTA of 1024
// threads per transform, gathering in digit-reversed order and running radix 4, 2, 3 and 5
// stages through shared memory, took 674 us for them and 489 us for the rows; this form takes
// 290 and 215 us, about 3 cycles per point and SM: four passes of FP64 arithmetic (1.3), shared
// memory (0.75) and global memory (0.5), which the two CTAs of an SM overlap only in part.
// Registers for three CTAs (80, with spills) gave 290 and 235.
#include <cuda_runtime.h>

#include <algorithm>

#include "jhtb_internal.cuh"

namespace jhtb {
namespace {

constexpr int kFftThreads = 256;   // of a CTA that shares its SM; twice that for one that does not
constexpr int kFftSmMax = 10240;   // longest transform held in shared memory (174 KB with the pads)
constexpr int kFftMaxPass = 12;
constexpr int kFftCtaBytes = 112 << 10;  // shared memory of each of two CTAs on an SM

constexpr int kFftMaxBytes = (kFftSmMax + kFftSmMax / 16 + 1) * 16;

// One length's passes: radices in the order they run, and for each the reciprocals its index
// arithmetic divides by.
struct FftShape {
    int n, npass, clog;  // 2^clog transforms per CTA
    int radix[kFftMaxPass], m[kFftMaxPass];
    unsigned inv_m[kFftMaxPass], inv_r[kFftMaxPass];  // ceil(2^31 / m), ceil(2^31 / radix)
    long long howmany;
    const double2 *roots;  // e^{-2 pi i k / n} for k < n, or null (sincospi)
};

// a / d for 0 <= a < 2^14, 1 <= d < 2^14, inv = ceil(2^31 / d): the excess a (inv d - 2^31) < 2^28.
__device__ __forceinline__ int f_div(int a, unsigned inv) { return (int)__umulhi(2u * (unsigned)a, inv); }

__device__ __forceinline__ double2 f_cmul(double2 a, double2 b) {
    return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ double2 f_add(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 f_sub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 f_conj(double2 a) { return make_double2(a.x, -a.y); }
__device__ __forceinline__ double2 f_scale(double2 a, double s) { return make_double2(s * a.x, s * a.y); }
__device__ __forceinline__ double2 f_mi(double2 a) { return make_double2(a.y, -a.x); }  // -i a

// e^{-2 pi i a / b} for integers 0 <= a < b.
__device__ __forceinline__ double2 f_root(long long a, long long b) {
    double s, c;
    sincospi(-2.0 * (double)a / (double)b, &s, &c);
    return make_double2(c, s);
}

// R-point DFTs in registers: X_k = sum_j x_j e^{-2 pi i j k / R}.
template <int R>
struct Dft;
template <>
struct Dft<1> {
    static __device__ __forceinline__ void run(double2 (&)[1]) {}
};
template <>
struct Dft<2> {
    static __device__ __forceinline__ void run(double2 (&v)[2]) {
        const double2 a = v[0], b = v[1];
        v[0] = f_add(a, b);
        v[1] = f_sub(a, b);
    }
};
template <>
struct Dft<3> {
    static __device__ __forceinline__ void run(double2 (&v)[3]) {
        constexpr double s3 = 0.86602540378443864676;  // sin(2 pi / 3)
        const double2 t1 = f_add(v[1], v[2]), d = f_sub(v[1], v[2]);
        const double2 t2 = make_double2(fma(-0.5, t1.x, v[0].x), fma(-0.5, t1.y, v[0].y));
        v[0] = f_add(v[0], t1);
        v[1] = make_double2(fma(s3, d.y, t2.x), fma(-s3, d.x, t2.y));
        v[2] = make_double2(fma(-s3, d.y, t2.x), fma(s3, d.x, t2.y));
    }
};
template <>
struct Dft<4> {
    static __device__ __forceinline__ void run(double2 (&v)[4]) {
        const double2 a = f_add(v[0], v[2]), b = f_sub(v[0], v[2]);
        const double2 c = f_add(v[1], v[3]), d = f_mi(f_sub(v[1], v[3]));
        v[0] = f_add(a, c);
        v[2] = f_sub(a, c);
        v[1] = f_add(b, d);
        v[3] = f_sub(b, d);
    }
};
template <>
struct Dft<5> {
    static __device__ __forceinline__ void run(double2 (&v)[5]) {
        constexpr double c1 = 0.30901699437494742410, c2 = -0.80901699437494742410;  // cos(2 pi / 5), cos(4 pi / 5)
        constexpr double s1 = 0.95105651629515357212, s2 = 0.58778525229247312917;   // sin(2 pi / 5), sin(4 pi / 5)
        const double2 a1 = f_add(v[1], v[4]), b1 = f_sub(v[1], v[4]);
        const double2 a2 = f_add(v[2], v[3]), b2 = f_sub(v[2], v[3]);
        const double2 x0 = v[0];
        const double2 r1 = make_double2(fma(c2, a2.x, fma(c1, a1.x, x0.x)), fma(c2, a2.y, fma(c1, a1.y, x0.y)));
        const double2 r2 = make_double2(fma(c1, a2.x, fma(c2, a1.x, x0.x)), fma(c1, a2.y, fma(c2, a1.y, x0.y)));
        const double2 i1 = f_mi(make_double2(fma(s1, b1.x, s2 * b2.x), fma(s1, b1.y, s2 * b2.y)));
        const double2 i2 = f_mi(make_double2(fma(s2, b1.x, -s1 * b2.x), fma(s2, b1.y, -s1 * b2.y)));
        v[0] = f_add(x0, f_add(a1, a2));
        v[1] = f_add(r1, i1);
        v[4] = f_sub(r1, i1);
        v[2] = f_add(r2, i2);
        v[3] = f_sub(r2, i2);
    }
};
// R = 2 B with B odd: the prime-factor map j = (B a + 2 b) mod R, k = (B ka + (B + 1) kb) mod R
// has no roots between the two transforms.
template <int B>
struct DftTwice {
    static __device__ __forceinline__ void run(double2 (&v)[2 * B]) {
        constexpr int R = 2 * B;
        double2 e[2][B];
#pragma unroll
        for (int a = 0; a < 2; ++a) {
#pragma unroll
            for (int b = 0; b < B; ++b) e[a][b] = v[(B * a + 2 * b) % R];
            Dft<B>::run(e[a]);
        }
#pragma unroll
        for (int b = 0; b < B; ++b) {
            v[((B + 1) * b) % R] = f_add(e[0][b], e[1][b]);
            v[(B + (B + 1) * b) % R] = f_sub(e[0][b], e[1][b]);
        }
    }
};
template <>
struct Dft<6> : DftTwice<3> {};
template <>
struct Dft<10> : DftTwice<5> {};
template <>
struct Dft<8> {
    static __device__ __forceinline__ void run(double2 (&v)[8]) {
        constexpr double h = 0.70710678118654752440;  // sqrt(1/2)
        double2 e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
        Dft<4>::run(e);
        Dft<4>::run(o);
        o[1] = make_double2(h * (o[1].x + o[1].y), h * (o[1].y - o[1].x));
        o[2] = f_mi(o[2]);
        o[3] = make_double2(h * (o[3].y - o[3].x), -h * (o[3].x + o[3].y));
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            v[k] = f_add(e[k], o[k]);
            v[k + 4] = f_sub(e[k], o[k]);
        }
    }
};
template <>
struct Dft<9> {
    static __device__ __forceinline__ void run(double2 (&v)[9]) {
        // cos and -sin of 2 pi k / 9, k = 1, 2, 4
        constexpr double2 w1{0.76604444311897803520, -0.64278760968653932632};
        constexpr double2 w2{0.17364817766693034885, -0.98480775301220805937};
        constexpr double2 w4{-0.93969262078590838405, -0.34202014332566873304};
        double2 e[3][3];
#pragma unroll
        for (int b = 0; b < 3; ++b) {
#pragma unroll
            for (int a = 0; a < 3; ++a) e[b][a] = v[3 * a + b];
            Dft<3>::run(e[b]);
        }
        e[1][1] = f_cmul(e[1][1], w1);
        e[1][2] = f_cmul(e[1][2], w2);
        e[2][1] = f_cmul(e[2][1], w2);
        e[2][2] = f_cmul(e[2][2], w4);
#pragma unroll
        for (int ka = 0; ka < 3; ++ka) {
            double2 u[3] = {e[0][ka], e[1][ka], e[2][ka]};
            Dft<3>::run(u);
#pragma unroll
            for (int kb = 0; kb < 3; ++kb) v[ka + 3 * kb] = u[kb];
        }
    }
};

// Shared-memory slot of element pos of transform c: one pad per 16 slots keeps the strided
// reads of the late passes off one bank.
__device__ __forceinline__ int f_slot(int pos, int c, int clog) {
    const int e = (pos << clog) + c;
    return e + (e >> 4);
}

// One pass of radix R over blocks of m R elements: butterfly j of a block takes the elements j +
// q m, transforms them and multiplies result q by e^{-2 pi i j q / (m R)}.  After the last pass
// the element of digits q0, q1, ... (the first pass's digit the most significant) is output
// q0 + R0 q1 + R0 R1 q2 + ...: its butterflies run in the order of their outputs.
template <int R, bool FIRST, bool LAST, class IO>
__device__ __forceinline__ void fft_pass(const FftShape &s, int p, const IO &io, double2 *buf, int c, bool on) {
    const int m = LAST ? 1 : s.m[p], nb = s.n / R;
    for (int b = threadIdx.x >> s.clog; b < nb; b += blockDim.x >> s.clog) {
        int j = 0, base = b;
        if (LAST) {
            base = 0;
            int r = b;
            for (int i = 0; i < p; ++i) {
                const int t = f_div(r, s.inv_r[i]);
                base += (r - t * s.radix[i]) * s.m[i];
                r = t;
            }
        } else if (FIRST) {
            j = b;
        } else {
            const int g = f_div(b, s.inv_m[p]);
            j = b - g * m;
            base = g * m * R + j;
        }
        double2 v[R];
#pragma unroll
        for (int q = 0; q < R; ++q)
            v[q] = FIRST ? (on ? io.load(base + q * m) : make_double2(0.0, 0.0)) : buf[f_slot(base + q * m, c, s.clog)];
        Dft<R>::run(v);
        if (!LAST) {
            const int step = FIRST ? j : j * (s.n / (m * R));  // e^{-2 pi i j / (m R)} = roots[step]
            double2 w[R];
#pragma unroll
            for (int q = 1; q < R; ++q) {
                if (q == 1 || q % 3 == 0) w[q] = s.roots ? __ldg(&s.roots[q * step]) : f_root(q * step, s.n);
                else if (q == 2) w[2] = f_cmul(w[1], w[1]);
                else w[q] = f_cmul(w[q - q % 3], w[q % 3]);
                v[q] = f_cmul(v[q], w[q]);
            }
#pragma unroll
            for (int q = 0; q < R; ++q) buf[f_slot(base + q * m, c, s.clog)] = v[q];
        } else if (on) {
#pragma unroll
            for (int q = 0; q < R; ++q) io.store(b + q * nb, v[q]);
        }
    }
}

template <bool FIRST, bool LAST, class IO>
__device__ __forceinline__ void fft_pass_of(const FftShape &s, int p, const IO &io, double2 *buf, int c, bool on) {
    switch (s.radix[p]) {
        case 1: if (FIRST && LAST) fft_pass<1, FIRST, LAST>(s, p, io, buf, c, on); break;
        case 2: fft_pass<2, FIRST, LAST>(s, p, io, buf, c, on); break;
        case 3: fft_pass<3, FIRST, LAST>(s, p, io, buf, c, on); break;
        case 4: fft_pass<4, FIRST, LAST>(s, p, io, buf, c, on); break;
        case 5: fft_pass<5, FIRST, LAST>(s, p, io, buf, c, on); break;
        case 6: fft_pass<6, FIRST, LAST>(s, p, io, buf, c, on); break;
        case 8: fft_pass<8, FIRST, LAST>(s, p, io, buf, c, on); break;
        case 9: fft_pass<9, FIRST, LAST>(s, p, io, buf, c, on); break;
        default: fft_pass<10, FIRST, LAST>(s, p, io, buf, c, on); break;
    }
}

template <class IO>
__global__ void __launch_bounds__(2 * kFftThreads, 1) fft_kernel(FftShape s, IO io) {
    extern __shared__ double2 fbuf[];
    const int c = threadIdx.x & ((1 << s.clog) - 1);
    const long long groups = (s.howmany + (1 << s.clog) - 1) >> s.clog;
    for (long long g = blockIdx.x; g < groups; g += gridDim.x) {
        const long long b = (g << s.clog) + c;
        const bool on = b < s.howmany;
        io.open(on ? b : 0);
        if (s.npass == 1) {
            fft_pass_of<true, true>(s, 0, io, fbuf, c, on);
        } else {
            fft_pass_of<true, false>(s, 0, io, fbuf, c, on);
            __syncthreads();
            for (int p = 1; p < s.npass - 1; ++p) {
                fft_pass_of<false, false>(s, p, io, fbuf, c, on);
                __syncthreads();
            }
            fft_pass_of<false, true>(s, s.npass - 1, io, fbuf, c, on);
        }
        __syncthreads();  // the next transforms reuse the buffer
    }
}

// sign +1 is the conjugate of the sign -1 transform of the conjugate input.
__device__ __forceinline__ double2 f_signed(double2 v, int sign) { return make_double2(v.x, sign > 0 ? -v.y : v.y); }

struct FftStrided {
    const double2 *in;
    double2 *out;
    long long inner;
    long long in_stride, in_dist_outer, in_dist_inner;
    long long out_stride, out_dist_outer, out_dist_inner;
    int sign;
    double scale;
    long long tw_n;  // 0: none; else output k of inner index t times e^{sign 2 pi i (t k mod tw_n) / tw_n}
    long long t;
    const double2 *src;
    double2 *dst;
    __device__ __forceinline__ void open(long long b) {
        const long long o = b / inner;
        t = b - o * inner;
        src = in + o * in_dist_outer + t * in_dist_inner;
        dst = out + o * out_dist_outer + t * out_dist_inner;
    }
    __device__ __forceinline__ double2 load(int i) const { return f_signed(src[(long long)i * in_stride], sign); }
    __device__ __forceinline__ void store(int k, double2 v) const {
        v = f_scale(v, scale);
        if (tw_n) v = f_cmul(v, f_root((t * (long long)k) % tw_n, tw_n));
        dst[(long long)k * out_stride] = f_signed(v, sign);
    }
};

// The off-grid path's geometry: ns rings (theta = 0 .. pi) extended to nd = 2 ns - 2 samples of
// the full circle, lmax orders either side of m = 0, and the nk x nm torus grid.
struct Torus {
    int lmax, ns, nd, spin, nk, nm;
    const double *ick, *icm;  // [nd] and [2 lmax + 1] deconvolution factors, centred
    __device__ __forceinline__ int Nm() const { return 2 * lmax + 1; }
    // (-1)^m (-1)^spin: the field's mirror image across a pole (spin is even or odd)
    __device__ __forceinline__ double mirror(int m) const { return ((m + spin) & 1) ? -1.0 : 1.0; }
    // grid row or column i of length n -> centred mode index, or -1 where the padding lies
    __device__ __forceinline__ int centred(int i, int n, int modes) const {
        const int lo = modes / 2;  // negative modes
        if (i < modes - lo) return i + lo;
        return i >= n - lo ? i - (n - lo) : -1;
    }
};

// Ring coefficients -> centred theta modes, T[nd][2 lmax + 1] (deconvolved).
struct ThetaFwd {
    Torus g;
    const double2 *Fp, *Fm;  // [ns][lmax + 1] of the +spin and the -spin channel
    double2 *T;
    int col;
    __device__ __forceinline__ void open(long long b) { col = (int)b; }
    __device__ __forceinline__ double2 load(int i) const {
        const int m = col - g.lmax, r = i < g.ns ? i : g.nd - i;
        const double2 f = m >= 0 ? Fp[(long long)r * (g.lmax + 1) + m] : f_conj(Fm[(long long)r * (g.lmax + 1) - m]);
        return i < g.ns ? f : f_scale(f, g.mirror(m < 0 ? -m : m));
    }
    __device__ __forceinline__ void store(int k, double2 v) const {
        const int row = k + g.nd / 2 < g.nd ? k + g.nd / 2 : k + g.nd / 2 - g.nd;
        T[(long long)row * g.Nm() + col] = f_scale(v, (1.0 / g.nd) * (g.ick[row] * g.icm[col]));
    }
};
// Rows of T, zero padded to nm -> R[nd][nm], sign +1.
struct RowFwd {
    Torus g;
    const double2 *T;
    double2 *R;
    long long row;
    __device__ __forceinline__ void open(long long b) { row = b; }
    __device__ __forceinline__ double2 load(int i) const {
        const int c = g.centred(i, g.nm, g.Nm());
        return c < 0 ? make_double2(0.0, 0.0) : f_conj(T[row * g.Nm() + c]);
    }
    __device__ __forceinline__ void store(int k, double2 v) const { R[row * g.nm + k] = f_conj(v); }
};
// Columns of R, zero padded to nk -> grid[nk][nm], sign +1.
struct ColFwd {
    Torus g;
    const double2 *R;
    double2 *grid;
    int col;
    __device__ __forceinline__ void open(long long b) { col = (int)b; }
    __device__ __forceinline__ double2 load(int i) const {
        const int r = g.centred(i, g.nk, g.nd);
        return r < 0 ? make_double2(0.0, 0.0) : f_conj(R[(long long)r * g.nm + col]);
    }
    __device__ __forceinline__ void store(int k, double2 v) const { grid[(long long)k * g.nm + col] = f_conj(v); }
};
// The transposes, in reverse order.  Columns of the grid -> the nd centred modes, R[nd][nm].
struct ColAdj {
    Torus g;
    const double2 *grid;
    double2 *R;
    int col;
    __device__ __forceinline__ void open(long long b) { col = (int)b; }
    __device__ __forceinline__ double2 load(int i) const { return grid[(long long)i * g.nm + col]; }
    __device__ __forceinline__ void store(int k, double2 v) const {
        const int r = g.centred(k, g.nk, g.nd);
        if (r >= 0) R[(long long)r * g.nm + col] = v;
    }
};
// Rows of R -> the centred orders, T[nd][2 lmax + 1] (deconvolved).
struct RowAdj {
    Torus g;
    const double2 *R;
    double2 *T;
    long long row;
    __device__ __forceinline__ void open(long long b) { row = b; }
    __device__ __forceinline__ double2 load(int i) const { return R[row * g.nm + i]; }
    __device__ __forceinline__ void store(int k, double2 v) const {
        const int c = g.centred(k, g.nm, g.Nm());
        if (c >= 0) T[row * g.Nm() + c] = f_scale(v, g.ick[row] * g.icm[c]);
    }
};
// Columns of T -> samples of the full circle, sign +1, in place (a CTA reads all of its columns
// before it writes the first).
struct ThetaAdj {
    Torus g;
    double2 *T;
    int col;
    __device__ __forceinline__ void open(long long b) { col = (int)b; }
    __device__ __forceinline__ double2 load(int i) const {
        const int row = i + g.nd / 2 < g.nd ? i + g.nd / 2 : i + g.nd / 2 - g.nd;
        return f_conj(T[(long long)row * g.Nm() + col]);
    }
    __device__ __forceinline__ void store(int k, double2 v) const {
        T[(long long)k * g.Nm() + col] = f_conj(f_scale(v, 1.0 / g.nd));
    }
};

// Samples of the full circle -> ring coefficients of both spin channels: a ring's mirror image
// joins it, order -m joins order m's conjugate.
__global__ void __launch_bounds__(256) torus_fold_kernel(Torus g, const double2 *d, double2 *V, int ncomp) {
    const long long idx = (long long)blockIdx.x * 256 + threadIdx.x;
    const int M = g.lmax + 1;
    if (idx >= (long long)g.ns * M) return;
    const int r = (int)(idx / M), m = (int)(idx - (long long)r * M);
    const bool both = r >= 1 && r <= g.nd - g.ns;
    const double sg = g.mirror(m);
    auto top = [&](int c) {
        double2 v = d[(long long)r * g.Nm() + c];
        if (both) {
            const double2 w = d[(long long)(g.nd - r) * g.Nm() + c];
            v = make_double2(fma(sg, w.x, v.x), fma(sg, w.y, v.y));
        }
        return v;
    };
    const double2 p = top(g.lmax + m);
    const double2 q = m > 0 ? f_conj(top(g.lmax - m)) : make_double2(0.0, 0.0);
    if (ncomp == 1) {
        V[idx] = f_add(p, q);
    } else {
        V[idx] = p;
        V[(long long)g.ns * M + idx] = q;
    }
}

int sm_count(int *nsm) {
    int dev = 0;
    JHTB_CUDA_TRY(cudaGetDevice(&dev));
    JHTB_CUDA_TRY(cudaDeviceGetAttribute(nsm, cudaDevAttrMultiProcessorCount, dev));
    return JHTB_OK;
}

// Radices of length n: the fewest passes, and among these the smallest sum, largest first.
void pick_radices(int n, int cap, int *cur, int depth, int sum, int *best, int *nbest, int *sbest) {
    if (n == 1) {
        if (depth < *nbest || (depth == *nbest && sum < *sbest)) {
            *nbest = depth;
            *sbest = sum;
            std::copy(cur, cur + depth, best);
        }
        return;
    }
    if (depth >= *nbest || depth >= kFftMaxPass) return;
    for (int r : {10, 9, 8, 6, 5, 4, 3, 2})
        if (r <= cap && n % r == 0) {
            cur[depth] = r;
            pick_radices(n / r, r, cur, depth + 1, sum + r, best, nbest, sbest);
        }
}

// apart: the transforms' elements lie apart in memory, and neighbouring transforms' next to each other.
template <class IO>
int launch_fft(const IO &io, int n, long long howmany, bool apart, const void *roots, int nsm, cudaStream_t stream) {
    if (howmany == 0) return JHTB_OK;
    FftShape s{};
    s.n = n;
    s.howmany = howmany;
    s.roots = (const double2 *)roots;
    int cur[kFftMaxPass], sum = 1 << 30;
    s.npass = kFftMaxPass + 1;
    pick_radices(n, 10, cur, 0, 0, s.radix, &s.npass, &sum);
    if (n == 1) s.npass = 1, s.radix[0] = 1;
    int m = n;
    for (int p = 0; p < s.npass; ++p) {
        m /= s.radix[p];
        s.m[p] = m;
        s.inv_m[p] = (unsigned)(((1u << 31) + (unsigned)m - 1) / (unsigned)m);
        s.inv_r[p] = (unsigned)(((1u << 31) + (unsigned)s.radix[p] - 1) / (unsigned)s.radix[p]);
    }
    // Transforms per CTA: up to a line's worth (8 x 16 bytes) while two CTAs of 256 threads fit an
    // SM and the batch still gives every SM two; two (a sector's worth) also where only one CTA of
    // 512 threads then fits (4320 columns of 4320 points: 391 us one by one, 290 us in pairs).
    auto bytes = [&](int clog) {
        const int e = n << clog;
        return (e + (e >> 4) + 1) * (int)sizeof(double2);
    };
    if (apart)
        while (s.clog < 3 && bytes(s.clog + 1) <= (s.clog ? kFftCtaBytes : kFftMaxBytes) &&
               (howmany >> (s.clog + 1)) >= 2 * nsm)
            ++s.clog;
    const int smem = s.npass > 1 ? bytes(s.clog) : 0;
    const int items = (n / s.radix[0]) << s.clog;
    const int threads = std::min(smem > kFftCtaBytes ? 2 * kFftThreads : kFftThreads, (items + 31) / 32 * 32);
    const long long groups = (howmany + (1 << s.clog) - 1) >> s.clog;
    JHTB_CUDA_TRY(cudaFuncSetAttribute(fft_kernel<IO>, cudaFuncAttributeMaxDynamicSharedMemorySize, kFftMaxBytes));
    fft_kernel<IO><<<(unsigned)std::min<long long>(groups, 1 << 20), threads, smem, stream>>>(s, io);
    JHTB_CUDA_TRY(cudaGetLastError());
    return JHTB_OK;
}

}  // namespace
}  // namespace jhtb

using namespace jhtb;

extern "C" int jhtb_fft_c2c(const void *in, void *out, int n, int64_t howmany, int64_t inner, int64_t in_stride,
                            int64_t in_dist_outer, int64_t in_dist_inner, int64_t out_stride, int64_t out_dist_outer,
                            int64_t out_dist_inner, int sign, double scale, int64_t twiddle_n, const void *roots,
                            void *stream) {
    if (!in || !out) return fail(JHTB_ERR_INVALID, "jhtb_fft_c2c: NULL argument");
    if (n < 1 || n > kFftSmMax)
        return fail(JHTB_ERR_INVALID, "jhtb_fft_c2c: n must be in [1, " + std::to_string(kFftSmMax) + "], got " +
                                          std::to_string(n));
    if (howmany < 0 || inner < 1) return fail(JHTB_ERR_INVALID, "jhtb_fft_c2c: howmany must be >= 0 and inner >= 1");
    if (sign != 1 && sign != -1) return fail(JHTB_ERR_INVALID, "jhtb_fft_c2c: sign must be +1 or -1");
    if (twiddle_n < 0) return fail(JHTB_ERR_INVALID, "jhtb_fft_c2c: twiddle_n must be >= 0");
    if (in == out && (in_stride != out_stride || in_dist_outer != out_dist_outer || in_dist_inner != out_dist_inner))
        return fail(JHTB_ERR_INVALID, "jhtb_fft_c2c: an in-place call needs the same input and output layout");
    int r = n;
    for (int f : {2, 3, 5})
        while (r % f == 0) r /= f;
    if (r != 1) return fail(JHTB_ERR_INVALID, "jhtb_fft_c2c: n must be 2,3,5-smooth, got " + std::to_string(n));
    FftStrided a{};
    a.in = (const double2 *)in;
    a.out = (double2 *)out;
    a.inner = inner;
    a.in_stride = in_stride;
    a.in_dist_outer = in_dist_outer;
    a.in_dist_inner = in_dist_inner;
    a.out_stride = out_stride;
    a.out_dist_outer = out_dist_outer;
    a.out_dist_inner = out_dist_inner;
    a.sign = sign;
    a.scale = scale;
    a.tw_n = twiddle_n;
    int nsm, rc;
    if ((rc = sm_count(&nsm))) return rc;
    return launch_fft(a, n, howmany, in_stride != 1 || out_stride != 1, roots, nsm, (cudaStream_t)stream);
}

namespace {
int torus_setup(const char *name, Torus *g, int ncomp, int lmax, int ns, int spin, int nk, int nm, const double *ick,
                const double *icm) {
    auto bad = [&](const char *what) { return fail(JHTB_ERR_INVALID, std::string(name) + ": " + what); };
    if (!ick || !icm) return bad("NULL argument");
    if (ncomp != 1 && ncomp != 2) return bad("ncomp must be 1 or 2");
    if (lmax < 0 || ns < 2) return bad("needs lmax >= 0 and ns >= 2");
    const long long nd = 2LL * ns - 2, Nm = 2LL * lmax + 1;
    if (nd > kFftSmMax || nk > kFftSmMax || nm > kFftSmMax) return bad("a length is above the one-CTA limit");
    if (nk < nd || nm < Nm) return bad("the grid must hold every mode");
    for (long long n : {nd, (long long)nk, (long long)nm}) {
        for (int f : {2, 3, 5})
            while (n % f == 0) n /= f;
        if (n != 1) return bad("lengths must be 2,3,5-smooth");
    }
    *g = Torus{lmax, ns, (int)nd, spin, nk, nm, ick, icm};
    return JHTB_OK;
}
}  // namespace

extern "C" int jhtb_torus_grid(const void *F, int ncomp, int lmax, int ns, int spin, int nk, int nm, const double *ick,
                               const double *icm, const void *roots_nd, const void *roots_nk, const void *roots_nm,
                               void *work, void *grid, void *stream) {
    Torus g;
    int nsm, rc;
    if (!F || !work || !grid) return fail(JHTB_ERR_INVALID, "jhtb_torus_grid: NULL argument");
    if ((rc = torus_setup("jhtb_torus_grid", &g, ncomp, lmax, ns, spin, nk, nm, ick, icm))) return rc;
    if ((rc = sm_count(&nsm))) return rc;
    const cudaStream_t st = (cudaStream_t)stream;
    const long long Nm = 2LL * lmax + 1;
    double2 *T = (double2 *)work, *R = T + g.nd * Nm;
    const double2 *Fp = (const double2 *)F, *Fm = Fp + (ncomp - 1) * (long long)ns * (lmax + 1);
    if ((rc = launch_fft(ThetaFwd{g, Fp, Fm, T, 0}, g.nd, Nm, true, roots_nd, nsm, st))) return rc;
    if ((rc = launch_fft(RowFwd{g, T, R, 0}, nm, g.nd, false, roots_nm, nsm, st))) return rc;
    return launch_fft(ColFwd{g, R, (double2 *)grid, 0}, nk, nm, true, roots_nk, nsm, st);
}

extern "C" int jhtb_torus_grid_adjoint(const void *grid, int ncomp, int lmax, int ns, int spin, int nk, int nm,
                                       const double *ick, const double *icm, const void *roots_nd, const void *roots_nk,
                                       const void *roots_nm, void *work, void *V, void *stream) {
    Torus g;
    int nsm, rc;
    if (!grid || !work || !V) return fail(JHTB_ERR_INVALID, "jhtb_torus_grid_adjoint: NULL argument");
    if ((rc = torus_setup("jhtb_torus_grid_adjoint", &g, ncomp, lmax, ns, spin, nk, nm, ick, icm))) return rc;
    if ((rc = sm_count(&nsm))) return rc;
    const cudaStream_t st = (cudaStream_t)stream;
    const long long Nm = 2LL * lmax + 1;
    double2 *T = (double2 *)work, *R = T + g.nd * Nm;
    if ((rc = launch_fft(ColAdj{g, (const double2 *)grid, R, 0}, nk, nm, true, roots_nk, nsm, st))) return rc;
    if ((rc = launch_fft(RowAdj{g, R, T, 0}, nm, g.nd, false, roots_nm, nsm, st))) return rc;
    if ((rc = launch_fft(ThetaAdj{g, T, 0}, g.nd, Nm, true, roots_nd, nsm, st))) return rc;
    const long long items = (long long)ns * (lmax + 1);
    torus_fold_kernel<<<(unsigned)((items + 255) / 256), 256, 0, st>>>(g, T, (double2 *)V, ncomp);
    JHTB_CUDA_TRY(cudaGetLastError());
    return JHTB_OK;
}
