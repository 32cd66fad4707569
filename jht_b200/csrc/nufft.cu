// 2D NUFFT interpolation and spreading on the oversampled torus grid (sm_100a), the
// point-dependent stages of the off-grid transforms (jht _nufft.py:150-191).
//
// The grid is complex128 [nk][nm] (theta axis k, phi axis m), row-major.  A point
// (theta, phi) touches the W x W window whose first cell is ceil(u - W/2), u = coord *
// n / 2 pi, on each axis (indices taken mod n), with the "exponential of semicircle"
// weights psi(u - idx) = exp(beta (sqrt(1 - (2 t / W)^2) - 1)) on |t| < W / 2
// (Barnett, Magland & af Klinteberg 2019; _nufft.py:69-84).
//
//   interp (type 2):  f_j = sum_ab wk_a wm_b grid[ik_a][im_b], optionally with
//                     d f_j / d theta and d f_j / d phi (the kernel's derivative
//                     weights times n / 2 pi);
//   spread (type 1):  grid[ik_a][im_b] += wk_a wm_b v_j for every point (FP64 atomic
//                     adds: the summation order over points is not fixed).
//
// Interpolation: eight lanes per point, a lane for columns b and b + 8 of the window.  A window
// row is then one or two contiguous reads of 128 bytes and the eight lanes share the window
// weights' exponentials; with a thread per point a warp read 32 scattered cells at a time and the
// L1 took one after the other.  3 million points of W = 14 on 4320 x 4320 cells: 1201 us with a
// thread per point, 784 us now; 20000 points on 864 x 810: 33 and 13 us.  (Sixteen lanes per
// point: 1292 us, 336 warp instructions per point, most of them row addresses and window starts.)
// What is left is the instructions: about 60 of each weight's exp and sqrt.
//
// Direct spread: a lane for each of the 2 W doubles of a window row, so that a row's additions
// leave as one request of whole sectors (20000 points: 70 us with a thread per point, now 18 us).
#include <cuda_runtime.h>

#include "jhtb_internal.cuh"

namespace jhtb {
namespace {

constexpr int kNuThreads = 256;
constexpr double kTwoPi = 6.283185307179586476925286766559;

// Window start of one coordinate: u is the position in cells, f the first cell, first f as an
// integer.  Far outside any sensible range (or NaN) the start saturates; every index is still
// reduced into [0, n) by wrap.
template <int W>
__device__ __forceinline__ void window_start(double coord, int n, double &u, double &f, long long &first) {
    u = coord * (double)n / kTwoPi;
    f = ceil(u - 0.5 * W);
    first = (f > -4.0e18 && f < 4.0e18) ? (long long)f : 0;
}

// Weight a of the window that starts at f, and its derivative d psi / d u.
template <int W, bool DERIV>
__device__ __forceinline__ double window_at(double u, double f, int a, double beta, double &dw) {
    const double t = u - (f + a);
    const double z = t * (2.0 / W);
    const double z2 = z * z;
    double w = 0.0;
    dw = 0.0;
    if (z2 < 1.0) {
        const double r = sqrt(1.0 - z2);
        w = exp(beta * (r - 1.0));
        if (DERIV) dw = -w * beta * z * (2.0 / W) / r;
    }
    return w;
}
template <int W>
__device__ __forceinline__ double window_at(double u, double f, int a, double beta) {
    const double t = u - (f + a);
    const double z = t * (2.0 / W);
    const double z2 = z * z;
    return z2 < 1.0 ? exp(beta * (sqrt(1.0 - z2) - 1.0)) : 0.0;
}

__device__ __forceinline__ int wrap(long long i, int n) {
    if (i == (int)i) {  // the ordinary case: 32-bit remainder
        const int r = (int)i % n;
        return r < 0 ? r + n : r;
    }
    const long long r = i % n;
    return (int)(r < 0 ? r + n : r);
}
// base + a reduced into [0, n), base already there.
__device__ __forceinline__ unsigned step_wrap(int base, int a, int n) {
    const unsigned r = (unsigned)base + (unsigned)a;
    return r < (unsigned)n ? r : r % (unsigned)n;
}

template <int L>
__device__ __forceinline__ double2 lane_sum(double2 v) {
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) {
        v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
        v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
    }
    return v;
}

constexpr int kInterpLanes = 8;                    // lanes of a point
constexpr int kInterpPts = kNuThreads / kInterpLanes;  // points of a CTA at a time
constexpr int kWinStride = 18;                     // of a point's row weights: 16-byte reads, points in other banks

// A warp takes `batch` points at a time: a lane per point finds the windows' starts (divisions,
// remainders), then the points go by four.  Lane b of a point has columns b and b + 8.
template <int W, bool DERIV>
__global__ void __launch_bounds__(kNuThreads) interp_kernel(const double2 *__restrict__ grid, int nk, int nm,
                                                            double beta, const double *__restrict__ theta,
                                                            const double *__restrict__ phi, long long npts, int batch,
                                                            const int *__restrict__ order, double2 *__restrict__ out, double2 *__restrict__ dth,
                                                            double2 *__restrict__ dph) {
    constexpr int L = kInterpLanes, PER = 32 / L, WARPS = kNuThreads / 32, NC = (W + L - 1) / L, ND = DERIV ? 2 : 1;
    static_assert(W % 2 == 0 && W <= 16, "rows in pairs, two columns a lane");
    __shared__ __align__(16) double sk[kInterpPts][ND][kWinStride];  // row weights (and derivatives) of each point
    __shared__ double2 su[WARPS][32], sf[WARPS][32];                 // (theta, phi) u and f of the batch
    __shared__ int2 sbase[WARPS][32];
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int b = lane % L, sub = lane / L, slot = threadIdx.x / L;
    // A CTA takes consecutive points, which the caller may have grouped by tiles of the grid: their
    // windows overlap in its L1.
    const long long batches = (npts + batch - 1) / batch;
    const long long b0 = batches * blockIdx.x / gridDim.x, b1 = batches * (blockIdx.x + 1) / gridDim.x;
    for (long long bi = b0 + warp; bi < b1; bi += WARPS) {
        const long long first = bi * batch;
        const int count = (int)min((long long)batch, npts - first);
        __syncwarp();  // the batch before is done
        bool inside = true;  // no row of this lane's point wraps
        if (lane < count) {
            double2 u, f;
            long long k0, m0;
            window_start<W>(theta[first + lane], nk, u.x, f.x, k0);
            window_start<W>(phi[first + lane], nm, u.y, f.y, m0);
            const int2 base = make_int2(wrap(k0, nk), wrap(m0, nm));
            su[warp][lane] = u;
            sf[warp][lane] = f;
            sbase[warp][lane] = base;
            inside = base.x <= nk - W;
        }
        inside = __all_sync(0xffffffffu, inside);
        __syncwarp();  // the batch's starts are written: a vote alone orders no memory
        for (int i0 = 0; i0 < count; i0 += PER) {
            const int i = min(i0 + sub, count - 1);  // the last points' partners repeat the last point
            const double2 u = su[warp][i], f0 = sf[warp][i];
            const int2 base = sbase[warp][i];
            double wm[NC], dm[NC];
            __syncwarp();  // the points before are read
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                double dk;
                const double wk = window_at<W, DERIV>(u.x, f0.x, b + L * c, beta, dk);
                sk[slot][0][b + L * c] = wk;
                if (DERIV) sk[slot][ND - 1][b + L * c] = dk;
                wm[c] = window_at<W, DERIV>(u.y, f0.y, b + L * c, beta, dm[c]);
            }
            __syncwarp();
            double2 s[NC], sd[NC];
            const double2 *col[NC];
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                s[c] = sd[c] = make_double2(0.0, 0.0);
                col[c] = grid + step_wrap(base.y, b + L * c, nm);
            }
            auto rows = [&](auto row_of) {
#pragma unroll
                for (int a = 0; a < W; a += 2) {
                    const double2 wk = *reinterpret_cast<const double2 *>(&sk[slot][0][a]);
                    double2 wd;
                    if (DERIV) wd = *reinterpret_cast<const double2 *>(&sk[slot][ND - 1][a]);
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const size_t r = row_of(a + h);
#pragma unroll
                        for (int c = 0; c < NC; ++c) {
                            if (b + L * c >= W) continue;
                            const double2 g = __ldg(col[c] + r);
                            const double w = h ? wk.y : wk.x;
                            s[c].x = fma(w, g.x, s[c].x);
                            s[c].y = fma(w, g.y, s[c].y);
                            if (DERIV) {
                                const double d = h ? wd.y : wd.x;
                                sd[c].x = fma(d, g.x, sd[c].x);
                                sd[c].y = fma(d, g.y, sd[c].y);
                            }
                        }
                    }
                }
            };
            if (inside) {
                const size_t r0 = (size_t)base.x * nm;
                rows([&](int a) { return r0 + (size_t)a * nm; });
            } else {
                rows([&](int a) { return (size_t)step_wrap(base.x, a, nk) * nm; });
            }
            // columns past the window hold zeros, whatever their weight
            double2 f = make_double2(0.0, 0.0), gk = f, gm = f;
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                if (b + L * c >= W) continue;
                f = make_double2(fma(wm[c], s[c].x, f.x), fma(wm[c], s[c].y, f.y));
                if (DERIV) {
                    gk = make_double2(fma(wm[c], sd[c].x, gk.x), fma(wm[c], sd[c].y, gk.y));
                    gm = make_double2(fma(dm[c], s[c].x, gm.x), fma(dm[c], s[c].y, gm.y));
                }
            }
            f = lane_sum<L>(f);
            if (DERIV) {
                gk = lane_sum<L>(gk);
                gm = lane_sum<L>(gm);
            }
            if (b == 0 && i0 + sub < count) {
                const long long j = order ? order[first + i] : first + i;
                out[j] = f;
                if (DERIV) {
                    // d/dcoord = (n / 2 pi) d/du
                    const double ck = (double)nk / kTwoPi, cm = (double)nm / kTwoPi;
                    dth[j] = make_double2(ck * gk.x, ck * gk.y);
                    dph[j] = make_double2(cm * gm.x, cm * gm.y);
                }
            }
        }
    }
}

template <int W>
constexpr int kSpreadLanes = W <= 8 ? 16 : 32;  // lanes of a point: 2 W doubles of a row

template <int W>
__global__ void __launch_bounds__(kNuThreads) spread_kernel(const double2 *__restrict__ vals,
                                                            const double *__restrict__ theta,
                                                            const double *__restrict__ phi, long long npts, int nk,
                                                            int nm, double beta, double2 *__restrict__ grid) {
    constexpr int L = kSpreadLanes<W>, H = L / 2, PER = 32 / L;
    const int l = threadIdx.x % L, slot = threadIdx.x / L;
    const long long step = (long long)gridDim.x * (kNuThreads / L);
    for (long long j0 = (long long)blockIdx.x * (kNuThreads / L) + slot / PER * PER; j0 < npts; j0 += step) {
        const long long jj = j0 + slot % PER, j = jj < npts ? jj : npts - 1;
        double uk, fk, um, fm;
        long long k0, m0;
        window_start<W>(theta[j], nk, uk, fk, k0);
        window_start<W>(phi[j], nm, um, fm, m0);
        // row weights in the lower lanes, column weights in the upper ones
        const double w = l < H ? window_at<W>(uk, fk, l, beta) : window_at<W>(um, fm, l - H, beta);
        const double wm = __shfl_sync(0xffffffffu, w, H + l / 2, L);
        const double2 v2 = vals[j];
        const double v = l & 1 ? v2.y : v2.x;
        const bool on = l < 2 * W && jj < npts;
        const int kb = wrap(k0, nk);
        double *col = reinterpret_cast<double *>(grid + wrap(m0 + l / 2, nm)) + (l & 1);
#pragma unroll 2
        for (int a = 0; a < W; ++a) {
            const double wk = __shfl_sync(0xffffffffu, w, a, L);
            if (on) atomicAdd(col + (size_t)step_wrap(kb, a, nk) * 2 * nm, wm * (wk * v));
        }
    }
}

// Tiled spread: the points arrive grouped by kTile x kTile-cell tiles of the grid (segments
// of one tile, at most kSegPoints points each).  A CTA sums its segment's windows over the tile and
// its W-cell halo on chip and adds that block to the grid once per cell, so the global atomics
// fall from 2 W^2 per point to 2 (kTile + W)^2 per segment.
//
// The sum over a segment's points is a matrix product, G[k][m] = sum_j wk_j[k] (v_j wm_j[m]), with
// each point's two windows as zero-padded rows of the 48 x 48-cell block (cells as re, im column
// pairs), so it runs on the FP64 matrix unit: 9 of the block's 6 x 12 products of 8 x 8 per warp,
// four points per step, accumulators in registers.  Products of blocks that none of the four points
// touches are left out: points grouped by the part of the tile their window starts in need about a
// third of them (3 million points of W = 14: all products 1417 us, those touched 1271 us, with the
// next round's points fetched a round ahead 1210 us; the window weights, their staging and the
// additions to the grid are now the larger part, and three CTAs an SM hide only some of their
// latency: two took 1561 us, four, with spills, 1240 us).  Adding the windows
// into shared memory took 392 shared FP64 atomics per point (compare-and-swap loops).  A point whose
// window leaves the block (it lies in another tile than its segment's, whole periods aside) and
// one with an infinite or NaN value is added straight to the grid.
constexpr int kTile = 32;
constexpr int kSpreadThreads = 256;
constexpr int kSpreadPts = 32;                    // points staged per round
constexpr int kBlkCells = 48;                     // block edge, >= kTile + 16
constexpr int kSA = kBlkCells + 4, kSB = 2 * kBlkCells + 4;  // strides = 4 mod 16: conflict-free fragment loads

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1},{%2},{%3},{%0,%1};" : "+d"(c[0]), "+d"(c[1]) : "d"(a), "d"(b));
}

template <int W>
__global__ void __launch_bounds__(kSpreadThreads, 3) spread_tiles_kernel(
    const double2 *__restrict__ vals, const double *__restrict__ theta, const double *__restrict__ phi,
    long long npts, const long long *__restrict__ seg_start, const int *__restrict__ seg_count,
    const long long *__restrict__ seg_tile, int tiles_m, int nk, int nm, double beta, double2 *__restrict__ grid) {
    constexpr int B = kTile + W;  // block edge: the tile and its halo
    static_assert(B <= kBlkCells, "block of 6 x 12 products");
    __shared__ __align__(16) double sa[kSpreadPts][kSA];  // wk of each point, row = grid row of the block
    __shared__ __align__(16) double sb[kSpreadPts][kSB];  // v wm, column pair = grid column of the block
    __shared__ unsigned smask[kSpreadPts / 4];  // blocks that four points touch: rows (bits 0-5), columns (6-17)
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int lr = lane >> 2, lk = lane & 3;
    // This warp's 3 x 3 products: row blocks rw + 2 r, column blocks cw + 4 c.  Dealt round, so that the
    // few blocks that neighbouring points touch fall on all warps.
    const int rw = warp & 1, cw = warp >> 1;
    const long long seg = blockIdx.x;
    const long long tile = seg_tile[seg];
    const long long k_org = (tile / tiles_m) * kTile - W / 2, m_org = (tile % tiles_m) * kTile - W / 2;
    const long long p0 = seg_start[seg];
    const int cnt = seg_count[seg];
    if (cnt <= 0) return;
    double acc[3][3][2];
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) acc[r][c][0] = acc[r][c][1] = 0.0;
    const int pt = threadIdx.x >> 3, sub = threadIdx.x & 7;  // eight threads stage a point
    // this thread's point of the next round, fetched while one runs
    double th = 0.0, ph = 0.0;
    double2 v = make_double2(0.0, 0.0);
    auto fetch = [&](int q0) {
        const long long j = p0 + q0 + pt;
        if (q0 + pt < cnt && j >= 0 && j < npts) {
            th = theta[j];
            ph = phi[j];
            v = vals[j];
        }
    };
    fetch(0);
    for (int q0 = 0; q0 < cnt; q0 += kSpreadPts) {
        __syncthreads();  // the round before is read
        for (int i = threadIdx.x; i < kSpreadPts * (kSA + kSB) / 2; i += kSpreadThreads) {
            double2 *z = i < kSpreadPts * kSA / 2 ? reinterpret_cast<double2 *>(&sa[0][0]) + i
                                                  : reinterpret_cast<double2 *>(&sb[0][0]) + (i - kSpreadPts * kSA / 2);
            *z = make_double2(0.0, 0.0);
        }
        __syncthreads();
        const long long j = p0 + q0 + pt;
        unsigned mask = 0;
        if (q0 + pt < cnt && j >= 0 && j < npts) {
            const double uk = th * (double)nk / kTwoPi, um = ph * (double)nm / kTwoPi;
            const double fk = ceil(uk - 0.5 * W), fm = ceil(um - 0.5 * W);
            const long long k0 = (fk > -4.0e18 && fk < 4.0e18) ? (long long)fk : 0;
            const long long m0 = (fm > -4.0e18 && fm < 4.0e18) ? (long long)fm : 0;
            // a coordinate outside [0, 2 pi) lies whole periods from the tile that its key named
            long long bk = k0 - k_org, bm = m0 - m_org;
            if (bk < 0 || bk + W > B) bk = wrap(bk, nk);
            if (bm < 0 || bm + W > B) bm = wrap(bm, nm);
            // an infinite value would reach the block's other cells as 0 x inf
            if (bk + W <= B && bm + W <= B && isfinite(v.x) && isfinite(v.y)) {
                mask = (2u << (bk + W - 1) / 8) - (1u << bk / 8) | ((2u << (bm + W - 1) / 4) - (1u << bm / 4)) << 6;
                for (int a = sub; a < W; a += 8) {
                    sa[pt][bk + a] = window_at<W>(uk, fk, a, beta);
                    const double wm = window_at<W>(um, fm, a, beta);
                    *reinterpret_cast<double2 *>(&sb[pt][2 * (bm + a)]) = make_double2(wm * v.x, wm * v.y);
                }
            } else {
                // the point's column weights once, in its own staged row: its row weights stay
                // zero, so nothing of them reaches the products
                for (int b = sub; b < W; b += 8) sb[pt][b] = window_at<W>(um, fm, b, beta);
                __syncwarp(0xffu << (lane & 24));  // the point's eight threads, which all came this way
                for (int a = sub; a < W; a += 8) {
                    double *row = reinterpret_cast<double *>(grid + (size_t)wrap(k0 + a, nk) * nm);
                    const double wk = window_at<W>(uk, fk, a, beta);
                    for (int b = 0; b < W; ++b) {
                        const double wm = sb[pt][b];
                        const int mi = wrap(m0 + b, nm);
                        atomicAdd(row + 2 * mi, wm * (wk * v.x));
                        atomicAdd(row + 2 * mi + 1, wm * (wk * v.y));
                    }
                }
            }
        }
        fetch(q0 + kSpreadPts);
        mask = __reduce_or_sync(0xffffffffu, mask);  // a warp stages the four points of a step
        if (lane == 0) smask[warp] = mask;
        __syncthreads();
        for (int ks = 0; ks < kSpreadPts / 4; ++ks) {
            const unsigned rows = smask[ks] >> rw, cols = smask[ks] >> (6 + cw);
            if (!(rows & 0x15) || !(cols & 0x111)) continue;
            double bf[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) bf[c] = sb[4 * ks + lk][8 * (cw + 4 * c) + lr];
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                if (!(rows >> 2 * r & 1)) continue;
                const double af = sa[4 * ks + lk][8 * (rw + 2 * r) + lr];
#pragma unroll
                for (int c = 0; c < 3; ++c)
                    if (cols >> 4 * c & 1) dmma(acc[r][c], af, bf[c]);
            }
        }
    }
    // this lane holds row 8 (rw + 2 r) + lr, cell 4 (cw + 4 c) + lk
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        const int a = 8 * (rw + 2 * r) + lr;
        if (a >= B) continue;
        double *row = reinterpret_cast<double *>(grid + (size_t)wrap(k_org + a, nk) * nm);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const int b = 4 * (cw + 4 * c) + lk;
            if (b >= B || (acc[r][c][0] == 0.0 && acc[r][c][1] == 0.0)) continue;
            double *cell = row + 2 * wrap(m_org + b, nm);
            atomicAdd(cell, acc[r][c][0]);
            atomicAdd(cell + 1, acc[r][c][1]);
        }
    }
}

// Grouping: a counting sort of the points by tile and, within a tile, by the 8 x 8-cell part that
// their window starts in, so that the four points of a spread step touch few blocks.  Each pass is
// bound by memory: 16 bytes per point read to count, 28 read and 20 scattered (36 with values) to place.
constexpr int kSub = 16;         // parts of a tile, 4 x 4
constexpr int kSegPoints = 1024; // points of a spread segment
constexpr int kScanTiles = 256;  // tiles of a scan CTA
constexpr long long kMaxScanCtas = 4096;  // 2^20 tiles: grids of 32768 x 32768 cells

// Tile and part of a coordinate.  Only approximate at a tile's edge, which costs a point its place
// in the block, not its sum: a window that leaves the block is added directly.
__device__ __forceinline__ int tile_part(double coord, int n, int tiles) {
    if (!isfinite(coord)) return 0;
    const double r = coord - kTwoPi * floor(coord / kTwoPi);
    const double c = floor(r * ((double)n / (kTwoPi * (kTile / 4))));
    return (int)fmin(fmax(c, 0.0), 4.0 * tiles - 1.0);
}

__global__ void __launch_bounds__(256) group_count_kernel(const double *__restrict__ theta,
                                                          const double *__restrict__ phi, long long npts, int nk, int nm,
                                                          int tiles_k, int tiles_m, int *__restrict__ count,
                                                          int *__restrict__ key, int *__restrict__ rank) {
    const int lane = threadIdx.x & 31;
    for (long long j0 = blockIdx.x * 256LL + (threadIdx.x & ~31); j0 < npts; j0 += gridDim.x * 256LL) {
        const long long j = j0 + lane;
        int k = -1;
        if (j < npts) {
            const int a = tile_part(theta[j], nk, tiles_k), b = tile_part(phi[j], nm, tiles_m);
            k = ((a / 4) * tiles_m + b / 4) * kSub + (a % 4) * 4 + b % 4;
        }
        // lanes of one key count together: points often arrive along a track
        const unsigned same = __match_any_sync(0xffffffffu, k);
        const int leader = __ffs(same) - 1;
        int base = 0;
        if (lane == leader && k >= 0) base = atomicAdd(&count[k], __popc(same));
        base = __shfl_sync(0xffffffffu, base, leader);
        if (k >= 0) {
            key[j] = k;
            rank[j] = base + __popc(same & ((1u << lane) - 1));
        }
    }
}

// Points (low word) and segments (high word) of a tile's counts.
__device__ __forceinline__ unsigned long long tile_total(const int *count, int (&c)[kSub]) {
    unsigned n = 0;
#pragma unroll
    for (int i = 0; i < kSub / 4; ++i) {
        const int4 q = reinterpret_cast<const int4 *>(count)[i];
        c[4 * i] = q.x, c[4 * i + 1] = q.y, c[4 * i + 2] = q.z, c[4 * i + 3] = q.w;
        n += q.x + q.y + q.z + q.w;
    }
    return (unsigned long long)((n + kSegPoints - 1) / kSegPoints) << 32 | n;
}
__device__ __forceinline__ unsigned long long cta_sum(unsigned long long v) {
    __shared__ unsigned long long part[kScanTiles / 32];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
    __syncthreads();
    unsigned long long s = 0;
    for (int i = 0; i < kScanTiles / 32; ++i) s += part[i];
    return s;
}

__global__ void __launch_bounds__(kScanTiles) group_sum_kernel(const int *count, int tiles, unsigned long long *total) {
    const int t = blockIdx.x * kScanTiles + threadIdx.x;
    int c[kSub];
    const unsigned long long s = cta_sum(t < tiles ? tile_total(count + (size_t)t * kSub, c) : 0);
    if (threadIdx.x == 0) total[blockIdx.x] = s;
}

// Start of every part (over its count) and the segments.
__global__ void __launch_bounds__(kScanTiles) group_start_kernel(int *count, int tiles, const unsigned long long *total,
                                                                 long long *seg_start, int *seg_count,
                                                                 long long *seg_tile) {
    __shared__ unsigned long long scan[kScanTiles / 32];
    unsigned long long before = 0;
    for (int i = threadIdx.x; i < blockIdx.x; i += kScanTiles) before += total[i];
    before = cta_sum(before);
    const int t = blockIdx.x * kScanTiles + threadIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int c[kSub];
    const unsigned long long own = t < tiles ? tile_total(count + (size_t)t * kSub, c) : 0;
    unsigned long long inc = own;
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long u = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += u;
    }
    if (lane == 31) scan[warp] = inc;
    __syncthreads();
    for (int i = 0; i < warp; ++i) before += scan[i];
    if (t >= tiles) return;
    before += inc - own;
    const int n = (int)(own & 0xffffffffu), start = (int)(before & 0xffffffffu);
    const long long seg = (long long)(before >> 32);
    int at = start;
#pragma unroll
    for (int i = 0; i < kSub; ++i) {
        count[(size_t)t * kSub + i] = at;
        at += c[i];
    }
    for (int i = 0; i * kSegPoints < n; ++i) {
        seg_start[seg + i] = start + i * kSegPoints;
        seg_count[seg + i] = min(kSegPoints, n - i * kSegPoints);
        seg_tile[seg + i] = t;
    }
}

__global__ void __launch_bounds__(256) group_place_kernel(const double *__restrict__ theta,
                                                          const double *__restrict__ phi,
                                                          const double2 *__restrict__ vals, long long npts,
                                                          const int *__restrict__ start, const int *__restrict__ key,
                                                          const int *__restrict__ rank, int *__restrict__ order,
                                                          double *__restrict__ theta_s, double *__restrict__ phi_s,
                                                          double2 *__restrict__ vals_s) {
    for (long long j = blockIdx.x * 256LL + threadIdx.x; j < npts; j += gridDim.x * 256LL) {
        const int p = start[key[j]] + rank[j];
        order[p] = (int)j;
        theta_s[p] = theta[j];
        phi_s[p] = phi[j];
        if (vals) vals_s[p] = vals[j];
    }
}

int sm_count() {
    int dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    return nsm;
}
// CTAs for `groups` units of work of a CTA each
int grid_blocks(long long groups) {
    return (int)std::max<long long>(1, std::min<long long>(groups, 16LL * sm_count()));
}

int check_args(int nk, int nm, int W, long long npts, const char *who) {
    if (W != 6 && W != 8 && W != 10 && W != 14 && W != 16)
        return fail(JHTB_ERR_UNSUPPORTED, std::string(who) + ": kernel width must be 6, 8, 10, 14 or 16");
    if (nk < 1 || nm < 1) return fail(JHTB_ERR_INVALID, std::string(who) + ": empty grid");
    if (npts < 0) return fail(JHTB_ERR_INVALID, std::string(who) + ": negative point count");
    return JHTB_OK;
}

template <int W>
void launch_interp(const double2 *g, int nk, int nm, double beta, const double *th, const double *ph, long long n,
                   const int *order, double2 *out, double2 *dth, double2 *dph, cudaStream_t s) {
    // points of a warp's batch: up to a lane each, while every SM has 32 warps' worth
    constexpr int per = 32 / kInterpLanes, warps = kNuThreads / 32;
    const int batch = (int)std::max<long long>(per, std::min<long long>(32, n / (32 * sm_count()) / per * per));
    const int blocks = grid_blocks((n + (long long)batch * warps - 1) / ((long long)batch * warps));
    if (dth && dph)
        interp_kernel<W, true><<<blocks, kNuThreads, 0, s>>>(g, nk, nm, beta, th, ph, n, batch, order, out, dth, dph);
    else
        interp_kernel<W, false><<<blocks, kNuThreads, 0, s>>>(g, nk, nm, beta, th, ph, n, batch, order, out, nullptr, nullptr);
}

template <int W>
void launch_spread(const double2 *v, const double *th, const double *ph, long long n, int nk, int nm, double beta,
                   double2 *g, cudaStream_t s) {
    constexpr int per = kNuThreads / kSpreadLanes<W>;
    spread_kernel<W><<<grid_blocks((n + per - 1) / per), kNuThreads, 0, s>>>(v, th, ph, n, nk, nm, beta, g);
}

template <int W>
void launch_spread_tiles(const double2 *v, const double *th, const double *ph, long long npts, long long nseg,
                         const long long *start, const int *count, const long long *tile, int tiles_m, int nk, int nm,
                         double beta, double2 *g, cudaStream_t s) {
    spread_tiles_kernel<W><<<(unsigned)nseg, kSpreadThreads, 0, s>>>(v, th, ph, npts, start, count, tile, tiles_m, nk,
                                                                    nm, beta, g);
}

}  // namespace
}  // namespace jhtb

using namespace jhtb;

extern "C" {

int jhtb_nufft_interp_grouped(const void *grid, int nk, int nm, int W, double beta, const double *theta,
                              const double *phi, const int *order, int64_t npts, void *out, void *dtheta, void *dphi, void *stream) {
    if (!grid || !theta || !phi || !out) return fail(JHTB_ERR_INVALID, "jhtb_nufft_interp: NULL argument");
    if ((dtheta == nullptr) != (dphi == nullptr))
        return fail(JHTB_ERR_INVALID, "jhtb_nufft_interp: pass both derivative outputs or neither");
    int rc = check_args(nk, nm, W, npts, "jhtb_nufft_interp");
    if (rc) return rc;
    if (npts == 0) return JHTB_OK;
    const double2 *g = (const double2 *)grid;
    double2 *o = (double2 *)out, *dt = (double2 *)dtheta, *dp = (double2 *)dphi;
    cudaStream_t s = (cudaStream_t)stream;
    switch (W) {
        case 6: launch_interp<6>(g, nk, nm, beta, theta, phi, npts, order, o, dt, dp, s); break;
        case 8: launch_interp<8>(g, nk, nm, beta, theta, phi, npts, order, o, dt, dp, s); break;
        case 10: launch_interp<10>(g, nk, nm, beta, theta, phi, npts, order, o, dt, dp, s); break;
        case 14: launch_interp<14>(g, nk, nm, beta, theta, phi, npts, order, o, dt, dp, s); break;
        default: launch_interp<16>(g, nk, nm, beta, theta, phi, npts, order, o, dt, dp, s); break;
    }
    JHTB_CUDA_TRY(cudaGetLastError());
    return JHTB_OK;
}

int jhtb_nufft_interp(const void *grid, int nk, int nm, int W, double beta, const double *theta, const double *phi,
                      int64_t npts, void *out, void *dtheta, void *dphi, void *stream) {
    return jhtb_nufft_interp_grouped(grid, nk, nm, W, beta, theta, phi, nullptr, npts, out, dtheta, dphi, stream);
}

int jhtb_nufft_group_points(const double *theta, const double *phi, const void *vals, int64_t npts, int nk, int nm,
                            int tiles_k, int tiles_m, int *work, int *order, double *theta_s, double *phi_s,
                            void *vals_s, int *seg_count, int64_t *seg_start, int64_t *seg_tile, void *stream) {
    if (!theta || !phi || !work || !order || !theta_s || !phi_s || !seg_count || !seg_start || !seg_tile ||
        (vals && !vals_s))
        return fail(JHTB_ERR_INVALID, "jhtb_nufft_group_points: NULL argument");
    if (nk < 1 || nm < 1 || tiles_k < 1 || tiles_m < 1)
        return fail(JHTB_ERR_INVALID, "jhtb_nufft_group_points: empty grid");
    const long long tiles = (long long)tiles_k * tiles_m, ctas = (tiles + kScanTiles - 1) / kScanTiles;
    if (npts < 0 || npts > 0x7fffffffLL - kSegPoints || ctas > kMaxScanCtas)
        return fail(JHTB_ERR_INVALID, "jhtb_nufft_group_points: too many points or tiles");
    if (((uintptr_t)work | (uintptr_t)vals | (uintptr_t)vals_s) & 15)
        return fail(JHTB_ERR_INVALID, "jhtb_nufft_group_points: work and values must be 16-byte aligned");
    cudaStream_t s = (cudaStream_t)stream;
    // work: [tiles * 16] counts, then starts; [kMaxScanCtas] CTA totals (8 bytes); [npts] keys; [npts] ranks
    int *count = work;
    unsigned long long *total = (unsigned long long *)(work + tiles * kSub);
    int *key = (int *)(total + kMaxScanCtas), *rank = key + npts;
    const long long nseg = tiles + npts / kSegPoints;
    JHTB_CUDA_TRY(cudaMemsetAsync(count, 0, sizeof(int) * tiles * kSub, s));
    JHTB_CUDA_TRY(cudaMemsetAsync(seg_count, 0, sizeof(int) * nseg, s));
    const int blocks = grid_blocks((npts + 255) / 256);
    group_count_kernel<<<blocks, 256, 0, s>>>(theta, phi, npts, nk, nm, tiles_k, tiles_m, count, key, rank);
    JHTB_CUDA_TRY(cudaGetLastError());
    group_sum_kernel<<<(unsigned)ctas, kScanTiles, 0, s>>>(count, (int)tiles, total);
    JHTB_CUDA_TRY(cudaGetLastError());
    group_start_kernel<<<(unsigned)ctas, kScanTiles, 0, s>>>(count, (int)tiles, total, (long long *)seg_start, seg_count,
                                                             (long long *)seg_tile);
    JHTB_CUDA_TRY(cudaGetLastError());
    group_place_kernel<<<blocks, 256, 0, s>>>(theta, phi, (const double2 *)vals, npts, count, key, rank, order, theta_s,
                                              phi_s, (double2 *)vals_s);
    JHTB_CUDA_TRY(cudaGetLastError());
    return JHTB_OK;
}

int jhtb_nufft_spread(const void *vals, const double *theta, const double *phi, int64_t npts, int nk, int nm, int W,
                      double beta, void *grid, void *stream) {
    if (!vals || !theta || !phi || !grid) return fail(JHTB_ERR_INVALID, "jhtb_nufft_spread: NULL argument");
    int rc = check_args(nk, nm, W, npts, "jhtb_nufft_spread");
    if (rc) return rc;
    if (npts == 0) return JHTB_OK;
    const double2 *v = (const double2 *)vals;
    double2 *g = (double2 *)grid;
    cudaStream_t s = (cudaStream_t)stream;
    switch (W) {
        case 6: launch_spread<6>(v, theta, phi, npts, nk, nm, beta, g, s); break;
        case 8: launch_spread<8>(v, theta, phi, npts, nk, nm, beta, g, s); break;
        case 10: launch_spread<10>(v, theta, phi, npts, nk, nm, beta, g, s); break;
        case 14: launch_spread<14>(v, theta, phi, npts, nk, nm, beta, g, s); break;
        default: launch_spread<16>(v, theta, phi, npts, nk, nm, beta, g, s); break;
    }
    JHTB_CUDA_TRY(cudaGetLastError());
    return JHTB_OK;
}

int jhtb_nufft_spread_tiles(const void *vals, const double *theta, const double *phi, int64_t npts, int64_t nseg,
                            const int64_t *seg_start, const int *seg_count, const int64_t *seg_tile, int tiles_m,
                            int nk, int nm, int W, double beta, void *grid, void *stream) {
    if (!vals || !theta || !phi || !grid || (nseg > 0 && (!seg_start || !seg_count || !seg_tile)))
        return fail(JHTB_ERR_INVALID, "jhtb_nufft_spread_tiles: NULL argument");
    int rc = check_args(nk, nm, W, npts, "jhtb_nufft_spread_tiles");
    if (rc) return rc;
    rc = nseg < 0 ? fail(JHTB_ERR_INVALID, "jhtb_nufft_spread_tiles: negative segment count") : JHTB_OK;
    if (rc) return rc;
    if (tiles_m < 1) return fail(JHTB_ERR_INVALID, "jhtb_nufft_spread_tiles: tiles_m must be >= 1");
    if (nseg > 0x7fffffffLL) return fail(JHTB_ERR_INVALID, "jhtb_nufft_spread_tiles: too many segments");
    if (nseg == 0) return JHTB_OK;
    const double2 *v = (const double2 *)vals;
    double2 *g = (double2 *)grid;
    const long long *st = (const long long *)seg_start, *tl = (const long long *)seg_tile;
    cudaStream_t s = (cudaStream_t)stream;
    switch (W) {
        case 6: launch_spread_tiles<6>(v, theta, phi, npts, nseg, st, seg_count, tl, tiles_m, nk, nm, beta, g, s); break;
        case 8: launch_spread_tiles<8>(v, theta, phi, npts, nseg, st, seg_count, tl, tiles_m, nk, nm, beta, g, s); break;
        case 10: launch_spread_tiles<10>(v, theta, phi, npts, nseg, st, seg_count, tl, tiles_m, nk, nm, beta, g, s); break;
        case 14: launch_spread_tiles<14>(v, theta, phi, npts, nseg, st, seg_count, tl, tiles_m, nk, nm, beta, g, s); break;
        default: launch_spread_tiles<16>(v, theta, phi, npts, nseg, st, seg_count, tl, tiles_m, nk, nm, beta, g, s); break;
    }
    JHTB_CUDA_TRY(cudaGetLastError());
    return JHTB_OK;
}

}  // extern "C"
