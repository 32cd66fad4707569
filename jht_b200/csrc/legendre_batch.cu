// FP64 Legendre stage of a batch of maps: one recursion for a group of maps, the sums on the
// FP64 matrix unit (mma.sync m8n8k4, sm_100a).
//
// The recursion values mu_l(t) of an order depend on the ring alone, so a group of maps shares
// them and the sums over l (synthesis) or over rings (adjoint) become small products:
//   synthesis  F[t, n] = sum_l mu_l(t) C[l, n]      rows = 8 rings, k = 4 degrees
//   adjoint    b[l, n] = sum_t mu_l(t) V[t, n]      rows = 8 degrees, k = 4 rings
// with 8 columns n per instruction: four spin-0 maps (re, im; even and odd degrees apart, jht
// _recursion.py:441-497) or two spin-2 maps (four columns per recursion, :512-572).
//
// Why the matrix unit: it runs at the FP64 FMA rate (37 TFLOP/s of either, they share the
// pipe), but an FMA with three different register operands issues only every 3 cycles per
// scheduler (the register file delivers one 64-bit operand a cycle), while an m8n8k4 product
// takes 16 cycles for 8 FMAs' worth per lane.  Per (l, ring, map) the one-map kernels spend about 11.6
// (spin 0) and 35 (spin 2) scheduler cycles; a group of 8 spin-0 maps spends 5/8 + 4, one of 4
// spin-2 maps 12/4 + 16.  Operands, accumulation and rounding stay FP64.
//
// Work: the tiles of 128 rings of the one-map adjoint (start states, first live degree), one
// CTA per item from a cost-sorted queue.  A synthesis item is (order, tile), a warp per 32
// rings; an adjoint item is (order, ring range), eight warps of 32 rings whose sums meet in
// shared memory, so that a range of 256 rings writes each degree once.  Rings in the underflow
// range count as zero and are rescaled once per 8 degrees, as in legendre.cu.
#include <cuda_runtime.h>

#include <algorithm>

#include "jhtb_internal.cuh"
#include "seed.cuh"

namespace jhtb {
namespace {

constexpr int kTileRings = 128;  // rings of a start-state tile (4 per lane of the one-map adjoint)
static_assert(kRA0 == 4 && kRA2 == 4, "start-state layout of 128-ring tiles");

struct BatchParams {
    int lmax, T, nrings, M, paired;
    long long K;
    const double *x;
    const SeedParam *seed;
    const double *alpha, *gamma, *cnorm;
    int ntiles;          // 128-ring tiles per order
    const int *lw;       // [M * ntiles] first degree of a tile
    const double2 *st;   // [M * ntiles][nrec][4][32] start states
    const int *stsc;
    const int *order;    // items by falling cost
    int nitems;
    int nsuper, nblk;    // adjoint: ring ranges per order, 256-ring blocks per range
    int blk_lo, blk_hi;  // 256-ring blocks of the plan's ring range
    unsigned *counter;
};

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1},{%2},{%3},{%0,%1};" : "+d"(c[0]), "+d"(c[1]) : "d"(a), "d"(b));
}

__device__ __forceinline__ void rescale_state(double &u, double &prev, int &sc) {
    if (sc < 0 && fabs(u) > kBig) {
        u *= kScaleDown;
        prev *= kScaleDown;
        sc += 1;
    }
}

// next item of the CTA's queue (all threads get it; two barriers)
__device__ __forceinline__ int next_cta_item(unsigned *counter, int *slot) {
    __syncthreads();
    if (threadIdx.x == 0) *slot = (int)atomicAdd(counter, 1u);
    __syncthreads();
    return *slot;
}

// One warp's 32 rings: the recursions of its lanes.
template <int SPIN>
struct Chains {
    static constexpr int NREC = SPIN ? 2 : 1;
    double x, u1[NREC], u2[NREC];
    int sc[NREC];

    __device__ __forceinline__ void load(const BatchParams &p, int m, int ring0, int lane) {
        const int t = ring0 + lane;
        x = 0.0;
#pragma unroll
        for (int h = 0; h < NREC; ++h) {
            u1[h] = u2[h] = 0.0;
            sc[h] = 0;
        }
        if (t >= p.T) return;
        const size_t item = (size_t)m * p.ntiles + ring0 / kTileRings;
        const int r = (ring0 / 32) & 3;
        x = __ldg(&p.x[t]);
#pragma unroll
        for (int h = 0; h < NREC; ++h) {
            const size_t o = ((item * NREC + h) * 4 + r) * 32 + lane;
            const double2 s = p.st[o];
            u1[h] = s.x;
            u2[h] = s.y;
            sc[h] = p.stsc[o];
        }
    }
    // 8 steps with the coefficients ag[0..8) = (alpha, gamma); out[h hstride + q stride] gets the
    // values (zero while scaled), then one rescale check.  PART: the states apply from step
    // `from` on, the values before are zero.
    template <bool PART>
    __device__ __forceinline__ void steps8(const double2 *ag, double *out, int stride, int hstride, int from) {
        bool live[NREC];
#pragma unroll
        for (int h = 0; h < NREC; ++h) live[h] = sc[h] == 0;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const double2 c = ag[q];
#pragma unroll
            for (int h = 0; h < NREC; ++h) {
                const double t = SPIN ? fma(c.x, x, h ? -c.y : c.y) : c.x * x;
                const double u = fma(t, u1[h], -u2[h]);
                const bool on = !PART || q >= from;
                if (on) {
                    u2[h] = u1[h];
                    u1[h] = u;
                }
                out[h * hstride + q * stride] = on && live[h] ? u : 0.0;
            }
        }
#pragma unroll
        for (int h = 0; h < NREC; ++h) rescale_state(u1[h], u2[h], sc[h]);
    }
};

// ---------------------------------------------------------------------------------
// synthesis
// ---------------------------------------------------------------------------------
constexpr int kSynWarps = 4;
constexpr int kSynL = 16;  // degrees staged per round

template <int SPIN, int NB>  // NB: blocks of 8 columns (4 spin-0 maps or 2 spin-2 maps each)
struct SynCfg {
    static constexpr int NREC = SPIN ? 2 : 1;
    static constexpr int MAPS = (SPIN ? 2 : 4) * NB;
    static constexpr int NC = 8 * NB;                  // columns per recursion
    static constexpr int SC = NC + (SPIN ? 4 : 2);     // column stride of a degree: k * SC (2 k SC for the parity
                                                       // split) and 4 lanes cover the 16 eight-byte banks
    static constexpr int SU = SPIN ? 36 : 34;          // ring stride of a degree, likewise
};

template <int SPIN, int NB>
struct SynSmem {
    using C = SynCfg<SPIN, NB>;
    double c[2][C::NREC][kSynL][C::SC];        // staged coefficients, double-buffered
    double2 ag[2][kSynL];
    double u[kSynWarps][C::NREC][8][C::SU];    // recursion values of one warp, 8 degrees
    int slot;
};

template <int SPIN, int NB>
__global__ void __launch_bounds__(kSynWarps * 32, 4) synth_batch_kernel(BatchParams p, const double2 *__restrict__ alm_all,
                                                                      double2 *__restrict__ F_all, int nb, int ngroups) {
    using C = SynCfg<SPIN, NB>;
    extern __shared__ __align__(16) unsigned char raw[];
    SynSmem<SPIN, NB> &sm = *reinterpret_cast<SynSmem<SPIN, NB> *>(raw);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int lr = lane >> 2, lk = lane & 3;
    constexpr int NCOMP = SPIN ? 2 : 1;
    for (;;) {
        const int it = next_cta_item(p.counter, &sm.slot);
        if (it >= p.nitems * ngroups) break;
        const int g = it / p.nitems;
        const int item = p.order[it - g * p.nitems];
        const int m = item / p.ntiles, tile = item - m * p.ntiles;
        const int b0map = g * C::MAPS, nmap = min(C::MAPS, nb - b0map);
        const double2 *alm = alm_all + (size_t)b0map * NCOMP * p.K;
        const int lmin = p.seed[m].lmin;
        const long long b0 = alm_index(lmin, m, p.lmax);
        const int nst = p.lmax - lmin + 1;
        const int i_start = min(p.lw[item] - lmin, nst);
        const int ring0 = tile * kTileRings + warp * 32;
        Chains<SPIN> ch;
        ch.load(p, m, ring0, lane);
        // spin 0: [parity][ring block][column block]; spin 2: [recursion][...]
        double acc[2][4][NB][2];
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < NB; ++b) acc[h][a][b][0] = acc[h][a][b][1] = 0.0;

        // a round's coefficients: thread = (map, degree); spin 0 with 8 maps fills the CTA
        const int sl = threadIdx.x % kSynL, sb = threadIdx.x / kSynL;
        double2 ra, rb, rag;
        double rc;
        auto fetch = [&](int i0) {
            ra = rb = rag = make_double2(0.0, 0.0);
            rc = 0.0;
            const long long idx = b0 + i0 + sl;
            if (i0 + sl < nst && JHTB_IN(idx, p.K, 206)) {
                if (sb < nmap) {
                    rc = p.cnorm[idx];
                    ra = alm[(size_t)sb * NCOMP * p.K + idx];
                    if (SPIN) rb = alm[((size_t)sb * NCOMP + 1) * p.K + idx];
                }
                if (sb == 0) rag = make_double2(p.alpha[idx], SPIN ? p.gamma[idx] : 0.0);
            }
        };
        auto stage = [&](int s) {
            if (sb < C::MAPS) {
                if (SPIN) {
                    // cp = -(aE + i aB) c, cm = -(aE - i aB) c (healpix.py:316-318); columns
                    // + : [cp, s cm], - : [cm, s cp], s = (-1)^(l - lmin)
                    const double sg = (sl & 1) ? -rc : rc;  // rounds start at even offsets from lmin
                    const double pr = -(ra.x - rb.y), pi = -(ra.y + rb.x), mr = -(ra.x + rb.y), mi = -(ra.y - rb.x);
                    double *cp = &sm.c[s][0][sl][4 * sb], *cm = &sm.c[s][C::NREC - 1][sl][4 * sb];
                    *reinterpret_cast<double2 *>(cp) = make_double2(pr * rc, pi * rc);
                    *reinterpret_cast<double2 *>(cp + 2) = make_double2(mr * sg, mi * sg);
                    *reinterpret_cast<double2 *>(cm) = make_double2(mr * rc, mi * rc);
                    *reinterpret_cast<double2 *>(cm + 2) = make_double2(pr * sg, pi * sg);
                } else {
                    *reinterpret_cast<double2 *>(&sm.c[s][0][sl][2 * sb]) = make_double2(ra.x * rc, ra.y * rc);
                }
            }
            if (sb == 0) sm.ag[s][sl] = rag;
        };
        fetch(i_start);
        int s = 0;
        for (int i0 = i_start; i0 < nst; i0 += kSynL, s ^= 1) {
            stage(s);
            __syncthreads();  // the other buffer's readers of the round before are past it as well
            if (i0 + kSynL < nst) fetch(i0 + kSynL);
#pragma unroll 1
            for (int half = 0; half < 2; ++half) {
                __syncwarp();
                ch.template steps8<false>(&sm.ag[s][half * 8], &sm.u[warp][0][0][lane], C::SU, 8 * C::SU, 0);
                __syncwarp();
#pragma unroll
                for (int kg = 0; kg < 2; ++kg) {
#pragma unroll
                    for (int h = 0; h < C::NREC; ++h) {
                        // spin 0: group kg holds the degrees of parity kg; spin 2: four consecutive ones
                        const int l = SPIN ? kg * 4 + lk : 2 * lk + kg;
                        const int slot = SPIN ? h : kg;
                        double bf[NB];
#pragma unroll
                        for (int b = 0; b < NB; ++b) bf[b] = sm.c[s][h][half * 8 + l][8 * b + lr];
#pragma unroll
                        for (int a = 0; a < 4; ++a) {
                            const double af = sm.u[warp][h][l][8 * a + lr];
#pragma unroll
                            for (int b = 0; b < NB; ++b) dmma(acc[slot][a][b], af, bf[b]);
                        }
                    }
                }
            }
        }
        // this lane holds ring 8 a + lr, columns 8 b + 2 lk, + 1
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const int t = ring0 + 8 * a + lr;
            if (t >= p.T || !JHTB_IN((long long)(p.nrings - 1 - t) * p.M + m, (long long)p.nrings * p.M, 207)) continue;
            const size_t rn = (size_t)t * p.M + m, rs = (size_t)(p.nrings - 1 - t) * p.M + m;
#pragma unroll
            for (int b = 0; b < NB; ++b) {
                if (SPIN) {
                    const int map = 2 * b + (lk >> 1);
                    if (map >= nmap) continue;
                    double2 *Fp = F_all + (size_t)(b0map + map) * 2 * p.nrings * p.M, *Fm = Fp + (size_t)p.nrings * p.M;
                    const double ssign = ((m + lmin) & 1) ? -1.0 : 1.0;  // the signed sums are relative to lmin
                    const double2 vp = make_double2(acc[0][a][b][0], acc[0][a][b][1]);
                    const double2 vm = make_double2(acc[1][a][b][0], acc[1][a][b][1]);
                    if (!(lk & 1)) {  // + : north of the +2 channel, - : north of the -2 channel
                        Fp[rn] = vp;
                        Fm[rn] = vm;
                    } else if (t < p.T - 1) {  // + : s cm with mu+, the south of -2; - : the south of +2
                        Fm[rs] = make_double2(ssign * vp.x, ssign * vp.y);
                        Fp[rs] = make_double2(ssign * vm.x, ssign * vm.y);
                    }
                } else {
                    const int map = 4 * b + lk;
                    if (map >= nmap) continue;
                    double2 *F = F_all + (size_t)(b0map + map) * p.nrings * p.M;
                    double2 n = make_double2(acc[0][a][b][0] + acc[1][a][b][0], acc[0][a][b][1] + acc[1][a][b][1]);
                    double2 so = make_double2(acc[0][a][b][0] - acc[1][a][b][0], acc[0][a][b][1] - acc[1][a][b][1]);
                    if (p.paired) spin0_pair(n, so, m == 0, t < p.T - 1);
                    F[rn] = n;
                    if (t < p.T - 1) F[rs] = so;
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------------
// adjoint
// ---------------------------------------------------------------------------------
constexpr int kAdjWarps = 8;
constexpr int kBlockRings = kAdjWarps * 32;

template <int SPIN, int NB>
struct AdjBCfg {
    static constexpr int NREC = SPIN ? 2 : 1;
    static constexpr int MAPS = (SPIN ? 2 : 4) * NB;
    static constexpr int NC = 8 * NB;
    static constexpr int LCH = SPIN ? 8 : 16;      // degrees per round: 8 rows of each recursion or parity
    static constexpr int NG = LCH / 8;             // recursion groups of 8 steps per round
    static constexpr int SU = SPIN ? 36 : 34;
    static constexpr int NOUT = 2 * 8 * NC;        // sums per round: (parity or recursion) x 8 rows x columns
    static constexpr int SO = NOUT + 2;            // per-warp stride of the round's sums
};

template <int SPIN, int NB>
struct AdjBSmem {
    using C = AdjBCfg<SPIN, NB>;
    double sum[2][kAdjWarps][C::SO];            // per-warp sums of a round, double-buffered
    double u[kAdjWarps][C::NREC][C::LCH][C::SU];
    double2 ag[2][16];
    int slot;
};

template <int SPIN, int NB>
__global__ void __launch_bounds__(kAdjWarps * 32, 2) adj_batch_kernel(BatchParams p, const double2 *__restrict__ V_all,
                                                                    double2 *__restrict__ part_all, int nb, int ngroups) {
    using C = AdjBCfg<SPIN, NB>;
    extern __shared__ __align__(16) unsigned char raw[];
    AdjBSmem<SPIN, NB> &sm = *reinterpret_cast<AdjBSmem<SPIN, NB> *>(raw);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int lr = lane >> 2, lk = lane & 3;
    constexpr int NCOMP = SPIN ? 2 : 1;
    for (;;) {
        const int it = next_cta_item(p.counter, &sm.slot);
        if (it >= p.nitems * ngroups) break;
        const int g = it / p.nitems;
        const int item = p.order[it - g * p.nitems];
        const int m = item / p.nsuper, sup = item - m * p.nsuper;
        const int b0map = g * C::MAPS, nmap = min(C::MAPS, nb - b0map);
        const int lmin = p.seed[m].lmin;
        const long long b0 = alm_index(lmin, m, p.lmax);
        const int nst = p.lmax - lmin + 1;
        const double ssign = ((m + lmin) & 1) ? -1.0 : 1.0;
        bool any = false;  // a block has written the rows
        // blocks nearest the equator start at the lowest degree: they go first, later ones add
        for (int blk = min(p.blk_lo + (sup + 1) * p.nblk, p.blk_hi) - 1; blk >= p.blk_lo + sup * p.nblk; --blk) {
            const int ring0 = blk * kBlockRings + warp * 32;
            const int my_start = ring0 < p.T ? min(p.lw[(size_t)m * p.ntiles + ring0 / kTileRings] - lmin, nst) : nst;
            int i_start = nst;  // even offsets, as every start
            for (int q = blk * (kBlockRings / kTileRings); q < (blk + 1) * (kBlockRings / kTileRings) && q < p.ntiles; ++q)
                i_start = min(i_start, p.lw[(size_t)m * p.ntiles + q] - lmin);
            if (i_start >= nst) continue;
            // rounds count from the block's start; a warp joins in the round that holds its own start
            const int wr_start = i_start + (max(0, my_start - i_start) & ~(C::LCH - 1));
            const int skip = my_start - wr_start;  // steps of its first round before its states apply
            Chains<SPIN> ch;
            ch.load(p, m, ring0, lane);
            // ring data of the warp's 32 rings as B operands: k block a, column block b
            double vf[2][8][NB];
#pragma unroll
            for (int a = 0; a < 8; ++a) {
                const int t = ring0 + 4 * a + lk;
                const bool in = t < p.T && JHTB_IN((long long)(p.nrings - 1 - t) * p.M + m, (long long)p.nrings * p.M, 208);
                const size_t rn = (size_t)t * p.M + m, rs = (size_t)(p.nrings - 1 - t) * p.M + m;
#pragma unroll
                for (int b = 0; b < NB; ++b) {
                    vf[0][a][b] = vf[1][a][b] = 0.0;
                    if (!in) continue;
                    if (SPIN) {
                        // column lr of the block: map, (north re, im, south re, im).  + : [Vp north | Vm south],
                        // - : [Vm north | Vp south] (signed)
                        const int map = 2 * b + (lr >> 2), e = lr & 3;
                        if (map >= nmap) continue;
                        const double2 *Vp = V_all + (size_t)(b0map + map) * 2 * p.nrings * p.M, *Vm = Vp + (size_t)p.nrings * p.M;
                        if (e < 2) {
                            const double2 vp = Vp[rn], vm = Vm[rn];
                            vf[0][a][b] = e ? vp.y : vp.x;
                            vf[1][a][b] = e ? vm.y : vm.x;
                        } else if (t < p.T - 1) {
                            const double2 vp = Vp[rs], vm = Vm[rs];
                            vf[0][a][b] = ssign * (e & 1 ? vm.y : vm.x);
                            vf[1][a][b] = ssign * (e & 1 ? vp.y : vp.x);
                        }
                    } else {
                        const int map = 4 * b + (lr >> 1);
                        if (map >= nmap) continue;
                        const double2 *V = V_all + (size_t)(b0map + map) * p.nrings * p.M;
                        double2 vn = V[rn], vs = make_double2(0.0, 0.0);
                        if (t < p.T - 1) {
                            vs = V[rs];
                            if (p.paired) spin0_unpair(vn, vs);
                        }
                        // even degrees sum vn + vs, odd ones vn - vs
                        vf[0][a][b] = lr & 1 ? vn.y + vs.y : vn.x + vs.x;
                        vf[1][a][b] = lr & 1 ? vn.y - vs.y : vn.x - vs.x;
                    }
                }
            }
            // rows below the block's start stay zero when no block has written them
            if (!any) {
                for (int i = threadIdx.x; i < i_start; i += blockDim.x)
                    for (int q = 0; q < nmap * NCOMP; ++q)
                        part_all[((size_t)(b0map + q / NCOMP) * p.nsuper + sup) * NCOMP * p.K + (size_t)(q % NCOMP) * p.K + b0 + i] =
                            make_double2(0.0, 0.0);
            }
            double2 rag = make_double2(0.0, 0.0);
            auto fetch = [&](int i0) {
                if (threadIdx.x >= C::LCH) return;
                const long long idx = b0 + i0 + threadIdx.x;
                rag = make_double2(0.0, 0.0);
                if (i0 + (int)threadIdx.x < nst && JHTB_IN(idx, p.K, 209)) rag = make_double2(p.alpha[idx], SPIN ? p.gamma[idx] : 0.0);
            };
            fetch(i_start);
            // the round's sums over the warps: thread = one output value, its running row value first
            auto finish = [&](int i0, int s) {
                for (int o = threadIdx.x; o < C::LCH * 2 * NCOMP * C::MAPS; o += blockDim.x) {
                    const int e = o % 2, map = (o / 2) % C::MAPS, comp = (o / (2 * C::MAPS)) % NCOMP, l = o / (2 * C::MAPS * NCOMP);
                    if (map >= nmap || i0 + l >= nst) continue;
                    double *dst = reinterpret_cast<double *>(part_all + ((size_t)(b0map + map) * p.nsuper + sup) * NCOMP * p.K +
                                                             (size_t)comp * p.K + b0 + i0 + l) + e;
                    double v = 0.0;
                    if (SPIN) {
                        // p2 = D+[Vp north] + s D-[Vp south], m2 = D-[Vm north] + s D+[Vm south], s = (-1)^(l - lmin)
                        const int a1 = (comp * 8 + l) * C::NC + 4 * map + e, a2 = ((1 - comp) * 8 + l) * C::NC + 4 * map + 2 + e;
                        double v2 = 0.0;
#pragma unroll
                        for (int w = 0; w < kAdjWarps; ++w) {
                            v += sm.sum[s][w][a1];
                            v2 += sm.sum[s][w][a2];
                        }
                        v = (l & 1) ? v - v2 : v + v2;
                    } else {
                        const int a1 = ((l & 1) * 8 + (l >> 1)) * C::NC + 2 * map + e;
#pragma unroll
                        for (int w = 0; w < kAdjWarps; ++w) v += sm.sum[s][w][a1];
                    }
                    *dst = any ? *dst + v : v;
                }
            };
            int s = 0;
            for (int i0 = i_start; i0 < nst; i0 += C::LCH, s ^= 1) {
                if (threadIdx.x < C::LCH) sm.ag[s][threadIdx.x] = rag;
                __syncthreads();  // coefficients staged; the sums of the round before are complete
                if (i0 + C::LCH < nst) fetch(i0 + C::LCH);
                double d[2][NB][2];
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int b = 0; b < NB; ++b) d[h][b][0] = d[h][b][1] = 0.0;
                if (i0 >= wr_start && my_start < nst) {
                    const int sk = i0 == wr_start ? skip : 0;
                    __syncwarp();
#pragma unroll 1
                    for (int gq = 0; gq < C::NG; ++gq) {
                        // 8 steps; in a warp's first round the steps before its start leave its states alone
                        double *out = &sm.u[warp][0][gq * 8][lane];
                        if (sk <= gq * 8) ch.template steps8<false>(&sm.ag[s][gq * 8], out, C::SU, C::LCH * C::SU, 0);
                        else ch.template steps8<true>(&sm.ag[s][gq * 8], out, C::SU, C::LCH * C::SU, sk - gq * 8);
                    }
                    __syncwarp();
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int row = SPIN ? lr : 2 * lr + h;
                        const double *ur = &sm.u[warp][SPIN ? h : 0][row][lk];
#pragma unroll
                        for (int a = 0; a < 8; ++a) {
                            const double af = ur[4 * a];
#pragma unroll
                            for (int b = 0; b < NB; ++b) dmma(d[h][b], af, vf[h][a][b]);
                        }
                    }
                }
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int b = 0; b < NB; ++b)
                        *reinterpret_cast<double2 *>(&sm.sum[s][warp][(h * 8 + lr) * C::NC + 8 * b + 2 * lk]) =
                            make_double2(d[h][b][0], d[h][b][1]);
                if (i0 > i_start) finish(i0 - C::LCH, s ^ 1);
            }
            __syncthreads();
            finish(i_start + ((nst - 1 - i_start) / C::LCH) * C::LCH, s ^ 1);
            __syncthreads();  // the buffers are reused by the next block or item
            any = true;
        }
        if (!any)
            for (int i = threadIdx.x; i < nst; i += blockDim.x)
                for (int q = 0; q < nmap * NCOMP; ++q)
                    part_all[((size_t)(b0map + q / NCOMP) * p.nsuper + sup) * NCOMP * p.K + (size_t)(q % NCOMP) * p.K + b0 + i] =
                        make_double2(0.0, 0.0);
    }
}

int sm_count() {
    int dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    return nsm;
}

BatchParams make_batch(const Plan &p, bool paired) {
    BatchParams q{};
    q.lmax = p.lmax;
    q.T = p.T;
    q.nrings = p.nrings;
    q.M = p.M;
    q.paired = paired;
    q.K = p.K;
    q.x = p.d_x;
    q.seed = p.d_seed;
    q.alpha = p.d_alpha;
    q.gamma = p.d_gamma;
    q.cnorm = p.d_cnorm;
    q.ntiles = p.a_ntiles;
    q.lw = p.d_a_lw;
    q.st = p.d_a_st;
    q.stsc = p.d_a_stsc;
    q.counter = p.d_counter;
    return q;
}

// persistent grid: the resident CTAs or the plan's tuned count, or fewer where the items do not fill them
template <typename K>
int batch_grid(const Plan &p, K k, int threads, int smem, long long items, int *grid) {
    JHTB_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, threads, smem) != cudaSuccess || n < 1) n = 1;
    if (p.leg_ctas > 0) n = std::min(n, p.leg_ctas);
    *grid = (int)std::max<long long>(1, std::min<long long>((long long)n * sm_count(), items));
    return JHTB_OK;
}

template <int SPIN, int NB>
int synth_groups(const Plan &p, BatchParams q, const double2 *alm, double2 *F, int nb, cudaStream_t s) {
    constexpr int MAPS = SynCfg<SPIN, NB>::MAPS;
    auto k = synth_batch_kernel<SPIN, NB>;
    const int smem = (int)sizeof(SynSmem<SPIN, NB>), groups = (nb + MAPS - 1) / MAPS;
    int rc, grid;
    if ((rc = batch_grid(p, k, kSynWarps * 32, smem, (long long)q.nitems * groups, &grid))) return rc;
    JHTB_CUDA_TRY(cudaMemsetAsync(p.d_counter, 0, sizeof(unsigned), s));
    k<<<grid, kSynWarps * 32, smem, s>>>(q, alm, F, nb, groups);
    JHTB_CUDA_TRY(cudaGetLastError());
    return JHTB_OK;
}

template <int SPIN, int NB>
int adj_groups(const Plan &p, BatchParams q, const double2 *V, double2 *part, int nb, cudaStream_t s) {
    constexpr int MAPS = AdjBCfg<SPIN, NB>::MAPS;
    auto k = adj_batch_kernel<SPIN, NB>;
    const int smem = (int)sizeof(AdjBSmem<SPIN, NB>), groups = (nb + MAPS - 1) / MAPS;
    int rc, grid;
    if ((rc = batch_grid(p, k, kAdjWarps * 32, smem, (long long)q.nitems * groups, &grid))) return rc;
    JHTB_CUDA_TRY(cudaMemsetAsync(p.d_counter, 0, sizeof(unsigned), s));
    k<<<grid, kAdjWarps * 32, smem, s>>>(q, V, part, nb, groups);
    JHTB_CUDA_TRY(cudaGetLastError());
    return JHTB_OK;
}

}  // namespace

JHTB_DEBUG_ACCESSOR(legendre_batch)

// The matrix-unit kernels pay where the one-map kernels would fill the GPU: below one wave of
// their items (16 warps on each of 148 SMs) both take the latency of the longest order (nside 64,
// lmax 96, 8 spin-2 maps: 24 and 45 us either way), and the one-map kernels keep a batch's results
// the bits of its single maps.  From there on two maps are already cheaper together (nside 256,
// lmax 512, spin 0: 0.099 against 2 x 0.067 ms).
constexpr long long kBatchMinItems = 148 * 16;

BatchSplit batch_split(const Plan &p, int nb) {
    const int per = p.spin ? 4 : 8, half = per / 2;
    BatchSplit s{};
    if ((long long)nb * p.M * p.ntiles < kBatchMinItems) {
        s.single = nb;
        return s;
    }
    int full = nb / per, rem = nb % per;
    if (rem > half) {
        ++full;
        rem = 0;
    }
    s.wide = std::min(nb, full * per);
    s.narrow = rem >= 2 ? rem : 0;
    s.single = nb - s.wide - s.narrow;
    return s;
}

int launch_batch_synth(const Plan &p, const double2 *alm, double2 *F, const BatchSplit &sp, bool paired, cudaStream_t s) {
    BatchParams q = make_batch(p, paired);
    q.order = p.d_b_synth_order;
    q.nitems = p.nb_synth;
    const size_t amap = (size_t)p.ncomp * p.K, fmap = (size_t)p.ncomp * p.nrings * p.M;
    int rc = JHTB_OK;
    if (sp.wide > 0) rc = p.spin ? synth_groups<2, 2>(p, q, alm, F, sp.wide, s) : synth_groups<0, 2>(p, q, alm, F, sp.wide, s);
    if (!rc && sp.narrow > 0) {
        const double2 *a = alm + sp.wide * amap;
        double2 *f = F + sp.wide * fmap;
        rc = p.spin ? synth_groups<2, 1>(p, q, a, f, sp.narrow, s) : synth_groups<0, 1>(p, q, a, f, sp.narrow, s);
    }
    return rc;
}

int launch_batch_adjoint(const Plan &p, const double2 *V, double2 *part, const BatchSplit &sp, bool paired, cudaStream_t s) {
    BatchParams q = make_batch(p, paired);
    q.order = p.d_b_adj_order;
    q.nitems = p.M * p.b_nsuper;
    q.nsuper = p.b_nsuper;
    q.blk_lo = p.ring_t0 / kBlockRings;
    q.blk_hi = (p.ring_t1 + kBlockRings - 1) / kBlockRings;
    q.nblk = (q.blk_hi - q.blk_lo + q.nsuper - 1) / q.nsuper;
    const size_t pmap = (size_t)p.b_nsuper * p.ncomp * p.K, fmap = (size_t)p.ncomp * p.nrings * p.M;
    int rc = JHTB_OK;
    if (sp.wide > 0) rc = p.spin ? adj_groups<2, 2>(p, q, V, part, sp.wide, s) : adj_groups<0, 2>(p, q, V, part, sp.wide, s);
    if (!rc && sp.narrow > 0) {
        const double2 *v = V + sp.wide * fmap;
        double2 *o = part + sp.wide * pmap;
        rc = p.spin ? adj_groups<2, 1>(p, q, v, o, sp.narrow, s) : adj_groups<0, 1>(p, q, v, o, sp.narrow, s);
    }
    return rc;
}

}  // namespace jhtb
