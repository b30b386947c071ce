// Gradients of the cubic delay-and-sum (no reference counterpart).
//
// Forward (per frame f, pixel p, summed over the taps that contribute):
//   img[p] += w * S_ch(x),  x = tau_tx(p) + tau_rx(p),  ch = (f, tx, rx)
//   S(x) = a y_j + b y_j+1 + (a^3 - a) z_j + (b^3 - b) z_j+1
// with the knot j, fractions a, b and (y, z) of the spline prefilter (whose
// float32 records hold the same cubic as a polynomial in b), z = 1/2 T^-1 D y (T = tridiag(0.5, 2, 0.5) on the interior
// samples, D the second difference; natural ends z_0 = z_nt-1 = 0).
//
// Three kernels, all deterministic (no atomics; every sum has a fixed order):
//   adj_delay_kernel    a warp per 32 pixels and share of the receives:
//                       dL/dx = g w S'(x) summed into dL/dtau_tx (ntx, np) and dL/dtau_rx (nrx, np) for
//                       Tabbed tables, or into dL/ds (np) for the Synthetic
//                       slowness form (x = (D_tx + D_rx) s + t0).
//   adj_scatter_kernel  one warp per (channel, part of the tiles): the transpose of
//                       the interpolation.  A tap adds (v, v b, v b^2, v b^3) to its
//                       interval's four moments in the warp's own shared-memory rows
//                       (512 intervals of the part's window at a time), lanes that
//                       share an interval in lane order; the moments then give dL/dy
//                       and dL/dz of the window's samples.  Parts are tiles of similar
//                       depth (adj_rank_kernel), so a part's window is short.
//   adj_finalize_kernel one warp per channel: adds the parts in order, then
//                       the adjoint of the prefilter, dL/drf = dL/dy +
//                       1/2 D^T T^-1 dL/dz (T is symmetric: the same chunked
//                       Thomas recurrences as the forward prefilter).
// Delays are recomputed from the tables or the geometry, never stored per tap;
// the tap decisions (range, threshold, correctly rounded knot) are the forward's.
#include <algorithm>

#include "das_rx.cuh"

namespace pgb {

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kWarmAdj = 32;  // warm-up of the chunked recurrences (0.268^32 ~ 5e-19)

// c_j = (xhi_j - xlo_j) / dt of the float32 knots (CoefRec<float>::make)
__device__ __forceinline__ float knot_step(const DasArgs &a, int j) {
    const float xlo = __fadd_rn(a.t0, __fmul_rn(a.dt, (float)j));
    const float xhi = __fadd_rn(a.t0, __fmul_rn(a.dt, (float)(j + 1)));
    return __fdiv_rn(__fsub_rn(xhi, xlo), a.dt);
}

// the upstream gradient of (frame f, receive r) at kernel-order pixel i (g.gk
// holds it in kernel order: gathered through pixel_index when there is one)
__device__ __forceinline__ long long grad_row(int sum, int f, int r, int nrx) {
    return sum == PYCBF_GB_SUM_TX_AND_RX ? (long long)f : (long long)f * nrx + r;
}

__global__ void adj_gather_kernel(const float *__restrict__ gout, const int *__restrict__ pidx,
                                  long long rows, long long np, float *__restrict__ gk) {
    const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= rows * np) return;
    const long long row = n / np, i = n - row * np;
    gk[n] = __ldg(gout + row * np + __ldg(pidx + i));
}

// ---------------------------------------------------------------------------
// delays / slowness: gather per pixel
// ---------------------------------------------------------------------------
// Bound by the issue rate and the latency of the gathers, as the forward: the taps
// are decided by its operations (knot_pairs), four at a time, in pairs, and the
// receives of 32 pixels are spread over the warps as in das_rx_kernel.  The warps share
// a column of delays and of weights (Tabbed) or path lengths (Synthetic); each has its
// own running dL/dtau_tx, added in warp order at the end.  11 transmits, 128 receives,
// 256 x 512 pixels: with a thread per pixel and all its receives 339 us from tables and
// 302 for the slowness (the whole call 955 and 1344 us); so 780 and 1113 (gathers from
// staged windows, as the TMA kernel of the forward makes them, measured 20 % slower).
//
// ONE: one frame on a time axis with packed decisions.  The gradient then goes into the
// weights, so a tap is its decisions, a gather, the slope of its cubic and two
// multiply-adds; otherwise the frames' products are summed per tap, and the knots of
// other axes are quotients.
//
// WARPS: eight, for tables of up to kFewRx receives four, or one or two for as many
// receives: each warp's running sums are a column of shared memory, which idle warps would
// hold too.  The whole call of 75 transmits, 512 samples, 256 x 512 pixels and 1 / 3 / 5 / 8
// receives 336 / 386 / 489 / 590 us, 458 / 619 / 717 / 810 with eight warps (373 / 482 / 661
// / 890 with a thread per pixel).
constexpr int kFewRx = 8;
template <int WARPS> constexpr int kDelayRun = WARPS < kRxWarps ? WARPS : kRxRun<GEOM_TABBED>;

template <int GEOM, int SUM, typename T, bool ONE, int WARPS>
__global__ void __launch_bounds__(32 * WARPS, 32 / WARPS) adj_delay_kernel(const __grid_constant__ AdjArgs g) {
    using rec = typename CoefRec<T>::raw;
    constexpr int G = kCubicGroup, kRun = kDelayRun<WARPS>;
    constexpr bool W = GEOM == GEOM_TABBED;
    const DasArgs &a = g.d;
    extern __shared__ float2 smp[];
    __shared__ float s_part[WARPS][32];  // largest weights; then dL/dslowness
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long long np = a.np;
    long long i = (long long)blockIdx.x * 32 + lane;
    const bool valid = i < np;
    if (!valid) i = np - 1;
    const int ntx = a.ntx, nrx = a.nrx, nfr = a.nframes, nt = a.nt;
    const int npair = (ntx + 3) / 4 * 2, ncol = 2 * npair;
    const float inf = __int_as_float(0x7f800000);
    const TapConst tc(a);
    float2 *stau = smp + lane, *sw = stau + (size_t)npair * 32,
           *sg = sw + (size_t)npair * 32 * (1 + w);  // Tabbed: [WARPS][npair][32]
    float *tabs = reinterpret_cast<float *>(smp + (size_t)npair * 32 * (2 + WARPS)) + lane;
    auto fetch_run = [&](int r0, int buf) {
        rx_fetch_run<kRun, WARPS>(a, tabs + (size_t)buf * 2 * kRun * 32, r0, min(kRun, nrx - r0), w, i);
    };
    if (W) fetch_run(0, 0);

    float pnt[3] = {0.f, 0.f, 0.f};
    float slow = 0.f;
    if (!W) {
        for (int k = 0; k < 3; ++k) if (k < a.ndim) pnt[k] = __ldg(a.geo.pnts + i * a.ndim + k);
        slow = __ldg(a.slow + i);
    }
    float amax = 0.f;
    for (int p = w; p < npair; p += WARPS) {
        float tau[2] = {inf, inf}, wt[2] = {0.f, 0.f};  // padding: never counts
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int t = 2 * p + h;
            if (t >= ntx) continue;
            if (W) {
                tau[h] = __ldg(a.tautx + (long long)t * np + i);
                wt[h] = __ldg(a.apodtx + (long long)t * np + i);
                amax = fmaxf(amax, fabsf(wt[h]));
            } else {
                float t0add;
                const bool ok = synth_tx_path(a, t, pnt, wt[h], t0add);
                tau[h] = slow_delay(ok, wt[h], slow, t0add);
            }
        }
        stau[(size_t)p * 32] = make_float2(tau[0], tau[1]);
        sw[(size_t)p * 32] = make_float2(wt[0], wt[1]);
    }
    if (W) {
        for (int p = 0; p < npair; ++p) sg[(size_t)p * 32] = make_float2(0.f, 0.f);
        s_part[w][lane] = amax;
    }
    __syncthreads();
    if (W) {
#pragma unroll
        for (int k = 0; k < WARPS; ++k) amax = fmaxf(amax, s_part[k][lane]);
    }
    const long long chs = (long long)nrx * nt;
    unsigned off[G];
#pragma unroll
    for (int k = 0; k < G; ++k) off[k] = (unsigned)k * (unsigned)chs - kKnotBits;

    const float gpix = nfr == 1 && SUM == PYCBF_GB_SUM_TX_AND_RX ? __ldg(g.gk + i) : 0.f;
    float gs = 0.f;
    // receive r by warp r % WARPS (a run is a multiple of WARPS)
    int buf = 1;
    for (int r = w; r < nrx; r += WARPS) {
        float trx, arx = 1.f, Drx = 0.f;
        bool live;
        if (W) {
            const int e = r % kRun;
            if (e == w) {  // the warp's first receive of a run
                buf ^= 1;
                fetch_run(min(r - w + kRun, nrx), buf ^ 1);  // none past the last: an empty group
                copy_wait_but_one();
            }
            const float *tab = tabs + (size_t)buf * 2 * kRun * 32;
            trx = tab[e * 32];
            arx = tab[(kRun + e) * 32];
            live = __fmul_rn(amax, fabsf(arx)) >= a.thresh;
        } else {
            live = synth_rx_path(a, r, pnt, Drx);
            trx = slow_delay(live, Drx, slow, 0.f);
        }
        float grx = 0.f;
        bool tap = false;  // some tap of this pixel and receive counts
        // the forward's exact reject, by warps: no tap of the others passes its tests
        if (__any_sync(kFull, live)) {
            const float gp0 = nfr == 1 && SUM == PYCBF_GB_SUM_TX_ONLY
                                  ? __ldg(g.gk + (long long)r * np + i) : gpix;
            const float gq = CoefRec<T>::kPoly ? gp0 * a.inv_dt : gp0;
            const rec *row = static_cast<const rec *>(a.data) + (long long)r * nt;
            for (int t0 = 0; t0 < ncol; t0 += G) {
                float2 tt2[G / 2], w2[G / 2], x2[G / 2], fj2[G / 2];
                unsigned rk[G];
#pragma unroll
                for (int p = 0; p < G / 2; ++p) {
                    tt2[p] = stau[(size_t)(t0 / 2 + p) * 32];
                    w2[p] = sw[(size_t)(t0 / 2 + p) * 32];
                    if (GEOM == GEOM_TABBED) w2[p] = mul2_rn(w2[p], make_float2(arx, arx));
                }
                knot_pairs<G / 2>(a, tc, tt2, trx, x2, fj2, rk);
                if (!ONE && !a.fast_axis) {  // knots past the record are clamped
#pragma unroll
                    for (int k = 0; k < G; ++k) {
                        const float fl = fminf(floorf(__fdiv_rn(__fsub_rn(pair_lane(x2, k), a.t0), a.dt)),
                                               (float)(nt - 1));
                        if (k & 1) fj2[k >> 1].y = fl;
                        else fj2[k >> 1].x = fl;
                        rk[k] = kKnotBits + (unsigned)(int)fl;
                    }
                }
                bool ok[G];
                float sum[G];
#pragma unroll
                for (int k = 0; k < G; ++k) {
                    const float x = pair_lane(x2, k);
                    ok[k] = (x >= tc.t0) && (x <= tc.xmax);
                    if (GEOM == GEOM_TABBED) ok[k] = ok[k] && (fabsf(pair_lane(w2, k)) >= tc.thresh);
                    sum[k] = 0.f;
                }
                if constexpr (ONE) {
                    rec c[G];
#pragma unroll
                    for (int k = 0; k < G; ++k)
                        if (ok[k]) c[k] = __ldg(row + (rk[k] + off[k]));
                    row += G * chs;
#pragma unroll
                    for (int p = 0; p < G / 2; ++p) {
                        float2 slope;
                        if constexpr (CoefRec<T>::kPoly) {  // c1 + 2 b (c2 + 1.5 b c3), times 1/dt (gq)
                            const float2 b2 = knot_frac2(tc, x2[p], fj2[p]);
                            const float2 u2 = add2_rn(b2, b2), v2 = mul2_rn(b2, make_float2(1.5f, 1.5f));
                            const rec &cx = c[2 * p], &cy = c[2 * p + 1];
                            slope.x = fmaf(fmaf(cx.w, v2.x, cx.z), u2.x, cx.y);
                            slope.y = fmaf(fmaf(cy.w, v2.y, cy.z), u2.y, cy.y);
                        } else {
                            slope.x = Kind<PYCBF_GB_INTERP_CUBIC, T>::slope(
                                CoefRec<T>::unpack(c[2 * p]), x2[p].x, fj2[p].x, a);
                            slope.y = Kind<PYCBF_GB_INTERP_CUBIC, T>::slope(
                                CoefRec<T>::unpack(c[2 * p + 1]), x2[p].y, fj2[p].y, a);
                        }
                        if (W) {
                            const float2 h = mul2_rn(w2[p], make_float2(gq, gq));
                            float2 d = sg[(size_t)(t0 / 2 + p) * 32];
                            if (ok[2 * p]) {
                                d.x = fmaf(h.x, slope.x, d.x);
                                grx = fmaf(h.x, slope.x, grx);
                            }
                            if (ok[2 * p + 1]) {
                                d.y = fmaf(h.y, slope.y, d.y);
                                grx = fmaf(h.y, slope.y, grx);
                            }
                            sg[(size_t)(t0 / 2 + p) * 32] = d;
                        } else {  // dx/ds = D_tx + D_rx; times gq at the end of the receive
                            const float2 D = add2_rn(w2[p], make_float2(Drx, Drx));
                            if (ok[2 * p]) grx = fmaf(slope.x, D.x, grx);
                            if (ok[2 * p + 1]) grx = fmaf(slope.y, D.y, grx);
                            tap = tap || ok[2 * p] || ok[2 * p + 1];
                        }
                    }
                    continue;
                }
                for (int f = 0; f < nfr; ++f) {
                    const float gp = nfr == 1 ? gp0 : __ldg(g.gk + grad_row(SUM, f, r, nrx) * np + i);
                    const rec *row = static_cast<const rec *>(a.data) +
                                     (((long long)f * ntx + t0) * nrx + r) * nt;
                    rec c[G];
#pragma unroll
                    for (int k = 0; k < G; ++k) {
                        if (ok[k])
                            c[k] = a.fast_axis ? __ldg(row + (rk[k] + off[k]))
                                               : __ldg(row + k * chs + (long long)(rk[k] - kKnotBits));
                    }
#pragma unroll
                    for (int k = 0; k < G; ++k) {
                        float slope;
                        if constexpr (CoefRec<T>::kPoly) {
                            const float2 b2 = knot_frac2(tc, x2[k >> 1], fj2[k >> 1]);
                            const float b = (k & 1) ? b2.y : b2.x;
                            slope = fmaf(fmaf(3.f * c[k].w, b, 2.f * c[k].z), b, c[k].y) * a.inv_dt;
                        } else {
                            slope = Kind<PYCBF_GB_INTERP_CUBIC, T>::slope(
                                CoefRec<T>::unpack(c[k]), pair_lane(x2, k), pair_lane(fj2, k), a);
                        }
                        if (ok[k]) sum[k] = fmaf(gp, slope, sum[k]);
                    }
                }
#pragma unroll
                for (int p = 0; p < G / 2; ++p) {
                    if (GEOM == GEOM_TABBED) {
                        float2 d = sg[(size_t)(t0 / 2 + p) * 32];
                        if (ok[2 * p]) {
                            d.x = fmaf(w2[p].x, sum[2 * p], d.x);
                            grx = fmaf(w2[p].x, sum[2 * p], grx);
                        }
                        if (ok[2 * p + 1]) {
                            d.y = fmaf(w2[p].y, sum[2 * p + 1], d.y);
                            grx = fmaf(w2[p].y, sum[2 * p + 1], grx);
                        }
                        sg[(size_t)(t0 / 2 + p) * 32] = d;
                    } else {  // dx/ds = D_tx + D_rx
                        if (ok[2 * p]) gs = fmaf(sum[2 * p], w2[p].x + Drx, gs);
                        if (ok[2 * p + 1]) gs = fmaf(sum[2 * p + 1], w2[p].y + Drx, gs);
                    }
                }
            }
            if (ONE && !W && tap) gs = fmaf(gq, grx, gs);  // else gq may be infinite or NaN
        }
        if (W && g.grad_taurx && valid) g.grad_taurx[(long long)r * np + i] = grx;
    }
    if (!W) s_part[w][lane] = gs;
    __syncthreads();
    if (!valid) return;
    if (W && g.grad_tautx) {
        const float2 *part = sw + (size_t)npair * 32;
        for (int p = w; p < npair; p += WARPS) {
            float2 d = part[(size_t)p * 32];
#pragma unroll
            for (int k = 1; k < WARPS; ++k) d = add2_rn(d, part[((size_t)k * npair + p) * 32]);
            if (2 * p < ntx) g.grad_tautx[(long long)(2 * p) * np + i] = d.x;
            if (2 * p + 1 < ntx) g.grad_tautx[(long long)(2 * p + 1) * np + i] = d.y;
        }
    }
    if (!W && w == 0 && g.grad_slow) {
#pragma unroll
        for (int k = 1; k < WARPS; ++k) gs += s_part[k][lane];
        g.grad_slow[i] = gs;
    }
}

// ---------------------------------------------------------------------------
// what the scatter needs to know of each tile of kBlock pixels: which receives can
// contribute to it (Tabbed: some pixel has fl(max_t |apodtx| * |apodrx|) >= thresh,
// so every tap of a dead pair fails the threshold; Synthetic: the receive's mask
// accepts some pixel), and the range of every transmit's and receive's delays (over
// the pixels that the receive reaches; empty: inf, -inf).  TABLES: also writes the
// Synthetic delays, NaN where masked.  One CTA per tile (blockIdx.x) and share of the
// receives (blockIdx.y).
// ---------------------------------------------------------------------------
// floats as integers of the same order (no NaN), for the warp's integer reductions
__device__ __forceinline__ int to_key(float v) {
    const int b = __float_as_int(v);
    return b < 0 ? b ^ 0x7fffffff : b;
}
__device__ __forceinline__ float from_key(int k) { return __int_as_float(k < 0 ? k ^ 0x7fffffff : k); }

template <int GEOM, bool TABLES>
__global__ void __launch_bounds__(kBlock) adj_range_kernel(const __grid_constant__ AdjArgs g) {
    constexpr int kWarps = kBlock / 32, M = kBlock / 32;  // a warp per element, M pixels a lane
    const DasArgs &a = g.d;
    const float inf = __int_as_float(0x7f800000), nan = __int_as_float(0x7fc00000);
    __shared__ float s_amax[kWarps][kBlock];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long long tile = blockIdx.x, tiles = gridDim.x;
    const long long i0 = tile * kBlock + lane;
    float2 *ranges = g.ranges ? g.ranges + tile * (a.ntx + a.nrx) : nullptr;
    float pnt[M][3], slow[M], amax[M];
#pragma unroll
    for (int m = 0; m < M; ++m) {
        const long long i = i0 + 32 * m;
        amax[m] = slow[m] = 0.f;
        for (int k = 0; k < 3; ++k)
            pnt[m][k] = (GEOM != GEOM_TABBED && i < a.np && k < a.ndim)
                            ? __ldg(a.geo.pnts + i * a.ndim + k) : 0.f;
        if (GEOM != GEOM_TABBED && i < a.np) slow[m] = __ldg(a.slow + i);
    }
    auto element = [&](int e) {
        const bool tx = e < a.ntx;
        const int r = e - a.ntx;
        float lo = inf, hi = -inf;
        bool any = false;
#pragma unroll
        for (int m = 0; m < M; ++m) {
            const long long i = i0 + 32 * m;
            if (i >= a.np) continue;
            float tau;
            bool live = true;
            if (GEOM == GEOM_TABBED) {
                tau = __ldg((tx ? a.tautx + (long long)e * a.np : a.taurx + (long long)r * a.np) + i);
                if (tx) amax[m] = fmaxf(amax[m], fabsf(__ldg(a.apodtx + (long long)e * a.np + i)));
                else live = __fmul_rn(amax[m], fabsf(__ldg(a.apodrx + (long long)r * a.np + i))) >= a.thresh;
            } else {
                float D, t0add = 0.f;
                live = tx ? synth_tx_path(a, e, pnt[m], D, t0add) : synth_rx_path(a, r, pnt[m], D);
                tau = slow_delay(live, D, slow[m], t0add);
                if (TABLES)
                    (tx ? g.tau_tx + (long long)e * a.np : g.tau_rx + (long long)r * a.np)[i] =
                        live ? tau : nan;
            }
            any |= live;
            if (live && fabsf(tau) < inf) {
                lo = fminf(lo, tau);
                hi = fmaxf(hi, tau);
            }
        }
        lo = from_key(__reduce_min_sync(kFull, to_key(lo)));
        hi = from_key(__reduce_max_sync(kFull, to_key(hi)));
        any = __any_sync(kFull, any);
        if (lane == 0 && !(tx && blockIdx.y > 0)) {
            if (ranges) ranges[e] = make_float2(lo, hi);
            if (ranges && tx && e == a.ntx / 2) g.depth[tile] = lo;
            if (!tx) g.live[(long long)r * tiles + tile] = any ? 1 : 0;
        }
    };
    // every share needs the Tabbed weights; the transmits are the first share's otherwise
    if (GEOM == GEOM_TABBED || blockIdx.y == 0)
        for (int t = w; t < a.ntx; t += kWarps) element(t);
    if (GEOM == GEOM_TABBED) {  // the largest weight over every warp's transmits
#pragma unroll
        for (int m = 0; m < M; ++m) s_amax[w][lane + 32 * m] = amax[m];
        __syncthreads();
#pragma unroll
        for (int m = 0; m < M; ++m)
            for (int k = 0; k < kWarps; ++k) amax[m] = fmaxf(amax[m], s_amax[k][lane + 32 * m]);
    }
    for (int r = blockIdx.y * kWarps + w; r < a.nrx; r += gridDim.y * kWarps) element(a.ntx + r);
}

// The tiles by depth -- the earliest delay of the middle transmit -- so that the
// consecutive tiles of a part share a short window of samples, in any pixel order:
// each tile's place is the number of tiles before it (ties by tile number, so the
// order is always the same).
constexpr long long kRankTiles = 1 << 16;  // above: the pixels' own order

__global__ void __launch_bounds__(256) adj_rank_kernel(const float *__restrict__ depth, int tiles,
                                                       int *__restrict__ order) {
    const int t = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;  // a warp per tile
    if (t >= tiles) return;
    const float key = __ldg(depth + t);
    int rank = 0;
    for (int k = lane; k < tiles; k += 32) {
        const float v = __ldg(depth + k);
        rank += (v < key || (v == key && k < t)) ? 1 : 0;
    }
    rank = __reduce_add_sync(kFull, rank);
    if (lane == 0) order[rank] = t;
}

// ---------------------------------------------------------------------------
// channel data: transpose of the interpolation, one warp per (channel, part).  The
// four warps of a CTA take four transmits of one receive (they share its delays,
// weights and gradient in L1) and never wait for one another.
//
// TABLES: delays from tau_tx / tau_rx (NaN: masked), weights Tabbed only.
//
// What the walk waits for is its loads, so a warp has the next live tile's inputs (20
// a lane) in flight, and which lanes share an interval: along image lines (neighbouring
// pixels some samples apart) none do, and a compare with the next lane shows it.  11 x
// 128 x 2048 samples, 256 x 512 pixels: 321 us along lines, 478 in Morton order with
// masks (59 and 52 % of the issue slots), against 920 and 1271 for one CTA a channel
// part whose warps took turns on full-length rows between barriers.
constexpr int kSeg = 512;  // intervals of a warp's rows: 8 KB, seven CTAs an SM
constexpr int kPartTiles = 16384;  // a part's tile list has to fit shared memory

template <int GEOM, int SUM, bool TABLES>
__global__ void __launch_bounds__(128, 5) adj_scatter_kernel(const __grid_constant__ AdjArgs g,
                                                             int per, int Lp) {
    const DasArgs &a = g.d;
    extern __shared__ float4 rows[];
    int *list = reinterpret_cast<int *>(rows + 4 * kSeg);  // [per] the part's live tiles
    __shared__ int s_count[4];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long long np = a.np;
    const int ntx = a.ntx, nrx = a.nrx, nt = a.nt, nel = ntx + nrx;
    const int r = blockIdx.x % nrx;
    const int tq = blockIdx.x / nrx, nq = (ntx + 3) / 4;  // group of four transmits, over frames
    const int f = tq / nq, t = tq % nq * 4 + w;
    const int q = blockIdx.y;
    const long long nch = (long long)a.nframes * ntx * nrx;
    const long long ch = ((long long)f * ntx + t) * nrx + r;
    const int tiles = (int)((np + kBlock - 1) / kBlock);
    // the part's tiles that receive r can reach, in order
    int nlist = 0;
    {
        const unsigned char *live = g.live + (long long)r * tiles;
        const int k1 = min(tiles, (q + 1) * per);
        for (int b = q * per; b < k1; b += 128) {
            const int k = b + threadIdx.x;
            const int tile = k < k1 ? (g.order ? __ldg(g.order + k) : k) : 0;
            const bool on = k < k1 && live[tile];
            const unsigned m = __ballot_sync(kFull, on);
            if (lane == 0) s_count[w] = __popc(m);
            __syncthreads();
            int at = nlist + __popc(m & ((1u << lane) - 1u));
            for (int v = 0; v < 4; ++v) {
                at += v < w ? s_count[v] : 0;
                nlist += s_count[v];
            }
            if (on) list[at] = tile;
            __syncthreads();
        }
    }
    if (t >= ntx) return;  // a whole warp; no barrier below
    float4 *row = rows + w * kSeg;
    float *py = g.partial + ((size_t)q * nch + ch) * 2 * Lp, *pz = py + Lp;

    // samples that those tiles' taps of this channel can touch: intervals [w0, w1)
    float4 rng = make_float4(__int_as_float(0x7f800000), -__int_as_float(0x7f800000),
                             __int_as_float(0x7f800000), -__int_as_float(0x7f800000));
    for (int k = lane; k < (g.ranges ? nlist : 0); k += 32) {
        const float2 u = __ldg(g.ranges + (long long)list[k] * nel + t);
        const float2 v = __ldg(g.ranges + (long long)list[k] * nel + ntx + r);
        rng = make_float4(fminf(rng.x, u.x), fmaxf(rng.y, u.y), fminf(rng.z, v.x), fmaxf(rng.w, v.y));
    }
    const float lo = __fadd_rn(from_key(__reduce_min_sync(kFull, to_key(rng.x))),
                               from_key(__reduce_min_sync(kFull, to_key(rng.z))));
    const float hi = __fadd_rn(from_key(__reduce_max_sync(kFull, to_key(rng.y))),
                               from_key(__reduce_max_sync(kFull, to_key(rng.w))));
    int w0 = 0, w1 = g.ranges ? 0 : nt;  // without the ranges: every interval
    if (g.ranges && lo <= hi && hi >= a.t0 && lo <= a.xmax) {
        w0 = lo <= a.t0 ? 0 : (int)floorf(__fdiv_rn(__fsub_rn(lo, a.t0), a.dt));
        w1 = hi >= a.xmax ? nt : min(nt, (int)floorf(__fdiv_rn(__fsub_rn(hi, a.t0), a.dt)) + 1);
        w0 = min(w0, nt - 1);
    }
    if (lane == 0) {  // samples w0 .. w1 of the rows: kept in the place past their last sample
        py[nt] = __int_as_float(w0);
        pz[nt] = __int_as_float(w1);
    }

    const float *ptx = (GEOM == GEOM_TABBED ? a.tautx : g.tau_tx) + (long long)t * np;
    const float *prx = (GEOM == GEOM_TABBED ? a.taurx : g.tau_rx) + (long long)r * np;
    const float *pat = a.apodtx + (long long)t * np, *par = a.apodrx + (long long)r * np;
    const float *grow = g.gk + grad_row(SUM, f, r, nrx) * np;
    constexpr int M = kBlock / 32;  // steps of 32 pixels in a tile
    struct In {
        float tx[M], rx[M], wt[M], wr[M], gp[M];
    };
    // the inputs of a lane's pixels of one tile: delays, weights and gradient
    auto fetch = [&](int tile, In &in) {
#pragma unroll
      for (int m = 0; m < M; ++m) {
        const long long i = (long long)tile * kBlock + 32 * m + lane;
        in.tx[m] = __int_as_float(0x7fc00000);  // NaN delay: no tap
        in.rx[m] = in.wt[m] = in.wr[m] = in.gp[m] = 0.f;
        if (i >= np) continue;
        if (GEOM == GEOM_TABBED || TABLES) {
            in.tx[m] = __ldg(ptx + i);
            in.rx[m] = __ldg(prx + i);
        } else {
            float pnt[3] = {0.f, 0.f, 0.f}, Dt, t0add, Dr;
            for (int k = 0; k < 3; ++k) if (k < a.ndim) pnt[k] = __ldg(a.geo.pnts + i * a.ndim + k);
            const float s = __ldg(a.slow + i);
            const bool okt = synth_tx_path(a, t, pnt, Dt, t0add);
            const bool okr = synth_rx_path(a, r, pnt, Dr);
            if (okt && okr) in.tx[m] = slow_delay(true, Dt, s, t0add);
            in.rx[m] = slow_delay(true, Dr, s, 0.f);
        }
        in.gp[m] = __ldg(grow + i);
        if (GEOM == GEOM_TABBED) {
            in.wt[m] = __ldg(pat + i);
            in.wr[m] = __ldg(par + i);
        }
      }
    };

    float4 carry = make_float4(0.f, 0.f, 0.f, 0.f);  // the interval before the segment
    for (int s0 = w0; s0 < w1; s0 += kSeg) {
        const int n = min(kSeg, w1 - s0);
        for (int m = lane; m < n; m += 32) row[m] = make_float4(0.f, 0.f, 0.f, 0.f);
        __syncwarp();
        // the live tiles in turn, the next one's inputs fetched meanwhile
        In cur, nxt;
        if (nlist > 0) fetch(list[0], cur);
        for (int k = 0; k < nlist; ++k, cur = nxt) {
          if (k + 1 < nlist) fetch(list[k + 1], nxt);
#pragma unroll
          for (int m = 0; m < M; ++m) {
            const float x = __fadd_rn(cur.tx[m], cur.rx[m]);
            int j;
            bool fix;
            using K = Kind<PYCBF_GB_INTERP_CUBIC, float>;
            bool hit = K::index(x, a, j, fix);
            if (fix) hit = K::index_exact(x, a, j);
            float v = cur.gp[m];
            if (GEOM == GEOM_TABBED) {
                const float wt = __fmul_rn(cur.wt[m], cur.wr[m]);
                hit = hit && fabsf(wt) >= a.thresh;
                v *= wt;
            }
            j -= s0;
            hit = hit && (unsigned)j < (unsigned)n;
            if (__any_sync(kFull, hit)) {
                const float xlo = __fadd_rn(a.t0, __fmul_rn(a.dt, (float)(j + s0)));
                const float b = __fmul_rn(__fsub_rn(x, xlo), a.inv_dt);
                const float m1 = v * b, m2 = m1 * b, m3 = m2 * b;
                // lanes of one interval add in lane order.  Along a line of pixels the
                // intervals mostly increase from lane to lane: then no two are alike.
                const int key = hit ? j : -1 - lane;
                const int up = __shfl_up_sync(kFull, j, 1);
                if (__all_sync(kFull, hit && (lane == 0 || j > up))) {
                    float4 c = row[j];
                    row[j] = make_float4(c.x + v, c.y + m1, c.z + m2, c.w + m3);
                } else {
                    const unsigned grp = __match_any_sync(kFull, key);
                    const int mine = __popc(grp & ((1u << lane) - 1u));
                    const int most = (int)__reduce_max_sync(kFull, hit ? (unsigned)mine : 0u);
                    for (int turn = 0; turn <= most; ++turn) {
                        if (hit && mine == turn) {
                            float4 c = row[j];
                            row[j] = make_float4(c.x + v, c.y + m1, c.z + m2, c.w + m3);
                        }
                        __syncwarp();
                    }
                }
                __syncwarp();
            }
          }
        }
        __syncwarp();
        // samples s0 .. s0 + n - 1 (and, past the last segment, s0 + n) from the moments of
        // the intervals on either side, with a = c_j - b as in the records
        const bool last = s0 + n >= w1;
        for (int m0 = 0; m0 < n + (last ? 1 : 0); m0 += 32) {
            const int m = m0 + lane;
            const float4 here = m < n ? row[m] : make_float4(0.f, 0.f, 0.f, 0.f);
            const float4 before = m == 0 ? carry : (m <= n ? row[m - 1] : here);
            if (s0 + m < nt && (m < n || (last && m == n))) {
                const float c = knot_step(a, s0 + m), c2 = c * c;
                py[s0 + m] = fmaf(c, here.x, -here.y) + before.y;
                pz[s0 + m] = fmaf(c2 * c - c, here.x,
                                  fmaf(1.f - 3.f * c2, here.y, fmaf(3.f * c, here.z, -here.w))) +
                             (before.w - before.y);
            }
        }
        carry = row[n - 1];
        __syncwarp();
    }
}

// v = T^-1 dL/dz in place of zv (one warp; u: scratch of nt floats), with v_0 =
// v_nt-1 = 0: the chunked recurrences of the forward prefilter (T symmetric)
__device__ __forceinline__ void prefilter_adjoint_warp(float *zv, float *u, int nt,
                                                       const SplineTable &tab, int lane) {
    if (lane == 0) u[0] = 0.f;
    __syncwarp();
    // T v = dL/dz on the interior samples 1..nt-2 (v_0 = v_nt-1 = 0)
    const int C = ((nt + 31) >> 5) | 1;
    const int s = lane * C;
    const int e = min(s + C, nt);
    {
        const int ib = max(s, 1), ie = min(e, nt - 1);
        if (ib < ie) {
            float up = 0.f;
            for (int k = max(1, ib - kWarmAdj); k < ie; ++k) {
                const float uk = fmaf(-0.5f, up, zv[k]) * tab.invp[min(k, kSplineTab - 1)];
                if (k >= ib) u[k] = uk;
                up = uk;
            }
        }
    }
    __syncwarp();  // every lane is past its reads of dL/dz
    {
        const int kb = max(s, 1), ke = min(e, nt - 1);
        if (kb < ke) {
            float vn = 0.f;
            for (int k = min(nt - 2, ke - 1 + kWarmAdj); k >= kb; --k) {
                const float vk = fmaf(tab.c[min(k, kSplineTab - 1)], vn, u[k]);
                if (k < ke) zv[k] = vk;
                vn = vk;
            }
        }
    }
    __syncwarp();
    if (lane == 0) {
        zv[0] = 0.f;
        zv[nt - 1] = 0.f;
    }
    __syncwarp();
}

// ---------------------------------------------------------------------------
// adjoint of the prefilter, one warp per channel
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
adj_finalize_kernel(const float *__restrict__ partial, int nparts, long long nch, int nt, int Lp,
                    float *__restrict__ grad_rf, const __grid_constant__ SplineTable tab) {
    extern __shared__ float smem[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, wpb = blockDim.x >> 5;
    const long long ch = (long long)blockIdx.x * wpb + w;
    if (ch >= nch) return;
    const int stride = (nt + 4) & ~3;
    float *zv = smem + (size_t)w * 2 * stride;  // dL/dz, then v = T^-1 dL/dz in place
    float *u = zv + stride;
    const float *p0 = partial + (size_t)ch * 2 * Lp;
    const size_t pstride = (size_t)nch * 2 * Lp;  // between parts
    // the parts' samples into dst, parts in order, each from its window only; sample n is
    // lane n % 32's in every part, so no lane adds to another's sum
    auto sum_parts = [&](float *dst, int off) {
        for (int n = lane; n < nt; n += 32) dst[n] = 0.f;
        int2 wins = make_int2(0, 0);  // of part q0 + lane
        for (int q = 0; q < nparts; ++q) {
            if (q % 32 == 0 && q + lane < nparts) {
                const float *row = p0 + (q + lane) * pstride;
                wins = make_int2(__float_as_int(row[nt]), __float_as_int(row[Lp + nt]));
            }
            const int2 win = make_int2(__shfl_sync(kFull, wins.x, q % 32), __shfl_sync(kFull, wins.y, q % 32));
            const float *src = p0 + q * pstride + off;
            if (win.x >= win.y) continue;
#pragma unroll 4
            for (int n = win.x + ((lane - win.x) & 31); n <= min(win.y, nt - 1); n += 32)
                dst[n] += src[n];
        }
    };
    sum_parts(zv, Lp);
    __syncwarp();
    prefilter_adjoint_warp(zv, u, nt, tab, lane);
    sum_parts(u, 0);
    __syncwarp();
    float *dst = grad_rf + ch * (long long)nt;
    for (int n = lane; n < nt; n += 32) {
        const float vm = n >= 1 ? zv[n - 1] : 0.f;
        const float vp = n + 1 < nt ? zv[n + 1] : 0.f;
        dst[n] = fmaf(0.5f, vm - 2.f * zv[n] + vp, u[n]);
    }
}


template <int WARPS> size_t delay_smem_bytes(int geom, int ntx) {
    const size_t column = (size_t)((ntx + 3) / 4 * 4) * 32 * sizeof(float);
    return geom == GEOM_TABBED ? (2 + WARPS) * column + 4 * kDelayRun<WARPS> * 32 * sizeof(float)
                               : 2 * column;
}

template <int GEOM, int SUM, typename T, int WARPS>
cudaError_t launch_delay_warps(const AdjArgs &g, cudaStream_t s) {
    auto kern = g.d.fast_axis && g.d.nframes == 1 ? adj_delay_kernel<GEOM, SUM, T, true, WARPS>
                                                  : adj_delay_kernel<GEOM, SUM, T, false, WARPS>;
    const size_t smem = delay_smem_bytes<WARPS>(GEOM, g.d.ntx);
    if (smem > 40 * 1024) {  // with the static part
        cudaError_t err = allow_smem(kern, delay_smem_bytes<WARPS>(GEOM, kMaxAdjTx));
        if (err != cudaSuccess) return err;
    }
    kern<<<(unsigned)((g.d.np + 31) / 32), 32 * WARPS, smem, s>>>(g);
    return cudaGetLastError();
}

template <int GEOM, int SUM, typename T>
cudaError_t launch_delay_one(const AdjArgs &g, cudaStream_t s) {
    if constexpr (GEOM == GEOM_TABBED) {
        if (g.d.nrx == 1) return launch_delay_warps<GEOM, SUM, T, 1>(g, s);
        if (g.d.nrx == 2) return launch_delay_warps<GEOM, SUM, T, 2>(g, s);
        if (g.d.nrx <= kFewRx) return launch_delay_warps<GEOM, SUM, T, 4>(g, s);
    }
    return launch_delay_warps<GEOM, SUM, T, kRxWarps>(g, s);
}

template <int GEOM, int SUM>
cudaError_t launch_scatter_one(const AdjArgs &g0, cudaStream_t s) {
    AdjArgs g = g0;
    const DasArgs &a = g.d;
    const long long nch = (long long)a.nframes * a.ntx * a.nrx;
    const long long tiles = (a.np + kBlock - 1) / kBlock;
    const int nparts = adjoint_parts(nch, a.np);
    const int per = (int)((tiles + nparts - 1) / nparts);
    const int Lp = (a.nt + 1 + 3) & ~3;
    // Synthetic delays once into tables where they fit (the scatter would take a root
    // and a quotient per tap again)
    const bool tables = GEOM == GEOM_TABBED || (g.tau_tx && g.tau_rx);
    constexpr bool kSynth = GEOM != GEOM_TABBED;
    const dim3 rgrid((unsigned)tiles, (unsigned)std::min(4, (a.nrx + 3) / 4));
    if (tables) adj_range_kernel<GEOM, kSynth><<<rgrid, kBlock, 0, s>>>(g);
    else adj_range_kernel<GEOM, false><<<rgrid, kBlock, 0, s>>>(g);
    cudaError_t err = cudaGetLastError();
    if (err != cudaSuccess) return err;
    if (tiles <= kRankTiles && g.ranges) {
        adj_rank_kernel<<<(unsigned)((tiles + 7) / 8), 256, 0, s>>>(g.depth, (int)tiles, g.order);
        if ((err = cudaGetLastError()) != cudaSuccess) return err;
    } else {
        g.order = nullptr;
    }
    const size_t smem = 4 * kSeg * sizeof(float4) + per * sizeof(int);
    const size_t most = 4 * kSeg * sizeof(float4) + kPartTiles * sizeof(int);
    err = allow_smem(
        tables ? adj_scatter_kernel<GEOM, SUM, true> : adj_scatter_kernel<GEOM, SUM, !kSynth>, most);
    if (err != cudaSuccess) return err;
    const long long groups = (long long)a.nframes * ((a.ntx + 3) / 4) * a.nrx;
    if (groups > 0x7fffffffLL) return cudaErrorInvalidValue;
    const dim3 grid((unsigned)groups, (unsigned)nparts);
    if (tables) adj_scatter_kernel<GEOM, SUM, true><<<grid, 128, smem, s>>>(g, per, Lp);
    else adj_scatter_kernel<GEOM, SUM, !kSynth><<<grid, 128, smem, s>>>(g, per, Lp);
    err = cudaGetLastError();
    if (err != cudaSuccess) return err;

    static SplineTable tab = [] {
        SplineTable t;
        make_spline_table(&t);
        return t;
    }();
    const size_t per_warp = sizeof(float) * 2 * (size_t)((a.nt + 4) & ~3);
    const int wpb = (int)std::min<size_t>(8, std::max<size_t>(1, (112 * 1024) / per_warp));
    const size_t fsmem = per_warp * wpb;
    err = allow_smem(adj_finalize_kernel, kSmemMax);
    if (err != cudaSuccess) return err;
    const long long blocks = (nch + wpb - 1) / wpb;
    adj_finalize_kernel<<<(unsigned)blocks, 32 * wpb, fsmem, s>>>(
        g.partial, nparts, nch, a.nt, Lp, g.grad_rf, tab);
    return cudaGetLastError();
}

template <int GEOM, int SUM, typename T>
cudaError_t launch_adjoint_gs(const AdjArgs &g, cudaStream_t s) {
    if (g.grad_tautx || g.grad_taurx || g.grad_slow) {
        cudaError_t err = launch_delay_one<GEOM, SUM, T>(g, s);
        if (err != cudaSuccess) return err;
    }
    if (g.grad_rf) return launch_scatter_one<GEOM, SUM>(g, s);
    return cudaSuccess;
}

template <typename T>
cudaError_t launch_adjoint_t(const AdjArgs &g0, cudaStream_t s) {
    AdjArgs g = g0;
    const bool both = g.sumtype == PYCBF_GB_SUM_TX_AND_RX;
    g.gk = g.gout;
    if (g.d.pixel_index) {
        const long long rows = (long long)g.d.nframes * (both ? 1 : g.d.nrx);
        const long long n = rows * g.d.np;
        adj_gather_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(g.gout, g.d.pixel_index, rows,
                                                                     g.d.np, g.gk_buf);
        cudaError_t err = cudaGetLastError();
        if (err != cudaSuccess) return err;
        g.gk = g.gk_buf;
    }
    if (g.geom == GEOM_TABBED)
        return both ? launch_adjoint_gs<GEOM_TABBED, PYCBF_GB_SUM_TX_AND_RX, T>(g, s)
                    : launch_adjoint_gs<GEOM_TABBED, PYCBF_GB_SUM_TX_ONLY, T>(g, s);
    return both ? launch_adjoint_gs<GEOM_SYNTH_SLOW, PYCBF_GB_SUM_TX_AND_RX, T>(g, s)
                : launch_adjoint_gs<GEOM_SYNTH_SLOW, PYCBF_GB_SUM_TX_ONLY, T>(g, s);
}

}  // namespace

int adjoint_parts(long long nch, long long np) {
    // enough (channel, part) CTAs to fill the GPU several times over (~11,000: the
    // 1408-channel workload measured 1.92 ms forward + adjoint at 8 parts against
    // 2.22 at 2), parts of >= 2048 pixels
    long long p = (11264 + nch - 1) / nch;
    p = std::min<long long>(p, std::max<long long>(1, np / 2048));
    p = std::max<long long>(1, std::min<long long>(p, 64));
    const long long tiles = (np + kBlock - 1) / kBlock;
    return (int)std::max<long long>(p, (tiles + kPartTiles - 1) / kPartTiles);
}

static size_t up256(size_t n) { return (n + 255) & ~(size_t)255; }
static size_t adjoint_grad_bytes(long long nframes, long long nrx, long long np) {
    return up256((size_t)nframes * nrx * np * sizeof(float));
}
static size_t adjoint_partial_bytes(long long nframes, long long ntx, long long nrx, long long np,
                                    int nt) {
    const long long nch = nframes * ntx * nrx;
    const size_t Lp = (size_t)((nt + 1 + 3) & ~3);
    return (size_t)adjoint_parts(nch, np) * (size_t)nch * 2 * Lp * sizeof(float);
}

// [gathered gradient][partial sums][live]
size_t adjoint_workspace_bytes(long long nframes, long long ntx, long long nrx, long long np, int nt) {
    const size_t tiles = (size_t)((np + kBlock - 1) / kBlock);
    return adjoint_grad_bytes(nframes, nrx, np) + adjoint_partial_bytes(nframes, ntx, nrx, np, nt) +
           up256((size_t)nrx * tiles);
}

// The rest takes space that is free: above the gathered gradient (one row a frame of the
// sum over receives; none without pixel_index), above the workspace's size, and, for the
// ranges, depths and order, which the last kernel no longer reads, in grad_rf before it is
// written.  Without room for them the scatter walks every tile for every interval (1717
// against 780 us for 11 x 128 x 2048 samples and 256 x 512 pixels; only channel data much
// smaller than the pixels' tables comes to that), and the Synthetic scatter computes its
// delays per tap (slowness gradients of the same size 1.71 against 1.13 ms).
constexpr size_t kAdjTableMax = (size_t)1 << 30;  // above: the scatter recomputes the delays

void adjoint_layout(char *ws, size_t bytes, AdjArgs *g) {
    const DasArgs &a = g->d;
    const size_t tiles = (size_t)((a.np + kBlock - 1) / kBlock), nel = (size_t)(a.ntx + a.nrx);
    const size_t np = (size_t)a.np;
    char *const partial = ws + adjoint_grad_bytes(a.nframes, a.nrx, np);
    g->gk_buf = reinterpret_cast<float *>(ws);
    g->partial = reinterpret_cast<float *>(partial);
    g->live = reinterpret_cast<unsigned char *>(
        partial + adjoint_partial_bytes(a.nframes, a.ntx, a.nrx, np, a.nt));
    const size_t need = adjoint_workspace_bytes(a.nframes, a.ntx, a.nrx, np, a.nt);
    const int rows = a.nframes * (g->sumtype == PYCBF_GB_SUM_TX_AND_RX ? 1 : a.nrx);
    struct Room { char *at, *end; } room[3] = {
        {ws + (a.pixel_index ? up256(rows * np * sizeof(float)) : 0), partial},
        {ws + need, ws + bytes},
        {reinterpret_cast<char *>(g->grad_rf),
         reinterpret_cast<char *>(g->grad_rf) + (size_t)a.nframes * a.ntx * a.nrx * a.nt * sizeof(float)}};
    auto take = [&](size_t n, int rooms) -> char * {
        for (int k = 0; k < rooms; ++k) {
            char *p = reinterpret_cast<char *>((reinterpret_cast<uintptr_t>(room[k].at) + 15) & ~(uintptr_t)15);
            if (p && p <= room[k].end && n <= (size_t)(room[k].end - p)) {
                room[k].at = p + n;
                return p;
            }
        }
        return nullptr;
    };
    if (!g->grad_rf) return;
    char *const small = take(tiles * (nel * sizeof(float2) + sizeof(float) + sizeof(int)), 3);
    if (small) {
        g->ranges = reinterpret_cast<float2 *>(small);
        g->depth = reinterpret_cast<float *>(g->ranges + tiles * nel);
        g->order = reinterpret_cast<int *>(g->depth + tiles);
    }
    if (g->geom != GEOM_TABBED && nel * np * sizeof(float) <= kAdjTableMax) {
        g->tau_rx = reinterpret_cast<float *>(take((size_t)a.nrx * np * sizeof(float), 2));
        if (g->tau_rx) g->tau_tx = reinterpret_cast<float *>(take((size_t)a.ntx * np * sizeof(float), 2));
    }
}

cudaError_t launch_adjoint(const AdjArgs &g, int dtype, cudaStream_t s) {
    switch (dtype) {
        case PYCBF_GB_F32: return launch_adjoint_t<float>(g, s);
        case PYCBF_GB_F16: return launch_adjoint_t<__half>(g, s);
        case PYCBF_GB_BF16: return launch_adjoint_t<__nv_bfloat16>(g, s);
        default: return cudaErrorInvalidValue;
    }
}

template <typename T>
static cudaError_t launch_synth_slow_t(const DasArgs &a, int sumtype, cudaStream_t s) {
    constexpr int CU = PYCBF_GB_INTERP_CUBIC, GE = GEOM_SYNTH_SLOW;
    constexpr int BOTH = PYCBF_GB_SUM_TX_AND_RX, EACH = PYCBF_GB_SUM_TX_ONLY;
    if (das_rx_ok(a, GE, CU, sumtype))
        return sumtype == BOTH ? launch_rx_one<GE, CU, BOTH, T>(a, s) : launch_rx_one<GE, CU, EACH, T>(a, s);
    return sumtype == BOTH ? launch_das_one<GE, CU, BOTH, T, false>(a, s)
                           : launch_das_one<GE, CU, EACH, T, false>(a, s);
}

cudaError_t launch_das_synth_slow(const DasArgs &a, int sumtype, int dtype, cudaStream_t s) {
    switch (dtype) {
        case PYCBF_GB_F32: return launch_synth_slow_t<float>(a, sumtype, s);
        case PYCBF_GB_F16: return launch_synth_slow_t<__half>(a, sumtype, s);
        case PYCBF_GB_BF16: return launch_synth_slow_t<__nv_bfloat16>(a, sumtype, s);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace pgb
