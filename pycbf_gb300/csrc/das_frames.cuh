// Cubic delay-and-sum of several frames that share one geometry, FG frames at a
// time per thread.
//
// A tap's delay, knot, fraction and weight do not depend on the frame: they are
// 14 of the 20 instructions of a tap (cubic_taps), so FG frames share them and
// each frame adds only its gather and its multiply-adds.  The prefilter stores the
// records of each pair of frames (a, b) together in planes of 16 bytes per sample
// (launch_spline_pairs), so that a warp's gather from a plane stays within a few
// lines (records of FG frames side by side spread it over FG times as many, and
// over the banks of the L1 FG times as badly):
//   float32: two planes, (p0a p0b p1a p1b) and (p2a p2b p3a p3b), evaluated two
//     frames per instruction in packed float32 pairs;
//   16-bit:  one plane, (y y z z) of a and of b; each frame's y and z terms are
//     summed side by side as in cubic_taps.
//
// The gathers and their latency bound it, so the receives are spread over the warps as
// in das_rx_kernel.  Against a thread per pixel and all its receives (128 pixels, 16
// warps an SM), with 11 transmits, 128 receives and 256 x 512 pixels from tables: four
// float32 frames 591 -> 364 us, eight float16 857 -> 541; 64 x 256 pixels, eight frames
// 567 -> 240 us; two synthetic frames of 75 transmits, 192 receives and 512 x 1024
// pixels 5.3 -> 4.7 ms; eight 3-D float16 volumes 53.8 -> 56.8 ms (a third of the sectors
// of their gathers hit L1 there, a ninth here; CTAs of 64 pixels gained 1 %).
// The operations on one frame and their order are those of cubic_taps and
// das_pixel, so the images are the single-frame ones bit for bit.
#pragma once

#include "das_rx.cuh"

namespace pgb {

// the running sums of FG frames over the transmits of a receive
template <typename T, int FG> struct FramesAcc {
    float2 v[FG];  // 16-bit: each frame's (y, z) sums
    __device__ __forceinline__ float total(int f) const { return v[f].x + v[f].y; }
    static constexpr int n = FG;
};
template <int FG> struct FramesAcc<float, FG> {
    float2 v[FG / 2];  // two frames each
    __device__ __forceinline__ float total(int f) const { return pair_lane(v, f); }
    static constexpr int n = FG / 2;
};

// FG frames' records of one interval, a 16-byte piece from each plane
template <typename T, int FG> struct FramesRec {
    static constexpr int kPlanes = FG * (int)sizeof(typename CoefRec<T>::raw) / 16;
    uint4 q[kPlanes];
    __device__ __forceinline__ void load(const char *rec, unsigned e, unsigned long long plane) {
#pragma unroll
        for (int k = 0; k < kPlanes; ++k)
            q[k] = __ldg(reinterpret_cast<const uint4 *>(rec + (unsigned long long)k * plane) + e);
    }
};

template <int FG>
__device__ __forceinline__ void frames_add(const FramesRec<float, FG> &rec, const TapConst &, float b,
                                           float, float, float w, bool weighted,
                                           FramesAcc<float, FG> &acc) {
    const float2 b2 = make_float2(b, b);
    auto f2 = [](unsigned x, unsigned y) {
        return make_float2(__uint_as_float(x), __uint_as_float(y));
    };
#pragma unroll
    for (int p = 0; p < FG / 2; ++p) {
        const uint4 lo = rec.q[2 * p], hi = rec.q[2 * p + 1];
        const float2 v = fma2_rn(
            fma2_rn(fma2_rn(f2(hi.z, hi.w), b2, f2(hi.x, hi.y)), b2, f2(lo.z, lo.w)), b2,
            f2(lo.x, lo.y));
        acc.v[p] = weighted ? fma2_rn(make_float2(w, w), v, acc.v[p]) : add2_rn(acc.v[p], v);
    }
}
template <typename T, int FG>
__device__ __forceinline__ void frames_add(const FramesRec<T, FG> &rec, const TapConst &c, float,
                                           float x, float fj, float w, bool weighted,
                                           FramesAcc<T, FG> &acc) {
    float2 wy, wz;
    if (weighted) half_weights<true>(c, x, fj, w, wy, wz);
    else half_weights<false>(c, x, fj, w, wy, wz);
#pragma unroll
    for (int f = 0; f < FG; ++f) {
        const uint4 q = rec.q[f / 2];
        const uint2 r = (f & 1) ? make_uint2(q.z, q.w) : make_uint2(q.x, q.y);
        acc.v[f] = half_add(CoefRec<T>::unpack(r), wy, wz, acc.v[f]);
    }
}

// Four taps of one receive for FG frames, gathered kLive taps at a time (128
// bytes of records a thread in flight)
template <int GEOM, typename T, int FG>
__device__ __forceinline__ void frames_taps(const DasArgs &a, const TapConst &c, const float2 *tt2,
                                            const float2 *at2, float trx, float arx,
                                            const char *rec, unsigned long long plane,
                                            const unsigned *off,
                                            FramesAcc<T, FG> &acc) {
    using Rec = FramesRec<T, FG>;
    constexpr int N = kCubicGroup, NP = N / 2;
    constexpr int kLive = Rec::kPlanes * N <= 8 ? N : (Rec::kPlanes * 2 <= 8 ? 2 : 1);
    constexpr bool W = GEOM == GEOM_TABBED;
    float2 x2[NP], fj2[NP], w2[NP];
    unsigned r[N];
    knot_pairs<NP>(a, c, tt2, trx, x2, fj2, r);
    if (W) {
#pragma unroll
        for (int p = 0; p < NP; ++p) w2[p] = mul2_rn(at2[p], make_float2(arx, arx));
    }
#pragma unroll
    for (int k0 = 0; k0 < N; k0 += kLive) {
        Rec pv[kLive];
        bool ok[kLive];
#pragma unroll
        for (int m = 0; m < kLive; ++m) {
            const int k = k0 + m;
            const float x = pair_lane(x2, k);
            ok[m] = (x >= c.t0) && (x <= c.xmax);
            if (W) ok[m] = ok[m] && (fabsf(pair_lane(w2, k)) >= c.thresh);
            if (ok[m]) pv[m].load(rec, r[k] + off[k], plane);
        }
#pragma unroll
        for (int m = 0; m < kLive; ++m) {
            const int k = k0 + m;
            float b = 0.f;
            if constexpr (CoefRec<T>::kPoly) {
                const float2 b2 = knot_frac2(c, x2[k >> 1], fj2[k >> 1]);
                b = (k & 1) ? b2.y : b2.x;
            }
            if (ok[m])
                frames_add(pv[m], c, b, pair_lane(x2, k), pair_lane(fj2, k),
                           W ? pair_lane(w2, k) : 1.f, W, acc);
        }
    }
}

// receives whose sums (and table rows) are in shared memory together
__host__ __device__ constexpr int frames_run(int geom, int fg) {
    return geom == GEOM_SYNTH && fg == 2 ? 2 * kRxBlockSum : kRxBlockSum;
}

constexpr size_t kFramesSmemMax = 200 * 1024;
inline size_t das_frames_smem(int geom, int sum, int fg, int ntx) {
    const size_t sums = sum == PYCBF_GB_SUM_TX_ONLY ? 0 : fg;
    const size_t rows = (sums + (geom == GEOM_TABBED ? 4 : 0)) * frames_run(geom, fg);
    return 32 * sizeof(float) * ((size_t)(ntx + 3) / 4 * 4 + rows);
}

// CTAs an SM.  Three (80 registers) hide more of the gathers: two 75-transmit float32
// frames 4.7 against 5.7 ms, four 8.5 against 10.9; Tabbed groups of four and eight hold
// the tables as well and gain nothing or spill (eight float16 frames 0.75 against 0.54 ms).
constexpr int frames_ctas(int geom, int fg) { return fg <= (geom == GEOM_TABBED ? 2 : 4) ? 3 : 2; }

// das_rx_kernel's division of the work for a group of FG frames (blockIdx.y): 32 pixels
// a CTA, the receives of a block of kRxBlockSum spread over the warps, each receive's FG
// sums in shared memory; warp f then adds frame f's, in order.
template <int GEOM, int SUM, typename T, int FG>
__global__ void __launch_bounds__(32 * kRxWarps, frames_ctas(GEOM, FG))
    das_frames_kernel(const __grid_constant__ DasArgs a) {
    constexpr unsigned kFull = 0xffffffffu;
    constexpr bool W = GEOM == GEOM_TABBED;
    constexpr bool kEach = SUM == PYCBF_GB_SUM_TX_ONLY;  // written per receive, nothing to add
    constexpr int kRun = frames_run(GEOM, FG);
    static_assert(FG <= kRxWarps, "a warp adds a frame");
    extern __shared__ float sm[];
    __shared__ float s_w[3][kRxWarps][32];  // Tabbed weights: largest magnitude, min, max
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long long np = a.np;
    long long i = (long long)blockIdx.x * 32 + lane;
    const bool valid = i < np;
    if (!valid) i = np - 1;
    const int ntx = a.ntx, nrx = a.nrx, ncol = (ntx + 3) / 4 * 4;
    const int f0 = (int)blockIdx.y * FG;
    const long long op = a.pixel_index ? (long long)__ldg(a.pixel_index + i) : i;
    const float inf = __int_as_float(0x7f800000);
    float2 *col = reinterpret_cast<float2 *>(sm) + lane;  // [ncol / 2][32] transmit delays
    float *sums = sm + (size_t)ncol * 32 + lane;          // [kRun][FG][32]
    float *tabs = sums + (kEach ? 0 : kRun * FG * 32);    // as in das_rx_kernel
    auto fetch_run = [&](int r0, int buf) {
        rx_fetch_run<kRun, kRxWarps>(a, tabs + (size_t)buf * 2 * kRun * 32, r0, min(kRun, a.r1 - r0), w, i);
    };
    if (W) fetch_run(a.r0, 0);

    float pnt[3] = {0.f, 0.f, 0.f};
    if (!W)
        for (int k = 0; k < 3; ++k) if (k < a.ndim) pnt[k] = __ldg(a.geo.pnts + i * a.ndim + k);
    float amax = 0.f, amin = inf, atop = -inf;
    rx_column<GEOM, kRxWarps>(a, pnt, 0.f, i, w, col, amax, amin, atop);
    if (W) {
        s_w[0][w][lane] = amax;
        s_w[1][w][lane] = amin;
        s_w[2][w][lane] = atop;
    }
    const TapConst tc(a);
    unsigned off[kCubicGroup];
#pragma unroll
    for (int k = 0; k < kCubicGroup; ++k) off[k] = (unsigned)k * (unsigned)nrx * (unsigned)a.nt - kKnotBits;
    __syncthreads();
    if (W) {
#pragma unroll 4
        for (int k = 0; k < kRxWarps; ++k) {
            amax = fmaxf(amax, s_w[0][k][lane]);
            amin = fminf(amin, s_w[1][k][lane]);
            atop = fmaxf(atop, s_w[2][k][lane]);
        }
    }
    const bool one_weight = W && __all_sync(kFull, amin == atop);
    const unsigned long long plane = 16ULL * ntx * nrx * a.nt;  // bytes
    const char *base = static_cast<const char *>(a.data) +
                       (unsigned long long)blockIdx.y * FramesRec<T, FG>::kPlanes * plane;
    const long long rstep = 16LL * a.nt;
    const long long gstep = (long long)kCubicGroup * nrx * rstep;
    // warp f < FG: frame f's image so far and DMAS's running sum
    float acc = 0.f, s1 = 0.f;
    if (SUM == PYCBF_GB_SUM_TX_AND_RX && a.r0 > 0 && w < FG)
        acc = a.out[(long long)(f0 + w) * np + op];
    int buf = 0;
    for (int r0 = a.r0; r0 < a.r1; r0 += kRun, buf ^= 1) {
        const int n = min(kRun, a.r1 - r0);
        if (W) {
            fetch_run(min(r0 + kRun, a.r1), buf ^ 1);  // none past the last: an empty group
            copy_wait_but_one();
        }
        const float *tab = tabs + (size_t)buf * 2 * kRun * 32;
        for (int e = w; e < n; e += kRxWarps) {
            const int r = r0 + e;
            float trx, arx = 1.f;
            bool live;
            if (W) {
                trx = tab[e * 32];
                arx = tab[(kRun + e) * 32];
                live = __fmul_rn(amax, fabsf(arx)) >= a.thresh;
            } else {
                trx = synth_rx_delay_warp(a, r, pnt);
                live = trx != inf;
            }
            FramesAcc<T, FG> sum;
#pragma unroll
            for (int k = 0; k < FramesAcc<T, FG>::n; ++k) sum.v[k] = make_float2(0.f, 0.f);
            if (__any_sync(kFull, live)) {
                const char *rec = base + r * rstep;
                for (int g = 0; g < ncol; g += kCubicGroup, rec += gstep) {
                    float2 t2[kCubicGroup / 2], w2[kCubicGroup / 2];
#pragma unroll
                    for (int p = 0; p < kCubicGroup / 2; ++p) {
                        t2[p] = col[(g / 2 + p) * 32];
                        w2[p] = make_float2(amin, amin);
                    }
                    if (W && !one_weight) {
                        float *v = reinterpret_cast<float *>(w2);
#pragma unroll
                        for (int k = 0; k < kCubicGroup; ++k)
                            v[k] = __ldg(a.apodtx + (long long)min(g + k, ntx - 1) * np + i);
                    }
                    frames_taps<GEOM, T, FG>(a, tc, t2, w2, trx, arx, rec, plane, off, sum);
                }
            }
#pragma unroll
            for (int f = 0; f < FG; ++f) {
                float v = sum.total(f);
                if (kEach) {
                    if (valid) a.out[((long long)(f0 + f) * nrx + r) * np + op] = v;
                } else {
                    if (SUM == PYCBF_GB_SUM_DMAS_SSR) {
                        if (!a.dmas_power) v = copysignf(sqrtf(fabsf(v)), v);
                        if (!live) v = __uint_as_float(kDeadSum);
                    }
                    sums[(e * FG + f) * 32] = v;
                }
            }
        }
        if (kEach) continue;
        __syncthreads();
        if (w < FG) {
            for (int e0 = 0; e0 < n; e0 += kRxBlockSum) {
                const int e1 = min(n, e0 + kRxBlockSum);
                float b = 0.f;
#pragma unroll 8
                for (int e = e0; e < e1; ++e) {
                    const float v = sums[(e * FG + w) * 32];
                    if (SUM == PYCBF_GB_SUM_TX_AND_RX) b += v;
                    else dmas_add(v, acc, s1);
                }
                acc += b;
            }
        }
        __syncthreads();
    }
    if (!kEach && w < FG && valid) a.out[(long long)(f0 + w) * np + op] = acc;
}

// Records of more than a gigabyte pass through L2 while the tiles run at every
// receive at once, so such launches go by kFramesStep receives at a time (whole blocks
// of kRxBlockSum: the sums so far carry over in the image).  Eight 3-D float16 volumes
// (3.4 GB of records): 59.4 ms in one launch, 56.8 by 256 or 128 receives, 57.7 by 64.
constexpr long long kFramesSplitBytes = 1LL << 30;
constexpr int kFramesStep = 256;

template <int GEOM, int SUM, typename T, int FG>
cudaError_t launch_das_frames_one(DasArgs a, cudaStream_t s) {
    auto kern = das_frames_kernel<GEOM, SUM, T, FG>;
    const size_t smem = das_frames_smem(GEOM, SUM, FG, a.ntx);
    if (smem > 40 * 1024) {  // with the static part
        cudaError_t err = allow_smem(kern, kFramesSmemMax);
        if (err != cudaSuccess) return err;
    }
    const dim3 grid((unsigned)((a.np + 31) / 32), (unsigned)(a.nframes / FG));
    const long long bytes = 16LL * FramesRec<T, FG>::kPlanes * a.ntx * a.nrx * a.nt;
    const bool split = SUM != PYCBF_GB_SUM_DMAS_SSR && bytes > kFramesSplitBytes;
    const int step = split ? kFramesStep : a.nrx;
    for (a.r0 = 0; a.r0 < a.nrx; a.r0 += step) {
        a.r1 = std::min(a.nrx, a.r0 + step);
        kern<<<grid, 32 * kRxWarps, smem, s>>>(a);
        cudaError_t err = cudaGetLastError();
        if (err != cudaSuccess) return err;
    }
    return cudaSuccess;
}

// a.nframes: a multiple of fg
template <int GEOM, int SUM, typename T>
cudaError_t launch_das_frames_fg(const DasArgs &a, int fg, cudaStream_t s) {
    if constexpr (!CoefRec<T>::kPoly)
        if (fg == 8) return launch_das_frames_one<GEOM, SUM, T, 8>(a, s);
    if (fg == 4) return launch_das_frames_one<GEOM, SUM, T, 4>(a, s);
    if (fg == 2) return launch_das_frames_one<GEOM, SUM, T, 2>(a, s);
    return cudaErrorInvalidValue;
}

template <int GEOM, typename T>
cudaError_t launch_das_frames_type(DasArgs a, int sum, int fg, cudaStream_t s) {
    a.dmas_power = sum == PYCBF_GB_SUM_DMAS_POWER;
    switch (sum) {
        case PYCBF_GB_SUM_TX_AND_RX: return launch_das_frames_fg<GEOM, PYCBF_GB_SUM_TX_AND_RX, T>(a, fg, s);
        case PYCBF_GB_SUM_TX_ONLY: return launch_das_frames_fg<GEOM, PYCBF_GB_SUM_TX_ONLY, T>(a, fg, s);
        case PYCBF_GB_SUM_DMAS_SSR:
        case PYCBF_GB_SUM_DMAS_POWER: return launch_das_frames_fg<GEOM, PYCBF_GB_SUM_DMAS_SSR, T>(a, fg, s);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace pgb
