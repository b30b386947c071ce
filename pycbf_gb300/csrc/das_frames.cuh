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
// The operations on one frame and their order are those of cubic_taps and
// das_pixel, so the images are the single-frame ones bit for bit.
#pragma once

#include "das_impl.cuh"

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

// One thread per pixel and group of FG frames (blockIdx.y); the transmit delays in
// the thread's column of shared memory, as das_pixel keeps them.
template <int GEOM, int SUM, typename T, int FG>
__global__ void __launch_bounds__(kBlock, 4) das_frames_kernel(const __grid_constant__ DasArgs a) {
    constexpr unsigned kFull = 0xffffffffu;
    constexpr bool W = GEOM == GEOM_TABBED;
    constexpr bool kDmas = SUM == PYCBF_GB_SUM_DMAS_SSR;  // or POWER, by a.dmas_power
    extern __shared__ float sm[];
    const long long np = a.np;
    long long i = (long long)blockIdx.x * kBlock + threadIdx.x;
    const bool valid = i < np;
    if (!valid) i = np - 1;
    const int ntx = a.ntx, nrx = a.nrx;
    const int f0 = (int)blockIdx.y * FG;
    const int ncol = cubic_column_padded(ntx);
    const long long op = a.pixel_index ? (long long)__ldg(a.pixel_index + i) : i;
    const float inf = __int_as_float(0x7f800000);
    const TapConst tc(a);
    unsigned off[kCubicGroup];
#pragma unroll
    for (int k = 0; k < kCubicGroup; ++k) off[k] = (unsigned)k * (unsigned)nrx * (unsigned)a.nt - kKnotBits;
    float2 *col = reinterpret_cast<float2 *>(sm) + threadIdx.x;
    float pnt[3] = {0.f, 0.f, 0.f};
    if (GEOM == GEOM_SYNTH)
        for (int k = 0; k < 3; ++k) if (k < a.ndim) pnt[k] = __ldg(a.geo.pnts + i * a.ndim + k);
    float amax = 0.f, amin = inf, atop = -inf;
    for (int k = 0; k < ncol; k += 2) {
        float2 t = make_float2(inf, inf);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (k + h < ntx) {
                float tau;
                if (W) {
                    tau = __ldg(a.tautx + (long long)(k + h) * np + i);
                    const float w = __ldg(a.apodtx + (long long)(k + h) * np + i);
                    amax = fmaxf(amax, fabsf(w));
                    weight_range(w, amin, atop);
                } else {
                    tau = synth_tx_delay(a, k + h, pnt);
                }
                if (h) t.y = tau;
                else t.x = tau;
            }
        }
        col[(size_t)(k >> 1) * kBlock] = t;
    }
    const bool one_weight = W && __all_sync(kFull, amin == atop);

    float acc[FG], s1[FG];  // s1: the current receive block's sum, or DMAS's running sum
#pragma unroll
    for (int f = 0; f < FG; ++f) acc[f] = s1[f] = 0.f;
    const unsigned long long plane = 16ULL * ntx * nrx * a.nt;  // bytes
    const char *base = static_cast<const char *>(a.data) +
                       (unsigned long long)blockIdx.y * FramesRec<T, FG>::kPlanes * plane;
    const long long rstep = 16LL * a.nt;
    const long long gstep = (long long)kCubicGroup * nrx * rstep;
    if (SUM == PYCBF_GB_SUM_TX_AND_RX && a.r0 > 0) {
#pragma unroll
        for (int f = 0; f < FG; ++f) acc[f] = a.out[(long long)(f0 + f) * np + op];
    }
    base += a.r0 * rstep;
    for (int r = a.r0; r < a.r1; ++r, base += rstep) {
        if (SUM == PYCBF_GB_SUM_TX_AND_RX && r > a.r0 && r % kRxBlockSum == 0) {
#pragma unroll
            for (int f = 0; f < FG; ++f) {
                acc[f] += s1[f];
                s1[f] = 0.f;
            }
        }
        float trx, arx = 1.f;
        bool live;
        if (W) {
            trx = __ldg(a.taurx + (long long)r * np + i);
            arx = __ldg(a.apodrx + (long long)r * np + i);
            live = __fmul_rn(amax, fabsf(arx)) >= a.thresh;
        } else {
            trx = synth_rx_delay_warp(a, r, pnt);
            live = trx != inf;
        }
        FramesAcc<T, FG> sum;
#pragma unroll
        for (int k = 0; k < FramesAcc<T, FG>::n; ++k) sum.v[k] = make_float2(0.f, 0.f);
        if (__any_sync(kFull, live)) {
            const char *rec = base;
            for (int g = 0; g < ncol; g += kCubicGroup, rec += gstep) {
                float2 t2[kCubicGroup / 2], w2[kCubicGroup / 2];
#pragma unroll
                for (int p = 0; p < kCubicGroup / 2; ++p) {
                    t2[p] = col[(size_t)(g / 2 + p) * kBlock];
                    w2[p] = make_float2(amin, amin);
                }
                if (W && !one_weight) {
                    float *w = reinterpret_cast<float *>(w2);
#pragma unroll
                    for (int k = 0; k < kCubicGroup; ++k)
                        w[k] = __ldg(a.apodtx + (long long)min(g + k, ntx - 1) * np + i);
                }
                frames_taps<GEOM, T, FG>(a, tc, t2, w2, trx, arx, rec, plane, off, sum);
            }
        } else if (SUM != PYCBF_GB_SUM_TX_ONLY) {
            continue;
        }
#pragma unroll
        for (int f = 0; f < FG; ++f) {
            const float v = sum.total(f);
            if (SUM == PYCBF_GB_SUM_TX_AND_RX) s1[f] += v;
            if (SUM == PYCBF_GB_SUM_TX_ONLY && valid)
                a.out[((long long)(f0 + f) * nrx + r) * np + op] = v;
            if (kDmas) {
                const float s = a.dmas_power ? v : copysignf(sqrtf(fabsf(v)), v);
                acc[f] = fmaf(s, s1[f], acc[f]);
                s1[f] += s;
            }
        }
    }
    if (!valid || SUM == PYCBF_GB_SUM_TX_ONLY) return;
#pragma unroll
    for (int f = 0; f < FG; ++f)
        a.out[(long long)(f0 + f) * np + op] =
            SUM == PYCBF_GB_SUM_TX_AND_RX ? acc[f] + s1[f] : acc[f];
}

// Records of more than a gigabyte pass through L2 while the tiles run at every
// receive at once, so such launches go block of receives by block of receives
// (kRxBlockSum: the sums so far carry over in the image).  Two 192-element float32
// frames of 75 transmits (1.9 GB): 6.06 -> 5.33 ms; eight 3-D float16 volumes (3.4
// GB): 75 -> 56 ms; 0.18 GB of Tabbed frames: 0.85 -> 0.89 ms, so they go in one.
constexpr long long kFramesSplitBytes = 1LL << 30;

template <int GEOM, int SUM, typename T, int FG>
cudaError_t launch_das_frames_one(DasArgs a, cudaStream_t s) {
    auto kern = das_frames_kernel<GEOM, SUM, T, FG>;
    const size_t smem = (size_t)kBlock * cubic_column_padded(a.ntx) * sizeof(float);
    if (smem > 48 * 1024) {
        cudaError_t err =
            cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (err != cudaSuccess) return err;
    }
    const dim3 grid((unsigned)((a.np + kBlock - 1) / kBlock), (unsigned)(a.nframes / FG));
    const long long bytes = 16LL * FramesRec<T, FG>::kPlanes * a.ntx * a.nrx * a.nt;
    const bool split = SUM != PYCBF_GB_SUM_DMAS_SSR && bytes > kFramesSplitBytes;
    const int step = split ? kRxBlockSum : a.nrx;
    for (a.r0 = 0; a.r0 < a.nrx; a.r0 += step) {
        a.r1 = std::min(a.nrx, a.r0 + step);
        kern<<<grid, kBlock, smem, s>>>(a);
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
