// Delay-and-sum with the receives of 32 pixels spread over the warps of a CTA.
//
// das_kernel gives a thread a pixel and all its receives.  Its transmit delays fill a
// column of shared memory per thread, which holds an SM to 20 warps at 75 transmits
// -- too few to cover the gathers (half of the issue slots used) -- and a small image
// is a few CTAs that walk the receives one after another.  Here the warps of a CTA
// share one column of 32 pixels and take the receives in turn; each receive's sum
// goes to shared memory, and the sums are added as the other kernels add them (in
// blocks of kRxBlockSum receives, then the blocks), so the image is theirs bit for bit.
// Receives go in runs of kRxRun, so that shared memory does not grow with them; the
// table rows of a run are copied to shared memory while the run before is summed (without
// that, 192 instead of 151 us for the tabled frame below).
//
// It is bound by issue and by the gathers' latency (half to two thirds of the issue slots
// used).  One float32 frame, cubic, 256 x 512 pixels and 128 receives unless said
// otherwise, against the kernels before (synthetic: das_kernel; tables: das_staged_kernel
// on its TMA windows up to 12 transmits, das_kernel beyond):
//   synthetic, 75 transmits, 192 receives,
//           512 x 1024 pixels              3910 -> 2880 us (64 x 128 pixels 2350 -> 610)
//   tables, 11 transmits                     170 ->  151 us (64 x 128 pixels 143 -> 40)
//           1 / 5 / 8 transmits      90 / 121 / 138 -> 82 / 116 / 122 us
//           11, 192 receives                 194 ->  187 us
//           11, float16                      183 ->  179 us
//           11, linear / nearest       177 / 149 -> 150 / 123 us
//           11, sums per receive             190 ->  164 us
//           31 / 75 (192 receives)    642 / 2200 -> 322 / 824 us
#pragma once

#include "das_impl.cuh"

namespace pgb {

constexpr int kRxWarps = 8;
// receives whose sums are in shared memory together; Tabbed: and their table rows,
// for this run and the next
template <int GEOM> constexpr int kRxRun = GEOM == GEOM_TABBED ? 64 : 256;
constexpr size_t kRxSmemMax = 100 * 1024;  // two CTAs an SM

// What DMAS keeps as the sum of a receive that does not reach a pixel, and then leaves out
// (a zero would turn an infinite sum before it into NaN): a NaN that no arithmetic gives.
constexpr unsigned kDeadSum = 0x7fc0dead;
// one receive's sum into DMAS's image and running sum: the pairs i < j as s_j * sum_i s_i
__device__ __forceinline__ void dmas_add(float s, float &acc, float &s1) {
    if (__float_as_uint(s) != kDeadSum) {
        acc = fmaf(s, s1, acc);
        s1 += s;
    }
}

inline size_t das_rx_smem(int geom, int ntx, int nrx) {
    const size_t rows = geom == GEOM_TABBED ? 5 * kRxRun<GEOM_TABBED>
                                            : std::min(nrx, kRxRun<GEOM_SYNTH>);
    return 32 * sizeof(float) * ((size_t)(ntx + 3) / 4 * 4 + rows);
}

// four bytes global -> shared without a register in between
__device__ __forceinline__ void copy_async4(float *dst, const float *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(
                     (unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src)
                 : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void copy_wait_but_one() {
    asm volatile("cp.async.wait_group 1;" ::: "memory");
}

// Warp w's rows of the receive tables for the n receives from r0, lane's pixel i, to
// t[delay, weight][RUN][32]: in flight while the run before is summed (a row read when
// its turn comes costs a trip to memory each).
template <int RUN, int WARPS>
__device__ __forceinline__ void rx_fetch_run(const DasArgs &a, float *t, int r0, int n, int w,
                                             long long i) {
    for (int e = w; e < n; e += WARPS) {
        copy_async4(t + e * 32, a.taurx + (long long)(r0 + e) * a.np + i);
        copy_async4(t + (RUN + e) * 32, a.apodrx + (long long)(r0 + e) * a.np + i);
    }
    copy_commit();
}

// Warp w's part of the transmit delays of pixel i, in pairs padded with infinite delays
// (never count) to whole groups, and of the range of its weights.
template <int GEOM, int WARPS>
__device__ __forceinline__ void rx_column(const DasArgs &a, const float *pnt, float slow,
                                          long long i, int w, float2 *col, float &amax, float &amin, float &atop) {
    const int npair = (a.ntx + 3) / 4 * 2;
    for (int p = w; p < npair; p += WARPS) {
        float tau[2] = {__int_as_float(0x7f800000), __int_as_float(0x7f800000)};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int k = 2 * p + h;
            if (k >= a.ntx) continue;
            if (GEOM == GEOM_TABBED) {
                tau[h] = __ldg(a.tautx + (long long)k * a.np + i);
                const float v = __ldg(a.apodtx + (long long)k * a.np + i);
                amax = fmaxf(amax, fabsf(v));
                weight_range(v, amin, atop);
            } else if (GEOM == GEOM_SYNTH) {
                tau[h] = synth_tx_delay(a, k, pnt);
            } else {
                float D, t0add;
                const bool ok = synth_tx_path(a, k, pnt, D, t0add);
                tau[h] = slow_delay(ok, D, slow, t0add);
            }
        }
        col[p * 32] = make_float2(tau[0], tau[1]);
    }
}

template <int GEOM, int KIND, int SUM, typename T>
__global__ void __launch_bounds__(32 * kRxWarps, GEOM == GEOM_TABBED ? 4 : 3)
    das_rx_kernel(const __grid_constant__ DasArgs a) {
    using S = TapSum<GEOM, KIND, T>;
    using Rec = typename S::Rec;
    constexpr unsigned kFull = 0xffffffffu;
    constexpr bool W = GEOM == GEOM_TABBED;
    constexpr bool kEach = SUM == PYCBF_GB_SUM_TX_ONLY;  // written per receive, nothing to add
    constexpr int kRun = kRxRun<GEOM>, kBlocks = kRun / kRxBlockSum;
    extern __shared__ float sm[];
    __shared__ float s_w[3][kRxWarps][32];      // Tabbed weights: largest magnitude, min, max
    __shared__ float s_block[kBlocks][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int ntx = a.ntx, nrx = a.nrx, ncol = (ntx + 3) / 4 * 4;
    const long long np = a.np;
    long long i = (long long)blockIdx.x * 32 + lane;
    const bool valid = i < np;
    if (!valid) i = np - 1;
    const int f = blockIdx.y;
    const long long op = a.pixel_index ? (long long)__ldg(a.pixel_index + i) : i;
    const float inf = __int_as_float(0x7f800000);
    float2 *col = reinterpret_cast<float2 *>(sm) + lane;  // [ncol / 2][32] transmit delays
    float *sums = sm + (size_t)ncol * 32 + lane;          // [receives of the run][32]
    float *tabs = sums + kRun * 32;  // Tabbed: [2 runs][delay, weight][kRun][32], own lane only
    auto fetch_run = [&](int r0, int buf) {
        rx_fetch_run<kRun, kRxWarps>(a, tabs + (size_t)buf * 2 * kRun * 32, r0, min(kRun, nrx - r0), w, i);
    };
    if (W) fetch_run(0, 0);

    float pnt[3] = {0.f, 0.f, 0.f};
    const float slow = GEOM == GEOM_SYNTH_SLOW ? __ldg(a.slow + i) : 0.f;
    if (!W)
        for (int k = 0; k < 3; ++k) if (k < a.ndim) pnt[k] = __ldg(a.geo.pnts + i * a.ndim + k);
    float amax = 0.f, amin = inf, atop = -inf;
    rx_column<GEOM, kRxWarps>(a, pnt, slow, i, w, col, amax, amin, atop);
    if (W) {
        s_w[0][w][lane] = amax;
        s_w[1][w][lane] = amin;
        s_w[2][w][lane] = atop;
    }
    const TapConst tc(a);
    const long long chs = (long long)nrx * a.nt;
    __syncthreads();
    if (W) {
#pragma unroll 4
        for (int k = 0; k < kRxWarps; ++k) {
            amax = fmaxf(amax, s_w[0][k][lane]);
            amin = fminf(amin, s_w[1][k][lane]);
            atop = fmaxf(atop, s_w[2][k][lane]);
        }
    }
    // one weight for every transmit of the warp's pixels (apodtx all ones), or the table
    const bool one_weight = W && __all_sync(kFull, amin == atop);
    float acc = 0.f, s1 = 0.f;  // warp 0: the image so far, DMAS's running sum
    int buf = 0;
    for (int r0 = 0; r0 < nrx; r0 += kRun, buf ^= 1) {
        const int n = min(kRun, nrx - r0);
        if (W) {
            fetch_run(min(r0 + kRun, nrx), buf ^ 1);  // none past the last: an empty group
            copy_wait_but_one();
        }
        const float *tab = tabs + (size_t)buf * 2 * kRun * 32;
        // receive r0 + e by warp e % kRxWarps: those that reach the pixels lie side by side
        for (int e = w; e < n; e += kRxWarps) {
            const int r = r0 + e;
            float trx, arx = 1.f;
            bool live;
            if (W) {
                trx = tab[e * 32];
                arx = tab[(kRun + e) * 32];
                live = __fmul_rn(amax, fabsf(arx)) >= a.thresh;
            } else if (GEOM == GEOM_SYNTH) {
                trx = synth_rx_delay_warp(a, r, pnt);
                live = trx != inf;
            } else {
                float D;
                const bool ok = synth_rx_path(a, r, pnt, D);
                trx = slow_delay(ok, D, slow, 0.f);
                live = trx != inf;
            }
            if (!__any_sync(kFull, live)) {
                if (kEach && valid) a.out[((long long)f * nrx + r) * np + op] = 0.f;
                if (!kEach)
                    sums[(size_t)e * 32] =
                        SUM == PYCBF_GB_SUM_DMAS_SSR ? __uint_as_float(kDeadSum) : 0.f;
                continue;
            }
            auto sum = S::zero();
            const Rec *rec = static_cast<const Rec *>(a.data) + ((long long)f * ntx * nrx + r) * a.nt;
            for (int g = 0; g < ncol; g += kCubicGroup, rec += kCubicGroup * chs) {
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
                sum = S::template taps<kCubicGroup, true>(a, tc, t2, w2, trx, arx, rec, chs, sum);
            }
            float v = S::total(sum);
            if (kEach) {
                if (valid) a.out[((long long)f * nrx + r) * np + op] = v;
            } else {
                if (SUM == PYCBF_GB_SUM_DMAS_SSR) {
                    if (!a.dmas_power) v = copysignf(sqrtf(fabsf(v)), v);
                    if (!live) v = __uint_as_float(kDeadSum);
                }
                sums[(size_t)e * 32] = v;
            }
        }
        __syncthreads();
        if (SUM == PYCBF_GB_SUM_TX_AND_RX) {
            if (w < kBlocks && w * kRxBlockSum < n) {  // block w of the run, in order
                const int e1 = min(n, (w + 1) * kRxBlockSum);
                float b = 0.f;
#pragma unroll 8
                for (int e = w * kRxBlockSum; e < e1; ++e) b += sums[(size_t)e * 32];
                s_block[w][lane] = b;
            }
            __syncthreads();
            if (w == 0)
                for (int b = 0; b * kRxBlockSum < n; ++b) acc += s_block[b][lane];
        } else if (SUM == PYCBF_GB_SUM_DMAS_SSR) {
            if (w == 0) {
#pragma unroll 8
                for (int e = 0; e < n; ++e) dmas_add(sums[(size_t)e * 32], acc, s1);
            }
            __syncthreads();
        }
    }
    if (!kEach && w == 0 && valid) a.out[(long long)f * np + op] = acc;
}

template <int GEOM, int KIND, int SUM, typename T>
cudaError_t launch_rx_one(const DasArgs &a, cudaStream_t s) {
    auto kern = das_rx_kernel<GEOM, KIND, SUM, T>;
    const size_t smem = das_rx_smem(GEOM, a.ntx, a.nrx);
    if (smem > 40 * 1024) {  // with the static part
        cudaError_t err = allow_smem(kern, kRxSmemMax);
        if (err != cudaSuccess) return err;
    }
    kern<<<dim3((unsigned)((a.np + 31) / 32), (unsigned)a.nframes), 32 * kRxWarps, smem, s>>>(a);
    return cudaGetLastError();
}

template <int GEOM, int KIND, typename T>
cudaError_t launch_rx_sum(DasArgs a, int sum, cudaStream_t s) {
    a.dmas_power = sum == PYCBF_GB_SUM_DMAS_POWER;
    switch (sum) {
        case PYCBF_GB_SUM_TX_AND_RX: return launch_rx_one<GEOM, KIND, PYCBF_GB_SUM_TX_AND_RX, T>(a, s);
        case PYCBF_GB_SUM_TX_ONLY: return launch_rx_one<GEOM, KIND, PYCBF_GB_SUM_TX_ONLY, T>(a, s);
        case PYCBF_GB_SUM_DMAS_SSR:
        case PYCBF_GB_SUM_DMAS_POWER: return launch_rx_one<GEOM, KIND, PYCBF_GB_SUM_DMAS_SSR, T>(a, s);
        default: return cudaErrorInvalidValue;
    }
}

template <int GEOM, typename T>
cudaError_t launch_rx_type(const DasArgs &a, int interp, int sum, cudaStream_t s) {
    switch (interp) {
        case PYCBF_GB_INTERP_CUBIC: return launch_rx_sum<GEOM, PYCBF_GB_INTERP_CUBIC, T>(a, sum, s);
        case PYCBF_GB_INTERP_LINEAR: return launch_rx_sum<GEOM, PYCBF_GB_INTERP_LINEAR, T>(a, sum, s);
        case PYCBF_GB_INTERP_NEAREST: return launch_rx_sum<GEOM, PYCBF_GB_INTERP_NEAREST, T>(a, sum, s);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace pgb
