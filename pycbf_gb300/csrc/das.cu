// Dispatch of the delay-and-sum kernels by geometry and channel-data type.
#include "das_frames.cuh"
#include "das_staged.cuh"

namespace pgb {

cudaError_t launch_das_tabbed_f32(const DasArgs &, int, int, bool, cudaStream_t);
cudaError_t launch_das_tabbed_f16(const DasArgs &, int, int, bool, cudaStream_t);
cudaError_t launch_das_tabbed_bf16(const DasArgs &, int, int, bool, cudaStream_t);
cudaError_t launch_das_synth_f32(const DasArgs &, int, int, bool, cudaStream_t);
cudaError_t launch_das_synth_f16(const DasArgs &, int, int, bool, cudaStream_t);
cudaError_t launch_das_synth_bf16(const DasArgs &, int, int, bool, cudaStream_t);
cudaError_t launch_plan_f32(const DasArgs &, int, int *, cudaStream_t);
cudaError_t launch_plan_f16(const DasArgs &, int, int *, cudaStream_t);
cudaError_t launch_plan_bf16(const DasArgs &, int, int *, cudaStream_t);
cudaError_t launch_staged_f32(const DasArgs &, int, int, const int *, int *, cudaStream_t);
cudaError_t launch_staged_f16(const DasArgs &, int, int, const int *, int *, cudaStream_t);
cudaError_t launch_staged_bf16(const DasArgs &, int, int, const int *, int *, cudaStream_t);
cudaError_t launch_das_frames_f32(const DasArgs &, int, int, int, cudaStream_t);
cudaError_t launch_das_frames_f16(const DasArgs &, int, int, int, cudaStream_t);
cudaError_t launch_das_frames_bf16(const DasArgs &, int, int, int, cudaStream_t);

// The kernels that spread a pixel's receives over warps (das_rx_kernel, das_frames_kernel)
// fill the GPU from few pixels and hide latency with many receives.  With few receives on an
// image that fills it anyway most of their warps only help to fetch the transmits' column,
// and das_kernel, a thread per pixel, is the faster one: up to 16 receives, more of them the
// more pixels there are (it walks them one after another) and fewer the longer the column of
// transmits that each thread holds.  us of a call, 2048 samples, das_kernel / das_rx_kernel:
//   tables      pixels   receives 1         4         8        16
//   5 tx        128 x 256   15 / 18   18 / 19   20 / 19   25 / 21
//               256 x 512   17 / 29   21 / 31   25 / 33   33 / 37
//              512 x 1024   26 / 68   35 / 78   46 / 84   90 / 115   (24 receives 144 / 138)
//   75 tx       128 x 256   25 / 31   45 / 37   69 / 40  124 / 55
//               256 x 512   37 / 78  70 / 103 114 / 127 204 / 160
//              512 x 1024 105 / 296 172 / 376 256 / 436 448 / 518     (24 receives 625 / 621)
//   200 tx      256 x 512          286 / 345 447 / 408
//              512 x 1024          822 / 1165 1234 / 1366 2142 / 1607
//   300 tx      256 x 512 373 / 580 740 / 708
//   Synthetic, 5 / 75 tx, 256 x 512 pixels, 4 receives 25 / 31 and 96 / 78 (every thread
//   computes its own transmit delays there: the more of them, the fewer receives)
// Up to twelve transmits and 16 to 64 receives on 512 x 1024 pixels and more are faster from
// staged windows than with either (5 transmits, 24 receives 103 us), but a staging plan
// holds the launch's queue, so it serves one stream at a time, and takes 64 bytes a tile and
// receive.
static bool few_receives(const DasArgs &a, int geom) {
    const long long px = a.np * a.nframes, rx = a.nrx, tx = a.ntx;
    if (geom == GEOM_SYNTH_SLOW) return false;  // gradients of the slowness: the rest of the step is far larger
    const bool regs = tx <= kTxReg;  // no column of shared memory: more warps an SM
    if (geom == GEOM_TABBED) {
        const long long each = regs ? 8192 : rx == 2 ? 12288 : std::max(12288LL, 160 * tx - 8192);
        return rx == 1 || (rx <= std::min(16LL, std::max(2LL, 1500 / tx)) && rx * each <= px);
    }
    // Synthetic: 48 receives of 5 transmits at 512 x 1024 pixels 176 us on either, 64 225 / 215
    return px >= 40000 && tx <= 100 && rx <= 48 && rx * (regs ? 8192 : 1365 * tx) <= px;
}

// Groups of frames share the decisions of a tap, so das_kernel is left fewer receives: groups
// of two or four float32 frames, 11 transmits, 256 x 512 pixels, 8 receives 42 / 44 and 64 /
// 66 us a call, 16 receives 63 / 53 and 105 / 76; of eight float16 frames, 2 receives 60 / 60,
// 4 82 / 68.  Three, five or seven frames are two or three launches each of two kernels: three,
// 128 x 128 pixels, 5 transmits, 2 receives 16 / 31.  Synthetic groups are the faster ones throughout.
bool das_frames_ok(const DasArgs &a, int geom, int sumtype, int group) {
    const bool odd = a.nframes < 8 && a.nframes % 2;
    const long long few = group == 8 ? 2 : odd ? 8 : std::max(2LL, std::min(a.np / 16384, 8LL));
    if (geom == GEOM_TABBED && a.nrx <= few) return false;
    return a.fast_axis && sumtype != PYCBF_GB_SUM_NONE && sumtype != PYCBF_GB_SUM_RX_ONLY &&
           das_frames_smem(GEOM_TABBED, sumtype, 8, a.ntx) <= kFramesSmemMax;
}

cudaError_t launch_das_frames(const DasArgs &a, int geom, int sumtype, int dtype, int fg,
                              cudaStream_t s) {
    switch (dtype) {
        case PYCBF_GB_F32: return launch_das_frames_f32(a, geom, sumtype, fg, s);
        case PYCBF_GB_F16: return launch_das_frames_f16(a, geom, sumtype, fg, s);
        case PYCBF_GB_BF16: return launch_das_frames_bf16(a, geom, sumtype, fg, s);
        default: return cudaErrorInvalidValue;
    }
}

long long tabbed_plan_words(long long np, int ntx, int nrx) {
    return plan_layout(np, ntx, nrx).total;
}

cudaError_t launch_tabbed_plan(const DasArgs &a, int interp, int dtype, int *plan, cudaStream_t s) {
    switch (dtype) {
        case PYCBF_GB_F32: return launch_plan_f32(a, interp, plan, s);
        case PYCBF_GB_F16: return launch_plan_f16(a, interp, plan, s);
        case PYCBF_GB_BF16: return launch_plan_bf16(a, interp, plan, s);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_das_staged(const DasArgs &a, int interp, int sumtype, int dtype, const int *plan,
                              int *status, cudaStream_t s) {
    switch (dtype) {
        case PYCBF_GB_F32: return launch_staged_f32(a, interp, sumtype, plan, status, s);
        case PYCBF_GB_F16: return launch_staged_f16(a, interp, sumtype, plan, status, s);
        case PYCBF_GB_BF16: return launch_staged_bf16(a, interp, sumtype, plan, status, s);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_rx_f32(const DasArgs &, int, int, int, cudaStream_t);
cudaError_t launch_rx_f16(const DasArgs &, int, int, int, cudaStream_t);
cudaError_t launch_rx_bf16(const DasArgs &, int, int, int, cudaStream_t);

// Sums over transmits of the kinds with packed decisions, on time axes that allow them
// (fast_axis): das_rx_kernel's (its figures are beside it) but for few receives.  Those and
// the other axes are das_kernel's; on other axes with a staging plan, das_staged_kernel's
// (nearest, 11 transmits, 128 receives, 256 x 512 pixels from 1 s at 40 ns: 178 us staged,
// 293 not).
bool das_rx_ok(const DasArgs &a, int geom, int interp, int sumtype) {
    if (interp != PYCBF_GB_INTERP_CUBIC && interp != PYCBF_GB_INTERP_LINEAR &&
        interp != PYCBF_GB_INTERP_NEAREST)
        return false;
    return a.fast_axis && !few_receives(a, geom) && sumtype != PYCBF_GB_SUM_NONE &&
           sumtype != PYCBF_GB_SUM_RX_ONLY && das_rx_smem(GEOM_TABBED, a.ntx, a.nrx) <= kRxSmemMax;
}

static cudaError_t launch_das_rx(const DasArgs &a, int geom, int interp, int sumtype, int dtype,
                                 cudaStream_t s) {
    switch (dtype) {
        case PYCBF_GB_F32: return launch_rx_f32(a, geom, interp, sumtype, s);
        case PYCBF_GB_F16: return launch_rx_f16(a, geom, interp, sumtype, s);
        case PYCBF_GB_BF16: return launch_rx_bf16(a, geom, interp, sumtype, s);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_das(const DasArgs &a, int geom, int interp, int sumtype, int dtype, bool census,
                       cudaStream_t s) {
    if (!census && geom != GEOM_SYNTH_SLOW && das_rx_ok(a, geom, interp, sumtype))
        return launch_das_rx(a, geom, interp, sumtype, dtype, s);
    if (geom == GEOM_TABBED) {
        switch (dtype) {
            case PYCBF_GB_F32: return launch_das_tabbed_f32(a, interp, sumtype, census, s);
            case PYCBF_GB_F16: return launch_das_tabbed_f16(a, interp, sumtype, census, s);
            case PYCBF_GB_BF16: return launch_das_tabbed_bf16(a, interp, sumtype, census, s);
        }
    } else {
        switch (dtype) {
            case PYCBF_GB_F32: return launch_das_synth_f32(a, interp, sumtype, census, s);
            case PYCBF_GB_F16: return launch_das_synth_f16(a, interp, sumtype, census, s);
            case PYCBF_GB_BF16: return launch_das_synth_bf16(a, interp, sumtype, census, s);
        }
    }
    return cudaErrorInvalidValue;
}

// receive masks of a synthetic geometry: mask[r, i] = 1 where receive r accepts pixel i
__global__ void synth_rx_mask_kernel(const __grid_constant__ DasArgs a, unsigned char *mask) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.np) return;
    float pnt[3] = {0.f, 0.f, 0.f};
    for (int k = 0; k < 3; ++k) if (k < a.ndim) pnt[k] = __ldg(a.geo.pnts + i * a.ndim + k);
    for (int r = 0; r < a.nrx; ++r)
        mask[(long long)r * a.np + i] = isinf(synth_rx_delay(a, r, pnt)) ? 0 : 1;
}

cudaError_t launch_synth_rx_mask(const DasArgs &a, unsigned char *mask, cudaStream_t s) {
    const long long bx = (a.np + 255) / 256;
    synth_rx_mask_kernel<<<(unsigned)bx, 256, 0, s>>>(a, mask);
    return cudaGetLastError();
}

}  // namespace pgb
