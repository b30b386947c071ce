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

// Receives enough for the kernels that spread them over warps.  From tables of one or two,
// most of a CTA's warps would only help to fetch the transmits' column and das_kernel is the
// faster one: a call of 256 x 512 pixels, 2048 samples, one receive and 13 / 31 / 75 / 300
// transmits 47 / 49 / 61 / 400 us against 56 / 66 / 97 / 580, two receives 49 / 54 / 71 / 558
// against 58 / 67 / 108 / 583 (three 51 / 56 / 80 / 694 against 58 / 68 / 112 / 590).
// Synthetic transmit delays are dearer to compute: 75 of them and one receive 88 us spread
// over warps or not, 300 215 against 537.
static bool receives_ok(const DasArgs &a, int geom) { return geom != GEOM_TABBED || a.nrx > 2; }

bool das_frames_ok(const DasArgs &a, int geom, int sumtype) {
    return a.fast_axis && receives_ok(a, geom) && sumtype != PYCBF_GB_SUM_NONE && sumtype != PYCBF_GB_SUM_RX_ONLY &&
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
// (fast_axis): das_rx_kernel is the faster one at every size (its figures are beside it)
// but the fewest receives.  Those and the other axes are das_kernel's; on other axes with a
// staging plan, das_staged_kernel's (nearest, 11 transmits, 128 receives, 256 x 512 pixels
// from 1 s at 40 ns: 178 us staged, 293 not; on ordinary axes with one or two receives the
// plan's launches cost more than the windows save, 47 against 41 us).
bool das_rx_ok(const DasArgs &a, int geom, int interp, int sumtype) {
    if (interp != PYCBF_GB_INTERP_CUBIC && interp != PYCBF_GB_INTERP_LINEAR &&
        interp != PYCBF_GB_INTERP_NEAREST)
        return false;
    return a.fast_axis && receives_ok(a, geom) && sumtype != PYCBF_GB_SUM_NONE &&
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
