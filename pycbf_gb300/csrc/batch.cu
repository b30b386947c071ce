// Uneven batches in one persistent launch (no reference counterpart).
//
// A batch is a list of jobs, each one frame of one beamformer (Tabbed or
// Synthetic, any ntx / nrx / nt / pixel count, float32 / float16 / bfloat16
// channel data), cubic interpolation, summed over transmits and receives.
// The work items are (job, run of tiles_per_item tiles of kBlock pixels) in
// an order the host chooses (largest first, or job order); a grid of `ctas`
// CTAs takes them from a queue head in global memory until it runs dry, so
// frames of very different cost share the GPU without a launch per frame.
//
// Two per-pixel forms, which the autotuner chooses between: the transmits
// taken TXC at a time into registers (TXC 4, 8 or 12; for each chunk every
// receive adds its chunk sum to the pixel's accumulator, so with one chunk,
// ntx <= TXC, the images are bitwise the single-frame ones), or (tx_chunk 0)
// the single-frame kernel's own body, bitwise the same for every ntx.
#include "das_impl.cuh"

namespace pgb {

namespace {

template <int GEOM, typename T, int TXC>
__device__ __forceinline__ void batch_tile(const DasArgs &a, long long tile) {
    using Rec = typename CoefRec<T>::raw;
    const long long i = tile * kBlock + threadIdx.x;
    if (i >= a.np) return;
    const long long np = a.np;
    const int ntx = a.ntx, nrx = a.nrx;
    const long long op = a.pixel_index ? (long long)__ldg(a.pixel_index + i) : i;
    const long long chs = (long long)nrx * a.nt;
    const float inf = __int_as_float(0x7f800000);
    const TapConst tc(a);
    float pnt[3] = {0.f, 0.f, 0.f};
    if (GEOM == GEOM_SYNTH)
        for (int k = 0; k < 3; ++k) if (k < a.ndim) pnt[k] = __ldg(a.geo.pnts + i * a.ndim + k);

    float acc = 0.f;
    for (int t0 = 0; t0 < ntx; t0 += TXC) {
        float2 tt2[TXC / 2], at2[TXC / 2];
        float amax = 0.f;
#pragma unroll
        for (int k = 0; k < TXC; ++k) {
            float tau = inf, apod = 0.f;  // padding: an infinite delay never counts
            const int t = t0 + k;
            if (t < ntx) {
                if (GEOM == GEOM_TABBED) {
                    tau = __ldg(a.tautx + (long long)t * np + i);
                    apod = __ldg(a.apodtx + (long long)t * np + i);
                    amax = fmaxf(amax, fabsf(apod));
                } else {
                    tau = synth_tx_delay(a, t, pnt);
                }
            }
            if (k & 1) {
                tt2[k >> 1].y = tau;
                at2[k >> 1].y = apod;
            } else {
                tt2[k >> 1].x = tau;
                at2[k >> 1].x = apod;
            }
        }
        const int nk_chunk = min(TXC, ntx - t0);
        float bacc = 0.f;  // blocks of kRxBlockSum receives, as the other kernels sum
        for (int r = 0; r < nrx; ++r) {
            if (r > 0 && r % kRxBlockSum == 0) {
                acc += bacc;
                bacc = 0.f;
            }
            float trx, arx;
            bool live;
            if (GEOM == GEOM_TABBED) {
                trx = __ldg(a.taurx + (long long)r * np + i);
                arx = __ldg(a.apodrx + (long long)r * np + i);
                live = __fmul_rn(amax, fabsf(arx)) >= a.thresh;
            } else {
                trx = synth_rx_delay(a, r, pnt);
                arx = 1.f;
                live = trx != inf;
            }
            if (!live) continue;
            const Rec *rec = static_cast<const Rec *>(a.data) + ((long long)t0 * nrx + r) * a.nt;
            auto sum = CubicAcc<T>::zero();
#pragma unroll
            for (int g = 0; g < TXC; g += kCubicGroup) {
                if (g < nk_chunk) {
                    const Rec *rg = rec + (long long)g * chs;
                    if (a.fast_axis)
                        sum = cubic_taps<GEOM, T, kCubicGroup>(a, tc, tt2 + g / 2, at2 + g / 2, trx,
                                                               arx, rg, (unsigned)chs, sum);
                    else
#pragma unroll
                        for (int k = 0; k < kCubicGroup; ++k)
                            sum = cubic_tap_clamped<T, GEOM == GEOM_TABBED>(
                                a, __fadd_rn(pair_lane(tt2 + g / 2, k), trx),
                                __fmul_rn(pair_lane(at2 + g / 2, k), arx), rg + k * chs, sum);
                }
            }
            bacc += CubicAcc<T>::total(sum);
        }
        acc += bacc;
    }
    a.out[op] = acc;
}

template <int TXC>
__global__ void __launch_bounds__(kBlock, 4)
batch_das_kernel(const BatchJob *__restrict__ jobs, const int2 *__restrict__ items,
                 long long nitems, int tiles_per_item, unsigned long long *counter) {
    __shared__ __align__(16) BatchJob s_job;
    __shared__ long long s_k;
    constexpr int kWords = (int)(sizeof(BatchJob) / sizeof(int));
    for (;;) {
        if (threadIdx.x == 0) s_k = (long long)atomicAdd(counter, 1ULL);
        __syncthreads();
        const long long k = s_k;
        if (k >= nitems) break;
        const int2 it = __ldg(items + k);
        const int *src = reinterpret_cast<const int *>(jobs + it.x);
        int *dst = reinterpret_cast<int *>(&s_job);
        for (int w = threadIdx.x; w < kWords; w += blockDim.x) dst[w] = __ldg(src + w);
        __syncthreads();
        const int geom = s_job.geom, dtype = s_job.dtype;
        for (int sub = 0; sub < tiles_per_item; ++sub) {
            const long long tile = (long long)it.y * tiles_per_item + sub;
            if (geom == GEOM_TABBED) {
                if (dtype == PYCBF_GB_F32) batch_tile<GEOM_TABBED, float, TXC>(s_job.a, tile);
                else if (dtype == PYCBF_GB_F16) batch_tile<GEOM_TABBED, __half, TXC>(s_job.a, tile);
                else batch_tile<GEOM_TABBED, __nv_bfloat16, TXC>(s_job.a, tile);
            } else {
                if (dtype == PYCBF_GB_F32) batch_tile<GEOM_SYNTH, float, TXC>(s_job.a, tile);
                else if (dtype == PYCBF_GB_F16) batch_tile<GEOM_SYNTH, __half, TXC>(s_job.a, tile);
                else batch_tile<GEOM_SYNTH, __nv_bfloat16, TXC>(s_job.a, tile);
            }
        }
        __syncthreads();  // every thread is done with s_job and s_k
    }
}

// One pixel by the single-frame kernels' cubic body in its shared-memory column
// form, whatever the job's ntx (per-receive sums are sequential over transmits
// either way, so the images are those of the single-frame calls bit for bit),
// behind a call of its own so that the compiler allocates each geometry's and
// type's registers apart from the others'.
template <int GEOM, typename T>
__device__ __noinline__ void batch_pixel(const DasArgs &a, long long i, float *sm) {
    das_pixel<GEOM, PYCBF_GB_INTERP_CUBIC, PYCBF_GB_SUM_TX_AND_RX, T, false, kTxSmem, true>(a, i, 0, sm);
}

// The same queue, each pixel run by the single-frame kernel's body
// (das_pixel): transmits in registers up to kTxReg, in the thread's column of
// shared memory beyond, every receive's delay and reject computed once.  The
// images are bitwise those of the single-frame calls for every ntx.
__global__ void __launch_bounds__(kBlock, 4)
batch_das_full_kernel(const BatchJob *__restrict__ jobs, const int2 *__restrict__ items,
                      long long nitems, int tiles_per_item, unsigned long long *counter) {
    extern __shared__ float sm[];
    __shared__ __align__(16) BatchJob s_job;
    __shared__ long long s_k;
    constexpr int kWords = (int)(sizeof(BatchJob) / sizeof(int));
    for (;;) {
        if (threadIdx.x == 0) s_k = (long long)atomicAdd(counter, 1ULL);
        __syncthreads();
        const long long k = s_k;
        if (k >= nitems) break;
        const int2 it = __ldg(items + k);
        const int *src = reinterpret_cast<const int *>(jobs + it.x);
        int *dst = reinterpret_cast<int *>(&s_job);
        for (int w = threadIdx.x; w < kWords; w += blockDim.x) dst[w] = __ldg(src + w);
        __syncthreads();
        const int geom = s_job.geom, dtype = s_job.dtype;
        for (int sub = 0; sub < tiles_per_item; ++sub) {
            const long long i0 = ((long long)it.y * tiles_per_item + sub) * kBlock;
            if (i0 >= s_job.a.np) break;  // past the job's last tile
            const long long i = i0 + threadIdx.x;
            if (geom == GEOM_TABBED) {
                if (dtype == PYCBF_GB_F32) batch_pixel<GEOM_TABBED, float>(s_job.a, i, sm);
                else if (dtype == PYCBF_GB_F16) batch_pixel<GEOM_TABBED, __half>(s_job.a, i, sm);
                else batch_pixel<GEOM_TABBED, __nv_bfloat16>(s_job.a, i, sm);
            } else {
                if (dtype == PYCBF_GB_F32) batch_pixel<GEOM_SYNTH, float>(s_job.a, i, sm);
                else if (dtype == PYCBF_GB_F16) batch_pixel<GEOM_SYNTH, __half>(s_job.a, i, sm);
                else batch_pixel<GEOM_SYNTH, __nv_bfloat16>(s_job.a, i, sm);
            }
        }
        __syncthreads();  // every thread is done with s_job and s_k
    }
}

// The same for a batch of one storage type T: the kernel carries the paths of
// that type only, and a CTA copies a job's descriptor only when its next item
// belongs to another job.  Measured on the 64-frame batch with the register form
// as well for ntx <= 12: 43 ms, without it 38 ms.
// five CTAs per SM for 16-bit records (42 against 43 ms), four for float32
// records, whose body spills under five's register cap (47 against 38 ms)
template <typename T>
__global__ void __launch_bounds__(kBlock, CoefRec<T>::kPoly ? 4 : 5)
batch_das_typed_kernel(const BatchJob *__restrict__ jobs, const int2 *__restrict__ items,
                       long long nitems, int tiles_per_item, unsigned long long *counter) {
    extern __shared__ float sm[];
    __shared__ __align__(16) BatchJob s_job;
    __shared__ long long s_k;
    constexpr int kWords = (int)(sizeof(BatchJob) / sizeof(int));
    int cur = -1;  // the job whose descriptor s_job holds
    for (;;) {
        if (threadIdx.x == 0) s_k = (long long)atomicAdd(counter, 1ULL);
        __syncthreads();
        const long long k = s_k;
        if (k >= nitems) break;
        const int2 it = __ldg(items + k);
        if (it.x != cur) {  // the same in every thread: the barrier below is uniform
            const int *src = reinterpret_cast<const int *>(jobs + it.x);
            int *dst = reinterpret_cast<int *>(&s_job);
            for (int w = threadIdx.x; w < kWords; w += blockDim.x) dst[w] = __ldg(src + w);
            __syncthreads();
            cur = it.x;
        }
        const bool tabbed = s_job.geom == GEOM_TABBED;
        for (int sub = 0; sub < tiles_per_item; ++sub) {
            const long long i0 = ((long long)it.y * tiles_per_item + sub) * kBlock;
            if (i0 >= s_job.a.np) break;  // past the job's last tile
            const long long i = i0 + threadIdx.x;
            if (tabbed) batch_pixel<GEOM_TABBED, T>(s_job.a, i, sm);
            else batch_pixel<GEOM_SYNTH, T>(s_job.a, i, sm);
        }
        __syncthreads();  // every thread is done with s_k (and, before a new job, s_job)
    }
}

}  // namespace

// the column of every job's transmit delays (the typed kernel uses the column
// form for every ntx, so this holds even when max_ntx <= kTxReg)
size_t batch_full_smem_bytes(int max_ntx) {
    return (size_t)cubic_column_padded(std::max(max_ntx, 1)) * kBlock * sizeof(float);
}

constexpr size_t kBatchFixedSmem = 512;  // room for the kernels' static part
static_assert(sizeof(BatchJob) + 32 <= kBatchFixedSmem, "");

cudaError_t prepare_batch_das(int max_ntx) {
    const size_t smem = batch_full_smem_bytes(max_ntx);
    if (smem > kSmemMax - kBatchFixedSmem) return cudaErrorInvalidValue;
    cudaError_t err = allow_smem(batch_das_full_kernel, kSmemMax - kBatchFixedSmem);
    if (err == cudaSuccess) err = allow_smem(batch_das_typed_kernel<float>, kSmemMax - kBatchFixedSmem);
    if (err == cudaSuccess) err = allow_smem(batch_das_typed_kernel<__half>, kSmemMax - kBatchFixedSmem);
    if (err == cudaSuccess) err = allow_smem(batch_das_typed_kernel<__nv_bfloat16>, kSmemMax - kBatchFixedSmem);
    return err;
}

cudaError_t launch_batch_das(const BatchJob *jobs, const int2 *items, long long nitems,
                             int tiles_per_item, unsigned long long *counter, int tx_chunk,
                             int ctas, cudaStream_t s, int max_ntx, int dtypes) {
    cudaError_t err = cudaMemsetAsync(counter, 0, sizeof(unsigned long long), s);
    if (err != cudaSuccess) return err;
    if (nitems <= 0) return cudaSuccess;
    const unsigned grid = (unsigned)std::max(1, ctas);
    if (tx_chunk == 0) {  // shared-memory size set by prepare_batch_das, outside any capture
        const size_t smem = batch_full_smem_bytes(max_ntx);
        if (dtypes == 1 << PYCBF_GB_F32)
            batch_das_typed_kernel<float><<<grid, kBlock, smem, s>>>(jobs, items, nitems,
                                                                     tiles_per_item, counter);
        else if (dtypes == 1 << PYCBF_GB_F16)
            batch_das_typed_kernel<__half><<<grid, kBlock, smem, s>>>(jobs, items, nitems,
                                                                      tiles_per_item, counter);
        else if (dtypes == 1 << PYCBF_GB_BF16)
            batch_das_typed_kernel<__nv_bfloat16><<<grid, kBlock, smem, s>>>(
                jobs, items, nitems, tiles_per_item, counter);
        else
            batch_das_full_kernel<<<grid, kBlock, smem, s>>>(jobs, items, nitems, tiles_per_item,
                                                             counter);
        return cudaGetLastError();
    }
    switch (tx_chunk) {
        case 4: batch_das_kernel<4><<<grid, kBlock, 0, s>>>(jobs, items, nitems, tiles_per_item, counter); break;
        case 8: batch_das_kernel<8><<<grid, kBlock, 0, s>>>(jobs, items, nitems, tiles_per_item, counter); break;
        case 12: batch_das_kernel<12><<<grid, kBlock, 0, s>>>(jobs, items, nitems, tiles_per_item, counter); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

}  // namespace pgb
