// Instantiations of the delay-and-sum with receives across warps for f16 channel data (split per
// storage type so the library's files compile in parallel).
#include "das_rx.cuh"

namespace pgb {

cudaError_t launch_rx_f16(const DasArgs &a, int geom, int interp, int sum, cudaStream_t s) {
    return geom == GEOM_TABBED ? launch_rx_type<GEOM_TABBED, __half>(a, interp, sum, s)
                               : launch_rx_type<GEOM_SYNTH, __half>(a, interp, sum, s);
}

}  // namespace pgb
