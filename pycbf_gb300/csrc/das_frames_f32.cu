// Instantiations of the several-frame delay-and-sum for f32 channel data (split
// per storage type so the library's files compile in parallel).
#include "das_frames.cuh"

namespace pgb {

cudaError_t launch_das_frames_f32(const DasArgs &a, int geom, int sum, int fg, cudaStream_t s) {
    return geom == GEOM_TABBED ? launch_das_frames_type<GEOM_TABBED, float>(a, sum, fg, s)
                               : launch_das_frames_type<GEOM_SYNTH, float>(a, sum, fg, s);
}

}  // namespace pgb
