// shade_full.cu — the single-frame shade kernel with every material feature
// compiled in: textures, specular-glossiness, volumes, debug mappings.  A unit
// of its own because its size is what bounds it (instruction fetch), so it
// compiles what repeats out of line.
#define GBRT_FULL_SHADE
#include "single_wave.cuh"

namespace gbrt {

__global__ void __launch_bounds__(kShadeThreads, kShadeMinBlocks)
    wf_shade(const __grid_constant__ SingleWave w, WfState st, uint32_t b) {
    after_previous();
    shade_body<SingleWave, false, kFeatAll>(w, st, b);
}

void launch_shade_full(const SingleWave& w, const WfState& st, uint32_t b, uint32_t blocks, uint32_t threads,
                       cudaStream_t stream) {
    launch_after(wf_shade, blocks, threads, stream, w, st, b);
}

const void* shade_full_kernel() { return reinterpret_cast<const void*>(wf_shade); }

cudaError_t init_shade_full_constants(const float* texel_lut) {
    return cudaMemcpyToSymbol(g_texel_lut, texel_lut, 512 * sizeof(float));
}

}  // namespace gbrt
