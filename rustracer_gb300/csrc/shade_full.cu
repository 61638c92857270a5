// shade_full.cu — single-frame shade kernels with every material feature
// compiled in: textures, specular-glossiness, volumes, debug mappings, and the
// radiance-cache form.  A unit of its own because their size is what bounds
// them (instruction fetch), so it compiles what repeats out of line.
#define GBRT_FULL_SHADE
#include "single_wave.cuh"

namespace gbrt {

__global__ void __launch_bounds__(kShadeThreads, kShadeMinBlocks)
    wf_shade(const __grid_constant__ SingleWave w, WfState st, uint32_t b) {
    shade_body<SingleWave, false, kFeatAll>(w, st, b);
}
__global__ void __launch_bounds__(kShadeThreads, kShadeMinBlocks)
    wf_shade_nrc(const __grid_constant__ SingleWave w, WfState st, uint32_t b, const __grid_constant__ NrcWave nrc) {
    shade_body<SingleWave, true>(w, st, b, &nrc);
}

void launch_shade_full(const SingleWave& w, const WfState& st, uint32_t b, const NrcWave* nrc, uint32_t blocks,
                       uint32_t threads, cudaStream_t stream) {
    if (nrc) wf_shade_nrc<<<blocks, threads, 0, stream>>>(w, st, b, *nrc);
    else wf_shade<<<blocks, threads, 0, stream>>>(w, st, b);
}

const void* shade_full_kernel(bool nrc) {
    return nrc ? reinterpret_cast<const void*>(wf_shade_nrc) : reinterpret_cast<const void*>(wf_shade);
}

cudaError_t init_shade_full_constants(const float* texel_lut) {
    return cudaMemcpyToSymbol(g_texel_lut, texel_lut, 512 * sizeof(float));
}

}  // namespace gbrt
