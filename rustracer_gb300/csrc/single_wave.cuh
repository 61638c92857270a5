// single_wave.cuh — the wave of a single frame: one job, one segment, passed to
// the kernels as a __grid_constant__ parameter (wavefront.cu, shade_full.cu).
#pragma once
#include "launch.cuh"
#include "wavefront.cuh"

namespace gbrt {

// One job and one segment; every block serves it.
struct SingleWave {
    WaveJob J;
    WaveSeg S;
    GB_D uint32_t block_job(int) const { return 0; }
    GB_D uint32_t blk0(int, uint32_t) const { return 0; }
    GB_D uint32_t nblk(int, uint32_t) const { return gridDim.x; }
    GB_D const WaveJob& job(uint32_t) const { return J; }
    GB_D const WaveSeg& seg(uint32_t) const { return S; }
    GB_D uint32_t seg_of_path(uint32_t) const { return 0; }
    GB_D uint32_t seg_of_fin(uint32_t) const { return 0; }
    GB_D uint32_t npaths() const { return S.k * S.npw; }
    GB_D uint32_t nfin() const { return S.npw; }
};

// shade_full.cu: the shade kernel with every material feature compiled in, and
// (for occupancy queries) its symbol.
void launch_shade_full(const SingleWave& w, const WfState& st, uint32_t b, uint32_t blocks, uint32_t threads,
                       cudaStream_t stream);
const void* shade_full_kernel();

}  // namespace gbrt
