// build_arena.h — device memory that the BVH builds of a context carve their
// scratch from.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <mutex>

namespace gbrt {

// Grown to the largest build's need (about 270 B per triangle) and kept, so
// that a rebuild of an animated scene does not allocate.  A build holds `mu`
// from its reserve to its last launch: a context's builds come from the
// caller's thread and, for skinned jobs, from the job worker's, each of many
// launches with host waits between them, and their order on the stream keeps
// two of them apart only when one is queued whole before the other.
struct BuildArena {
    void* p = nullptr;
    size_t bytes = 0;
    std::mutex mu;
    BuildArena() = default;
    BuildArena(const BuildArena&) = delete;
    BuildArena& operator=(const BuildArena&) = delete;
    ~BuildArena() { release(); }
    // With mu held.
    cudaError_t reserve(size_t n) {
        if (n <= bytes) return cudaSuccess;
        release();
        const cudaError_t e = cudaMalloc(&p, n);
        if (e == cudaSuccess) bytes = n;
        else p = nullptr;
        return e;
    }
    void release() {  // cudaFree waits for the launches that use it
        if (p) cudaFree(p);
        p = nullptr;
        bytes = 0;
    }
};

}  // namespace gbrt
