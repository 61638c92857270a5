// build_arena.h — device memory that the BVH builds of a context carve their
// scratch from.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <mutex>

namespace gbrt {

// Grown to the largest build's need (about 270 B per triangle) and kept up to
// kKeep, so that a rebuild of an animated scene does not allocate: scenes of up
// to four million triangles rebuild in it, larger ones give theirs back.  A build holds `mu`
// from its reserve to its last launch: a context's builds come from the
// caller's thread and, for skinned jobs, from the job worker's, each of many
// launches with host waits between them, and their order on the stream keeps
// two of them apart only when one is queued whole before the other.
struct BuildArena {
    static constexpr size_t kKeep = size_t(1) << 30;
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
    // Gives memory back beyond `keep` bytes.
    void trim(size_t keep) {
        std::lock_guard<std::mutex> hold(mu);
        if (bytes > keep) release();
    }
};

// The life of one call's builds: when it ends the arena keeps at most kKeep,
// and nothing unless the call says done(), since a call that fails is likely
// short of memory.
struct BuildCall {
    BuildArena& arena;
    size_t keep = 0;
    explicit BuildCall(BuildArena& a) : arena(a) {}
    BuildCall(const BuildCall&) = delete;
    BuildCall& operator=(const BuildCall&) = delete;
    ~BuildCall() { arena.trim(keep); }
    void done() { keep = BuildArena::kKeep; }
};

}  // namespace gbrt
