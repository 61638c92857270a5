// rays.cu — gbrt_trace_rays: ray queries through the persistent world
// traversal (8-wide when the scene carries it).
#include "wavefront.cuh"

namespace gbrt {

#ifndef GBRT_RAYS_MINB
#define GBRT_RAYS_MINB 8
#endif
// traceRayEXT queries (gbrt_trace_rays) through the persistent traversal of
// the world BVH in the layout the scene carries.  Bound by instruction issue at
// a third of the lanes, as the frame's traversal, and compiled in its forms and
// at its occupancy.
template <bool kAny, int kMode>
__global__ void __launch_bounds__(128, GBRT_RAYS_MINB)
    trace_rays_persistent(DevScene s, const gbrt_ray* rays, uint32_t n, uint32_t flags, gbrt_hit* hits, uint32_t* work,
                          DeviceCounters* cnt) {
    TraceStats ts{0, 0, 0};
    world_trace<kAny, kMode, true>(
        s, n, work, flags, ts, gridDim.x * (blockDim.x >> 5),
        [&](uint32_t q, float3& o, float3& d, float& tmin, float& tmax, AnyCtx& ctx) {
            const gbrt_ray r = rays[q];
            o = f3(r.org[0], r.org[1], r.org[2]);
            d = f3(r.dir[0], r.dir[1], r.dir[2]);
            tmin = r.tmin;
            tmax = r.tmax;
            ctx = AnyCtx{q, 0u, 0u, 0u};
        },
        [&](uint32_t q, bool hit, const Hit& h) {
            gbrt_hit g;
            g.t = hit ? h.t : -1.0f;
            g.u = hit ? h.u : 0.0f;
            g.v = hit ? h.v : 0.0f;
            g.instance_id = hit ? h.inst : 0xFFFFFFFFu;
            g.primitive_id = hit ? h.prim : 0xFFFFFFFFu;
            g.custom_index = hit ? s.inst[h.inst].custom : 0xFFFFFFFFu;
            hits[q] = g;
        });
    if (cnt) flush_trace_stats(ts, cnt);
}

cudaError_t init_rays_constants(const float* texel_lut) {
    return cudaMemcpyToSymbol(g_texel_lut, texel_lut, 512 * sizeof(float));
}

cudaError_t launch_trace_rays_persistent(const DevScene& s, const gbrt_ray* rays, uint32_t n, uint32_t flags,
                                         gbrt_hit* hits, uint32_t* work, DeviceCounters* cnt, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    // The form: as the frame's (launch constants of persistent.cuh).  One form with
    // the TLAS walk and the alpha test for every scene took 254 us for 1,500,001
    // random closest hits on an opaque icosphere of 327,680 triangles, its own
    // 176 (any hits 255 and 197; with alpha tests, material zoo, 367 and 266).  With
    // 8, 7, 6 and 5 blocks per SM: 174, 179, 188 and 205.  The forms that spill at 64
    // registers are within 8% of their best at 8 too: closest hits in the zoo 264,
    // 258, 271 and 300, in the binary layout 413, 397, 400 and 418 (zoo 479, 488, 465,
    // 488), under the TLAS of instanced tori 674, 653, 669 and 695, of a city 421,
    // 405, 397 and 420.
    using Kernel = void (*)(DevScene, const gbrt_ray*, uint32_t, uint32_t, gbrt_hit*, uint32_t*, DeviceCounters*);
    static constexpr Kernel kernels[2][6] = {
        {trace_rays_persistent<false, 0>, trace_rays_persistent<false, 1>, trace_rays_persistent<false, 2>,
         trace_rays_persistent<false, 4>, trace_rays_persistent<false, 5>, trace_rays_persistent<false, 6>},
        {trace_rays_persistent<true, 0>, trace_rays_persistent<true, 1>, trace_rays_persistent<true, 2>,
         trace_rays_persistent<true, 4>, trace_rays_persistent<true, 5>, trace_rays_persistent<true, 6>}};
    const int form = trace_mode(s) + (s.all_opaque || (flags & GBRT_RAY_OPAQUE) ? 3 : 0);
    const Kernel kernel = kernels[flags & GBRT_RAY_TERMINATE_ON_FIRST ? 1 : 0][form];
    int dev = 0, sms = 0, per = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, 128, 0)) != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(work, 0, sizeof(uint32_t), st)) != cudaSuccess) return e;
    const TraceGrid g = trace_grid(sms * (per > 0 ? per : 1), n);
    kernel<<<g.blocks, g.threads, 0, st>>>(s, rays, n, flags, hits, work, cnt);
    return cudaGetLastError();
}

}  // namespace gbrt
