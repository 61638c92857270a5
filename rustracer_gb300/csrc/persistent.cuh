// persistent.cuh — persistent-lane traversal of the world BVH with ray
// refill (after Aila & Laine 2009, "Understanding the Efficiency of Ray
// Traversal on GPUs").
//
// Every lane owns one ray at a time.  Each outer iteration a lane descends
// inner nodes until it reaches a leaf (or its stack empties), then tests that
// leaf's triangles (while-while).  A lane whose ray finished goes idle; once
// at least kRefill lanes of the warp are idle they take new rays from the
// queue together (one atomic per warp).  The warp therefore no longer waits
// for its longest ray, which is what kept SIMT efficiency low when a warp
// traced a fixed group of 32 rays.  The stack holds (node, entry distance)
// pairs so entries behind the current closest hit are dropped when popped.
//
// Scenes with transformed instances finish each ray with the two-level pass
// of trace.cuh after the world BVH (same exactness rules).
#pragma once
#include "trace.cuh"

namespace gbrt {

constexpr int kEmpty = 0x7FFFFFFF;  // "stack exhausted"
// Idle lanes that trigger a refill: icosphere frame at 12 / 16 / 20 lanes 86.1 /
// 86.5 / 88.1 ms, instanced tori 13.6 / 13.7 / 14.0 ms (with triangles tested
// lane by lane 16 was best: the idle lanes now work).
#ifndef GBRT_REFILL
#define GBRT_REFILL 12
#endif
constexpr uint32_t kRefill = GBRT_REFILL;  // idle lanes that trigger a refill

// Rays a warp takes from the queue at a time.  A queue of few rays is spread
// over half of the launch's warps instead of filling the first ones: a warp's
// time grows with the rays whose ways through the tree it serialises, and the
// other warps would idle.  Frames of one sample at depth 8, us of device time
// with 32 / 8 / 4 / 2 / 1 rays at least (all of the warps: half): 64 x 64
// Cornell 214 / 185 / 184 / 183 / 204, 128 x 128 instanced tori 1636 / 1402 /
// 1310 / 1255 / 1198; half of the warps instead of all: 512 x 256 icosphere 626
// against 659, 128 x 128 tori 1338 against 1310.
#ifndef GBRT_MIN_QUOTA
#define GBRT_MIN_QUOTA 2
#endif
constexpr uint32_t kMinQuota = GBRT_MIN_QUOTA;
GB_D uint32_t ray_quota(uint32_t n, uint32_t warps) {
    const unsigned long long q = (2ull * n + warps - 1u) / warps;
    return q < kMinQuota ? kMinQuota : (q < 32u ? (uint32_t)q : 32u);
}

// Loader: bool load(uint32_t q, float3& o, float3& d, float& tmin, float& tmax, AnyCtx& ctx)
// Finisher: void finish(uint32_t q, bool hit, const Hit& h)
template <bool kAny, bool kAlpha, class Loader, class Finisher>
GB_D void persistent_trace(const DevScene& s, uint32_t n, uint32_t* work, uint32_t flags, TraceStats& ts,
                           uint32_t quota, Loader&& load, Finisher&& finish) {
    const uint32_t lane = threadIdx.x & 31u;
    const bool test_alpha = kAlpha && !(flags & GBRT_RAY_OPAQUE) && !s.all_opaque;
    int stack_node[kStack];
    float stack_t[kStack];
    bool has = false, exhausted = false;
    uint32_t q = 0;
    TRay r;
    Hit best;
    float best_det = 1.0f;  // any-hit queries: best.u, best.v hold V, W of the world hit until the ray is done
    AnyCtx ctx{0, 0, 0, 0};
    float tmin = 0.0f, tmax = 0.0f;
    int cur = kEmpty, sp = 0;
    uint32_t iter = 0;
    for (;;) {
        if (!exhausted) {
            const uint32_t idle = __ballot_sync(0xFFFFFFFFu, !has);
            if (__popc(idle) >= (int)kRefill) {
                const uint32_t take = min((uint32_t)__popc(idle), quota);
                uint32_t base = 0;
                if (lane == 0) base = atomicAdd(work, take);
                base = __shfl_sync(0xFFFFFFFFu, base, 0);
                if (base + take >= n) exhausted = true;
                const uint32_t rank = __popc(idle & ((1u << lane) - 1u));
                if (!has && rank < take) {
                    q = base + rank;
                    if (q < n) {
                        float3 o, d;
                        load(q, o, d, tmin, tmax, ctx);
                        best.t = tmax;
                        best.u = best.v = 0.0f;
                        best_det = 1.0f;
                        best.inst = best.prim = best.bgeo = 0xFFFFFFFFu;
                        iter = 0;
                        if (d.x == 0.0f && d.y == 0.0f && d.z == 0.0f) {
                            finish(q, false, best);
                        } else {
                            has = true;
                            setup_ray(r, o, d);
                            sp = 0;
                            cur = kEmpty;
                            float tn;
                            if (s.has_world && box_hit(r, s.world_lo.x, s.world_hi.x, s.world_lo.y, s.world_hi.y,
                                                       s.world_lo.z, s.world_hi.z, tmin, best.t, tn))
                                cur = s.world_root;
                        }
                    }
                }
            }
        }
        if (!__any_sync(0xFFFFFFFFu, has)) {
            if (exhausted) break;
            continue;
        }
        if (!has) continue;
        // --- descend to a leaf ------------------------------------------------
        int leaf = 0;
        while (cur != kEmpty) {
            if (++iter > kMaxIter) {
                ts.status |= GBRT_STATUS_ITER_LIMIT;
                cur = kEmpty;
                break;
            }
            if (cur < 0) {  // leaf: take it, resume from the stack afterwards
                leaf = cur;
                cur = kEmpty;
                while (sp > 0) {
                    --sp;
                    if (stack_t[sp] <= best.t * kBoxSlack) {
                        cur = stack_node[sp];
                        break;
                    }
                }
                break;
            }
            const BNode2* nd = s.nodes + cur;
            const float4 a = __ldg(&nd->lxy), b = __ldg(&nd->rxy), z = __ldg(&nd->lrz);
            const int4 c = __ldg(&nd->c);
            ts.nodes++;
            float tn0, tn1;
            const bool h0 = box_hit(r, a.x, a.y, a.z, a.w, z.x, z.y, tmin, best.t, tn0);
            const bool h1 = box_hit(r, b.x, b.y, b.z, b.w, z.z, z.w, tmin, best.t, tn1);
            if (h0 && h1) {
                const bool swap = tn1 < tn0;
                if (sp < kStack) {
                    stack_node[sp] = swap ? c.x : c.y;
                    stack_t[sp] = swap ? tn0 : tn1;
                    ++sp;
                } else {
                    ts.status |= GBRT_STATUS_STACK_OVERFLOW;
                }
                cur = swap ? c.y : c.x;
            } else if (h0) {
                cur = c.x;
            } else if (h1) {
                cur = c.y;
            } else {
                cur = kEmpty;
                while (sp > 0) {
                    --sp;
                    if (stack_t[sp] <= best.t * kBoxSlack) {
                        cur = stack_node[sp];
                        break;
                    }
                }
            }
        }
        // --- test the leaf ------------------------------------------------------
        bool done = false;
        if (leaf != 0) {
            const uint32_t first = leaf_first(leaf), count = leaf_count(leaf);
            for (uint32_t i = 0; i < count; ++i) {
                const TriRec* tr = s.tris + first + i;
                const float4 pa = __ldg(&tr->a), pb = __ldg(&tr->b), pc = __ldg(&tr->c);
                ts.tris++;
                // any-hit queries keep V, W and det of the hit and divide once the ray is done (if
                // their caller reads u, v at all); closest-hit queries divide per accepted hit
                float t, u, v, det = 1.0f;
                if constexpr (kAny) {
                    if (!isect_tri_t(r, f3(pa), f3(pb), f3(pc), tmin, best.t, t, u, v, det)) continue;
                } else {
                    if (!isect_tri(r, f3(pa), f3(pb), f3(pc), tmin, best.t, t, u, v)) continue;
                }
                const uint32_t inst = __float_as_uint(pa.w);
                const uint32_t prim = __float_as_uint(pb.w);
                const uint32_t gw = __float_as_uint(pc.w);
                if (!closer(t, inst, prim, best)) continue;
                if (test_alpha && !(gw >> 31) &&
                    anyhit_ignore(s, s.inst[inst].custom, prim, inst, kAny ? __fdiv_rn(u, det) : u,
                                  kAny ? __fdiv_rn(v, det) : v, ctx))
                    continue;
                best.t = t;
                best.u = u;
                best.v = v;
                best_det = det;
                best.inst = inst;
                best.prim = prim;
                best.bgeo = gw & 0x7FFFFFFFu;
                if (kAny) {
                    done = true;
                    break;
                }
            }
        }
        if (!done && cur == kEmpty) done = true;
        if (done) {
            if constexpr (kAny) {
                best.u = __fdiv_rn(best.u, best_det);
                best.v = __fdiv_rn(best.v, best_det);
            }
            if (s.has_tlas && !(kAny && best.inst != 0xFFFFFFFFu)) {
                // transformed instances: finish the ray with the two-level pass
                trace_tlas<kAny>(s, r, r.o, r.d, tmin, best, test_alpha, ctx, ts);
            }
            finish(q, best.inst != 0xFFFFFFFFu, best);
            has = false;
        }
    }
}

}  // namespace gbrt

namespace gbrt {

// Inclusive prefix sum over the warp.
GB_D uint32_t warp_scan(uint32_t v) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
        asm volatile("{\n.reg .u32 t;\n.reg .pred p;\nshfl.sync.up.b32 t|p, %0, %1, 0, 0xFFFFFFFF;\n@p add.u32 %0, %0, t;\n}\n"
                     : "+r"(v)
                     : "r"(o));
    return v;
}

// What the lanes of a warp need of each other's rays to test triangles for
// one another, and the triangles of one round.
struct WarpTris {
    float4 o[32];     // origin, tmin
    float4 s[32];     // shear constants, axis permutation kx | ky << 2 | kz << 4
    uint2 pair[32];   // triangle slot, lane of its ray; or work handed to an idle lane
    uint32_t helpers[32];  // lanes that work on this lane's ray besides itself
};

// Idle lanes of a warp that make it worth handing work out (2, 8 and 16 measure
// the same within 2%).
constexpr int kSteal = 8;

// Persistent-lane traversal of the 8-wide world BVH; same interface and
// refill policy as persistent_trace.
//
// Every lane visits the nodes of its own ray, but the triangles that a step
// of the warp turned up (none to a dozen a lane) are dealt out over all 32
// lanes through shared memory, one each: the kernel is bound by instruction
// issue, and testing them lane by lane kept about 4 of 32 lanes busy while the
// lane with the most triangles finished.  The owner of a ray then takes the
// results of its triangles in slot order, so hits are those of the
// lane-by-lane loop.  Icosphere frame (1080p x 64): extend 41.5 -> 36.7 ms,
// shadow 22.4 -> 18.0; 1.5M incoherent ray queries 383 -> 310 us.
//
// Once the queue is empty (exhausted), idle lanes take subtrees from lanes
// that have some pending, with a copy of the ray: a launch ends with its
// longest rays, whose dozens of steps in a row took most of the time of waves
// of up to a million rays while the rest of the GPU was idle.  A helper hands
// every hit to the ray's owner, which settles ties as ever and reports once
// nobody works on its ray (WarpTris::helpers), so hits do not depend on who
// helps; the statistics' node and triangle counts do, by a few percent.  64 x
// 64 frames of instanced tori 820 -> 519 us, of an icosphere 348 -> 301, 854 x
// 480 x 3 viewer 1.10 -> 1.00 ms; 1080p x 64 icosphere 77.0 -> 77.3.
//
// kHit: the finisher reads the hit of an any-hit query, not only whether there
// is one; such a query takes no help, so that it reports the first hit of the
// traversal order whatever its neighbours do.  Every block has at most 128
// threads.
template <bool kAny, bool kTlas, bool kAlpha, bool kHit, class Loader, class Finisher>
GB_D void persistent_trace_cw(const DevScene& s, uint32_t n, uint32_t* work, uint32_t flags, TraceStats& ts,
                              uint32_t quota, Loader&& load, Finisher&& finish) {
    constexpr uint32_t kAll = 0xFFFFFFFFu, kInner = 0xFF000000u;
    constexpr bool kHelp = !(kAny && kHit);
    __shared__ WarpTris s_tris[4];
    WarpTris& sw = s_tris[threadIdx.x >> 5];
    const uint32_t lane = threadIdx.x & 31u;
    const bool test_alpha = kAlpha && !(flags & GBRT_RAY_OPAQUE) && !s.all_opaque;
    uint2 stack[kCwStack];
    bool has = false, exhausted = false;
    uint32_t q = 0, oct = 0;
    TRay r;
    Hit best;
    AnyCtx ctx{0, 0, 0, 0};
    float tmin = 0.0f, tmax = 0.0f;
    uint2 ng = make_uint2(0, 0);
    int sp = 0;
    uint32_t own = lane;  // the lane whose ray this one works on (itself until idle lanes help)
    uint32_t iter = 0;
    if (kHelp) sw.helpers[lane] = 0u;
    for (;;) {
        if (!exhausted) {
            const uint32_t idle = __ballot_sync(kAll, !has);
            if (__popc(idle) >= (int)kRefill) {
                const uint32_t take = min((uint32_t)__popc(idle), quota);
                uint32_t base = 0;
                if (lane == 0) base = atomicAdd(work, take);
                base = __shfl_sync(kAll, base, 0);
                if (base + take >= n) exhausted = true;
                const uint32_t rank = __popc(idle & ((1u << lane) - 1u));
                if (!has && rank < take) {
                    q = base + rank;
                    if (q < n) {
                        float3 o, d;
                        load(q, o, d, tmin, tmax, ctx);
                        best.t = tmax;
                        best.u = best.v = 0.0f;
                        best.inst = best.prim = best.bgeo = 0xFFFFFFFFu;
                        iter = 0;
                        if (d.x == 0.0f && d.y == 0.0f && d.z == 0.0f) {
                            finish(q, false, best);
                        } else {
                            has = true;
                            setup_ray(r, o, d);
                            oct = (d.x < 0.0f ? 1u : 0u) | (d.y < 0.0f ? 2u : 0u) | (d.z < 0.0f ? 4u : 0u);
                            sw.o[lane] = make_float4(o.x, o.y, o.z, tmin);
                            sw.s[lane] = make_float4(r.Sx, r.Sy, r.Sz, __int_as_float(r.kx | r.ky << 2 | r.kz << 4));
                            cw_ray<!kTlas>(r);
                            sp = 0;
                            // virtual parent: one inner child (the root, node 0) in slot 0
                            ng = s.has_world ? make_uint2(0u, (1u << (24u + oct)) | 1u) : make_uint2(0u, 0u);
                        }
                    }
                }
            }
        }
        if (!__any_sync(kAll, has)) {
            if (exhausted) break;
            continue;
        }
        // --- no more rays: idle lanes take work from busy ones ------------------
        if (kHelp && exhausted) {
            const uint32_t idle = __ballot_sync(kAll, !has), inner = ng.y & kInner;
            const bool rich = has && (sp > 0 || (inner & (inner - 1u)));
            const uint32_t donors = __ballot_sync(kAll, rich);
            const int pairs = min(__popc(idle), __popc(donors)), rank = __popc((rich ? donors : idle) & ((1u << lane) - 1u));
            if (pairs && __popc(idle) >= kSteal) {
                if (rich && rank < pairs) {  // the last stack entry, or all but the next child; bits 8..12: from whom
                    uint2 give;
                    if (sp > 0) {
                        give = stack[--sp];
                    } else {
                        give = make_uint2(ng.x, ng.y & ~(inner & (0u - inner)));
                        ng.y = (inner & (0u - inner)) | (ng.y & 0xFFu);
                    }
                    sw.pair[rank] = make_uint2(give.x, give.y | lane << 8);
                }
                __syncwarp();
                const bool take = !has && rank < pairs;
                uint2 got = make_uint2(0u, lane << 8);
                if (take) got = sw.pair[rank];
                const uint32_t from = (got.y >> 8) & 31u;
                const float ix = __shfl_sync(kAll, r.inv.x, from), iy = __shfl_sync(kAll, r.inv.y, from),
                            iz = __shfl_sync(kAll, r.inv.z, from), bt = __shfl_sync(kAll, best.t, from);
                const uint32_t o2 = __shfl_sync(kAll, oct, from), w2 = __shfl_sync(kAll, own, from);
                AnyCtx c2{0, 0, 0, 0};
                if constexpr (kAlpha)
                    c2 = AnyCtx{__shfl_sync(kAll, ctx.px, from), __shfl_sync(kAll, ctx.py, from),
                                __shfl_sync(kAll, ctx.sample, from), __shfl_sync(kAll, ctx.tag, from)};
                if (take) {
                    const float4 o4 = sw.o[from];
                    sw.o[lane] = o4;
                    sw.s[lane] = sw.s[from];
                    r.o = f3(o4);
                    r.inv = f3(ix, iy, iz);
                    tmin = o4.w;
                    oct = o2;
                    own = w2;
                    if constexpr (kAlpha) ctx = c2;
                    best.t = bt;
                    best.inst = best.prim = 0xFFFFFFFFu;
                    ng = make_uint2(got.x, got.y & (kInner | 0xFFu));
                    sp = 0;
                    iter = 0;
                    has = true;
                    atomicAdd(&sw.helpers[own], 1u);
                }
                __syncwarp();
            }
            const float ot = __shfl_sync(kAll, best.t, own);
            if (own != lane && ot < best.t) {  // ties with the owner's hit are settled by the owner
                best.t = ot;
                best.inst = best.prim = 0xFFFFFFFFu;
            }
        }
        // --- one node per ray -------------------------------------------------
        bool done = false;
        uint32_t tri_bits = 0, tri_base = 0;
        if (has) {
            if (!(ng.y & kInner) && sp > 0) ng = stack[--sp];
            if (++iter > kMaxIter) {
                ts.status |= GBRT_STATUS_ITER_LIMIT;
                done = true;
            } else if (ng.y & kInner) {
                const uint32_t bit = __ffs(ng.y & kInner) - 1u;
                ng.y &= ~(1u << bit);
                const uint32_t slot = (bit - 24u) ^ oct;
                const uint32_t child = ng.x + __popc((ng.y & 0xFFu) & ((1u << slot) - 1u));
                if (ng.y & kInner) {
                    if (sp < kCwStack) stack[sp++] = ng;
                    else ts.status |= GBRT_STATUS_STACK_OVERFLOW;
                }
                uint32_t cb, im;
                const uint32_t hm = cw_intersect(s.cw_nodes, child, r, oct * 0x01010101u, tmin, best.t, cb, tri_base, im);
                ts.nodes++;
                ng = make_uint2(cb, (hm & kInner) | im);
                tri_bits = hm & 0x00FFFFFFu;
            }
        }
        // --- the triangles of all rays, 32 at a time ----------------------------
        const uint32_t cnt = __popc(tri_bits);
        const uint32_t incl = warp_scan(cnt), total = __shfl_sync(kAll, incl, 31);
        uint32_t pos = incl - cnt;  // place of this lane's next triangle in the round
        for (uint32_t base = 0; base < total; base += 32) {
            uint32_t mine = 0;
            while (tri_bits && pos < 32u) {
                const uint32_t tbit = __ffs(tri_bits) - 1u;
                tri_bits &= tri_bits - 1u;
                sw.pair[pos] = make_uint2(tri_base + tbit, lane);
                mine |= 1u << pos;
                ++pos;
            }
            pos -= 32u;
            __syncwarp();
            const bool live = lane < total - base;
            uint2 pr = make_uint2(0u, lane);
            if (live) pr = sw.pair[lane];
            const float tcur = __shfl_sync(kAll, best.t, pr.y);
            AnyCtx pc{0, 0, 0, 0};
            if (kAlpha && test_alpha)
                pc = AnyCtx{__shfl_sync(kAll, ctx.px, pr.y), __shfl_sync(kAll, ctx.py, pr.y),
                            __shfl_sync(kAll, ctx.sample, pr.y), __shfl_sync(kAll, ctx.tag, pr.y)};
            bool hit = false;
            float t = 0.0f, u = 0.0f, v = 0.0f;
            uint32_t inst = 0, prim = 0;
            if (live) {
                const float4 po = sw.o[pr.y], ps = sw.s[pr.y];
                const int k = __float_as_int(ps.w);
                TRay pray;
                pray.o = f3(po);
                pray.Sx = ps.x;
                pray.Sy = ps.y;
                pray.Sz = ps.z;
                pray.kx = k & 3;
                pray.ky = (k >> 2) & 3;
                pray.kz = k >> 4;
                const TriRec* tr = s.cw_tris + pr.x;
                const float4 pa = __ldg(&tr->a), pb = __ldg(&tr->b), pcv = __ldg(&tr->c);
                ts.tris++;
                inst = __float_as_uint(pa.w);
                prim = __float_as_uint(pb.w);
                if constexpr (kAny && !kHit && !kAlpha) {
                    float V, W, det;
                    hit = isect_tri_t(pray, f3(pa), f3(pb), f3(pcv), po.w, tcur, t, V, W, det);
                } else {
                    hit = isect_tri(pray, f3(pa), f3(pb), f3(pcv), po.w, tcur, t, u, v);
                    if (kAlpha && hit && test_alpha && !(__float_as_uint(pcv.w) >> 31) &&
                        anyhit_ignore(s, s.inst[inst].custom, prim, inst, u, v, pc))
                        hit = false;
                }
            }
            uint32_t my = __ballot_sync(kAll, hit) & mine;  // hits of this lane's own ray
            __syncwarp();                                   // the pairs have been read
            if constexpr (kAny) {
                if constexpr (kHit) {
                    const uint32_t f = my && !done ? __ffs(my) - 1u : lane;
                    const float t2 = __shfl_sync(kAll, t, f), u2 = __shfl_sync(kAll, u, f),
                                v2 = __shfl_sync(kAll, v, f);
                    const uint32_t i2 = __shfl_sync(kAll, inst, f), p2 = __shfl_sync(kAll, prim, f);
                    if (my && !done) {
                        best.t = t2;
                        best.u = u2;
                        best.v = v2;
                        best.inst = i2;
                        best.prim = p2;
                    }
                } else if (my) {
                    best.inst = 0u;
                }
                done = done || my;
                if constexpr (kHelp) {
                    if (exhausted) {
                        uint32_t up = __ballot_sync(kAll, my && own != lane);  // helpers' hits end their owners' rays
                        for (; up; up &= up - 1u)
                            if (lane == __shfl_sync(kAll, own, __ffs(up) - 1)) best.inst = 0u;
                    }
                }
            } else {
                bool fresh = false;
                while (__any_sync(kAll, my != 0u)) {
                    const uint32_t f = my ? __ffs(my) - 1u : lane;
                    const float t2 = __shfl_sync(kAll, t, f), u2 = __shfl_sync(kAll, u, f),
                                v2 = __shfl_sync(kAll, v, f);
                    const uint32_t i2 = __shfl_sync(kAll, inst, f), p2 = __shfl_sync(kAll, prim, f);
                    if (my && closer(t2, i2, p2, best)) {
                        best.t = t2;
                        best.u = u2;
                        best.v = v2;
                        best.inst = i2;
                        best.prim = p2;
                        fresh = true;
                    }
                    my &= my - 1u;
                }
                if constexpr (kHelp) {
                    if (exhausted) {  // helpers' hits go to their owners at once
                        for (uint32_t up = __ballot_sync(kAll, fresh && own != lane); up; up &= up - 1u) {
                            const int f = __ffs(up) - 1;
                            const float t2 = __shfl_sync(kAll, best.t, f), u2 = __shfl_sync(kAll, best.u, f),
                                        v2 = __shfl_sync(kAll, best.v, f);
                            const uint32_t i2 = __shfl_sync(kAll, best.inst, f), p2 = __shfl_sync(kAll, best.prim, f);
                            if (lane == __shfl_sync(kAll, own, f) && closer(t2, i2, p2, best)) {
                                best.t = t2;
                                best.u = u2;
                                best.v = v2;
                                best.inst = i2;
                                best.prim = p2;
                            }
                        }
                    }
                }
            }
        }
        bool last = true;  // nobody else works on this ray
        if (kHelp && exhausted) {
            const uint32_t found = __shfl_sync(kAll, best.inst, own);  // by every lane, done or not
            if (kAny && found != 0xFFFFFFFFu) done = true;
            if (has && own != lane && (done || (!(ng.y & kInner) && sp == 0))) {
                has = false;
                atomicSub(&sw.helpers[own], 1u);
            }
            __syncwarp();
            last = own == lane && sw.helpers[lane] == 0u;
        }
        if (has && (done || (!(ng.y & kInner) && sp == 0)) && last) {
            if constexpr (kTlas) {
                if (s.has_tlas && !(kAny && best.inst != 0xFFFFFFFFu))
                    trace_tlas<kAny, true>(s, r, r.o, r.d, tmin, best, test_alpha, ctx, ts);
            }
            finish(q, best.inst != 0xFFFFFFFFu, best);
            has = false;
        }
    }
}

// Traversal forms of a world query (chosen per launch by trace_mode):
//   kTraceBinary  binary world BVH, binary BLASes (scenes without 8-wide nodes)
//   kTraceWide    8-wide world BVH, no transformed instances
//   kTraceWideTlas 8-wide world BVH, then the TLAS with 8-wide BLASes
// Keeping the TLAS code out of the common form keeps its registers free.
// A form | kTraceOpaque is compiled without the any-hit alpha test, for
// launches where no geometry can need it (all-opaque scenes or frames); the
// code it leaves out cost the 8-wide traversal kernels spills.
constexpr int kTraceBinary = 0, kTraceWide = 1, kTraceWideTlas = 2, kTraceOpaque = 4;

template <bool kAny, int kMode, bool kHit, class Loader, class Finisher>
GB_D void world_trace(const DevScene& s, uint32_t n, uint32_t* work, uint32_t flags, TraceStats& ts,
                      uint32_t warps, Loader&& load, Finisher&& finish) {
    constexpr int kForm = kMode & 3;
    constexpr bool kAlpha = !(kMode & kTraceOpaque);
    const uint32_t quota = ray_quota(n, warps);
    if constexpr (kForm == kTraceBinary) persistent_trace<kAny, kAlpha>(s, n, work, flags, ts, quota, load, finish);
    else persistent_trace_cw<kAny, kForm == kTraceWideTlas, kAlpha, kHit>(s, n, work, flags, ts, quota, load, finish);
}

// Launch shape of a traversal kernel over at most n rays, `resident` blocks
// of 128 threads filling the GPU: full blocks when every resident warp gets
// rays, else one-warp blocks, one per kMinQuota rays, which spread over all
// SMs and leave no warp that only finds its queue empty.  The 64 x 64 Cornell
// frame takes 246 us instead of 284 with the quota, these grids, the shade
// blocks of shade_threads and queue_done.
struct TraceGrid {
    uint32_t blocks, threads;
};
inline TraceGrid trace_grid(int resident, uint64_t n) {
    const uint64_t full = (uint64_t)resident * 4, warps = (n + kMinQuota - 1) / kMinQuota;
    if (warps >= full) return {(uint32_t)resident, 128u};
    return {warps ? (uint32_t)warps : 1u, 32u};
}

// The form a scene needs: binary when it has a world BVH without its
// 8-wide copy (after gbrt_scene_rebuild_noalloc) or when the autotuner chose
// it, else 8-wide, with the TLAS when it has transformed instances.
inline int trace_mode(const DevScene& s) {
    if (s.prefer_binary || (s.has_world && !s.cw_nodes)) return kTraceBinary;
    return s.has_tlas ? kTraceWideTlas : kTraceWide;
}

}  // namespace gbrt
