// bvh_build.cu — GPU BVH construction.
//
// 30-bit Morton codes of the item centroids and a CUB radix sort, then a
// binary tree: by default parallel locally-ordered clustering
// (ploc_build.inc), or, for allocation-free rebuilds, the linear BVH of Karras 2012
// ("Maximizing Parallelism in the Construction of BVHs, Octrees, and k-d
// Trees": one thread per inner node finds its key range and split); then one
// bottom-up pass (atomic arrival counters) that computes the boxes
// and the SAH cost of every subtree and collapses subtrees of at most
// kMaxLeaf items into leaves when that lowers the SAH cost.  The result is
// written in the traversal layout (BNode2 with both child boxes; leaves as
// codes over a contiguous range of TriRec slots in Morton order).
#include <cub/device/device_radix_sort.cuh>
#include <algorithm>
#include <cmath>
#include <cstring>
#include <utility>
#include <float.h>
#include "kernels.h"
#include "launch.cuh"

namespace gbrt {

namespace {

#ifndef GBRT_SAH_TRAVERSE
#define GBRT_SAH_TRAVERSE 1.2f
#endif
constexpr float kCostTraverse = GBRT_SAH_TRAVERSE;  // SAH cost of an inner node relative to one triangle test
constexpr float kCostTri = 1.0f;

__device__ __forceinline__ uint32_t expand_bits(uint32_t v) {
    v = (v * 0x00010001u) & 0xFF0000FFu;
    v = (v * 0x00000101u) & 0x0F00F00Fu;
    v = (v * 0x00000011u) & 0xC30C30C3u;
    v = (v * 0x00000005u) & 0x49249249u;
    return v;
}

// float <-> order-preserving uint for atomic min/max of bounds
__device__ __forceinline__ uint32_t f2o(float f) {
    uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float o2f(uint32_t u) {
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u);
}

struct Scratch {
    float4* lo;           // [n] item boxes
    float4* hi;
    uint32_t* morton_in;  // [n]
    uint32_t* morton;     // [n] sorted
    uint32_t* idx_in;     // [n]
    uint32_t* idx;        // [n] sorted item index
    int32_t* left;        // [n-1] inner children: >= 0 inner, < 0 ~leaf(sorted position)
    int32_t* right;
    int32_t* parent_i;    // [n-1] parent of inner node (-1 root)
    int32_t* parent_l;    // [n] parent of leaf
    uint32_t* range_lo;   // [n-1]
    uint32_t* range_hi;
    float4* ilo;          // [n-1] inner boxes
    float4* ihi;
    float* cost;          // [n-1] SAH cost (area-weighted)
    uint32_t* collapse;   // [n-1] 1 = becomes a leaf
    uint32_t* arrive;     // [n-1]
    uint32_t* cbounds;    // 6 order-encoded centroid bounds
    TriRec* unsorted;     // [n]
    void* cub_tmp;
    size_t cub_bytes;
    // 8-wide collapse
    float* dp_cost;         // [n-1][8]
    uint8_t* dp_split;      // [n-1][8]
    uint32_t* cw_collapse;  // [n-1] 1 = one leaf slot of a wide node
    int32_t* cw_task;       // [n] binary node of each wide node
    uint2* cw_level;        // [n + 16] first node and node count of each level
    uint32_t* counters;     // 4
    // clustering (ploc_build.inc); the boxes share memory with what is written after it
    int32_t* p_cid[2];
    float4 *p_lo[2], *p_hi[2];
    int32_t *p_partner, *p_left, *p_right, *p_parent, *p_lparent;
    uint32_t *p_cnt, *p_pre, *p_off, *p_loff, *p_tile, *p_state;
};

// Adds a centroid of every thread with ok to the bounds cb: over the warp, the
// block, then six atomics a block (per warp they took most of tri_boxes_kernel:
// 48.8 -> 21 us for 327,714 triangles).
__device__ __forceinline__ void add_centroid(bool ok, float3 c, uint32_t* cb) {
    __shared__ uint32_t s_cb[6];
    if (threadIdx.x < 6) s_cb[threadIdx.x] = threadIdx.x < 3 ? 0xFFFFFFFFu : 0u;
    __syncthreads();
    const float v[3] = {c.x, c.y, c.z};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const bool in = ok && v[a] == v[a];  // a NaN does not count
        const uint32_t mn = __reduce_min_sync(0xFFFFFFFFu, f2o(in ? v[a] : FLT_MAX));
        const uint32_t mx = __reduce_max_sync(0xFFFFFFFFu, f2o(in ? v[a] : -FLT_MAX));
        if ((threadIdx.x & 31) == 0) {
            atomicMin(&s_cb[a], mn);
            atomicMax(&s_cb[3 + a], mx);
        }
    }
    __syncthreads();
    if (threadIdx.x < 3) atomicMin(cb + threadIdx.x, s_cb[threadIdx.x]);
    else if (threadIdx.x < 6) atomicMax(cb + threadIdx.x, s_cb[threadIdx.x]);
}

// Item i's triangle (world space when `inst` is given and the item's
// instance is a flattened transformed one), its box and TriRec.
__global__ void tri_boxes_kernel(const gbrt_vertex* V, const uint32_t* I, const gbrt_priminfo* P, const uint4* items,
                                 uint32_t n, float4* lo, float4* hi, TriRec* unsorted, uint32_t* cb,
                                 const DevInstance* inst) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    float3 c = f3(0.0f);
    bool ok = i < n;
    if (ok) {
        const uint4 it = items[i];
        const gbrt_priminfo pi = P[it.y];
        const uint32_t io = pi.i_offset + 3u * it.z;
        const float* a = V[pi.v_offset + I[io]].pos;
        const float* b = V[pi.v_offset + I[io + 1]].pos;
        const float* d = V[pi.v_offset + I[io + 2]].pos;
        float3 p0 = f3(a[0], a[1], a[2]), p1 = f3(b[0], b[1], b[2]), p2 = f3(d[0], d[1], d[2]);
        if (inst && !inst[it.x].identity) {
            const float* xf = inst[it.x].xf;
            p0 = xform34_rn(xf, p0, 1.0f);
            p1 = xform34_rn(xf, p1, 1.0f);
            p2 = xform34_rn(xf, p2, 1.0f);
        }
        const float3 l = fmin3(fmin3(p0, p1), p2), h = fmax3(fmax3(p0, p1), p2);
        lo[i] = f4(l, 0.0f);
        hi[i] = f4(h, 0.0f);
        TriRec r;
        r.a = f4(p0, __uint_as_float(it.x));
        r.b = f4(p1, __uint_as_float(it.z));
        r.c = f4(p2, __uint_as_float(it.y | (it.w ? 0x80000000u : 0u)));
        unsorted[i] = r;
        c = (l + h) * 0.5f;
    }
    add_centroid(ok, c, cb);
}

__global__ void box_centroid_bounds_kernel(const float4* lo, const float4* hi, uint32_t n, uint32_t* cb) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool ok = i < n;
    add_centroid(ok, ok ? (f3(lo[i]) + f3(hi[i])) * 0.5f : f3(0.0f), cb);
}

__global__ void morton_kernel(const float4* lo, const float4* hi, uint32_t n, const uint32_t* cb, uint32_t* codes,
                              uint32_t* idx) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float3 mn = f3(o2f(cb[0]), o2f(cb[1]), o2f(cb[2]));
    const float3 mx = f3(o2f(cb[3]), o2f(cb[4]), o2f(cb[5]));
    const float3 ext = mx - mn;
    const float3 c = (f3(lo[i]) + f3(hi[i])) * 0.5f;
    auto q = [](float v, float m, float e) {
        float t = e > 0.0f ? (v - m) / e : 0.5f;
        return (uint32_t)fminf(fmaxf(t * 1024.0f, 0.0f), 1023.0f);
    };
    const uint32_t x = q(c.x, mn.x, ext.x), y = q(c.y, mn.y, ext.y), z = q(c.z, mn.z, ext.z);
    codes[i] = (expand_bits(x) << 2) | (expand_bits(y) << 1) | expand_bits(z);
    idx[i] = i;
}

__device__ __forceinline__ int delta(const uint32_t* k, int n, int i, int j) {
    if (j < 0 || j >= n) return -1;
    const uint32_t a = k[i], b = k[j];
    if (a == b) return 32 + __clz((uint32_t)i ^ (uint32_t)j);
    return __clz(a ^ b);
}

// Karras 2012, Figure 4: one thread per inner node.
__global__ void karras_kernel(const uint32_t* k, int n, int32_t* left, int32_t* right, int32_t* parent_i,
                              int32_t* parent_l, uint32_t* rlo, uint32_t* rhi) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n - 1) return;
    const int d = (delta(k, n, i, i + 1) - delta(k, n, i, i - 1)) >= 0 ? 1 : -1;
    const int dmin = delta(k, n, i, i - d);
    int lmax = 2;
    while (delta(k, n, i, i + lmax * d) > dmin) lmax <<= 1;
    int l = 0;
    for (int t = lmax >> 1; t >= 1; t >>= 1)
        if (delta(k, n, i, i + (l + t) * d) > dmin) l += t;
    const int j = i + l * d;
    const int dnode = delta(k, n, i, j);
    int s = 0;
    int t = l;
    do {
        t = (t + 1) >> 1;
        if (delta(k, n, i, i + (s + t) * d) > dnode) s += t;
    } while (t > 1);
    const int gamma = i + s * d + min(d, 0);
    const int lo = min(i, j), hi = max(i, j);
    int32_t lc, rc;
    if (lo == gamma) { lc = ~gamma; parent_l[gamma] = i; } else { lc = gamma; parent_i[gamma] = i; }
    if (hi == gamma + 1) { rc = ~(gamma + 1); parent_l[gamma + 1] = i; } else { rc = gamma + 1; parent_i[gamma + 1] = i; }
    left[i] = lc;
    right[i] = rc;
    rlo[i] = (uint32_t)lo;
    rhi[i] = (uint32_t)hi;
    if (i == 0) parent_i[0] = -1;
}

__device__ __forceinline__ float half_area(float3 l, float3 h) {
    const float3 e = fmax3(h - l, f3(0.0f));
    return e.x * e.y + e.y * e.z + e.z * e.x;
}

// Wide collapse: costs of a wide node and of a triangle in a leaf slot, per
// unit of area, and the most triangles a slot holds (cwbvh_build.inc).
constexpr uint32_t kCwMaxLeaf = 3;
#ifndef GBRT_CW_COST_NODE
#define GBRT_CW_COST_NODE 1.0f
#endif
#ifndef GBRT_CW_COST_TRI
#define GBRT_CW_COST_TRI 0.3f
#endif
constexpr float kCwCostNode = GBRT_CW_COST_NODE, kCwCostTri = GBRT_CW_COST_TRI;

// Bottom-up: one thread per leaf climbs while it is the second child to
// arrive at a node.  Child data is read with L1-bypassing loads.  Per inner
// node: its box, its SAH cost and whether it becomes a leaf of the binary
// tree; with kWide also the optimal distribution of the wide collapse
// (cwbvh_build.inc), in the same climb: a climb is bound by its chain of
// atomics and loads over the tree's depth, so a second one would cost as much
// again.
//
// The distribution: dp_cost[p][j-1] = least cost of p's subtree with at most
// j slots; dp_split[p][j-1] = 0 when that is the cost with j - 1 slots, else
// the slots k of the left child (the right one gets j - k); dp_split[p][0] =
// the left child's slots when p is a wide node (a distribution over `width`
// slots).  cw_collapse[p] = 1 when p is best a single leaf slot.
template <bool kWide>
__global__ void bottom_up_kernel(int n, const uint32_t* idx, const float4* lo, const float4* hi,
                                 const int32_t* left, const int32_t* right, const int32_t* parent_i,
                                 const int32_t* parent_l, const uint32_t* rlo, const uint32_t* rhi, float4* ilo,
                                 float4* ihi, float* cost, uint32_t* collapse, uint32_t* arrive, float* dp_cost,
                                 uint8_t* dp_split, uint32_t* cw_collapse, int width) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int p = parent_l[i];
    while (p >= 0) {
        __threadfence();
        if (atomicAdd(&arrive[p], 1u) == 0u) return;  // the sibling will finish p
        __threadfence();
        float3 bl[2], bh[2];
        float c[2];
        float4 d[2][2];  // the children's costs with 1..8 slots
        const int32_t ch[2] = {__ldcg(&left[p]), __ldcg(&right[p])};
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            if (ch[k] < 0) {
                const uint32_t item = __ldcg(&idx[~ch[k]]);
                bl[k] = f3(__ldcg(&lo[item]));
                bh[k] = f3(__ldcg(&hi[item]));
                const float a = half_area(bl[k], bh[k]);
                c[k] = kCostTri * a;
                const float w = kCwCostTri * a;  // one triangle: a leaf slot whatever the budget
                d[k][0] = d[k][1] = f4(w, w, w, w);
            } else {
                bl[k] = f3(__ldcg(&ilo[ch[k]]));
                bh[k] = f3(__ldcg(&ihi[ch[k]]));
                c[k] = __ldcg(&cost[ch[k]]);
                if constexpr (kWide) {
                    const float4* q = reinterpret_cast<const float4*>(dp_cost + (size_t)ch[k] * 8);
                    d[k][0] = __ldcg(q);
                    d[k][1] = __ldcg(q + 1);
                }
            }
        }
        const float3 l = fmin3(bl[0], bl[1]), h = fmax3(bh[0], bh[1]);
        const float a = half_area(l, h);
        const uint32_t count = rhi[p] - rlo[p] + 1u;
        const float split = kCostTraverse * a + c[0] + c[1];
        const float as_leaf = kCostTri * a * (float)count;
        const bool col = count <= kMaxLeaf && as_leaf <= split;
        ilo[p] = f4(l, 0.0f);
        ihi[p] = f4(h, 0.0f);
        cost[p] = col ? as_leaf : split;
        collapse[p] = col ? 1u : 0u;
        if constexpr (kWide) {
            const float cc[2][8] = {{d[0][0].x, d[0][0].y, d[0][0].z, d[0][0].w, d[0][1].x, d[0][1].y, d[0][1].z, d[0][1].w},
                                    {d[1][0].x, d[1][0].y, d[1][0].z, d[1][0].w, d[1][1].x, d[1][1].y, d[1][1].z, d[1][1].w}};
            float dist[8], out[8];
            uint32_t kbest[8], best[8];
            dist[0] = FLT_MAX;
            kbest[0] = 0;
            float all = FLT_MAX;  // over `width` slots
            uint32_t kall = 0;
#pragma unroll
            for (int j = 2; j <= 8; ++j) {  // j slots shared by the two children
                float b = FLT_MAX;
                uint32_t bk = 1;
#pragma unroll
                for (int k = 1; k < j; ++k) {
                    const float v = cc[0][k - 1] + cc[1][j - k - 1];
                    if (v < b) {
                        b = v;
                        bk = k;
                    }
                }
                dist[j - 1] = b;
                kbest[j - 1] = bk;
                if (j == width) {
                    all = b;
                    kall = bk;
                }
            }
            const float leaf_cost = count <= kCwMaxLeaf ? kCwCostTri * a * (float)count : FLT_MAX;
            const float node_cost = kCwCostNode * a + all;
            const bool leaf = count <= kCwMaxLeaf && leaf_cost <= node_cost;  // an area can be infinite
            float v = leaf ? leaf_cost : node_cost;
            out[0] = v;
            best[0] = kall;
#pragma unroll
            for (int j = 2; j <= 8; ++j) {
                const bool better = j <= width && dist[j - 1] < v;
                if (better) v = dist[j - 1];
                out[j - 1] = v;
                best[j - 1] = better ? kbest[j - 1] : 0u;
            }
            float4* q = reinterpret_cast<float4*>(dp_cost + (size_t)p * 8);
            q[0] = f4(out[0], out[1], out[2], out[3]);
            q[1] = f4(out[4], out[5], out[6], out[7]);
            *reinterpret_cast<uint2*>(dp_split + (size_t)p * 8) =
                make_uint2(best[0] | best[1] << 8 | best[2] << 16 | best[3] << 24,
                           best[4] | best[5] << 8 | best[6] << 16 | best[7] << 24);
            cw_collapse[p] = leaf ? 1u : 0u;
        }
        p = parent_i[p];
    }
}

// Writes the traversal nodes.  Inner node p of the radix tree becomes pool
// node node_base + p; a child that is a radix-tree leaf or a collapsed inner
// node becomes a leaf code over its contiguous sorted range.
__global__ void emit_nodes_kernel(int n, const uint32_t* idx, const float4* lo, const float4* hi,
                                  const int32_t* left, const int32_t* right, const uint32_t* rlo,
                                  const uint32_t* rhi, const float4* ilo, const float4* ihi,
                                  const uint32_t* collapse, const int32_t* parent_i, BNode2* nodes,
                                  uint32_t node_base, uint32_t tri_base) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n - 1) return;
    // inside a leaf's range (an ancestor or p itself collapsed): no node of the tree
    bool inside = false;
    for (int q = p; q >= 0 && rhi[q] - rlo[q] < kMaxLeaf && !inside; q = parent_i[q]) inside = collapse[q] != 0;
    if (inside) {
        nodes[node_base + p].c = make_int4(0, 0, -2, 0);
        return;
    }
    float3 bl[2], bh[2];
    int code[2];
    const int32_t ch[2] = {left[p], right[p]};
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        if (ch[k] < 0) {
            const uint32_t item = idx[~ch[k]];
            bl[k] = f3(lo[item]);
            bh[k] = f3(hi[item]);
            code[k] = leaf_code(tri_base + (uint32_t)~ch[k], 1u);
        } else {
            bl[k] = f3(ilo[ch[k]]);
            bh[k] = f3(ihi[ch[k]]);
            code[k] = collapse[ch[k]] ? leaf_code(tri_base + rlo[ch[k]], rhi[ch[k]] - rlo[ch[k]] + 1u)
                                      : (int)(node_base + ch[k]);
        }
    }
    BNode2 o;
    o.lxy = f4(bl[0].x, bh[0].x, bl[0].y, bh[0].y);
    o.rxy = f4(bl[1].x, bh[1].x, bl[1].y, bh[1].y);
    o.lrz = f4(bl[0].z, bh[0].z, bl[1].z, bh[1].z);
    const int32_t up = parent_i[p];
    o.c = make_int4(code[0], code[1], up < 0 ? -1 : (int)((node_base + up) * 2u + (right[up] == p ? 1u : 0u)), 0);
    nodes[node_base + p] = o;
}

// Threads to a block of the kernels that climb the tree: a block stays until
// its longest climb ends (refit of 1.95 million triangles with 32, 64, 128 and
// 256: 657, 642, 653 and 670 us; builds differ by 1%).
constexpr uint32_t kClimb = 64;

// Boxes of a built tree over triangle records that have moved.  A thread per
// node: the one of a node with leaf children makes their boxes and, if no inner
// child is missing, climbs; at each parent the last of its boxes goes on.  Bound
// by the climb's chain of atomics and loads, as the build's bottom-up pass, but
// without that one's costs, and it replaces the whole rebuild of the tree
// (Morton codes, sort, tree, bottom-up pass, emission: 625 -> 310 us, records
// included, at 1.95 million triangles).
__global__ void refit_nodes_kernel(int n, BNode2* nodes, const TriRec* tris) {
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n - 1) return;
    int4 c = nodes[p].c;
    if (c.z == -2 || (c.x >= 0 && c.y >= 0)) return;
    float3 bl[2], bh[2];
    bool own[2];
    const int code[2] = {c.x, c.y};
    int arrived = 0;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        own[k] = code[k] < 0;
        if (!own[k]) continue;
        ++arrived;
        const TriRec* t = tris + leaf_first(code[k]);
        bl[k] = f3(FLT_MAX);
        bh[k] = f3(-FLT_MAX);
        for (uint32_t i = 0; i < leaf_count(code[k]); ++i) {
            const float3 v0 = f3(t[i].a), v1 = f3(t[i].b), v2 = f3(t[i].c);
            bl[k] = fmin3(bl[k], fmin3(fmin3(v0, v1), v2));
            bh[k] = fmax3(bh[k], fmax3(fmax3(v0, v1), v2));
        }
    }
    for (;;) {
        BNode2* o = nodes + p;
        float2* z = reinterpret_cast<float2*>(&o->lrz);
        if (own[0]) {
            __stcg(&o->lxy, f4(bl[0].x, bh[0].x, bl[0].y, bh[0].y));
            __stcg(z, make_float2(bl[0].z, bh[0].z));
        }
        if (own[1]) {
            __stcg(&o->rxy, f4(bl[1].x, bh[1].x, bl[1].y, bh[1].y));
            __stcg(z + 1, make_float2(bl[1].z, bh[1].z));
        }
        if (!(own[0] && own[1])) {
            __threadfence();
            if (atomicAdd(&o->c.w, arrived) + arrived < 2) return;  // the other box's thread goes on
            __threadfence();
            o->c.w = 0;  // for the next refit
            const float4 xy = __ldcg(own[0] ? &o->rxy : &o->lxy);
            const float2 oz = __ldcg(own[0] ? z + 1 : z);
            const float3 l = f3(xy.x, xy.z, oz.x), h = f3(xy.y, xy.w, oz.y);
            const int m = own[0] ? 0 : 1;
            bl[0] = fmin3(bl[m], l);
            bh[0] = fmax3(bh[m], h);
        } else {
            bl[0] = fmin3(bl[0], bl[1]);
            bh[0] = fmax3(bh[0], bh[1]);
        }
        const int up = o->c.z;
        if (up < 0) return;
        p = up >> 1;
        const bool right = up & 1;
        own[0] = !right;
        own[1] = right;
        bl[1] = bl[0];
        bh[1] = bh[0];
        arrived = 1;
    }
}

__global__ void gather_tris_kernel(const uint32_t* idx, uint32_t n, const TriRec* unsorted, TriRec* tris,
                                   uint32_t tri_base) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) tris[tri_base + i] = unsorted[idx[i]];
}

__global__ void gather_inst_kernel(const uint32_t* idx, uint32_t n, const uint32_t* ids, TriRec* tris,
                                   uint32_t tri_base) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        TriRec r;
        r.a = f4(0.0f, 0.0f, 0.0f, __uint_as_float(ids[idx[i]]));
        r.b = f4(0.0f, 0.0f, 0.0f, 0.0f);
        r.c = f4(0.0f, 0.0f, 0.0f, 0.0f);
        tris[tri_base + i] = r;
    }
}

__global__ void init_bounds_kernel(uint32_t* cb) {
    if (threadIdx.x < 3) cb[threadIdx.x] = 0xFFFFFFFFu;
    else if (threadIdx.x < 6) cb[threadIdx.x] = 0u;
}

#define CK(x)                                   \
    do {                                        \
        cudaError_t e_ = (x);                   \
        if (e_ != cudaSuccess) return e_;       \
    } while (0)

inline uint32_t blocks(uint32_t n, uint32_t b = 256) { return (n + b - 1) / b; }

// Lays the scratch of one build over n items out in the context's arena, which the build holds.
cudaError_t scratch_carve(Scratch& s, uint32_t n, BuildArena& arena, cudaStream_t st) {
    std::memset(&s, 0, sizeof(s));
    const size_t m = n > 1 ? n - 1 : 1;
    CK(cub::DeviceRadixSort::SortPairs(nullptr, s.cub_bytes, s.morton_in, s.morton, s.idx_in, s.idx, (int)n, 0, 30,
                                       st));
    for (int pass = 0; pass < 2; ++pass) {  // measure, then place
        char* p = static_cast<char*>(arena.p);
        size_t used = 0;
        auto take = [&](auto*& ptr, size_t count) {
            if (pass) ptr = reinterpret_cast<std::remove_reference_t<decltype(ptr)>>(p + used);
            used += (count * sizeof(*ptr) + 255) & ~size_t(255);
        };
        take(s.lo, n);
        take(s.hi, n);
        take(s.morton_in, n);
        take(s.morton, n);
        take(s.idx_in, n);
        take(s.idx, n);
        take(s.left, m);
        take(s.right, m);
        take(s.parent_i, m);
        take(s.parent_l, n);
        take(s.range_lo, m);
        take(s.range_hi, m);
        take(s.cost, m);
        take(s.collapse, m);
        take(s.arrive, m);
        take(s.cbounds, 8);
        take(s.unsorted, n);
        char* tmp = nullptr;
        take(tmp, s.cub_bytes ? s.cub_bytes : 16);
        s.cub_tmp = tmp;
        take(s.dp_split, m * 8);
        take(s.cw_collapse, m);
        take(s.cw_task, n);
        take(s.cw_level, (size_t)n + 16);
        take(s.counters, 4);
        for (int k = 0; k < 2; ++k) take(s.p_cid[k], n);
        take(s.p_partner, n);
        take(s.p_left, m);
        take(s.p_right, m);
        take(s.p_parent, m);
        take(s.p_lparent, n);
        take(s.p_cnt, m);
        take(s.p_pre, m);
        take(s.p_off, m);
        take(s.p_loff, n);
        take(s.p_tile, n / 256 + 1);
        take(s.p_state, 8);
        // clusters' boxes; after the clustering inner boxes and the collapse's costs
        for (int k = 0; k < 2; ++k) {
            take(s.p_lo[k], n);
            take(s.p_hi[k], n);
        }
        s.ilo = s.p_lo[0];
        s.ihi = s.p_hi[0];
        s.dp_cost = reinterpret_cast<float*>(s.p_lo[1]);
        if (!pass) CK(arena.reserve(used));
    }
    return cudaSuccess;
}

}  // namespace

#include "ploc_build.inc"

namespace {

// Morton codes, sort, binary tree (PLOC clustering, or the Karras radix tree
// when quality is kBvhFast) and the bottom-up pass (boxes, SAH costs, leaf
// collapse; for width > 0 also the wide collapse's distribution).  Item boxes
// in s.lo/hi and centroid bounds in s.cbounds must be ready.
cudaError_t binary_tree(Scratch& s, uint32_t n, cudaStream_t st, int quality, int width) {
    morton_kernel<<<blocks(n), 256, 0, st>>>(s.lo, s.hi, n, s.cbounds, s.morton_in, s.idx_in);
    CK(cudaGetLastError());
    CK(cub::DeviceRadixSort::SortPairs(s.cub_tmp, s.cub_bytes, s.morton_in, s.morton, s.idx_in, s.idx, (int)n, 0,
                                       30, st));
    if (n > 1) {
        cudaError_t pe = quality == kBvhPloc ? ploc_tree(s, n, st) : cudaErrorNotReady;
        if (pe != cudaSuccess && pe != cudaErrorNotReady) return pe;
        if (pe == cudaErrorNotReady) {  // radix tree (asked for, or clustering did not converge)
            karras_kernel<<<blocks(n - 1), 256, 0, st>>>(s.morton, (int)n, s.left, s.right, s.parent_i, s.parent_l,
                                                        s.range_lo, s.range_hi);
            CK(cudaGetLastError());
        }
        CK(cudaMemsetAsync(s.arrive, 0, (n - 1) * sizeof(uint32_t), st));
        if (width)
            bottom_up_kernel<true><<<blocks(n, kClimb), kClimb, 0, st>>>((int)n, s.idx, s.lo, s.hi, s.left, s.right, s.parent_i,
                                                              s.parent_l, s.range_lo, s.range_hi, s.ilo, s.ihi, s.cost,
                                                              s.collapse, s.arrive, s.dp_cost, s.dp_split,
                                                              s.cw_collapse, width);
        else
            bottom_up_kernel<false><<<blocks(n, kClimb), kClimb, 0, st>>>((int)n, s.idx, s.lo, s.hi, s.left, s.right, s.parent_i,
                                                               s.parent_l, s.range_lo, s.range_hi, s.ilo, s.ihi,
                                                               s.cost, s.collapse, s.arrive, nullptr, nullptr,
                                                               nullptr, 0);
        CK(cudaGetLastError());
    }
    return cudaSuccess;
}

// Common tail: binary tree with leaves of up to kMaxLeaf items, emit BNode2.
cudaError_t build_common(Scratch& s, uint32_t n, BNode2* nodes, uint32_t node_base, uint32_t tri_base,
                         BvhResult* res, cudaStream_t st, int quality, int width = 0) {
    CK(binary_tree(s, n, st, quality, width));
    if (n > 1) {
        emit_nodes_kernel<<<blocks(n - 1), 256, 0, st>>>((int)n, s.idx, s.lo, s.hi, s.left, s.right, s.range_lo,
                                                        s.range_hi, s.ilo, s.ihi, s.collapse, s.parent_i, nodes,
                                                        node_base, tri_base);
        CK(cudaGetLastError());
    }
    // root: inner node 0 (or a leaf if it collapsed / n == 1)
    float4 rl, rh;
    uint32_t col = 0;
    if (n > 1) {
        CK(cudaMemcpyAsync(&rl, s.ilo, sizeof(float4), cudaMemcpyDeviceToHost, st));
        CK(cudaMemcpyAsync(&rh, s.ihi, sizeof(float4), cudaMemcpyDeviceToHost, st));
        CK(cudaMemcpyAsync(&col, s.collapse, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
    } else {
        CK(cudaMemcpyAsync(&rl, s.lo, sizeof(float4), cudaMemcpyDeviceToHost, st));
        CK(cudaMemcpyAsync(&rh, s.hi, sizeof(float4), cudaMemcpyDeviceToHost, st));
    }
    CK(cudaStreamSynchronize(st));
    res->lo = rl;
    res->hi = rh;
    if (n == 1) res->root = leaf_code(tri_base, 1u);
    else if (col) res->root = leaf_code(tri_base, n);
    else res->root = (int32_t)node_base;
    return cudaSuccess;
}

}  // namespace

#include "cwbvh_build.inc"

namespace {
// Writes 16 bytes an item (22 us for 1.95 million items); a list made on the
// host and copied cost 6.9 ms more of a build of that many.
__global__ void expand_spans_kernel(const uint4* spans, uint32_t nspans, uint32_t n, uint4* items) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t lo = 0, hi = nspans;  // the last span that starts at or before i
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (spans[mid].x <= i) lo = mid;
        else hi = mid;
    }
    const uint4 s = spans[lo];
    items[i] = make_uint4(s.y, s.z, i - s.x, s.w);
}
}  // namespace

cudaError_t expand_spans(const uint4* spans, uint32_t nspans, uint32_t n, uint4* items, cudaStream_t st) {
    expand_spans_kernel<<<blocks(n), 256, 0, st>>>(spans, nspans, n, items);
    return cudaGetLastError();
}

cudaError_t build_triangle_bvh(BuildArena& arena, const gbrt_vertex* vertices, const uint32_t* indices,
                               const gbrt_priminfo* prims, const uint4* items, uint32_t n, BNode2* nodes,
                               uint32_t node_base, TriRec* tris, uint32_t tri_base, BvhResult* res, cudaStream_t st,
                               const DevInstance* inst, int quality, const WideBuild* wide) {
    if (n == 0 || (wide && (wide->width < 2 || wide->width > 8))) return cudaErrorInvalidValue;
    std::lock_guard<std::mutex> hold(arena.mu);
    Scratch s;
    CK(scratch_carve(s, n, arena, st));
    init_bounds_kernel<<<1, 32, 0, st>>>(s.cbounds);
    tri_boxes_kernel<<<blocks(n), 256, 0, st>>>(vertices, indices, prims, items, n, s.lo, s.hi, s.unsorted, s.cbounds,
                                                inst);
    CK(cudaGetLastError());
    CK(build_common(s, n, nodes, node_base, tri_base, res, st, quality, wide ? wide->width : 0));
    gather_tris_kernel<<<blocks(n), 256, 0, st>>>(s.idx, n, s.unsorted, tris, tri_base);
    CK(cudaGetLastError());
    return wide ? emit_wide(s, n, *wide, *res, st) : cudaSuccess;
}

cudaError_t refit_triangle_bvh(const gbrt_vertex* vertices, const uint32_t* indices, const gbrt_priminfo* prims,
                               BNode2* nodes, TriRec* tris, uint32_t n, cudaStream_t st, const DevInstance* inst) {
    if (n < 2) return cudaErrorInvalidValue;
    cw_refit_tris_kernel<<<blocks(n), 256, 0, st>>>(vertices, indices, prims, tris, n, inst);
    refit_nodes_kernel<<<blocks(n - 1, kClimb), kClimb, 0, st>>>((int)n, nodes, tris);
    return cudaGetLastError();
}

cudaError_t read_root(const BNode2* nodes, BvhResult* res, cudaStream_t st) {
    BNode2 root;
    CK(cudaMemcpyAsync(&root, nodes, sizeof(root), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    const float4 a = root.lxy, b = root.rxy, z = root.lrz;
    res->lo = make_float4(std::min(a.x, b.x), std::min(a.z, b.z), std::min(z.x, z.z), 0.0f);
    res->hi = make_float4(std::max(a.y, b.y), std::max(a.w, b.w), std::max(z.y, z.w), 0.0f);
    res->root = 0;
    return cudaSuccess;
}

cudaError_t build_instance_bvh(BuildArena& arena, const float4* lo, const float4* hi, const uint32_t* ids, uint32_t n,
                               BNode2* nodes, uint32_t node_base, TriRec* tris, uint32_t tri_base, BvhResult* res,
                               cudaStream_t st, int quality) {
    if (n == 0) return cudaErrorInvalidValue;
    std::lock_guard<std::mutex> hold(arena.mu);
    Scratch s;
    CK(scratch_carve(s, n, arena, st));
    CK(cudaMemcpyAsync(s.lo, lo, n * sizeof(float4), cudaMemcpyDeviceToDevice, st));
    CK(cudaMemcpyAsync(s.hi, hi, n * sizeof(float4), cudaMemcpyDeviceToDevice, st));
    init_bounds_kernel<<<1, 32, 0, st>>>(s.cbounds);
    box_centroid_bounds_kernel<<<blocks(n), 256, 0, st>>>(s.lo, s.hi, n, s.cbounds);
    CK(cudaGetLastError());
    CK(build_common(s, n, nodes, node_base, tri_base, res, st, quality));
    gather_inst_kernel<<<blocks(n), 256, 0, st>>>(s.idx, n, ids, tris, tri_base);
    return cudaGetLastError();
}

size_t bvh_sort_temp_bytes(uint32_t n) {
    size_t bytes = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, bytes, (const uint32_t*)nullptr, (uint32_t*)nullptr,
                                    (const uint32_t*)nullptr, (uint32_t*)nullptr, (int)n, 0, 30);
    return bytes;
}

namespace {
inline size_t al256(size_t x) { return (x + 255) & ~size_t(255); }
}  // namespace

size_t bvh_scratch_bytes(uint32_t cap) {
    const size_t n = cap, m = cap > 1 ? cap - 1 : 1;
    return 4 * al256(n * sizeof(float4)) + 4 * al256(n * sizeof(uint32_t)) + 2 * al256(m * sizeof(uint32_t)) +
           2 * al256(m * sizeof(uint32_t)) + al256(32) + 4 * al256(n * sizeof(int32_t)) +
           al256(m * sizeof(float)) + al256(n * sizeof(TriRec)) + al256(bvh_sort_temp_bytes(cap));
}

BuildScratch bvh_scratch_carve(void* base, uint32_t cap) {
    const size_t n = cap, m = cap > 1 ? cap - 1 : 1;
    char* p = static_cast<char*>(base);
    auto take = [&](size_t bytes) {
        void* r = p;
        p += al256(bytes);
        return r;
    };
    BuildScratch s;
    s.capacity = cap;
    s.lo = (float4*)take(n * sizeof(float4));
    s.hi = (float4*)take(n * sizeof(float4));
    s.ilo = (float4*)take(n * sizeof(float4));
    s.ihi = (float4*)take(n * sizeof(float4));
    s.morton_in = (uint32_t*)take(n * sizeof(uint32_t));
    s.morton = (uint32_t*)take(n * sizeof(uint32_t));
    s.idx_in = (uint32_t*)take(n * sizeof(uint32_t));
    s.idx = (uint32_t*)take(n * sizeof(uint32_t));
    s.range_lo = (uint32_t*)take(m * sizeof(uint32_t));
    s.range_hi = (uint32_t*)take(m * sizeof(uint32_t));
    s.collapse = (uint32_t*)take(m * sizeof(uint32_t));
    s.arrive = (uint32_t*)take(m * sizeof(uint32_t));
    s.cbounds = (uint32_t*)take(32);
    s.left = (int32_t*)take(n * sizeof(int32_t));
    s.right = (int32_t*)take(n * sizeof(int32_t));
    s.parent_i = (int32_t*)take(n * sizeof(int32_t));
    s.parent_l = (int32_t*)take(n * sizeof(int32_t));
    s.cost = (float*)take(m * sizeof(float));
    s.unsorted = (TriRec*)take(n * sizeof(TriRec));
    s.sort_tmp_bytes = bvh_sort_temp_bytes(cap);
    s.sort_tmp = take(s.sort_tmp_bytes);
    return s;
}

cudaError_t build_triangle_bvh_scratch(const BuildScratch& bs, const gbrt_vertex* vertices, const uint32_t* indices,
                                       const gbrt_priminfo* prims, const uint4* items, uint32_t n, BNode2* nodes,
                                       uint32_t node_base, TriRec* tris, uint32_t tri_base, BvhResult* res,
                                       cudaStream_t st) {
    if (n == 0 || n > bs.capacity) return cudaErrorInvalidValue;
    Scratch s;
    std::memset(&s, 0, sizeof(s));
    s.lo = bs.lo;
    s.hi = bs.hi;
    s.morton_in = bs.morton_in;
    s.morton = bs.morton;
    s.idx_in = bs.idx_in;
    s.idx = bs.idx;
    s.left = bs.left;
    s.right = bs.right;
    s.parent_i = bs.parent_i;
    s.parent_l = bs.parent_l;
    s.range_lo = bs.range_lo;
    s.range_hi = bs.range_hi;
    s.ilo = bs.ilo;
    s.ihi = bs.ihi;
    s.cost = bs.cost;
    s.collapse = bs.collapse;
    s.arrive = bs.arrive;
    s.cbounds = bs.cbounds;
    s.cub_tmp = bs.sort_tmp;
    s.cub_bytes = bvh_sort_temp_bytes(n);  // the sort of n items needs no more than the capacity's size
    if (s.cub_bytes > bs.sort_tmp_bytes) return cudaErrorInvalidValue;
    init_bounds_kernel<<<1, 32, 0, st>>>(s.cbounds);
    tri_boxes_kernel<<<blocks(n), 256, 0, st>>>(vertices, indices, prims, items, n, s.lo, s.hi, bs.unsorted,
                                                s.cbounds, nullptr);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = build_common(s, n, nodes, node_base, tri_base, res, st, kBvhFast);  // no allocation
    if (e == cudaSuccess) {
        gather_tris_kernel<<<blocks(n), 256, 0, st>>>(s.idx, n, bs.unsorted, tris, tri_base);
        e = cudaGetLastError();
    }
    return e;
}

// World box of a transformed instance: the 8 transformed corners of its BLAS
// root box, widened by a relative 1e-6 of the box size plus 1e-6 of the
// largest coordinate so float rounding of the transform cannot make it
// smaller than the exact image.
__global__ void inst_boxes_kernel(const DevInstance* inst, const uint32_t* ids, const float4* blo,
                                  const float4* bhi, uint32_t n, float4* lo, float4* hi) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const DevInstance& in = inst[ids[i]];
    const float4 l = blo[i], h = bhi[i];
    float3 mn = f3(FLT_MAX), mx = f3(-FLT_MAX);
    for (int c = 0; c < 8; ++c) {
        const float3 p = f3((c & 1) ? h.x : l.x, (c & 2) ? h.y : l.y, (c & 4) ? h.z : l.z);
        const float3 q = f3(in.xf[0] * p.x + in.xf[1] * p.y + in.xf[2] * p.z + in.xf[3],
                            in.xf[4] * p.x + in.xf[5] * p.y + in.xf[6] * p.z + in.xf[7],
                            in.xf[8] * p.x + in.xf[9] * p.y + in.xf[10] * p.z + in.xf[11]);
        mn = fmin3(mn, q);
        mx = fmax3(mx, q);
    }
    const float3 ext = mx - mn;
    const float m = fmaxf(fmaxf(fmaxf(fabsf(mn.x), fabsf(mn.y)), fmaxf(fabsf(mn.z), fabsf(mx.x))),
                          fmaxf(fabsf(mx.y), fabsf(mx.z)));
    const float pad = 1e-6f * (fmaxf(fmaxf(ext.x, ext.y), ext.z) + m) + 1e-30f;
    lo[i] = f4(mn - pad, 0.0f);
    hi[i] = f4(mx + pad, 0.0f);
}

cudaError_t instance_world_boxes(const DevInstance* inst, const uint32_t* ids, const float4* blas_lo,
                                 const float4* blas_hi, uint32_t n, float4* lo, float4* hi, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    inst_boxes_kernel<<<blocks(n), 256, 0, st>>>(inst, ids, blas_lo, blas_hi, n, lo, hi);
    return cudaGetLastError();
}

}  // namespace gbrt
