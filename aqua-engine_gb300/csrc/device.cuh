// device.cuh — the scene as the device sees it, and the traversal routine
// shared by every kernel that casts rays (render wavefront, aqua_trace,
// batched rendering).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "aq_math.h"
#include "bvh.h"
#include "walk_nodes.h"

namespace aq {

struct DevMaterial {
    float4 a;  // base colour rgb (linear), texture index (int bits, -1 none)
    float4 b;  // metallic, roughness, specular, 0
};
struct DevLight {
    float4 p0;  // xyz, type (int bits)
    float4 e1;  // xyz, area
    float4 e2;  // xyz, selection pmf
    float4 le;  // radiance (quad, triangle) or intensity (point), cdf
};
struct DevTexture {
    uint32_t offset;  // first texel in the texel pool
    int32_t w, h;
    int32_t pad;
};
struct DevCamera {
    float pos[3], right[3], up[3], back[3];
    float tan_half, aspect, lens_radius, focal;
    int32_t width, height;
};
struct DevScene {
    const float4* __restrict__ nodes;  // 8 words per four-wide node, or 4 per quantized node (bvh.h)
    const float4* __restrict__ wnodes; // 4 words per walk node (load_walk); null for small trees and with qbvh
    const float4* __restrict__ tris;   // 3 words per triangle, leaf order
    const float2* __restrict__ uvs;    // 3 per triangle, leaf order
    const DevMaterial* __restrict__ mats;
    const DevLight* __restrict__ lights;
    const DevTexture* __restrict__ texs;
    const uint32_t* __restrict__ texels;  // RGBA8, sRGB
    const float4* __restrict__ nrm;    // 3 vertex normals per triangle (xyz, 0), leaf order; null = flat
    // 2 words per material: (specular_tint, sheen, sheen_tint, clearcoat),
    // (clearcoat_roughness, transmission, ior, 0); null when no material
    // sets any of those lobes (the base-model kernels run then).
    const float4* __restrict__ mext;
    int32_t n_nodes, n_tris, n_mats, n_lights, n_texs;
    int32_t qbvh;  // 1: `nodes` holds quantized 64-byte nodes
    float env[3];
    DevCamera cam;
};

// Result of a traversal: leaf-order triangle index (or -1), its scene index,
// distance and barycentrics.
struct TraceResult {
    float t, u, v;
    int32_t tri;
    int32_t id;
};

// Node formats a walk is compiled for, chosen on the host (walk_format).
// kNodesOwn: full-precision or quantized, whichever the scene holds (a
// warp-uniform branch).
enum { kNodesFull = 0, kNodesQuantized = 1, kNodesWalk = 2, kNodesOwn = 3 };

#if defined(__CUDACC__)

template <class T>
__device__ __forceinline__ T ldg_(const T* p) { return __ldg(p); }

// Programmatic dependent launch: wait until the kernel this one was chained
// to (launched with programmatic stream serialization) has completed and
// its writes are visible. Returns at once for a kernel launched normally.
__device__ __forceinline__ void grid_dep_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
// Lets the kernel chained after this one be scheduled once every block of
// this grid has passed this point (its blocks then take SM slots as this
// grid's blocks exit, and wait in grid_dep_wait). No effect without a
// chained kernel.
__device__ __forceinline__ void grid_dep_launch() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }

// Two consecutive 16-byte words in one 256-bit load through the read-only
// (non-coherent) path (sm_100 and later); p must be 32-byte aligned. Only
// for data that nothing writes during the render (scene nodes): kernels
// chained by programmatic dependent launch may begin before their
// predecessor has finished, and the non-coherent path is outside what
// griddepcontrol.wait makes visible, so they read what earlier kernels of
// the chain wrote through coherent loads (plain or __ldcg).
__device__ __forceinline__ void ldg2x4(const float4* p, float4& a, float4& b) {
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
        : "l"(p));
}

constexpr int kStackSize = kBvhStackSize;  // the builder checks its trees fit
constexpr int32_t kTraversalDone = (int32_t)0x80000000;

// One compare-exchange of the child-ordering network: (ta, ca) gets the
// nearer entry, ties keep their order.
__device__ __forceinline__ void order2(float& ta, int32_t& ca, float& tb, int32_t& cb) {
    const bool sw = tb < ta;
    const float t = sw ? tb : ta;
    const int32_t c = sw ? cb : ca;
    tb = sw ? ta : tb;
    cb = sw ? ca : cb;
    ta = t;
    ca = c;
}

// Entry distances (INFINITY = missed) and links of a node's four children.
struct Children {
    float t0, t1, t2, t3;
    int32_t c0, c1, c2, c3;
};

// Full-precision node (128-byte aligned): the four child boxes through
// slab_entry. It comes in three 256-bit loads and one 128-bit load (the
// counts word is not read): scattered lanes cost the L1 one request per
// load instruction, so fewer, wider loads relieve it.
__device__ __forceinline__ Children load_wide(const DevScene& S, int32_t node, const RayPre& rp, float tfar) {
    const float4* np = S.nodes + 8 * (size_t)node;
    float4 lx, hx, ly, hy, lz, hz;
    ldg2x4(np, lx, hx);
    ldg2x4(np + 2, ly, hy);
    ldg2x4(np + 4, lz, hz);
    const int4 ch = ldg_(reinterpret_cast<const int4*>(np + 6));
    Children c;
    c.t0 = slab_entry(lx.x, hx.x, ly.x, hy.x, lz.x, hz.x, rp, tfar);
    c.t1 = slab_entry(lx.y, hx.y, ly.y, hy.y, lz.y, hz.y, rp, tfar);
    c.t2 = slab_entry(lx.z, hx.z, ly.z, hy.z, lz.z, hz.z, rp, tfar);
    c.t3 = slab_entry(lx.w, hx.w, ly.w, hy.w, lz.w, hz.w, rp, tfar);
    c.c0 = ch.x, c.c1 = ch.y, c.c2 = ch.z, c.c3 = ch.w;
    return c;
}

// Plane of child byte k of a quantized word: fmaf(q, scale, origin), the
// byte turned into a float exactly by placing it under the exponent of 2^23
// (one byte permute and one subtraction).
__device__ __forceinline__ float qplane(uint32_t word, int k, float scale, float origin) {
    // result bytes: word byte k, zero, zero, 0x4B  ->  2^23 + q
    const float q = __uint_as_float(__byte_perm(word, 0x4B000000u, 0x7540u | (uint32_t)k)) - 8388608.0f;
    return fmaf(q, scale, origin);
}

// Quantized 64-byte node (two 256-bit loads): the child planes are decoded
// (bvh.h) and tested with the same slab_entry; empty slots (link ~0) are
// skipped.
__device__ __forceinline__ Children load_quantized(const DevScene& S, int32_t node, const RayPre& rp, float tfar) {
    const float4* np = S.nodes + 4 * (size_t)node;
    float4 w0, w1, w2, w3;
    ldg2x4(np, w0, w1);
    ldg2x4(np + 2, w2, w3);
    const uint32_t ex = __float_as_uint(w0.w);
    const float sx = __uint_as_float((ex & 0xffu) << 23), sy = __uint_as_float(((ex >> 8) & 0xffu) << 23),
                sz = __uint_as_float(((ex >> 16) & 0xffu) << 23);
    const uint32_t lx = __float_as_uint(w2.x), hx = __float_as_uint(w2.y), ly = __float_as_uint(w2.z),
                   hy = __float_as_uint(w2.w), lz = __float_as_uint(w3.x), hz = __float_as_uint(w3.y);
    Children c;
    c.c0 = __float_as_int(w1.x), c.c1 = __float_as_int(w1.y), c.c2 = __float_as_int(w1.z),
    c.c3 = __float_as_int(w1.w);
    float t[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
        t[k] = slab_entry(qplane(lx, k, sx, w0.x), qplane(hx, k, sx, w0.x), qplane(ly, k, sy, w0.y),
                          qplane(hy, k, sy, w0.y), qplane(lz, k, sz, w0.z), qplane(hz, k, sz, w0.z), rp, tfar);
    c.t0 = c.c0 == ~0 ? INFINITY : t[0], c.t1 = c.c1 == ~0 ? INFINITY : t[1];
    c.t2 = c.c2 == ~0 ? INFINITY : t[2], c.t3 = c.c3 == ~0 ? INFINITY : t[3];
    return c;
}

// Walk node (64 bytes, two 256-bit loads; walk_nodes.h).
__device__ __forceinline__ Children load_walk(const DevScene& S, int32_t node, const RayPre& rp, float tfar) {
    const float4* np = S.wnodes + 4 * (size_t)node;
    float4 w0, w1, w2, w3;
    ldg2x4(np, w0, w1);
    ldg2x4(np + 2, w2, w3);
    const WalkBoxes w{w0.x, w0.y, w0.z, w0.w, w3.z, w3.w, __float_as_uint(w2.x), __float_as_uint(w2.y),
                      __float_as_uint(w2.z), __float_as_uint(w2.w), __float_as_uint(w3.x), __float_as_uint(w3.y)};
    float t[4];
    walk_entries(w, rp, tfar, t);
    Children c;
    c.t0 = t[0], c.t1 = t[1], c.t2 = t[2], c.t3 = t[3];
    c.c0 = __float_as_int(w1.x), c.c1 = __float_as_int(w1.y), c.c2 = __float_as_int(w1.z), c.c3 = __float_as_int(w1.w);
    return c;
}

template <int NODES>
__device__ __forceinline__ Children load_children(const DevScene& S, int32_t node, const RayPre& rp, float tfar) {
    if constexpr (NODES == kNodesFull) return load_wide(S, node, rp, tfar);
    if constexpr (NODES == kNodesQuantized) return load_quantized(S, node, rp, tfar);
    if constexpr (NODES == kNodesWalk) return load_walk(S, node, rp, tfar);
    return S.qbvh ? load_quantized(S, node, rp, tfar) : load_wide(S, node, rp, tfar);
}

// Orders the hit children with a five-comparator sorting network, pushes all
// but the nearest, farthest first, and returns the nearest. With no box hit
// it returns the top of the stack, or kTraversalDone when the stack is empty.
__device__ __forceinline__ int32_t push_ordered(Children c, int32_t* stack, int& sp) {
    order2(c.t0, c.c0, c.t1, c.c1);
    order2(c.t2, c.c2, c.t3, c.c3);
    order2(c.t0, c.c0, c.t2, c.c2);
    order2(c.t1, c.c1, c.t3, c.c3);
    order2(c.t1, c.c1, c.t2, c.c2);
    if (c.t3 != INFINITY) stack[sp++] = c.c3;
    if (c.t2 != INFINITY) stack[sp++] = c.c2;
    if (c.t1 != INFINITY) stack[sp++] = c.c1;
    if (c.t0 != INFINITY) return c.c0;
    return sp > 0 ? stack[--sp] : kTraversalDone;
}

// Turns the hit children's entry distances into keys that sort the one
// entered last to the front (misses stay behind).
__device__ __forceinline__ void farthest_first(Children& c) {
    c.t0 = c.t0 == INFINITY ? INFINITY : -c.t0;
    c.t1 = c.t1 == INFINITY ? INFINITY : -c.t1;
    c.t2 = c.t2 == INFINITY ? INFINITY : -c.t2;
    c.t3 = c.t3 == INFINITY ? INFINITY : -c.t3;
}

// Order for occlusion: descend into the child entered last, push the other
// hit children as three of the comparators leave them. The answer does not
// depend on the order, and near the origin a ray mostly passes by what it
// left; the far children hold its occluder sooner (visits per ray, random
// segments: interior 11.4 nearest first, 8.5 farthest first; sphere field
// 10.0 and 3.7; rays to the lights 17.9 and 18.1, 16.7 and 15.5).
__device__ __forceinline__ int32_t push_occlusion(Children c, int32_t* stack, int& sp) {
    farthest_first(c);
    order2(c.t0, c.c0, c.t1, c.c1);
    order2(c.t2, c.c2, c.t3, c.c3);
    order2(c.t0, c.c0, c.t2, c.c2);
    if (c.t3 != INFINITY) stack[sp++] = c.c3;
    if (c.t2 != INFINITY) stack[sp++] = c.c2;
    if (c.t1 != INFINITY) stack[sp++] = c.c1;
    if (c.t0 != INFINITY) return c.c0;
    return sp > 0 ? stack[--sp] : kTraversalDone;
}

// Visits node `node` in the scene's own format, nearest child first (the
// canonical walk, whose work is counted).
__device__ __forceinline__ int32_t visit_node(const DevScene& S, int32_t node, const RayPre& rp, float tfar,
                                              int32_t* stack, int& sp) {
    return push_ordered(S.qbvh ? load_quantized(S, node, rp, tfar) : load_wide(S, node, rp, tfar), stack, sp);
}

// Whether the result of a walk over S.wnodes is the full-precision walk's.
// That walk tests a triangle only when its leaf's box, and with it every
// ancestor's, passes slab_entry; the wider boxes of the walk nodes also let
// through hits that the rounding of the triangle test puts just outside
// (about one ray in 10^7, at corners with flat axis-aligned surfaces). The
// nearest (or any) hit of the wider set is the full walk's when it belongs to
// the smaller one, which the triangle's own box, part of its leaf's, proves
// for practically every hit; a ray whose hit fails it is walked again
// through the full-precision nodes.
__device__ __forceinline__ bool walk_confirmed(const DevScene& S, const RayPre& rp, const TraceResult& r) {
    if (r.tri < 0) return true;
    const float4* tp = S.tris + 3 * (size_t)r.tri;
    const float4 a = ldg_(tp), b = ldg_(tp + 1), c = ldg_(tp + 2);
    return slab_entry(fminf(fminf(a.x, b.x), c.x), fmaxf(fmaxf(a.x, b.x), c.x), fminf(fminf(a.y, b.y), c.y),
                      fmaxf(fmaxf(a.y, b.y), c.y), fminf(fminf(a.z, b.z), c.z), fmaxf(fmaxf(a.z, b.z), c.z), rp,
                      rp.tmax) != INFINITY;
}

// The walk of one ray through the full-precision nodes (`stack` is free).
__device__ __forceinline__ void walk_full(const DevScene& S, const RayPre& rp, const RayShear& sh, bool any,
                                          int32_t* stack, TraceResult& r) {
    r.t = rp.tmax; r.u = 0.0f; r.v = 0.0f; r.tri = -1; r.id = 0x7fffffff;
    int sp = 0;
    int32_t node = 0;
    while (true) {
#pragma unroll 1
        while (node >= 0) node = push_ordered(load_wide(S, node, rp, r.t), stack, sp);
        if (node == kTraversalDone) return;
        const int32_t code = ~node, first = code >> 3, cnt = code & 7;
#pragma unroll 1
        for (int k = 0; k < cnt; ++k) {
            const float4* tp = S.tris + 3 * (size_t)(first + k);
            const float4 a = ldg_(tp), b = ldg_(tp + 1), c = ldg_(tp + 2);
            const TriHit h = intersect_tri(sh, mk(a.x, a.y, a.z), mk(b.x, b.y, b.z), mk(c.x, c.y, c.z), rp.tmin,
                                           rp.tmax);
            const int32_t id = __float_as_int(a.w);
            if (!h.hit || !(h.t < r.t || (h.t == r.t && id < r.id))) continue;
            r.t = h.t; r.u = h.u; r.v = h.v; r.tri = first + k; r.id = id;
            if (any) return;
        }
        if (sp == 0) return;
        node = stack[--sp];
    }
}

// Stack-based traversal of the four-wide BVH (nearest child first, the other
// hit children pushed farthest first). ANY: stop at the first hit in (tmin,
// tmax). Otherwise the result is the lexicographic minimum (t, scene index)
// over all triangles hit: boxes are tested conservatively (slab_entry), a
// child is skipped only when its entry distance exceeds the best t, so the
// answer does not depend on visit order.
// COUNT: add inner-node visits and triangle tests to the counters.
template <bool ANY, bool COUNT>
__device__ __forceinline__ TraceResult traverse(const DevScene& S, v3 o, v3 d, float tmin, float tmax,
                                                uint32_t& n_nodes, uint32_t& n_tris) {
    RayPre rp;
    rp.o = o;
    rp.invd = mk(safe_inv(d.x), safe_inv(d.y), safe_inv(d.z));
    rp.tmin = tmin;
    rp.tmax = tmax;
    RayShear sh = make_shear(o, d);
    TraceResult r;
    r.t = tmax; r.u = 0.0f; r.v = 0.0f; r.tri = -1; r.id = 0x7fffffff;
    int32_t stack[kStackSize];
    int sp = 0;
    int32_t node = 0;
    while (true) {
        while (node >= 0) {
            if (COUNT) ++n_nodes;
            node = visit_node(S, node, rp, r.t, stack, sp);
        }
        if (node == kTraversalDone) return r;
        // Leaf.
        int32_t code = ~node;
        int32_t first = code >> 3, cnt = code & 7;
        for (int k = 0; k < cnt; ++k) {
            const float4* tp = S.tris + 3 * (size_t)(first + k);
            float4 a = ldg_(tp), b = ldg_(tp + 1), c = ldg_(tp + 2);
            if (COUNT) ++n_tris;
            TriHit h = intersect_tri(sh, mk(a.x, a.y, a.z), mk(b.x, b.y, b.z), mk(c.x, c.y, c.z), tmin, tmax);
            if (h.hit) {
                int32_t id = __float_as_int(a.w);
                if (ANY) {
                    r.t = h.t; r.tri = first + k; r.id = id;
                    return r;
                }
                if (h.t < r.t || (h.t == r.t && id < r.id)) {
                    r.t = h.t; r.u = h.u; r.v = h.v; r.tri = first + k; r.id = id;
                }
            }
        }
        if (sp == 0) return r;
        node = stack[--sp];
    }
}

// Persistent traversal of a queue of n rays with ray replacement (Aila &
// Laine 2009, sec. 4: "replacing terminated rays"): each lane holds its own
// ray; once at least kRefillLanes lanes of the warp have finished theirs (or
// all have), the idle lanes take the next rays from *cursor together (one
// atomic per warp). Between refills every lane runs rounds with postponed
// leaves (same paper): a lane that reaches a leaf parks it and keeps walking
// inner nodes until the warp vote says the walking lanes hold one, then all
// test triangles together. Boxes, culling and triangle tests are those of
// traverse(), so the result (the minimum (t, scene index) over all triangles
// hit, or any hit) is identical; only the order of visits differs.
//   load(i, o, d, tmin, tmax) -> uint32_t tag: fetches ray i of the queue;
//   done(tag, r): called once per ray, by the lanes finishing in the same
//                 round together (warp collectives inside are allowed).
constexpr int kRefillLanes = 16;
// Over walk nodes, a round leaves the inner nodes once fewer than this many
// of the lanes still walking hold no leaf; waiting for the last of them left
// 17 of 32 lanes active per visit on the interior and 15 on its occlusion
// rays, 6 leaves 22 and 21. (4, 8 and 12 were slower there; over the
// full-precision nodes of small trees, where rays are short, waiting for the
// last lane stays the faster by 0.5%.)
constexpr int kWalkLanes = 6;
// Resident 128-thread blocks per SM the traversal kernels are compiled for:
// 9 keep them within 56 registers. Against 8 (64 registers) and 10 (48): Cornell
// GGX 1024^2 at 64 spp 37.8 / 38.6 / 38.9 ms, interior 1080p at 8 spp 40.3 /
// 41.2 / 42.1 ms, 2.07M interior rays 475 / 486 / 512 us.
constexpr int kTraceBlocks = 9;

// Kinds of queue: closest hits, any hits, or both mixed (the load callback
// then sets `any` per ray: load(i, o, d, tmin, tmax, any)).
enum { kQueueClosest = 0, kQueueAny = 1, kQueueMixed = 2 };

template <int KIND, int NODES, bool SPARSE, class Load, class Done>
__device__ __forceinline__ void traverse_lanes(const DevScene& S, uint32_t n, uint32_t width, uint32_t* cursor,
                                               Load load, Done done) {
    const unsigned kFull = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    RayPre rp;
    RayShear sh;
    TraceResult r;
    int32_t stack[kStackSize];
    int sp = 0;
    int32_t node = kTraversalDone, leaf = 0;
    uint32_t tag = 0;
    bool have = false, drained = false, any = KIND == kQueueAny;
    auto take = [&](uint32_t i) {
        v3 o, d;
        float tmin, tmax;
        if constexpr (KIND == kQueueMixed) tag = load(i, o, d, tmin, tmax, any);
        else tag = load(i, o, d, tmin, tmax);
        rp.o = o;
        rp.invd = mk(safe_inv(d.x), safe_inv(d.y), safe_inv(d.z));
        rp.tmin = tmin;
        rp.tmax = tmax;
        sh = make_shear(o, d);
        r.t = tmax; r.u = 0.0f; r.v = 0.0f; r.tri = -1; r.id = 0x7fffffff;
        sp = 0;
        node = 0;
        leaf = 0;
        have = true;
    };
    if constexpr (SPARSE) {
        // The warp's share, dealt without the counter: thousands of warps
        // asking one address take microseconds.
        const uint32_t i = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * width + (uint32_t)lane;
        if ((uint32_t)lane < width && i < n) take(i);
    }
    while (true) {
        if constexpr (!SPARSE) {
            const unsigned idle = __ballot_sync(kFull, !have);
            if (!drained && __popc(idle) >= kRefillLanes) {
                const int leader = __ffs(idle) - 1;
                uint32_t base = 0;
                if (lane == leader) base = atomicAdd(cursor, (uint32_t)__popc(idle));
                base = __shfl_sync(kFull, base, leader);
                if (base + (uint32_t)__popc(idle) >= n) drained = true;
                if (!have) {
                    const uint32_t i = base + (uint32_t)__popc(idle & ((1u << lane) - 1u));
                    if (i < n) take(i);
                }
            }
        }
        if (!__any_sync(kFull, have)) break;
        if (!have) continue;
        // One round.
        while (node >= 0) {
            Children c = load_children<NODES>(S, node, rp, r.t);
            if constexpr (KIND == kQueueAny && NODES == kNodesWalk) {
                node = push_occlusion(c, stack, sp);
            } else {
                if constexpr (KIND == kQueueMixed && NODES == kNodesWalk)
                    if (any) farthest_first(c);
                node = push_ordered(c, stack, sp);
            }
            if (node < 0 && node != kTraversalDone && leaf == 0) {
                leaf = node;
                node = sp > 0 ? stack[--sp] : kTraversalDone;
            }
            if constexpr (NODES == kNodesWalk && !SPARSE) {
                if (__popc(__ballot_sync(__activemask(), leaf == 0)) < kWalkLanes) break;
            } else {
                if (!__any_sync(__activemask(), leaf == 0)) break;
            }
        }
        while (leaf < 0) {
            int32_t code = ~leaf;
            int32_t first = code >> 3, cnt = code & 7;
            bool stop = false;
            for (int k = 0; k < cnt; ++k) {
                const float4* tp = S.tris + 3 * (size_t)(first + k);
                float4 a = ldg_(tp), b = ldg_(tp + 1), c = ldg_(tp + 2);
                TriHit h = intersect_tri(sh, mk(a.x, a.y, a.z), mk(b.x, b.y, b.z), mk(c.x, c.y, c.z), rp.tmin,
                                         rp.tmax);
                if (h.hit) {
                    int32_t id = __float_as_int(a.w);
                    if (KIND == kQueueAny || (KIND == kQueueMixed && any)) {
                        r.t = h.t; r.tri = first + k; r.id = id;
                        stop = true;
                        break;
                    }
                    if (h.t < r.t || (h.t == r.t && id < r.id)) {
                        r.t = h.t; r.u = h.u; r.v = h.v; r.tri = first + k; r.id = id;
                    }
                }
            }
            leaf = 0;
            if (stop) {
                node = kTraversalDone;
                break;
            }
            if (node < 0 && node != kTraversalDone) {
                leaf = node;
                node = sp > 0 ? stack[--sp] : kTraversalDone;
            }
        }
        if (node == kTraversalDone) {
            if (NODES == kNodesWalk && !walk_confirmed(S, rp, r)) walk_full(S, rp, sh, any, stack, r);
            done(tag, r);
            have = false;
        }
    }
}

// A queue shorter than the grid's lanes is spread over all its warps, few
// lanes each: a warp then takes as long as the longest of its few rays, not as
// the union of 32 divergent ones, and more warps hide each other's fetches (a
// cached 1080p frame, whose last ten iterations trace 10-40k rays: 3.39 -> 3.24
// ms; a 64 x 64 thumbnail 0.57 -> 0.41 ms). Two copies of the loop, because one
// with a variable width spills registers on full queues (Cornell GGX 1024^2
// 155.1 -> 157.4 ms).
template <int KIND, int NODES, class Load, class Done>
__device__ __forceinline__ void traverse_queue(const DevScene& S, uint32_t n, uint32_t* cursor, Load load,
                                               Done done) {
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    const uint32_t width = (n + warps - 1u) / warps;
    if (width < 32u) traverse_lanes<KIND, NODES, true>(S, n, width, cursor, load, done);
    else traverse_lanes<KIND, NODES, false>(S, n, 32u, cursor, load, done);
}

// Warp-aggregated append: lanes with pred set get consecutive slots of *ctr.
__device__ __forceinline__ uint32_t warp_append(uint32_t* ctr, bool pred) {
    unsigned mask = __ballot_sync(__activemask(), pred);
    if (!pred) return 0;
    int lane = threadIdx.x & 31;
    int leader = __ffs(mask) - 1;
    uint32_t base = 0;
    if (lane == leader) base = atomicAdd(ctr, (uint32_t)__popc(mask));
    base = __shfl_sync(mask, base, leader);
    return base + (uint32_t)__popc(mask & ((1u << lane) - 1u));
}

#endif  // __CUDACC__

}  // namespace aq
