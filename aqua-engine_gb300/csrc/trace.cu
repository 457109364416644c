// trace.cu — aqua_trace: closest-hit or any-hit queries for a caller's ray
// set. This is the traversal the parity tests compare, ray for ray, with the
// FP32 CPU traversal of the same flattened BVH.
#include <algorithm>
#include <cstring>

#include "internal.h"

namespace aq {

template <bool ANY>
__device__ __forceinline__ void store_hit(float4* hits, size_t i, const TraceResult& r) {
    float4 h;
    if (ANY) h = make_float4(0.0f, 0.0f, 0.0f, __int_as_float(r.tri >= 0 ? 1 : -1));
    else if (r.tri < 0) h = make_float4(0.0f, 0.0f, 0.0f, __int_as_float(-1));
    else h = make_float4(r.t, r.u, r.v, __int_as_float(r.id));
    hits[i] = h;
}

// The renderer's traversal over the caller's rays.
template <bool ANY, int NODES>
__global__ void __launch_bounds__(128, kTraceBlocks) k_trace_user(DevScene S, const float4* __restrict__ rays,
                                                                  uint32_t n, float4* __restrict__ hits,
                                                                  uint32_t* cursor) {
    traverse_queue<ANY ? kQueueAny : kQueueClosest, NODES>(
        S, n, cursor,
        [&](uint32_t i, v3& o, v3& d, float& tmin, float& tmax) -> uint32_t {
            float4 a = ldg_(rays + 2 * (size_t)i), b = ldg_(rays + 2 * (size_t)i + 1);
            o = mk(a.x, a.y, a.z);
            d = mk(b.x, b.y, b.z);
            tmin = a.w;
            tmax = b.w;
            return i;
        },
        [&](uint32_t i, const TraceResult& r) { store_hit<ANY>(hits, i, r); });
}

// The canonical walk, counted: stats[0] += node visits, stats[1] += triangle tests.
template <bool ANY>
__global__ void __launch_bounds__(128) k_trace_count(DevScene S, const float4* __restrict__ rays, size_t n,
                                                     float4* __restrict__ hits, unsigned long long* stats) {
    uint32_t nodes = 0, tris = 0;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        float4 a = ldg_(rays + 2 * i), b = ldg_(rays + 2 * i + 1);
        store_hit<ANY>(hits, i, traverse<ANY, true>(S, mk(a.x, a.y, a.z), mk(b.x, b.y, b.z), a.w, b.w, nodes, tris));
    }
    for (int o = 16; o > 0; o >>= 1) {
        nodes += __shfl_down_sync(0xffffffffu, nodes, o);
        tris += __shfl_down_sync(0xffffffffu, tris, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&stats[0], (unsigned long long)nodes);
        atomicAdd(&stats[1], (unsigned long long)tris);
    }
}

// One thread per node: the walk node of full-precision node k (walk_nodes.h).
__global__ void k_walk_nodes(const float4* __restrict__ nodes, int32_t n, float4* __restrict__ out) {
    const int32_t k = (int32_t)(blockIdx.x * blockDim.x + threadIdx.x);
    if (k >= n) return;
    const float* w = reinterpret_cast<const float*>(nodes + 8 * (size_t)k);
    const int32_t* link = reinterpret_cast<const int32_t*>(w + 24);
    float org[3], step[3];
    uint32_t lo_bytes[3], hi_bytes[3];
    for (int a = 0; a < 3; ++a) walk_axis(w + 8 * a, w + 8 * a + 4, link, org[a], step[a], lo_bytes[a], hi_bytes[a]);
    float4* o = out + 4 * (size_t)k;
    o[0] = make_float4(org[0], org[1], org[2], step[0]);
    o[1] = nodes[8 * (size_t)k + 6];
    o[2] = make_float4(__uint_as_float(lo_bytes[0]), __uint_as_float(hi_bytes[0]), __uint_as_float(lo_bytes[1]),
                       __uint_as_float(hi_bytes[1]));
    o[3] = make_float4(__uint_as_float(lo_bytes[2]), __uint_as_float(hi_bytes[2]), step[1], step[2]);
}

void build_walk_nodes(aqua_ctx* ctx, const DevScene& S, float4* out) {
    k_walk_nodes<<<(S.n_nodes + 127) / 128, 128, 0, ctx->stream>>>(S.nodes, S.n_nodes, out);
    AQ_CUDA(cudaGetLastError());
}

void trace_rays(aqua_ctx* ctx, aqua_scene* sc, const aqua_ray* rays, size_t n, aqua_hit* out, uint32_t flags,
                aqua_trace_counts* counts) {
    static_assert(sizeof(aqua_ray) == 32, "aqua_ray must be 32 bytes");
    static_assert(sizeof(aqua_hit) == 16, "aqua_hit must be 16 bytes");
    cudaStream_t st = ctx->stream;
    bool dev = (flags & AQUA_TRACE_DEVICE_PTRS) != 0;
    bool any = (flags & AQUA_TRACE_ANY_HIT) != 0;
    bool count = (flags & AQUA_TRACE_COUNT) != 0;
    if (counts) memset(counts, 0, sizeof(*counts));
    if (n == 0) return;
    const float4* d_rays;
    float4* d_hits;
    if (dev) {
        if (((uintptr_t)rays & 15) || ((uintptr_t)out & 15))
            throw Error(AQUA_ERR_INVALID_ARG, "device ray and hit arrays must be 16-byte aligned");
        d_rays = (const float4*)rays;
        d_hits = (float4*)out;
    } else {
        if (ctx->trace_rays.bytes < 32 * n) { dev_free(ctx->trace_rays); dev_alloc(ctx, ctx->trace_rays, 32 * n); }
        if (ctx->trace_hits.bytes < 16 * n) { dev_free(ctx->trace_hits); dev_alloc(ctx, ctx->trace_hits, 16 * n); }
        AQ_CUDA(cudaMemcpyAsync(ctx->trace_rays.ptr, rays, 32 * n, cudaMemcpyHostToDevice, st));
        d_rays = (const float4*)ctx->trace_rays.ptr;
        d_hits = (float4*)ctx->trace_hits.ptr;
    }
    if (!ctx->trace_stats.ptr) dev_alloc(ctx, ctx->trace_stats, 64);
    unsigned long long* d_stats = (unsigned long long*)ctx->trace_stats.ptr;
    AQ_CUDA(cudaMemsetAsync(d_stats, 0, 24, st));  // node and triangle counters, queue cursor
    using Walk = void (*)(DevScene, const float4*, uint32_t, float4*, uint32_t*);
    static constexpr Walk walks[2][3] = {  // by any, walk_format
        {k_trace_user<false, kNodesFull>, k_trace_user<false, kNodesQuantized>, k_trace_user<false, kNodesWalk>},
        {k_trace_user<true, kNodesFull>, k_trace_user<true, kNodesQuantized>, k_trace_user<true, kNodesWalk>}};
    const Walk walk = walks[any][walk_format(sc->ds)];
    const auto counted = any ? k_trace_count<true> : k_trace_count<false>;
    const int per_sm = count ? resident_blocks(ctx, counted, 128) : resident_blocks(ctx, walk, 128);
    // A short queue is dealt to all warps (traverse_queue): down to one ray each.
    const size_t need = count ? (n + 127) / 128 : (n + 3) / 4;
    int grid = (int)std::min<size_t>(need, (size_t)ctx->num_sms * (size_t)per_sm);
    EventPair* ev = counts ? &timer(ctx) : nullptr;
    if (ev) AQ_CUDA(cudaEventRecord(ev->e[0], st));
    if (count) {
        counted<<<grid, 128, 0, st>>>(sc->ds, d_rays, n, d_hits, d_stats);
        AQ_CUDA(cudaGetLastError());
    }
    constexpr size_t kChunk = (size_t)1 << 30;  // rays per launch: the queue counts in 32 bits
    for (size_t i = 0; !count && i < n; i += kChunk) {
        if (i > 0) AQ_CUDA(cudaMemsetAsync(d_stats + 2, 0, 8, st));
        walk<<<grid, 128, 0, st>>>(sc->ds, d_rays + 2 * i, (uint32_t)std::min(kChunk, n - i), d_hits + i,
                                   reinterpret_cast<uint32_t*>(d_stats + 2));
        AQ_CUDA(cudaGetLastError());
    }
    if (ev) AQ_CUDA(cudaEventRecord(ev->e[1], st));
    if (!dev) AQ_CUDA(cudaMemcpyAsync(out, d_hits, 16 * n, cudaMemcpyDeviceToHost, st));
    const bool read = counts && count;
    if (read) AQ_CUDA(cudaMemcpyAsync(ctx->pinned_stats, d_stats, 16, cudaMemcpyDeviceToHost, st));
    AQ_CUDA(cudaStreamSynchronize(st));
    if (counts) {
        counts->node_visits = read ? ctx->pinned_stats[0] : 0;
        counts->tri_tests = read ? ctx->pinned_stats[1] : 0;
        counts->kernel_ms = ev->ms();
    }
}

}  // namespace aq
