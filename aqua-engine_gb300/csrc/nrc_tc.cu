// nrc_tc.cu — radiance-cache inference on the 5th-generation tensor cores:
// tcgen05.mma with the accumulator in tensor memory (TMEM), inputs brought in
// by TMA.
//
// One persistent CTA per SM holds the network's bf16 weights (42 KB) in shared
// memory once and runs kTcFwdGroups independent warpgroups. A warpgroup owns
// 96 TMEM columns (64 for the FP32 accumulator, 32 for the next layer's bf16
// activations; five groups fill 480 of the SM's 512) and a 128-row input
// tile in shared memory, and works through its tiles alone:
//   - its first thread loads the next input tile with TMA (eight 128 x 8-column
//     boxes) as soon as layer 1 has read the current one;
//   - per layer one of its warps, a different one in each group so that the
//     four schedulers share the work, issues four tcgen05.mma.kind::f16 (M =
//     128, N = 64, or 16 for the output layer, K = 16 each; BF16 x BF16 ->
//     FP32) and commits them to the group's mbarrier. Layer 1 reads A from
//     shared memory, layers 2-6 read it from TMEM;
//   - each warp reads its 32 TMEM lanes (rows) of the accumulator with
//     tcgen05.ld, applies ReLU, rounds to bf16 pairs and stores them back to
//     the activation columns with tcgen05.st.
// Activations never leave TMEM, and while one group is in its epilogue the
// tensor core serves the others. Bound: the chain MMA -> epilogue -> MMA of six
// layers, about 1000 cycles each with five tiles in flight. 16.8M rows: 774 us
// when a single lane issued (110 cycles per MMA), 563 us issued by the
// converged first warps, 536 us (31.3 G rows/s, 0.67 of the copy rate) spread
// over the schedulers; 2.0M rows 107 -> 79 us.
//
// Shared-memory operands use the K-major layout without swizzle, with the
// 8-row x 16-byte core matrices of one 8-column K slice stored back to back:
// element (r, k) of an R-row tile sits at (k / 8) * R * 16 + r * 16 + (k % 8) * 2.
// So the leading byte offset (next core matrix along K) is R * 16 and the
// stride byte offset (next 8 rows) is 128, and a TMA box of 8 columns x 128
// rows lands as one contiguous K slice.
//
// Every mbarrier wait is bounded. A group whose wait expires agrees on it
// with a barrier reduction, records an error flag, waits (bounded) for what
// it still has in flight and leaves; TMEM is freed on every path.
#include <algorithm>
#include <mutex>

#include <cuda.h>
#include <cuda_bf16.h>
#include <cudaTypedefs.h>

#include "internal.h"
#include "nrc.h"

namespace aq {

constexpr int kTcRows = 128;                      // rows per tile (MMA M)
constexpr int kTcTileBytes = kTcRows * 64 * 2;    // 16 KB per input or activation tile
constexpr int kTcLayerBytes = kNrcTcLayerBytes;  // 8 KB hidden-layer weights
constexpr int kTcOutRows = kNrcTcOutRows;        // output layer padded to N = 16 (3 used)
constexpr int kTcOutBytes = kTcOutRows * 64 * 2;  // 2 KB
constexpr int kTcWeightBytes = 5 * kTcLayerBytes + kTcOutBytes;  // 42 KB
constexpr uint32_t kTcTmemCols = 512;              // a power of two >= 32
constexpr uint32_t kTcWaitLimit = 1u << 22;       // try_wait rounds before a wait gives up
// Inference: five groups (tiles in flight; four measured 9% slower),
// accumulators at columns 64 g, activations after all accumulators at
// 64 * 5 + 32 g. The weights and five input tiles take 123 KB of shared
// memory, which keeps two CTAs (and two full TMEM allocations) off one SM.
constexpr int kTcFwdGroups = 5;
constexpr int kTcFwdThreads = 128 * kTcFwdGroups;
constexpr int kTcFwdSmemBytes = std::max(kTcWeightBytes + kTcFwdGroups * kTcTileBytes + 1024, 120 * 1024);
constexpr uint32_t kTcFwdActBase = 64u * kTcFwdGroups;
static_assert(kTcFwdActBase + 32u * kTcFwdGroups <= kTcTmemCols, "inference TMEM columns");
static_assert(kTcFwdSmemBytes <= 227 * 1024, "shared memory per CTA");
static_assert((kTcTmemCols & (kTcTmemCols - 1)) == 0 && kTcTmemCols >= 32 && kTcTmemCols <= 512, "TMEM alloc");
static_assert(kTcWeightBytes % 1024 == 0 && kTcTileBytes % 1024 == 0, "tiles stay 1024-byte aligned");

// Byte offset of element (r, k) in an R-row operand tile.
__host__ __device__ constexpr uint32_t tc_offset(int rows, int r, int k) { return nrc_tc_offset(rows, r, k); }

// Both weight images from the FP32 weights w (training) and the inference
// weights inf (nrc_tc_param_offsets; the caller zeroes the padding first).
__global__ void k_nrc_pack_tc(const float* __restrict__ w, const float* __restrict__ inf, uint8_t* __restrict__ img_w,
                              uint8_t* __restrict__ img_inf) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;  // one parameter
    if (p >= kNrcParams) return;
    uint32_t fwd;
    int32_t bwd;
    nrc_tc_param_offsets(p, fwd, bwd);
    *reinterpret_cast<__nv_bfloat16*>(img_w + fwd) = __float2bfloat16_rn(w[p]);
    *reinterpret_cast<__nv_bfloat16*>(img_inf + fwd) = __float2bfloat16_rn(inf[p]);
}

// ---------------------------------------------------------------- PTX wrappers
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Instruction descriptor, kind::f16: D = F32 (bits 4-5), A = B = BF16 (bits
// 7-9, 10-12), both K-major, N >> 3 at bit 17, M >> 4 at bit 24.
__host__ __device__ constexpr uint32_t tc_idesc(int m, int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// Descriptors from a shared address >> 4 (no swizzle). K-major: `lbo` bytes
// between groups of 8 along K, 128 between groups of 8 rows of the result.
// MN-major: 128 between groups of 8 along K, `sbo` between groups of 8 rows.
__device__ __forceinline__ uint64_t desc_k(uint32_t a, uint32_t lbo) {
    return (uint64_t)(a | ((lbo >> 4) << 16)) | ((uint64_t)((128u >> 4) | (1u << 14)) << 32);
}
__device__ __forceinline__ uint64_t desc_mn(uint32_t a, uint32_t sbo) {
    return (uint64_t)(a | ((128u >> 4) << 16)) | ((uint64_t)((sbo >> 4) | (1u << 14)) << 32);
}

// True in one lane of the (converged) warp.
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "elect.sync _|p, 0xffffffff;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(p));
    return p != 0;
}

// tc_mma by the elected lane of a warp that runs converged.
__device__ __forceinline__ void tc_issue(bool lead, uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p, q;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "setp.ne.b32 q, %5, 0;\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
        "}\n" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"((uint32_t)lead));
}
// Same with A (128 rows x 16 bf16, two per 32-bit column) read from TMEM.
__device__ __forceinline__ void tc_issue_ts(bool lead, uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc,
                                            uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p, q;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "setp.ne.b32 q, %5, 0;\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
        "}\n" ::"r"(tmem_d),
        "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"((uint32_t)lead));
}

__device__ __forceinline__ void tc_commit(uint32_t mbar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(mbar)
                 : "memory");
}

// Bounded wait on an mbarrier phase; false when the limit expired.
__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t parity) {
    for (uint32_t it = 0; it < kTcWaitLimit; ++it) {
        uint32_t done;
        asm volatile(
            "{\n"
            ".reg .pred p;\n"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
            "selp.u32 %0, 1, 0, p;\n"
            "}\n"
            : "=r"(done)
            : "r"(mbar), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

// Barrier over one warpgroup (named barrier `id`, 128 threads) that also
// returns whether any of its threads passed `pred`.
__device__ __forceinline__ bool group_any(int id, bool pred) {
    uint32_t r;
    asm volatile(
        "{\n"
        ".reg .pred p, q;\n"
        "setp.ne.u32 p, %1, 0;\n"
        "bar.red.or.pred q, %2, 128, p;\n"
        "selp.u32 %0, 1, 0, q;\n"
        "}\n"
        : "=r"(r)
        : "r"((uint32_t)pred), "r"(id)
        : "memory");
    return r != 0;
}

// Barrier over one warpgroup (named barrier `id`, 128 threads).
__device__ __forceinline__ void group_sync(int id) { asm volatile("bar.sync %0, 128;\n" ::"r"(id) : "memory"); }

// One input tile: eight boxes of 8 columns x 128 rows, 16 KB on one mbarrier.
__device__ __forceinline__ void tma_load_tile(const CUtensorMap* map, uint32_t dst, uint32_t mbar, int row0) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(mbar), "r"((uint32_t)kTcTileBytes)
                 : "memory");
#pragma unroll
    for (int kc = 0; kc < 8; ++kc)
        asm volatile(
            "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n" ::"r"(
                dst + (uint32_t)(kc * kTcRows * 16)),
            "l"(reinterpret_cast<uint64_t>(map)), "r"(kc * 8), "r"(row0), "r"(mbar)
            : "memory");
}

#define AQ_TC_LD16(taddr, r)                                                                               \
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, " \
                 "[%16];\n"                                                                                \
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),     \
                   "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), \
                   "=r"(r[14]), "=r"(r[15])                                                                \
                 : "r"(taddr))

#define AQ_TC_ST16(taddr, r)                                                                               \
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "                                          \
                 "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n" ::"r"(taddr),              \
                 "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),    \
                 "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) \
                 : "memory")

__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }

// ReLU and round-to-nearest-even to a bf16 pair: `lo` (the even K index) in
// the low half, `hi` in the high half.
__device__ __forceinline__ uint32_t relu_pack2(uint32_t lo, uint32_t hi) {
    uint32_t d;
    asm("cvt.rn.relu.bf16x2.f32 %0, %1, %2;\n" : "=r"(d) : "f"(__uint_as_float(hi)), "f"(__uint_as_float(lo)));
    return d;
}

// ---------------------------------------------------------------- kernel
// X (through `xmap`): n rows x 64 bf16; out: n x 3 fp32; err: set to 1 when a
// wait expired.
__global__ void __launch_bounds__(kTcFwdThreads, 1)
    k_nrc_forward_tc(const __grid_constant__ CUtensorMap xmap, int n, const uint4* __restrict__ wimg,
                     float* __restrict__ out, uint32_t* __restrict__ err) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bar_in[kTcFwdGroups], bar_mma[kTcFwdGroups];
    __shared__ uint32_t tmem_base_slot;

    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // known to be uniform
    const int g = warp >> 2, q = warp & 3, gt = tid & 127;
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* sbase = smem_raw + (base - smem_u32(smem_raw));
    const uint32_t sI = base + kTcWeightBytes + (uint32_t)g * kTcTileBytes;  // this group's input tile

    grid_dep_wait();  // the weights and inputs come from the kernels before
    grid_dep_launch();
    for (int i = tid; i < kTcWeightBytes / 16; i += kTcFwdThreads) reinterpret_cast<uint4*>(sbase)[i] = __ldcg(wimg + i);
    if (tid < kTcFwdGroups) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&bar_in[tid])) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&bar_mma[tid])) : "memory");
    }
    if (tid == 0) {
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        asm volatile("prefetch.tensormap [%0];\n" ::"l"(reinterpret_cast<uint64_t>(&xmap)) : "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(
                         smem_u32(&tmem_base_slot)),
                     "r"(kTcTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();

    // All 512 columns were allocated, so they start at 0; with a constant the
    // MMAs' TMEM addresses stay in uniform registers.
    const uint32_t tmem = (uint32_t)g * 64u;                    // this group's accumulator
    const uint32_t tact = kTcFwdActBase + (uint32_t)g * 32u;   // and activations
    const uint32_t lanes = (uint32_t)(q * 32) << 16;                             // this warp's lanes
    const uint32_t mb_in = smem_u32(&bar_in[g]), mb_mma = smem_u32(&bar_mma[g]);
    const int bar_id = 1 + g;
    const int tiles = (n + kTcRows - 1) / kTcRows;
    const int stride = (int)gridDim.x * kTcFwdGroups;
    const int row = q * 32 + lane;  // TMEM lane = tile row
    uint32_t ph_in = 0, ph_mma = 0;      // parity of the next phase to wait for
    uint32_t tma_par = 0, mma_par = 0;   // parity the work in flight will complete
    bool fail = false, tma_pending = false, mma_pending = false;
    const bool lead = q == (g & 3) && elect_one();

    // Tiles interleave across CTAs first, so a small batch still spreads
    // over many SMs.
    int tile = (int)blockIdx.x + g * (int)gridDim.x;
    if (gt == 0 && tile < tiles) {
        tma_load_tile(&xmap, sI, mb_in, tile * kTcRows);
        tma_pending = true;
        tma_par = ph_in;
    }
    while (tile < tiles) {
        bool ok = true;
        if (gt == 0) {
            ok = mbar_wait(mb_in, ph_in);
            if (ok) tma_pending = false;
        }
        ph_in ^= 1u;
        if (group_any(bar_id, !ok)) { fail = true; break; }
        const int next = tile + stride;
#pragma unroll
        for (int l = 0; l < 6; ++l) {
            const bool last = l == 5;
            if (q == (g & 3)) {
                // One of the group's warps issues, converged and with uniform
                // operands (a single lane's code moves them to uniform
                // registers for every MMA): K = 64 as four K = 16 steps, two
                // core matrices of B each, and of A two core matrices (layer
                // 1) or eight TMEM columns.
                tc_fence_after();
                const uint32_t idesc = tc_idesc(kTcRows, last ? kTcOutRows : 64);
                const uint32_t blbo = (last ? kTcOutRows : 64) * 16;
                const uint32_t b0 = (base >> 4) + (uint32_t)l * (kTcLayerBytes / 16);
#pragma unroll
                for (uint32_t k = 0; k < 4; ++k) {
                    const uint64_t bd = desc_k(b0 + k * 2u * (blbo / 16), blbo);
                    if (l == 0) tc_issue(lead, tmem, desc_k((sI >> 4) + k * 256u, kTcRows * 16), bd, idesc, k > 0);
                    else tc_issue_ts(lead, tmem, tact + k * 8u, bd, idesc, k > 0);
                }
                if (lead) tc_commit(mb_mma);
                mma_pending = true;
                mma_par = ph_mma;
            }
            ok = mbar_wait(mb_mma, ph_mma);
            ph_mma ^= 1u;
            ok = __all_sync(0xffffffffu, ok);  // tcgen05.ld below is warp-collective
            if (ok) mma_pending = false;
            // The input tile is free once layer 1 has read it: fetch the next one.
            if (l == 0 && gt == 0 && ok && next < tiles) {
                tma_load_tile(&xmap, sI, mb_in, next * kTcRows);
                tma_pending = true;
                tma_par = ph_in;
            }
            tc_fence_after();
            if (ok) {
                if (!last) {
                    uint32_t r[64], a[32];
                    AQ_TC_LD16(tmem + lanes + 0u, (r + 0));
                    AQ_TC_LD16(tmem + lanes + 16u, (r + 16));
                    AQ_TC_LD16(tmem + lanes + 32u, (r + 32));
                    AQ_TC_LD16(tmem + lanes + 48u, (r + 48));
                    tc_wait_ld();
#pragma unroll
                    for (int c = 0; c < 32; ++c) a[c] = relu_pack2(r[2 * c], r[2 * c + 1]);
                    AQ_TC_ST16(tact + lanes + 0u, (a + 0));
                    AQ_TC_ST16(tact + lanes + 16u, (a + 16));
                    tc_wait_st();
                } else {
                    uint32_t r[16];
                    AQ_TC_LD16(tmem + lanes, r);
                    tc_wait_ld();
                    const int grow = tile * kTcRows + row;
                    if (grow < n) {
                        out[(size_t)grow * 3 + 0] = __uint_as_float(r[0]);
                        out[(size_t)grow * 3 + 1] = __uint_as_float(r[1]);
                        out[(size_t)grow * 3 + 2] = __uint_as_float(r[2]);
                    }
                }
            }
            tc_fence_before();
            if (group_any(bar_id, !ok)) { fail = true; break; }
        }
        if (fail) break;
        tile = next;
    }
    if (fail) {
        // Let what this group still has in flight land (bounded) before TMEM is freed.
        if (gt == 0) atomicExch(err, 1u);
        if (lead && mma_pending) mbar_wait(mb_mma, mma_par);
        if (gt == 0 && tma_pending) mbar_wait(mb_in, tma_par);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base_slot),
                     "r"(kTcTmemCols)
                     : "memory");
    }
}

// ---------------------------------------------------------------- training
// One optimisation step's forward pass, backward pass and weight gradients in
// one persistent kernel (relative L2 loss of Mueller et al. 2021 with y^2 held
// constant, as k_nrc_backward). Separate kernels wrote the five activations
// and deltas of every row to memory and read them back, 3.6 KB per row, and
// the step was bound by that traffic and the launches' ramps; here a row's
// activations live in shared memory from its forward pass to its weight
// gradients, and a row costs its 128 B of input and 12 B of target.
//
// A CTA holds the forward weight image (42 KB) and runs two groups of 256
// threads, each with a 128-row tile in flight: five 16 KB buffers (the input
// and H1..H4; H5 takes the input's place) and dY (4 KB). One more warp issues
// every MMA:
//   steps 0-5   layer l's accumulator = H_{l-1} W_l^T
//   step 6      dH5 = dY W6, and dW6^T += H5^T dY
//   steps 7-10  dH_l = delta_{l+1} W_{l+1}, and dW_{l+1} += delta_{l+1}^T H_l
//   step 11     dW1 += delta1^T X
// and a group's threads (two per row, 32 columns each) turn an accumulator
// into the next operand: ReLU and bf16 for H_l, the loss gradient for dY,
// ReLU' for delta_l, which overwrites H_l once the MMAs that read it are done.
// While one group is in its epilogue the tensor core works for the other. The
// input comes in by TMA twice, before layer 1 and, into the buffer that
// delta5 leaves, for dW1; the next tile's input is fetched into delta4's.
//
// All operands share one storage: element (row, feature) of a tile at
// (feature / 8) slice + row 16 + (feature % 8) 2 bytes. Read with 128-byte
// steps between 8-row groups it is K-major over features (the layer MMAs' A),
// read with 128-byte steps along K it is MN-major with K = rows (the weight
// gradients' A and B); likewise one weight image serves W_l^T and W_l.
// The weight gradients of all layers accumulate in TMEM over every tile of
// the CTA (336 columns; a layer's 64 outputs are lanes 0-63 of an M = 128 MMA
// whose upper rows read, and ignore, the neighbouring buffer) and leave once,
// as this CTA's partial for the Adam kernel. One thread issues all MMAs, so
// the accumulations of both groups are ordered and a step is reproducible.
//
// Bound: the chain of eleven dependent MMA -> epilogue steps per tile, about
// 1400 cycles each, with two tiles in flight (the activations fill shared
// memory); without any weight-gradient MMA 250,007 rows take 73 us instead of
// 78. Measured (one step with Adam, device time): 250,007 rows 302 -> 78 us,
// 65,536 rows 85 -> 36 us, 16,384 rows 40 -> 25 us.
//
// Every wait is bounded: a wait that expires raises a flag that ends all
// others, and TMEM is freed on every path.
constexpr int kTrGroups = 2;
constexpr int kTrThreads = 256 * kTrGroups + 32;   // two threads per row, and the issuing warp
// Bytes between the 8-feature slices of a tile and of a layer's weights.
// (16 bytes of padding, which put the slices on different banks for the
// MN-major reads, changed nothing.)
constexpr uint32_t kTrSlice = kTcRows * 16, kTrWSlice = 64 * 16, kTrW6Slice = kTcOutRows * 16;
constexpr int kTrDyBytes = 2 * kTrSlice;           // dY, 16 columns (3 used)
constexpr int kTrGroupBytes = 5 * kTcTileBytes;
// dY of both groups, the groups' buffers, then the weights: an M = 128 weight
// gradient reads up to 16 KB past its buffer, which stays inside.
constexpr int kTrSmemBytes = kTrGroups * (kTrDyBytes + kTrGroupBytes) + kTcWeightBytes + 1024;
constexpr uint32_t kTrW6Col = 320, kTrAccCol = 352;  // dW1..dW5 at 64 L, dW6^T, the groups' accumulators
constexpr float kTcLossEps = 0.01f;
static_assert(kTrSmemBytes <= 227 * 1024, "shared memory per CTA");
static_assert(kTrAccCol + 64 * kTrGroups <= 512, "TMEM columns");

__device__ __forceinline__ uint32_t pack2_rn(float lo, float hi) {
    uint32_t d;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;\n" : "=r"(d) : "f"(hi), "f"(lo));
    return d;
}

// 0xffff in each half of a bf16 pair that is above zero.
__device__ __forceinline__ uint32_t positive2(uint32_t h) {
    __nv_bfloat162 a;
    *reinterpret_cast<uint32_t*>(&a) = h;
    return __hgt2_mask(a, __floats2bfloat162_rn(0.0f, 0.0f));
}

constexpr uint32_t kIdescAMn = 1u << 15, kIdescBMn = 1u << 16;  // A, B are MN-major

__device__ __forceinline__ void mbar_arrive(uint32_t mbar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(mbar) : "memory");
}

// Bounded wait that also ends when another wait of the CTA has expired.
__device__ __forceinline__ bool mbar_wait_or(uint32_t mbar, uint32_t parity, volatile uint32_t* failed) {
    for (uint32_t it = 0; it < kTcWaitLimit; ++it) {
        uint32_t done;
        asm volatile(
            "{\n"
            ".reg .pred p;\n"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
            "selp.u32 %0, 1, 0, p;\n"
            "}\n"
            : "=r"(done)
            : "r"(mbar), "r"(parity)
            : "memory");
        if (done) return true;
        if ((it & 15u) == 15u && *failed) return false;
    }
    *failed = 1u;
    return false;
}

// T: n x 3 targets; partial: one kNrcParams vector per CTA; loss: one sum of
// per-element losses per CTA; err: set to 1 when a wait expired.
__global__ void __launch_bounds__(kTrThreads, 1)
    k_nrc_train_tc(const __grid_constant__ CUtensorMap xmap, const float* __restrict__ T, int n, float inv_count,
                   const uint4* __restrict__ wimg, float* __restrict__ partial, double* __restrict__ loss,
                   uint32_t* __restrict__ err) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bars[5 * kTrGroups];
    __shared__ float s_loss[8 * kTrGroups];
    __shared__ uint32_t tmem_slot, s_failed;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* sbase = smem_raw + (base - smem_u32(smem_raw));
    constexpr uint32_t kBuf0 = kTrGroups * kTrDyBytes, kW0 = kBuf0 + kTrGroups * kTrGroupBytes;
    // Barriers of group g: input landed, input landed again, operand ready
    // (8 warps), accumulator complete, weight-gradient MMAs complete.
    enum { kX = 0, kR = 1, kReady = 2, kAcc = 3, kWg = 4 };
    auto bar = [&](int g, int k) { return smem_u32(&bars[5 * g + k]); };

    if (tid < 5 * kTrGroups)
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(&bars[tid])),
                     "r"(tid % 5 == kReady ? 8u : 1u)
                     : "memory");
    if (tid == 0) {
        s_failed = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        asm volatile("prefetch.tensormap [%0];\n" ::"l"(reinterpret_cast<uint64_t>(&xmap)) : "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_slot)),
                     "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    grid_dep_wait();  // the weights and inputs come from the kernels before
    grid_dep_launch();
    for (int i = tid; i < kTcWeightBytes / 16; i += kTrThreads)
        reinterpret_cast<uint4*>(sbase + kW0)[i] = __ldcg(wimg + i);
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();

    // All 512 columns were allocated, so they start at 0; the constant keeps
    // the issuing warp's TMEM addresses uniform.
    constexpr uint32_t tmem = 0u;
    if (tid == 0 && tmem_slot != 0u) s_failed = 1u;
    const int tiles = (n + kTcRows - 1) / kTcRows;
    const int stride = (int)gridDim.x * kTrGroups;
    float lsum = 0.0f;

    if (warp == 8 * kTrGroups) {
        // ------------------------------------------------ the issuing warp
        // All lanes run it with warp-uniform values, so that addresses and
        // descriptors live in uniform registers, and one lane issues: code
        // run by a single lane moved four registers to the uniform file for
        // every MMA, 110 cycles each, and bound the kernel (250,007 rows
        // 120 us).
        const bool lead = elect_one();
        const uint32_t idesc = tc_idesc(kTcRows, 64);
        // Low descriptor words: the groups' buffers (input, H1..H4), dY, weights.
        uint32_t b[kTrGroups][5], dy[kTrGroups];
#pragma unroll
        for (int g = 0; g < kTrGroups; ++g) {
            dy[g] = (base + (uint32_t)g * kTrDyBytes) >> 4;
#pragma unroll
            for (int k = 0; k < 5; ++k)
                b[g][k] = (base + kBuf0 + (uint32_t)g * kTrGroupBytes + (uint32_t)k * kTcTileBytes) >> 4;
        }
        const uint32_t w0 = (base + kW0) >> 4;
        uint32_t par = 0;      // parity of kX and kR (one phase per tile)
        uint32_t par_rdy = 0;  // bit g: parity of the group's kReady
        uint32_t sums = 0;     // 1 once the dW accumulators hold sums (group 0 starts them)
        bool ok = true;
        for (int t0 = (int)blockIdx.x; t0 < tiles; t0 += stride) {
#pragma unroll
            for (int step = 0; step < 12; ++step) {
#pragma unroll
                for (int g = 0; g < kTrGroups; ++g) {
                    if (t0 + g * (int)gridDim.x >= tiles || !ok) break;
                    const uint32_t acc = kTrAccCol + 64u * (uint32_t)g;
                    if (step == 0) {
                        ok = mbar_wait_or(bar(g, kX), par, &s_failed);
                    } else {
                        ok = mbar_wait_or(bar(g, kReady), (par_rdy >> g) & 1u, &s_failed);
                        par_rdy ^= 1u << g;
                    }
                    if (step == 11) ok = ok && mbar_wait_or(bar(g, kR), par, &s_failed);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    tc_fence_after();
                    // The layer MMAs: A is K-major over features.
                    constexpr uint32_t kStep = 2 * kTrSlice / 16, kWStep = 2 * kTrWSlice / 16, kW6Step = 2 * kTrW6Slice / 16;
                    if (step < 5) {  // H_{step+1}, from buffer `step` (0: the input)
#pragma unroll
                        for (uint32_t k = 0; k < 4; ++k)
                            tc_issue(lead, acc, desc_k(b[g][step] + k * kStep, kTrSlice),
                                     desc_k(w0 + (uint32_t)step * (kTcLayerBytes / 16) + k * kWStep, kTrWSlice), idesc, k > 0);
                    } else if (step == 5) {  // the outputs, from H5 in buffer 0
#pragma unroll
                        for (uint32_t k = 0; k < 4; ++k)
                            tc_issue(lead, acc, desc_k(b[g][0] + k * kStep, kTrSlice),
                                     desc_k(w0 + 5u * (kTcLayerBytes / 16) + k * kW6Step, kTrW6Slice),
                                     tc_idesc(kTcRows, kTcOutRows), k > 0);
                    } else if (step == 6) {  // dH5 = dY W6, K = 16 outputs
                        tc_issue(lead, acc, desc_k(dy[g], kTrSlice), desc_mn(w0 + 5u * (kTcLayerBytes / 16), kTrW6Slice),
                                 idesc | kIdescBMn, 0u);
                    } else if (step < 11) {  // dH_{11-step}, from delta_{12-step}
#pragma unroll
                        for (uint32_t k = 0; k < 4; ++k)
                            tc_issue(lead, acc, desc_k(b[g][(12 - step) % 5] + k * kStep, kTrSlice),
                                     desc_mn(w0 + (uint32_t)(11 - step) * (kTcLayerBytes / 16) + k * 16u, kTrWSlice),
                                     idesc | kIdescBMn, k > 0);
                    }
                    if (step < 11 && lead) tc_commit(bar(g, kAcc));
                    // The weight gradients: K = rows, both operands MN-major.
                    const uint32_t add = g > 0 ? 1u : sums;
                    if (step == 6) {
#pragma unroll
                        for (uint32_t k = 0; k < 8; ++k)
                            tc_issue(lead, kTrW6Col, desc_mn(b[g][0] + k * 16u, kTrSlice),
                                     desc_mn(dy[g] + k * 16u, kTrSlice),
                                     tc_idesc(kTcRows, kTcOutRows) | kIdescAMn | kIdescBMn, k > 0 ? 1u : add);
                    } else if (step > 6) {  // dW_{12-step}: delta_{12-step} with H_{11-step} (step 11: the input)
#pragma unroll
                        for (uint32_t k = 0; k < 8; ++k)
                            tc_issue(lead, 64u * (uint32_t)(11 - step),
                                     desc_mn(b[g][(12 - step) % 5] + k * 16u, kTrSlice),
                                     desc_mn(b[g][11 - step] + k * 16u, kTrSlice),
                                     idesc | kIdescAMn | kIdescBMn, k > 0 ? 1u : add);
                    }
                    if (step >= 6 && lead) tc_commit(bar(g, kWg));
                }
            }
            if (!ok) break;
            sums = 1u;
            par ^= 1u;
#pragma unroll
            for (int g = 0; g < kTrGroups; ++g) {  // the next input lies where delta4 was
                const uint32_t last = b[g][4];
#pragma unroll
                for (int k = 4; k > 0; --k) b[g][k] = b[g][k - 1];
                b[g][0] = last;
            }
        }
    } else {
        // ------------------------------------------------ a group's rows
        const int g = warp >> 3, q = warp & 3, gt = tid & 255;
        const uint32_t half = (uint32_t)(warp >> 2) & 1u;  // columns 32 half .. 32 half + 31
        const uint32_t row = (uint32_t)(q * 32 + lane);  // TMEM lane = tile row
        const uint32_t lanes = (uint32_t)(q * 32) << 16;
        const uint32_t acc = tmem + kTrAccCol + 64u * (uint32_t)g + 32u * half + lanes;
        const uint32_t b0 = base + kBuf0 + (uint32_t)g * kTrGroupBytes;
        uint8_t* gbuf = sbase + kBuf0 + (size_t)g * kTrGroupBytes;
        uint32_t ph_acc = 0, ph_wg = 0, o = 0;
        bool ok = true, wg_open = false;  // wg_open: the last tile's dW1 not yet waited for
        auto wait_acc = [&]() {
            ok = ok && mbar_wait_or(bar(g, kAcc), ph_acc, &s_failed);
            ph_acc ^= 1u;
            ok = __all_sync(0xffffffffu, ok);  // tcgen05.ld is warp-collective
            tc_fence_after();
            return ok;
        };
        auto wait_wg = [&]() {
            ok = ok && mbar_wait_or(bar(g, kWg), ph_wg, &s_failed);
            ph_wg ^= 1u;
            ok = __all_sync(0xffffffffu, ok);
            return ok;
        };
        auto ready = [&]() {  // this warp's rows of the next operand are in place
            fence_async_smem();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(g, kReady));
        };
        auto half_row = [&](uint32_t k) {  // this thread's 32 features in buffer k, 8 every 2048 bytes
            return gbuf + (o + k) % 5u * (uint32_t)kTcTileBytes + half * 4u * kTrSlice + row * 16u;
        };
        int tile = (int)blockIdx.x + g * (int)gridDim.x;
        if (gt == 0 && tile < tiles) tma_load_tile(&xmap, b0, bar(g, kX), tile * kTcRows);
        for (; tile < tiles; tile += stride) {
            const int grow = tile * kTcRows + (int)row;
            const bool valid = grow < n;
            float t[3] = {0.0f, 0.0f, 0.0f};
            if (valid)
                for (int c = 0; c < 3; ++c) t[c] = __ldcg(T + (size_t)grow * 3 + c);
            uint32_t r[32];
            for (uint32_t l = 0; l < 5; ++l) {  // H_{l+1} into buffer l + 1 (H5 into 0)
                if (!wait_acc()) break;
                if (l == 0 && wg_open) {
                    if (!wait_wg()) break;
                    wg_open = false;
                }
                AQ_TC_LD16(acc + 0u, (r + 0));
                AQ_TC_LD16(acc + 16u, (r + 16));
                tc_wait_ld();
                uint8_t* dst = half_row(l + 1);
#pragma unroll
                for (uint32_t j = 0; j < 4; ++j)
                    *reinterpret_cast<uint4*>(dst + j * kTrSlice) =
                        make_uint4(relu_pack2(r[8 * j], r[8 * j + 1]), relu_pack2(r[8 * j + 2], r[8 * j + 3]),
                                   relu_pack2(r[8 * j + 4], r[8 * j + 5]), relu_pack2(r[8 * j + 6], r[8 * j + 7]));
                ready();
            }
            if (!ok) break;
            if (!wait_acc()) break;
            if (half == 0) {  // dY = dLoss / dY, columns 0..2 of 16
                uint32_t y[16];
                AQ_TC_LD16(acc, y);
                tc_wait_ld();
                float gy[3] = {0.0f, 0.0f, 0.0f};
                if (valid) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        const float yc = __uint_as_float(y[c]);
                        const float den = yc * yc + kTcLossEps, d = yc - t[c];
                        lsum += d * d / den;
                        gy[c] = 2.0f * d / den * inv_count;
                    }
                }
                uint8_t* dy = sbase + (size_t)g * kTrDyBytes + row * 16u;
                *reinterpret_cast<uint4*>(dy) = make_uint4(pack2_rn(gy[0], gy[1]), pack2_rn(gy[2], 0.0f), 0u, 0u);
                *reinterpret_cast<uint4*>(dy + kTrSlice) = make_uint4(0u, 0u, 0u, 0u);
            }
            ready();
            for (uint32_t l = 5; l >= 1; --l) {  // delta_l over H_l, in buffer l % 5
                if (!wait_acc()) break;
                uint8_t* dst = half_row(l);
                uint4 h[4];
#pragma unroll
                for (uint32_t j = 0; j < 4; ++j) h[j] = *reinterpret_cast<const uint4*>(dst + j * kTrSlice);
                AQ_TC_LD16(acc + 0u, (r + 0));
                AQ_TC_LD16(acc + 16u, (r + 16));
                tc_wait_ld();
#pragma unroll
                for (uint32_t j = 0; j < 4; ++j)  // ReLU'(Z) from H = ReLU(Z)
                    h[j] = make_uint4(pack2_rn(__uint_as_float(r[8 * j]), __uint_as_float(r[8 * j + 1])) & positive2(h[j].x),
                                      pack2_rn(__uint_as_float(r[8 * j + 2]), __uint_as_float(r[8 * j + 3])) & positive2(h[j].y),
                                      pack2_rn(__uint_as_float(r[8 * j + 4]), __uint_as_float(r[8 * j + 5])) & positive2(h[j].z),
                                      pack2_rn(__uint_as_float(r[8 * j + 6]), __uint_as_float(r[8 * j + 7])) & positive2(h[j].w));
                if (!wait_wg()) break;  // the weight gradient that reads H_l is done
#pragma unroll
                for (uint32_t j = 0; j < 4; ++j) *reinterpret_cast<uint4*>(dst + j * kTrSlice) = h[j];
                ready();
                // delta5's buffer is free after step 7, delta4's after step 8.
                if (gt == 0 && l == 4) tma_load_tile(&xmap, b0 + o * (uint32_t)kTcTileBytes, bar(g, kR), tile * kTcRows);
                if (gt == 0 && l == 3 && tile + stride < tiles)
                    tma_load_tile(&xmap, b0 + (o + 4u) % 5u * (uint32_t)kTcTileBytes, bar(g, kX),
                                  (tile + stride) * kTcRows);
            }
            if (!ok) break;
            wg_open = true;  // dW1
            o = (o + 4u) % 5u;
        }
        if (wg_open) wait_wg();
        for (int k = 16; k > 0; k >>= 1) lsum += __shfl_down_sync(0xffffffffu, lsum, k);
        if (lane == 0) s_loss[warp] = lsum;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (s_failed) {
        if (tid == 0) atomicExch(err, 1u);
        // Whatever is still in flight (TMA, MMAs) lands within these bounded waits.
        if (tid < 5 * kTrGroups)
            for (uint32_t it = 0; it < 2; ++it) mbar_wait(smem_u32(&bars[tid]), it);
    } else if (warp < 8 * kTrGroups && (warp & 3) < 2) {
        // Lanes 0..63 hold the outputs of a layer (dW6^T: the inputs), which warps 0
        // and 1 of every four can read; the fours share the layers.
        const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
        const int orow = (warp & 3) * 32 + lane;
        float* P = partial + (size_t)blockIdx.x * kNrcParams;
        for (int L = warp >> 2; L < 6; L += 2 * kTrGroups) {
            if (L < 5) {
                uint32_t r[64];
                const uint32_t col = tmem + 64u * (uint32_t)L + lanes;
                AQ_TC_LD16(col + 0u, (r + 0));
                AQ_TC_LD16(col + 16u, (r + 16));
                AQ_TC_LD16(col + 32u, (r + 32));
                AQ_TC_LD16(col + 48u, (r + 48));
                tc_wait_ld();
                float4* dst = reinterpret_cast<float4*>(P + (size_t)L * 4096 + (size_t)orow * 64);
#pragma unroll
                for (int c = 0; c < 16; ++c)
                    dst[c] = make_float4(__uint_as_float(r[4 * c]), __uint_as_float(r[4 * c + 1]),
                                         __uint_as_float(r[4 * c + 2]), __uint_as_float(r[4 * c + 3]));
            } else {
                uint32_t r[16];
                AQ_TC_LD16(tmem + kTrW6Col + lanes, r);
                tc_wait_ld();
                for (int c = 0; c < kNrcOut; ++c) P[5 * 4096 + c * 64 + orow] = __uint_as_float(r[c]);
            }
        }
    }
    if (tid == 0) {
        double sum = 0.0;
        for (int k = 0; k < 8 * kTrGroups; ++k) sum += (double)s_loss[k];
        loss[blockIdx.x] = sum;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_slot), "r"(512u) : "memory");
}

// ---------------------------------------------------------------- host side
size_t nrc_tc_weight_bytes() { return (size_t)kTcWeightBytes; }

void nrc_pack_tc(aqua_ctx* ctx, const float* w, const float* inf, void* img_w, void* img_inf) {
    AQ_CUDA(cudaMemsetAsync(img_w, 0, kTcWeightBytes, ctx->stream));
    AQ_CUDA(cudaMemsetAsync(img_inf, 0, kTcWeightBytes, ctx->stream));
    k_nrc_pack_tc<<<(kNrcParams + 255) / 256, 256, 0, ctx->stream>>>(w, inf, (uint8_t*)img_w, (uint8_t*)img_inf);
    AQ_CUDA(cudaGetLastError());
}

static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, []() {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
        (void)cudaGetLastError();
    });
    if (!fn) throw Error(AQUA_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    return fn;
}

// n rows of 64 bf16 as boxes of 8 columns x 128 rows (zero past n).
static CUtensorMap row_map(const uint16_t* X, int n) {
    if (((uintptr_t)X & 15) != 0) throw Error(AQUA_ERR_INVALID_ARG, "x must be 16-byte aligned");
    CUtensorMap map;
    const cuuint64_t dims[2] = {64, (cuuint64_t)n};
    const cuuint64_t strides[1] = {128};  // bytes per row
    const cuuint32_t box[2] = {8, (cuuint32_t)kTcRows};
    const cuuint32_t estr[2] = {1, 1};
    CUresult r = tensor_map_encoder()(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<uint16_t*>(X), dims,
                                      strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                                      CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) throw Error(AQUA_ERR_CUDA, "cuTensorMapEncodeTiled failed for the network's rows");
    return map;
}

void nrc_forward_tc_dev(aqua_ctx* ctx, const void* img, const uint16_t* X, int n, float* out, uint32_t* err) {
    if (n <= 0) return;
    const CUtensorMap map = row_map(X, n);
    if (!ctx->nrc_tc_ready) {  // once per context (one device)
        AQ_CUDA(cudaFuncSetAttribute(k_nrc_forward_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, kTcFwdSmemBytes));
        ctx->nrc_tc_ready = true;
    }
    const int tiles = (n + kTcRows - 1) / kTcRows;
    const int grid = std::max(1, std::min(tiles, ctx->num_sms));
    launch_chained(k_nrc_forward_tc, dim3(grid), dim3(kTcFwdThreads), kTcFwdSmemBytes, ctx->stream, map, n,
                   reinterpret_cast<const uint4*>(img), out, err);
    AQ_CUDA(cudaGetLastError());
}


// One training step's gradients: per-CTA partials (kNrcParams each) and loss
// sums for the Adam kernel; returns how many.
int nrc_train_tc_dev(aqua_ctx* ctx, const void* img, const uint16_t* X, const float* T, int n, float inv_count,
                     float* partial, double* loss, uint32_t* err) {
    if (n <= 0) return 0;
    const CUtensorMap map = row_map(X, n);
    if (!ctx->nrc_tc_train_ready) {
        AQ_CUDA(cudaFuncSetAttribute(k_nrc_train_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, kTrSmemBytes));
        ctx->nrc_tc_train_ready = true;
    }
    const int grid = std::min(nrc_train_tc_max_partials(ctx), (n + kTcRows - 1) / kTcRows);
    launch_chained(k_nrc_train_tc, dim3(grid), dim3(kTrThreads), kTrSmemBytes, ctx->stream, map, T, n, inv_count,
                   reinterpret_cast<const uint4*>(img), partial, loss, err);
    AQ_CUDA(cudaGetLastError());
    return grid;
}

int nrc_train_tc_max_partials(const aqua_ctx* ctx) { return ctx->num_sms; }

}  // namespace aq
