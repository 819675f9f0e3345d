// extend.cuh — the traversal loop of a BVH kind and the launch shape of the
// kernels built around it (trace.cu, paths.cu, siblings.cu).
#pragma once

#include <algorithm>

#include "bvh2_2l.cuh"
#include "bvh2_ww.cuh"
#include "bvh4_ww.cuh"
#include "bvh8_ww.cuh"
#include "internal.h"

namespace solrt {

// Rays of `io` until the work counter passes n, with the kind's loop.
template <int KIND, bool kCount, class IO>
SOLRT_D void extend_kind(IO& io, uint32_t n, unsigned int* work, const StackMem& mem, TraceCounters& cnt,
                         uint32_t& ef) {
    if constexpr (KIND == SOLRT_BVH2) extend_bvh2_ww<IO, kCount, false>(io, n, work, mem, cnt, ef);
    else if constexpr (KIND == SOLRT_BVH2_Q16) extend_bvh2_ww<IO, kCount, true>(io, n, work, mem, cnt, ef);
    else if constexpr (KIND == SOLRT_BVH2_TWO_LEVEL) extend_bvh2_2l_ww<IO, kCount>(io, n, work, mem, cnt, ef);
    else if constexpr (KIND == SOLRT_BVH4_Q8) extend_bvh4_ww<IO, kCount>(io, n, work, mem, cnt, ef);
    else if constexpr (KIND == SOLRT_BVH8_F32) extend_bvh8_ww<IO, kCount, true>(io, n, work, mem, cnt, ef);
    else extend_bvh8_ww<IO, kCount, false>(io, n, work, mem, cnt, ef);
}

// Closest hit of one ray with the kind's per-ray loop.
template <int KIND>
SOLRT_D void trace_one(const TravScene& ts, const float4& o, const float4& d, HitRec& h, TraceCounters& cnt,
                       uint32_t& ef) {
    if (KIND == SOLRT_BVH8_Q8) trace_bvh8<false>(ts, o.x, o.y, o.z, d.x, d.y, d.z, o.w, d.w, h, cnt, ef);
    else if (KIND == SOLRT_BVH8_F32) trace_bvh8<false, true>(ts, o.x, o.y, o.z, d.x, d.y, d.z, o.w, d.w, h, cnt, ef);
    else if (KIND == SOLRT_BVH4_Q8) trace_bvh4_ray(ts, o.x, o.y, o.z, d.x, d.y, d.z, o.w, d.w, h, cnt, ef);
    else if (KIND == SOLRT_BVH2_Q16) trace_bvh2_ray<true>(ts, o.x, o.y, o.z, d.x, d.y, d.z, o.w, d.w, h, cnt, ef);
    else if (KIND == SOLRT_BVH2_TWO_LEVEL) trace_bvh2_2l_ray(ts, o.x, o.y, o.z, d.x, d.y, d.z, o.w, d.w, h, cnt, ef);
    else trace_bvh2_ray(ts, o.x, o.y, o.z, d.x, d.y, d.z, o.w, d.w, h, cnt, ef);
}

// Shared-memory stack slots of a launch: the context's choice for the kinds
// with a node stack, none for the 8-wide kinds (group stack in local memory).
template <int KIND>
constexpr bool kind_has_smem_stack() {
    return KIND != SOLRT_BVH8_Q8 && KIND != SOLRT_BVH8_F32;
}

extern __shared__ int s_dyn[];

// Traversal memory of the calling thread: its stack column at the start of
// the block's shared memory, its ray column (RayMem) behind the stacks, and its
// entries of `deep` (Context::deep_stack).
SOLRT_D StackMem stack_mem(uint32_t slots, int* deep) {
    const uint32_t threads = gridDim.x * blockDim.x;
    return StackMem{smem_addr(s_dyn + threadIdx.x), 4u * blockDim.x, (int)slots,
                    deep + blockIdx.x * blockDim.x + threadIdx.x - (size_t)kMinStackSlots * threads, threads,
                    smem_addr(s_dyn + slots * blockDim.x + threadIdx.x)};
}
// The thread's column of the block's program state (word w at address
// column + 4 * w * blockDim.x), behind the stacks and the rays.
SOLRT_D uint32_t state_column(uint32_t slots) {
    return smem_addr(s_dyn + (slots + kRayWords) * blockDim.x + threadIdx.x);
}

// Zeroes the work counter for the next launch on the stream once every block
// is done with it: `work` is (next ray, finished blocks), both 0 between
// launches.
SOLRT_D void release_work(unsigned int* work) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(work + 1, 1u) == gridDim.x - 1u) {
            work[0] = 0u;
            work[1] = 0u;
        }
    }
}

// A thread's words of program state in shared memory (state_column).
struct StateMem {
    uint32_t base, stride;
    SOLRT_D explicit StateMem(uint32_t slots) : base(state_column(slots)), stride(4u * blockDim.x) {}
    SOLRT_D uint32_t get(uint32_t w) const { return lds_u32(base + w * stride); }
    SOLRT_D void put(uint32_t w, uint32_t v) const { sts_u32(base + w * stride, v); }
    SOLRT_D void bump(uint32_t w) const { put(w, get(w) + 1u); }
    SOLRT_D float getf(uint32_t w) const { return __uint_as_float(get(w)); }
    SOLRT_D void putf(uint32_t w, float v) const { put(w, __float_as_uint(v)); }
    SOLRT_D f3 get3(uint32_t w) const { return f3{getf(w), getf(w + 1), getf(w + 2)}; }
    SOLRT_D void put3(uint32_t w, float x, float y, float z) const {
        putf(w, x);
        putf(w + 1, y);
        putf(w + 2, z);
    }
};

SOLRT_D void flush_traversal(DevStats* stats, const TraceCounters& cnt, uint32_t ef, bool count_nodes) {
    const uint32_t fb = __reduce_add_sync(0xffffffffu, cnt.fallbacks);
    const uint32_t e = __reduce_or_sync(0xffffffffu, ef);
    uint32_t nn = 0, nt = 0;
    if (count_nodes) {
        nn = __reduce_add_sync(0xffffffffu, cnt.nodes);
        nt = __reduce_add_sync(0xffffffffu, cnt.tris);
    }
    if ((threadIdx.x & 31) == 0) {
        if (fb) atomicAdd(&stats->fp64_fallbacks, (unsigned long long)fb);
        if (e) atomicOr(&stats->eflags, e);
        if (nn) atomicAdd(&stats->node_visits, (unsigned long long)nn);
        if (nt) atomicAdd(&stats->tri_tests, (unsigned long long)nt);
    }
}

// Blocks of 256 threads that an SM must hold, for the register allocator: 5
// (48 registers, 1280 threads), for the wide kinds 4 (64 registers: their node
// tests hold more). 4 / 5 / 6: a 64-spp soup frame through FP32 binary
// nodes 132.9 / 131.9 / 134.0 ms, 4.2M incoherent rays 2.80 / 2.72 / 2.86 ms,
// two-level scenes 9.41 / 9.12 / 9.99 ms; the 8-wide tree on a tunnel frame
// 60.3 / 55.3 / 58.0 ms with 3 / 4 / 5, the 4-wide one 57.4 / 57.6 with 4 / 5
// (next-event estimation through it 15.3 / 15.9 ms).
template <int KIND>
constexpr int traverse_min_blocks() {
    return KIND == SOLRT_BVH4_Q8 || KIND == SOLRT_BVH8_Q8 || KIND == SOLRT_BVH8_F32 ? 4 : 5;
}

// Shape of one launch of `kern`: the context's block size and stack slots,
// state_words words of program state per thread, a grid of (SMs x resident
// blocks) or fewer blocks when `units` rays or paths need fewer, and how many
// lanes of each warp take work: 32, or, for up to spread_units units with
// `spread`, as few as spread them over all warps of a full grid. A warp with
// fewer rays steps faster, but beyond that its idle lanes cost more than the
// shorter steps gain (microseconds for one call, few lanes / 32: 2000 rays
// through 20k triangles 94 / 134, 8000 117 / 143, 30k 159 / 152, 100k 214 / 194;
// with three calls in flight 34 / 47, 43 / 47, 68 / 56, 98 / 74; the 8-wide tree
// 7400 rays 88 / 92 and 30.9 / 29.9, 4000 97 / 117 and 37.1 / 39.1).
template <int KIND>
constexpr uint32_t spread_units() {
    return KIND == SOLRT_BVH8_Q8 || KIND == SOLRT_BVH8_F32 ? 4096 : 8192;
}
struct LaunchShape {
    uint32_t grid = 0, block = 0, smem = 0, slots = 0, lanes = 32;
};

template <int KIND, auto kern>
solrt_status launch_shape(const Context& ctx, uint32_t state_words, uint32_t units, bool spread, LaunchShape& s) {
    if (host_fault(kFaultLaunch)) {
        set_error("launch refused by a test");
        return SOLRT_ERR_DEVICE;
    }
    s.block = ctx.tune.block;
    s.slots = kind_has_smem_stack<KIND>() ? stack_slots(ctx.tune.smem) : 0u;
    s.smem = 4u * s.block * (s.slots + kRayWords + state_words);
    static LaunchTable table;
    const int shape = (s.block == 64 ? 0 : s.block == 128 ? 2 : 4) + (ctx.tune.smem == 16 ? 0 : 1);
    const auto query = [&](int* fits) -> solrt_status {
        const uint32_t most = 4u * 256u * (32u + kRayWords + state_words);
        SOLRT_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most));
        SOLRT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(fits, kern, (int)s.block, s.smem));
        return SOLRT_OK;
    };
    int b = 0;
    SOLRT_TRY(table.blocks(ctx.device, shape, s.block, query, &b));
    const uint32_t full = (uint32_t)ctx.sm_count * (uint32_t)b;
    const uint32_t warps = full * (s.block / 32u);
    s.lanes = spread && units <= spread_units<KIND>() ? std::min(32u, std::max(1u, (units + warps - 1u) / warps)) : 32u;
    s.grid = std::min(full, (units + s.lanes * (s.block / 32u) - 1u) / (s.lanes * (s.block / 32u)));
    return SOLRT_OK;
}

}  // namespace solrt
