// extend.cu — the `extend` stage: closest hits for a queue of rays. This is
// the work traceRayEXT hands to RT cores in the reference
// (assets/glsl/pathtrace.rgen:65-76). Persistent kernels: one grid of
// (SMs x resident blocks) whose warps take rays from an atomic work counter,
// so the queue length can stay on the device (no host round trip). The
// traversal loops are those of trace.cu.
#include "extend.cuh"

namespace solrt {

namespace {

// Wavefront queue: o_tmin / d_tmax SoA, hit = (t, prim bits, u, v). kSingle: all
// rays in `scene`, else ray i in the scene of its job (meta[i].y >> kDepthBits),
// or in `scene` when there is no job table.
template <bool kSingle>
struct QueueIO : FetchLoop {
    const float4* __restrict__ o_tmin;
    const float4* __restrict__ d_tmax;
    const uint2* __restrict__ meta;
    const DevJob* __restrict__ jobs;
    float4* __restrict__ hits;
    const TravScene& scene;
    int lanes;
    bool any_hit;  // occlusion queries (shadow rays): any hit in (tmin, tmax)
    SOLRT_D TravScene first_scene() const { return kSingle ? scene : TravScene{}; }
    SOLRT_D void load(uint32_t i, float4& o, float4& d, TravScene& ts) const {
        load_ray(i, o, d);
        if (!kSingle) ts = jobs ? trav_scene(jobs[meta[i].y >> kDepthBits].sc) : scene;
    }
    SOLRT_D void load_ray(uint32_t i, float4& o, float4& d) const {
        o = o_tmin[i];
        d = d_tmax[i];
    }
    SOLRT_D bool next(uint32_t i, float, const HitRec& h, float4&, float4&, const TraceCounters&, uint32_t&) const {
        hits[i] = make_float4(h.t, __uint_as_float(h.prim), h.u, h.v);
        return false;
    }
};

struct ExtendArgs {
    TravScene scene;
    const DevJob* jobs;
    PathQueue q;
    float4* hits;
    const unsigned int* count;
    uint32_t slots;
    int lanes;
    bool any_hit;
    unsigned int* work;
    int* deep;
    DevStats* stats;
};

template <int KIND, bool kSingle, bool kCount>
__global__ void __launch_bounds__(256, traverse_min_blocks<KIND>()) k_extend(const __grid_constant__ ExtendArgs a) {
    const uint32_t n = *a.count;
    if (blockIdx.x == 0 && threadIdx.x == 0 && n) atomicAdd(&a.stats->segments, (unsigned long long)n);
    QueueIO<kSingle> io{{}, a.q.o_tmin, a.q.d_tmax, a.q.meta, a.jobs, a.hits, a.scene, a.lanes, a.any_hit};
    TraceCounters cnt{0, 0, 0};
    uint32_t ef = 0;
    extend_kind<KIND, kCount>(io, n, a.work, stack_mem(a.slots, a.deep), cnt, ef);
    flush_traversal(a.stats, cnt, ef, kCount);
    release_work(a.work);
}

template <int KIND, bool kSingle, bool kCount>
solrt_status launch_extend_variant(Context& ctx, ExtendArgs a, uint32_t most) {
    LaunchShape s;
    SOLRT_TRY((launch_shape<KIND, k_extend<KIND, kSingle, kCount>>(ctx, 0, most, true, s)));
    a.slots = s.slots;
    a.lanes = (int)s.lanes;
    k_extend<KIND, kSingle, kCount><<<s.grid, s.block, s.smem, ctx.stream>>>(a);
    return SOLRT_OK;
}

// Counting launches have one variant (its scenes per ray).
template <int KIND>
solrt_status launch_extend_kind(Context& ctx, const ExtendArgs& a, uint32_t most) {
    if (ctx.counters) return launch_extend_variant<KIND, false, true>(ctx, a, most);
    if (!a.jobs) return launch_extend_variant<KIND, true, false>(ctx, a, most);
    return launch_extend_variant<KIND, false, false>(ctx, a, most);
}

}  // namespace

bool extend_variant_ok(uint32_t block, uint32_t smem) {
    return (block == 64 || block == 128 || block == 256) && (smem == 16 || smem == 32);
}

solrt_status launch_extend(Context& ctx, uint32_t kind, const DevScene* scene, const DevJob* jobs, const PathQueue& q,
                           float4* hits, const unsigned int* count, uint32_t most, DevStats* st, bool any_hit) {
    ctx.last_kind = kind;
    const ExtendArgs a{scene ? trav_scene(*scene) : TravScene{}, scene ? nullptr : jobs, q, hits, count, 0, 32, any_hit,
                       ctx.trace_work.as<unsigned int>(), ctx.deep_stack.as<int>(),
                       st ? st : ctx.stats.as<DevStats>()};
    if (kind == SOLRT_BVH8_Q8) SOLRT_TRY(launch_extend_kind<SOLRT_BVH8_Q8>(ctx, a, most));
    else if (kind == SOLRT_BVH4_Q8) SOLRT_TRY(launch_extend_kind<SOLRT_BVH4_Q8>(ctx, a, most));
    else if (kind == SOLRT_BVH8_F32) SOLRT_TRY(launch_extend_kind<SOLRT_BVH8_F32>(ctx, a, most));
    else if (kind == SOLRT_BVH2_Q16) SOLRT_TRY(launch_extend_kind<SOLRT_BVH2_Q16>(ctx, a, most));
    else if (kind == SOLRT_BVH2_TWO_LEVEL)
        SOLRT_TRY(launch_extend_kind<SOLRT_BVH2_TWO_LEVEL>(ctx, a, most));
    else SOLRT_TRY(launch_extend_kind<SOLRT_BVH2>(ctx, a, most));
    ++ctx.launches;
    SOLRT_CUDA(cudaGetLastError());
    return SOLRT_OK;
}

}  // namespace solrt
