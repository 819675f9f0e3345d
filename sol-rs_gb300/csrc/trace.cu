// trace.cu — closest-hit queries for arrays of rays (solrt_trace_rays*): the
// work traceRayEXT hands to RT cores in the reference
// (assets/glsl/pathtrace.rgen:65-76). Persistent kernels: one grid of
// (SMs x resident blocks) whose warps take rays from an atomic work counter.
//   BVH2: while-while traversal with per-lane refill (bvh2_ww.cuh); two-level
//   scenes: the same loop over a TLAS and object-space BLASes (bvh2_2l.cuh).
//   BVH8 / BVH4: the same warp-uniform organisation over quantised wide
//   nodes (bvh8_ww.cuh, bvh4_ww.cuh).
#include "extend.cuh"

namespace solrt {

namespace {

// AoS solrt_ray (2 float4) -> solrt_hit (float4), one scene.
struct RayFileIO : FetchLoop {
    const float4* __restrict__ rays;
    float4* __restrict__ hits;
    const TravScene& scene;
    int lanes;
    static constexpr bool any_hit = false;
    SOLRT_D TravScene first_scene() const { return scene; }
    SOLRT_D void load(uint32_t i, float4& o, float4& d, TravScene&) const { load_ray(i, o, d); }
    SOLRT_D void load_ray(uint32_t i, float4& o, float4& d) const { 
        o = rays[2 * (size_t)i];
        d = rays[2 * (size_t)i + 1];
    }
    SOLRT_D bool next(uint32_t i, float, const HitRec& h, float4&, float4&, const TraceCounters&, uint32_t&) const {
        hits[i] = make_float4(h.t, __uint_as_float(h.prim), h.u, h.v);
        return false;
    }
};

struct TraceArgs {
    TravScene scene;
    const float4* rays;
    float4* hits;
    uint32_t n, slots;
    int lanes;
    unsigned int* work;
    int* deep;
    DevStats* stats;
};

template <int KIND, bool kCount>
__global__ void __launch_bounds__(256, traverse_min_blocks<KIND>()) k_trace(const __grid_constant__ TraceArgs a) {
    RayFileIO io{{}, a.rays, a.hits, a.scene, a.lanes};
    TraceCounters cnt{0, 0, 0};
    uint32_t ef = 0;
    extend_kind<KIND, kCount>(io, a.n, a.work, stack_mem(a.slots, a.deep), cnt, ef);
    flush_traversal(a.stats, cnt, ef, kCount);
    release_work(a.work);
}

template <int KIND>
solrt_status launch_kind(Context& ctx, TraceArgs a) {
    auto kern = ctx.counters ? k_trace<KIND, true> : k_trace<KIND, false>;
    LaunchShape s;
    if (ctx.counters) SOLRT_TRY((launch_shape<KIND, k_trace<KIND, true>>(ctx, 0, a.n, true, s)));
    else SOLRT_TRY((launch_shape<KIND, k_trace<KIND, false>>(ctx, 0, a.n, true, s)));
    a.slots = s.slots;
    a.lanes = (int)s.lanes;
    kern<<<s.grid, s.block, s.smem, ctx.stream>>>(a);
    return SOLRT_OK;
}

}  // namespace

solrt_status launch_trace_rays(Context& ctx, const Scene& sc, const solrt_ray* rays, uint32_t n, solrt_hit* hits) {
    if (n == 0) return SOLRT_OK;
    const DevScene d = sc.view();
    ctx.last_kind = d.bvh_kind;
    const TraceArgs a{trav_scene(d), reinterpret_cast<const float4*>(rays), reinterpret_cast<float4*>(hits), n, 0, 32,
                      ctx.trace_work.as<unsigned int>(), ctx.deep_stack.as<int>(),
                      ctx.stats.as<DevStats>()};
    if (d.bvh_kind == SOLRT_BVH8_Q8) SOLRT_TRY(launch_kind<SOLRT_BVH8_Q8>(ctx, a));
    else if (d.bvh_kind == SOLRT_BVH4_Q8) SOLRT_TRY(launch_kind<SOLRT_BVH4_Q8>(ctx, a));
    else if (d.bvh_kind == SOLRT_BVH8_F32) SOLRT_TRY(launch_kind<SOLRT_BVH8_F32>(ctx, a));
    else if (d.bvh_kind == SOLRT_BVH2_Q16) SOLRT_TRY(launch_kind<SOLRT_BVH2_Q16>(ctx, a));
    else if (d.bvh_kind == SOLRT_BVH2_TWO_LEVEL) SOLRT_TRY(launch_kind<SOLRT_BVH2_TWO_LEVEL>(ctx, a));
    else SOLRT_TRY(launch_kind<SOLRT_BVH2>(ctx, a));
    ++ctx.launches;
    SOLRT_CUDA(cudaGetLastError());
    return SOLRT_OK;
}

}  // namespace solrt
