// paths.cuh — a frame of one job as one persistent launch: the path kernel.
//
// The reference runs one raygen invocation per pixel that loops over 8
// samples and up to maxBounces+1 traceRayEXT calls, each resuming in the
// closest-hit or miss shader (assets/glsl/pathtrace.rgen:39-104,
// pathtrace.rchit:56-113, pathtrace.rmiss:8-21). Here a warp holds up to 32
// paths in the traversal loop of the BVH kind; when enough of its lanes have
// finished their rays (12 of 32, 24 where traversal is short or shading long:
// PathArgs::refill), those lanes shade their hits and go on with the next ray of
// their path, or end it and take another one from the launch's work counter
// (warp_feed). Path state that traversal does not touch waits in shared memory.
//
// What it saves over the wavefront (pathtrace.cu) is the launches, two per
// bounce level, and the end of each extend launch, which lasts as long as its
// longest ray with few other rays left to trace. What it costs is shading with
// part of a warp while the other lanes wait: on frames large enough to fill
// the wavefront's launches it is a third slower (path_kernel_pays in
// pathtrace.cu draws the line).
//
// A unit of work is a path, or, for jobs with one random stream per pixel
// (SOLRT_RNG_REF_STREAM), a pixel whose samples the lane traces one after
// the other. Every sample writes its radiance to its own slot and per-pixel
// sums run in sample order, so the image equals a sequential per-pixel
// evaluation, and the wavefront's, bit for bit.
#pragma once

#include "extend.cuh"
#include "path_ops.cuh"

#ifndef SOLRT_PATH_MINB
#define SOLRT_PATH_MINB 4
#endif

namespace solrt {

// One launch: the samples of one work item of one job, `units` units of work.
struct PathArgs {
    DevJob job;
    DevItem item;
    uint32_t units, slots;
    int refill;  // warp_feed's threshold
    unsigned int* work;
    int* deep;
    float4* rad;
    DevStats* stats;
};

// Shared-memory words per thread.
enum PathWord {
    kWDir = 0,      // direction of the ray in flight (3)
    kWThr = 3,      // throughput (3)
    kWRng = 6,      // random stream
    kWSlot = 7,     // radiance slot in the pass
    kWDepth = 8,    // bounces so far
    kWSegs = 9,     // rays traced by this thread, shadow rays apart
    kWOrg = 10,     // origin of the ray in flight (3; two-level scenes and next-event estimation)
    kWNext = 13,    // next-event estimation: direction after the shadow ray (3)
    kWLight = 16,   // what the shadow ray adds when it is unoccluded (3)
    kWSum = 19,     // sum of the path's light terms (3)
    kWPrev = 22,    // normal of the vertex the ray left, pdf of its direction (4)
    kWMark = 26,    // FP64 fallbacks when the last ray ended
    kWShadow = 27,  // FP64 fallbacks of shadow rays
    kWShadowSegs = 28,  // shadow rays traced, and those that reached their light (2)
    kWNeeEnd = 30,
};
template <int KIND, bool kNee>
constexpr uint32_t path_words() {
    return kNee ? kWNeeEnd : KIND == SOLRT_BVH2_TWO_LEVEL ? kWNext : kWOrg;
}

// The any-hit switch of the traversal loops: a per-lane flag where shadow
// rays are traced, a constant elsewhere.
template <bool kNee> struct PathAnyHit { bool any_hit = false; };
template <> struct PathAnyHit<false> { static constexpr bool any_hit = false; };

template <int KIND, bool kNee>
struct PathIO : PathAnyHit<kNee>, ShadeLoop {
    const PathArgs& a;
    const StateMem st;
    const int refill;
    static constexpr int lanes = 32;  // fewer make a lone small frame no faster and several at once slower
    static constexpr bool kOrg = kNee || KIND == SOLRT_BVH2_TWO_LEVEL;

    SOLRT_D PathIO(const PathArgs& args) : a(args), st(args.slots), refill(args.refill) {
        st.put(kWSegs, 0u);
        if (kNee)
            for (int w = kWMark; w < kWNeeEnd; ++w) st.put(w, 0u);
    }
    SOLRT_D TravScene first_scene() const { return trav_scene(a.job.sc); }

    // The camera ray of a sample of pixel pix (rgen:47-61).
    SOLRT_D void start(uint32_t pix, uint32_t rng, uint32_t slot, float4& o, float4& d) {
        camera_ray(a.job, pix, rng, o, d);
        st.put3(kWDir, d.x, d.y, d.z);
        st.put3(kWThr, 1.0f, 1.0f, 1.0f);
        st.put(kWRng, rng);
        st.put(kWSlot, slot);
        st.put(kWDepth, 0u);
        if (kOrg) st.put3(kWOrg, o.x, o.y, o.z);
        if (kNee) st.put3(kWSum, 0.0f, 0.0f, 0.0f);
        st.bump(kWSegs);
    }
    SOLRT_D void load(uint32_t unit, float4& o, float4& d, TravScene&) {
        const DevItem& it = a.item;
        const bool chain = a.job.rng_mode == SOLRT_RNG_REF_STREAM;
        const uint32_t lp = chain ? unit : unit / it.k, j = chain ? 0u : unit - lp * it.k;
        const uint32_t pix = it.pix0 + lp, s = it.s0 + j;
        const uint32_t rng = sample_seed(a.job, pix, s, chain && s > 0 ? a.job.rng_state[pix] : 0u);
        start(pix, rng, lp * it.k + j, o, d);
    }
    SOLRT_D void load_ray(uint32_t, float4& o, float4& d) const {
        const f3 p = st.get3(kWOrg), q = st.get3(kWDir);
        o = make_float4(p.x, p.y, p.z, 0.0f);
        d = make_float4(q.x, q.y, q.z, 0.0f);
    }
    // The lane's ray is done: shades its hit. True with the path's next ray
    // (or its pixel's next sample).
    SOLRT_D bool next(uint32_t unit, float tmin, const HitRec& best, float4& o, float4& d, const TraceCounters& cnt,
                      uint32_t& ef) {
        const DevJob& J = a.job;
        const f3 dir = st.get3(kWDir);
        f3 org{0.0f, 0.0f, 0.0f};
        if (kOrg) org = st.get3(kWOrg);
        if constexpr (kNee) {
            if (this->any_hit) st.put(kWShadow, st.get(kWShadow) + cnt.fallbacks - st.get(kWMark));
            st.put(kWMark, cnt.fallbacks);
            if (this->any_hit) {  // a shadow ray: its term, then the bounce ray from the same vertex
                this->any_hit = false;
                if (best.prim == SOLRT_NO_HIT) {
                    const f3 c = st.get3(kWLight), s = st.get3(kWSum);
                    st.put3(kWSum, s.x + c.x, s.y + c.y, s.z + c.z);
                    st.bump(kWShadowSegs + 1);
                }
                const f3 q = st.get3(kWNext);
                st.put3(kWDir, q.x, q.y, q.z);
                o = make_float4(org.x, org.y, org.z, tmin);
                d = make_float4(q.x, q.y, q.z, J.tmax);
                st.bump(kWSegs);
                return true;
            }
        }
        f3 acc = st.get3(kWThr);
        uint32_t rng = st.get(kWRng), depth = st.get(kWDepth);
        const float4 h = make_float4(best.t, __uint_as_float(best.prim), best.u, best.v);
        const bool nee = kNee && J.integrator == SOLRT_INTEGRATOR_PATH_NEE;
        f3 n_o{0.0f, 0.0f, 0.0f};
        float4 prev = make_float4(0.0f, 0.0f, 0.0f, 0.0f), prev_out = prev;
        if (nee && depth > 0u) {
            const f3 n = st.get3(kWPrev);
            prev = make_float4(n.x, n.y, n.z, st.getf(kWPrev + 3));
        }
        if (shade_step<kNee>(J, make_float4(org.x, org.y, org.z, tmin), make_float4(dir.x, dir.y, dir.z, J.tmax), h, acc,
                             rng, depth, o, d, ef, &n_o, prev, &prev_out)) {
            st.put3(kWThr, acc.x, acc.y, acc.z);
            st.put(kWDepth, depth);
            if (kOrg) st.put3(kWOrg, o.x, o.y, o.z);
            if constexpr (kNee) {
                if (nee) {
                    st.put3(kWPrev, prev_out.x, prev_out.y, prev_out.z);
                    st.putf(kWPrev + 3, prev_out.w);
                    float4 so, sd;
                    f3 c;
                    if (nee_sample(J.sc, f3{o.x, o.y, o.z}, n_o, acc, tmin, rng, so, sd, c)) {
                        st.put3(kWNext, d.x, d.y, d.z);
                        st.put3(kWLight, c.x, c.y, c.z);
                        d = sd;
                        this->any_hit = true;
                        st.bump(kWShadowSegs);
                    }
                }
            }
            st.put(kWRng, rng);
            st.put3(kWDir, d.x, d.y, d.z);
            if (!this->any_hit) st.bump(kWSegs);
            return true;
        }
        if (nee) acc = st.get3(kWSum) + acc;  // light terms in bounce order, then the end term
        const uint32_t slot = st.get(kWSlot);
        a.rad[slot] = make_float4(acc.x, acc.y, acc.z, 0.0f);
        if (J.rng_mode == SOLRT_RNG_REF_STREAM) {  // the pixel's next sample continues the stream
            const uint32_t pix = a.item.pix0 + unit;
            if (slot - unit * a.item.k + 1u < a.item.k) {
                start(pix, rng, slot + 1u, o, d);
                return true;
            }
            J.rng_state[pix] = rng;
        }
        return false;
    }
};

// Registers capped at 64 (1024 threads per SM): shading holds more than
// traversal does.
// kPlain: the small-scene loop (extend_bvh2_plain).
template <int KIND, bool kNee, bool kPlain>
__global__ void __launch_bounds__(256, SOLRT_PATH_MINB) k_paths(const __grid_constant__ PathArgs a) {
    PathIO<KIND, kNee> io(a);
    TraceCounters cnt{0, 0, 0};
    uint32_t ef = 0;
    if constexpr (kPlain) extend_bvh2_plain(io, a.units, a.work, stack_mem(a.slots, a.deep), cnt, ef);
    else extend_kind<KIND, false>(io, a.units, a.work, stack_mem(a.slots, a.deep), cnt, ef);
    if constexpr (kNee) {
        const TraceCounters sc{0u, 0u, io.st.get(kWShadow)};
        cnt.fallbacks -= sc.fallbacks;
        flush_traversal(a.stats + 1, sc, 0u, false);
        const uint32_t ws = __reduce_add_sync(0xffffffffu, io.st.get(kWShadowSegs));
        const uint32_t wu = __reduce_add_sync(0xffffffffu, io.st.get(kWShadowSegs + 1));
        if ((threadIdx.x & 31) == 0) {
            if (ws) atomicAdd(&a.stats[1].segments, (unsigned long long)ws);
            if (wu) atomicAdd(&a.stats[1].unoccluded, (unsigned long long)wu);
        }
    }
    flush_traversal(a.stats, cnt, ef, false);
    const uint32_t wsegs = __reduce_add_sync(0xffffffffu, io.st.get(kWSegs));
    if ((threadIdx.x & 31) == 0 && wsegs) atomicAdd(&a.stats->segments, (unsigned long long)wsegs);
    if (blockIdx.x == 0 && threadIdx.x == 0)
        atomicAdd(&a.stats->paths, (unsigned long long)a.item.npix * a.item.k);
    release_work(a.work);
}

template <int KIND, bool kNee, bool kPlain = false>
solrt_status launch_paths_kind(Context& ctx, PathArgs a) {
    LaunchShape s;
    SOLRT_TRY((launch_shape<KIND, k_paths<KIND, kNee, kPlain>>(ctx, path_words<KIND, kNee>(), a.units, false, s)));
    a.slots = s.slots;
    k_paths<KIND, kNee, kPlain><<<s.grid, s.block, s.smem, ctx.stream>>>(a);
    ++ctx.launches;
    SOLRT_CUDA(cudaGetLastError());
    return SOLRT_OK;
}

template <bool kNee>
solrt_status launch_paths_any(Context& ctx, uint32_t kind, const PathArgs& a) {
    ctx.last_kind = kind;
    switch (kind) {
        case SOLRT_BVH8_Q8: return launch_paths_kind<SOLRT_BVH8_Q8, kNee>(ctx, a);
        case SOLRT_BVH4_Q8: return launch_paths_kind<SOLRT_BVH4_Q8, kNee>(ctx, a);
        case SOLRT_BVH8_F32: return launch_paths_kind<SOLRT_BVH8_F32, kNee>(ctx, a);
        case SOLRT_BVH2_Q16: return launch_paths_kind<SOLRT_BVH2_Q16, kNee>(ctx, a);
        case SOLRT_BVH2_TWO_LEVEL: return launch_paths_kind<SOLRT_BVH2_TWO_LEVEL, kNee>(ctx, a);
        default:
            return a.job.sc.tri_count < kSmallScene ? launch_paths_kind<SOLRT_BVH2, kNee, true>(ctx, a)
                                                    : launch_paths_kind<SOLRT_BVH2, kNee>(ctx, a);
    }
}

// Queues one launch of the path kernel on the context stream (paths.cu,
// paths_nee.cu).
solrt_status launch_paths(Context& ctx, uint32_t kind, const PathArgs& a);
solrt_status launch_paths_nee(Context& ctx, uint32_t kind, const PathArgs& a);

}  // namespace solrt
