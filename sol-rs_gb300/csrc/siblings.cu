// siblings.cu — the reference's sibling ray-tracing pipelines over the same
// traversal: DEBUG (debug.rgen / .rchit / .rmiss) and AO (ao.rgen / .rchit /
// .rmiss).
//
// Their shaders run one invocation per pixel, and so do k_debug and k_ao_plain.
// AO frames of large scenes run k_ao instead (ao_plain, below): a persistent
// launch that holds 32 pixels per warp in the traversal loop of the BVH kind
// (warp_feed), where lanes whose ray is done shade and go on with their pixel's
// next ray or sample, or take another pixel, instead of waiting for the warp's
// longest chain: a 1280x720 frame (4 samples) of a 300k-triangle soup 7.1 -> 4.4
// ms.
#include "extend.cuh"
#include "path_ops.cuh"

namespace solrt {

namespace {

struct SiblingArgs {
    DevJob job;
    uint32_t units, slots;
    unsigned int* work;
    int* deep;
    DevStats* stats;
};

// Primary direction of debug.rgen:20-27 / ao.rgen:56-61 for pixel position
// (px, py): origin and direction through the inverse matrices.
SOLRT_D void pixel_ray(const DevJob& J, float px, float py, float4& o, float4& d) {
    const float ux = px / __uint2float_rn(J.width), uy = py / __uint2float_rn(J.height);
    const float dx = ux * 2.0f - 1.0f, dy = uy * 2.0f - 1.0f;
    float org[4], tgt[4], dir[4];
    mat4_mul(J.vinv, 0.0f, 0.0f, 0.0f, 1.0f, org);
    mat4_mul(J.pinv, dx, dy, 1.0f, 1.0f, tgt);
    const f3 tn = normalize(f3{tgt[0], tgt[1], tgt[2]});
    mat4_mul(J.vinv, tn.x, tn.y, tn.z, 0.0f, dir);
    o = make_float4(org[0], org[1], org[2], 0.0f);
    d = make_float4(dir[0], dir[1], dir[2], 0.0f);
}

// State words: the ray in flight and the rays traced by this thread, then
// those of AO.
enum SiblingWord {
    kSDir = 0,
    kSOrg = 3,
    kSSegs = 6,
    kSRng = 7,
    kSDepth = 8,    // hits so far
    kSSample = 9,   // sample of the pixel
    kSHits = 10,    // occlusions of the sample
    kSSum = 11,     // occlusion sum over the pixel's samples
    kSWords = 12,
};

// Statistics of a thread that traced `segs` rays of its pixel.
SOLRT_D void flush_plain(const SiblingArgs& a, const TraceCounters& cnt, uint32_t ef, uint32_t segs, uint32_t paths) {
    flush_traversal(a.stats, cnt, ef, false);
    const uint32_t ws = __reduce_add_sync(0xffffffffu, segs);
    if ((threadIdx.x & 31) == 0 && ws) atomicAdd(&a.stats->segments, (unsigned long long)ws);
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(&a.stats->paths, (unsigned long long)a.units * paths);
}

// debug.rgen:18-36, debug.rchit:9-13, debug.rmiss: barycentrics of the
// primary hit through the pixel centre, else the ray direction; stored
// without accumulation (imageStore of vec4(hitValue, 0)).
SOLRT_D void debug_ray(const DevJob& J, uint32_t pix, float4& o, float4& d) {
    const uint32_t x = pix % J.width, y = pix / J.width;
    pixel_ray(J, __uint2float_rn(x) + 0.5f, __uint2float_rn(y) + 0.5f, o, d);
    o.w = 0.001f;
    d.w = 1000.0f;
}
SOLRT_D void debug_write_pixel(const DevJob& J, uint32_t pix, const HitRec& h, f3 dir) {
    float4 v = make_float4(dir.x, dir.y, dir.z, 0.0f);
    if (h.prim != SOLRT_NO_HIT) v = make_float4((1.0f - h.u) - h.v, h.u, h.v, 0.0f);
    J.accum[pix] = v;
    J.rgba8[pix] = make_uchar4(to_unorm8(v.x), to_unorm8(v.y), to_unorm8(v.z), 0);
}

template <int KIND>
__global__ void __launch_bounds__(128, 1) k_debug(const __grid_constant__ SiblingArgs a) {
    const uint32_t pix = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t ef = 0;
    TraceCounters cnt{0, 0, 0};
    if (pix < a.units) {
        float4 o, d;
        debug_ray(a.job, pix, o, d);
        HitRec h;
        trace_one<KIND>(trav_scene(a.job.sc), o, d, h, cnt, ef);
        debug_write_pixel(a.job, pix, h, f3{d.x, d.y, d.z});
    }
    flush_plain(a, cnt, ef, pix < a.units ? 1u : 0u, 1u);
}

// ao.rgen:37-83, ao.rchit:53-88, ao.rmiss: `spp` jittered samples; each
// follows cosine-weighted rays (directions from the blue-noise texture)
// until a miss or max_bounces + 1 hits, counting every hit after the first.

// The camera ray of a sample (ao.rgen:53-72).
SOLRT_D void ao_camera_ray(const DevJob& J, uint32_t pix, uint32_t& rng, float4& o, float4& d) {
    const uint32_t x = pix % J.width, y = pix / J.width;
    const float j0 = next_rand(rng);                                          // nextRand2 (ao.rgen:53)
    const float j1 = next_rand(rng);
    pixel_ray(J, __uint2float_rn(x) + j0, __uint2float_rn(y) + j1, o, d);
    o.w = glsl_max(1.0f, length(f3{o.x, o.y, o.z})) * 1e-3f;                  // preparePayload
    d.w = 10000.0f;
}

// The ray that leaves hit `h` of the ray along `dir`, the depth-th of a sample
// (ao.rchit:53-88). False for a miss (or a bad index): the sample ends.
SOLRT_D bool ao_bounce(const DevJob& J, uint32_t pix, uint32_t sample, uint32_t depth, const HitRec& h, f3 dir,
                       uint32_t& rng, float4& o, float4& d, uint32_t& ef) {
    const DevScene& sc = J.sc;
    if (h.prim == SOLRT_NO_HIT) return false;                                 // ao.rmiss
    if (h.prim >= sc.tri_count) {
        ef |= SOLRT_EFLAG_INDEX;
        return false;
    }
    const uint32_t x = pix % J.width, y = pix / J.width;
    const uint4 ti = __ldg(sc.tri_idx + h.prim);
    const float b1 = h.u, b2 = h.v;
    const float b0 = (1.0f - b1) - b2;
    f3 normal, pos;
    hit_frame(sc, ti, b0, b1, b2, normal, pos);                               // ao.rchit:66-75
    const f3 no = pos + 0.00001f * dir;                                       // ao.rchit:78
    // getBlueRand2(depth + depth * sampleId) (ao.rchit:43-49)
    const uint32_t bi = (depth + depth * sample) & 3u;
    const float r0 = next_rand(rng);
    const float r1 = next_rand(rng);
    const float tw = __uint2float_rn(J.noise_w), th = __uint2float_rn(J.noise_h);
    float cx = __uint2float_rn(x) + r0 * tw, cy = __uint2float_rn(y) + r1 * th;
    cx = cx - tw * floorf(cx / tw);                                           // GLSL mod
    cy = cy - th * floorf(cy / th);
    const int ix = min(max((int)cx, 0), (int)J.noise_w - 1);
    const int iy = min(max((int)cy, 0), (int)J.noise_h - 1);
    const uchar4 t = __ldg(J.noise + (size_t)iy * J.noise_w + ix);
    const uint32_t u0 = bi == 0 ? t.x : bi == 1 ? t.y : bi == 2 ? t.z : t.w;
    const uint32_t u1 = bi == 0 ? t.y : bi == 1 ? t.z : bi == 2 ? t.w : t.x;
    const f3 hit_n = normal * glsl_sign(dot(-dir, normal));
    const f3 nd = sample_cosine(hit_n, __uint2float_rn(u0) / 255.0f, __uint2float_rn(u1) / 255.0f);
    o = make_float4(no.x, no.y, no.z, 0.001f);
    d = make_float4(nd.x, nd.y, nd.z, 10.0f);
    return true;
}

// The pixel's occlusion sum after a sample of `hits` occlusions (ao.rgen:77).
SOLRT_D float ao_add_sample(const DevJob& J, float sum, float hits) {
    return sum + (1.0f / __uint2float_rn(J.max_bounces)) * hits;
}

// The images of pixel pix from its occlusion sum (ao.rgen:79-82).
SOLRT_D void ao_write_pixel(const DevJob& J, uint32_t pix, float sum) {
    const float c = 1.0f - sum / __uint2float_rn(J.spp);
    f3 color{c, c, c};
    const float w = 1.0f / __uint2float_rn(J.frame - J.start + 1u);
    const float4 old = J.accum[pix];
    color = mix(f3{old.x, old.y, old.z}, color, w);
    J.accum[pix] = make_float4(color.x, color.y, color.z, 1.0f);
    J.rgba8[pix] = make_uchar4(to_unorm8(color.x), to_unorm8(color.y), to_unorm8(color.z), 255);
}

struct AoIO : ShadeLoop {
    const SiblingArgs& a;
    const StateMem st;
    static constexpr int lanes = 32, refill = kShadeRefill;
    static constexpr bool any_hit = false;
    SOLRT_D explicit AoIO(const SiblingArgs& args) : a(args), st(args.slots) { st.put(kSSegs, 0u); }
    SOLRT_D TravScene first_scene() const { return trav_scene(a.job.sc); }
    SOLRT_D void load_ray(uint32_t, float4& o, float4& d) const {
        const f3 p = st.get3(kSOrg), q = st.get3(kSDir);
        o = make_float4(p.x, p.y, p.z, 0.0f);
        d = make_float4(q.x, q.y, q.z, 0.0f);
    }
    SOLRT_D void keep_ray(const float4& o, const float4& d) const {
        st.put3(kSOrg, o.x, o.y, o.z);
        st.put3(kSDir, d.x, d.y, d.z);
        st.bump(kSSegs);
    }
    SOLRT_D void start(uint32_t pix, uint32_t sample, uint32_t rng, float4& o, float4& d) const {
        ao_camera_ray(a.job, pix, rng, o, d);
        st.put(kSRng, rng);
        st.put(kSDepth, 0u);
        st.put(kSSample, sample);
        st.putf(kSHits, 0.0f);
        keep_ray(o, d);
    }
    SOLRT_D void load(uint32_t pix, float4& o, float4& d, TravScene&) const {
        st.putf(kSSum, 0.0f);
        start(pix, 0u, tea(pix, a.job.frame), o, d);                          // ao.rgen:49
    }
    SOLRT_D bool next(uint32_t pix, float, const HitRec& h, float4& o, float4& d, const TraceCounters&,
                      uint32_t& ef) const {
        const DevJob& J = a.job;
        const uint32_t sample = st.get(kSSample);
        uint32_t rng = st.get(kSRng), depth = st.get(kSDepth);
        if (ao_bounce(J, pix, sample, depth, h, st.get3(kSDir), rng, o, d, ef)) {
            if (depth > 0) st.putf(kSHits, st.getf(kSHits) + 1.0f);
            ++depth;
            if (depth <= J.max_bounces) {                                     // ao.rgen:75
                st.put(kSRng, rng);
                st.put(kSDepth, depth);
                keep_ray(o, d);
                return true;
            }
        }
        const float sum = ao_add_sample(J, st.getf(kSSum), st.getf(kSHits));
        if (sample + 1u < J.spp) {
            st.putf(kSSum, sum);
            start(pix, sample + 1u, rng, o, d);
            return true;
        }
        ao_write_pixel(J, pix, sum);
        return false;
    }
};

// AO with one thread per pixel, 8 blocks per SM (64 registers).
template <int KIND>
__global__ void __launch_bounds__(128, 8) k_ao_plain(const __grid_constant__ SiblingArgs a) {
    const DevJob& J = a.job;
    const uint32_t pix = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t segs = 0, ef = 0;
    TraceCounters cnt{0, 0, 0};
    if (pix < a.units) {
        const TravScene ts = trav_scene(J.sc);
        uint32_t rng = tea(pix, J.frame);                                     // ao.rgen:49
        float sum = 0.0f;
        for (uint32_t i = 0; i < J.spp; ++i) {
            float4 o, d;
            ao_camera_ray(J, pix, rng, o, d);
            float hits = 0.0f;
            for (uint32_t depth = 0; depth <= J.max_bounces; ++depth) {       // ao.rgen:75
                HitRec h;
                trace_one<KIND>(ts, o, d, h, cnt, ef);
                ++segs;
                if (!ao_bounce(J, pix, i, depth, h, f3{d.x, d.y, d.z}, rng, o, d, ef)) break;
                if (depth > 0) hits = hits + 1.0f;
            }
            sum = ao_add_sample(J, sum, hits);
        }
        ao_write_pixel(J, pix, sum);
    }
    flush_plain(a, cnt, ef, segs, J.spp);
}

template <int KIND>
__global__ void __launch_bounds__(256, 4) k_ao(const __grid_constant__ SiblingArgs a) {
    AoIO io(a);
    TraceCounters cnt{0, 0, 0};
    uint32_t ef = 0;
    extend_kind<KIND, false>(io, a.units, a.work, stack_mem(a.slots, a.deep), cnt, ef);
    flush_traversal(a.stats, cnt, ef, false);
    const uint32_t segs = __reduce_add_sync(0xffffffffu, io.st.get(kSSegs));
    if ((threadIdx.x & 31) == 0 && segs) atomicAdd(&a.stats->segments, (unsigned long long)segs);
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(&a.stats->paths, (unsigned long long)a.units * a.job.spp);
    release_work(a.work);
}

template <int KIND>
solrt_status launch_kind(const Context& ctx, SiblingArgs a, bool plain) {
    const uint32_t blocks = (a.units + 127) / 128;
    if (a.job.integrator != SOLRT_INTEGRATOR_AO) {
        k_debug<KIND><<<blocks, 128, 0, ctx.stream>>>(a);
    } else if (plain) {
        k_ao_plain<KIND><<<blocks, 128, 0, ctx.stream>>>(a);
    } else {
        LaunchShape s;
        SOLRT_TRY((launch_shape<KIND, k_ao<KIND>>(ctx, kSWords, a.units, false, s)));
        a.slots = s.slots;
        k_ao<KIND><<<s.grid, s.block, s.smem, ctx.stream>>>(a);
    }
    return SOLRT_OK;
}

}  // namespace

// Whether a frame runs one thread per pixel. Always for DEBUG: its one ray per
// pixel leaves no chain to wait for, and neighbouring camera rays stay together
// in a plain loop (1280x720, three frames in flight, per pixel / persistent: a
// 300k-triangle tube 112 / 147 us, a 300k soup 297 / 251). For AO the
// persistent launch pays once traversals are long: a soup ends its chains at
// many lengths, a tube hardly, and what its refills cost in coherence there
// shrinks with the size of the tree (640x360, 4 samples, us: tubes of 5k
// triangles 830 / 1088, 50k 1294 / 1584, 300k 2105 / 2179, 1M 2571 / 2629;
// soups 1007 / 802, 1584 / 1187, 1927 / 1430, 2140 / 1560; 320x180 of the 300k
// tube 653 / 577). Frames of few pixels leave the GPU idle either way and take
// the shorter steps of the plain loop (64x48 of a tube 134 / 160).
bool sibling_plain(const Scene& sc, const solrt_render_params& p) {
    return p.integrator != SOLRT_INTEGRATOR_AO || sc.tri_count < 196608u || (uint64_t)p.width * p.height <= 16384u;
}

solrt_status launch_sibling(Context& ctx, uint32_t kind, const DevJob& J, bool plain) {
    ctx.last_kind = kind;
    const SiblingArgs a{J, J.width * J.height, 0, ctx.trace_work.as<unsigned int>(), ctx.deep_stack.as<int>(),
                        ctx.stats.as<DevStats>()};
    switch (kind) {
        case SOLRT_BVH8_Q8: SOLRT_TRY(launch_kind<SOLRT_BVH8_Q8>(ctx, a, plain)); break;
        case SOLRT_BVH4_Q8: SOLRT_TRY(launch_kind<SOLRT_BVH4_Q8>(ctx, a, plain)); break;
        case SOLRT_BVH8_F32: SOLRT_TRY(launch_kind<SOLRT_BVH8_F32>(ctx, a, plain)); break;
        case SOLRT_BVH2_Q16: SOLRT_TRY(launch_kind<SOLRT_BVH2_Q16>(ctx, a, plain)); break;
        case SOLRT_BVH2_TWO_LEVEL: SOLRT_TRY(launch_kind<SOLRT_BVH2_TWO_LEVEL>(ctx, a, plain)); break;
        default: SOLRT_TRY(launch_kind<SOLRT_BVH2>(ctx, a, plain)); break;
    }
    ++ctx.launches;
    SOLRT_CUDA(cudaGetLastError());
    return SOLRT_OK;
}

}  // namespace solrt
