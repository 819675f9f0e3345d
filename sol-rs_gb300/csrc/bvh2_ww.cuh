// bvh2_ww.cuh — BVH2 traversal organised for SIMT efficiency.
//
// A warp keeps 32 rays in flight. Every step of its loop is warp-uniform
// (full-warp votes decide the phases), so lanes re-converge at each step:
//   refill  lanes whose ray has finished take new rays from the global queue
//           (one atomic per warp), once enough lanes are free (warp_feed);
//   nodes   lanes visit inner nodes, up to IO::kNodeSteps between two
//           votes, until every lane has parked a leaf or has no inner node
//           left, or until fewer than IO::kNodeMin lanes still have
//           inner nodes while others hold leaves; a lane that
//           already parked a leaf keeps descending until it reaches a second
//           one ("while-while" with speculative traversal, after Aila &
//           Laine, HPG 2009);
//   leaves  lanes test their parked leaves together.
// Each lane carries its own scene (IO::load), so one launch can serve rays of
// many scenes. The closest hit does not depend on visiting order, so results
// equal those of a plain per-ray loop.
#pragma once

#include "traverse.cuh"

namespace solrt {

constexpr int kBvh2Sentinel = 0x7fffffff;
// Inner nodes a lane may visit between two votes of its warp (IO::kNodeSteps,
// unrolled IO::kNodeUnroll times). The votes and the phase tests are about a
// quarter of a step's instructions: 4.2M incoherent rays through a 1M-triangle
// tree (32-byte nodes) take 2.47 / 2.26 / 2.20 / 2.20 ms with 1 / 2 / 3 / 4 steps,
// a 64-spp soup frame 121.4 / 117.7 / 116.2 ms with 2 / 3 / 4. Kernels that shade
// between traversals roll the loop: unrolled, the two no longer fit the
// instruction cache together (640x360 Cornell frame with per-pixel streams
// 2.62 ms unrolled, 2.31 as a loop of 8 steps; next-event estimation in a
// tunnel 1105 / 907 us).
//
// kNodeMin (kWideMin and kWideTriMin: the wide kinds, see bvh8_ww.cuh): the
// node phase ends early when fewer lanes have inner nodes to visit and some lane
// holds a leaf. refill: see warp_feed; a lane that only fetches its next ray
// should not wait long for it, one that shades in between should have company. 4.2M incoherent rays /
// a soup frame (16 spp) / a batch of 24 jobs: refill 16, kNodeMin 12 2160 us /
// 30.5 ms / 6.61 ms, 8 and 12 2075 / 30.1 / 6.48, 8 and 18 2023 / 29.6 / 6.22,
// 6 and 16 2013 / 29.5 / 6.27, 2 and 16 2018 / 29.8 / 6.30. Shading programs:
// an AO frame 4.66 ms with 16 and 12, 4.58 with 12 and 16; kWideMin 10 / 12 / 16
// a 64x48 preview through 8-wide nodes 53.8 / 54.8 / 56.9 us.
//
// kLeafMin: the leaf phase ends early when fewer lanes still hold a leaf and
// kNodeMin lanes have inner nodes (the rays with two or three leaves in a row
// then wait for the next leaf phase; below kNodeMin, so that the node phase has
// work). 1 / 4 / 8 / 13: 4.2M incoherent rays 1928 / 1865 / 1853 / 1854 us, a
// 64-spp soup frame 111.6 / 108.6 / 108.0 / 108.3 ms, next-event estimation in a
// tunnel 12.78 / 12.57 / 12.54 / 12.64 ms.
struct FetchLoop {
    static constexpr int kNodeSteps = 4, kNodeUnroll = 4, kNodeMin = 18, kLeafMin = 8;
    static constexpr int kWideMin = 16, kWideEnd = 6, kWideTriMin = 8;
    static constexpr int refill = 6;
};
struct ShadeLoop {
    static constexpr int kNodeSteps = 8, kNodeUnroll = 1, kNodeMin = 16, kLeafMin = 8;
    static constexpr int kWideMin = 10, kWideEnd = 6, kWideTriMin = 8;
};
constexpr int kShadeRefill = 12;

// A thread's traversal-stack memory: entry k at shared address base + k *
// stride for k < slots (stride = 4 x threads per block, so lanes at different
// depths hit different banks), the rest at deep[k * deep_stride] in global
// memory. A 1M-triangle tree's rays hold at most about 20 entries, so `deep` is
// hardly ever touched; it is global and not local memory because a local load
// cannot fault, so the compiler issues it for every pop, ahead of the test
// (4.2M incoherent rays through a 1M-triangle tree: 4.12 ms with local memory
// behind the shared slots, 3.19 with a ring of shared slots that spills,
// 2.95 with global memory behind them).
struct StackMem {
    uint32_t base;
    uint32_t stride;
    int slots;
    int* deep;
    uint32_t deep_stride;
    uint32_t ray;  // shared address of the thread's RayMem column (same stride)
    SOLRT_D RayMem ray_mem() const { return RayMem{ray, stride}; }
};

// Per-thread traversal stack of SOLRT_BVH2_STACK + 1 entries.
struct Bvh2Stack {
    StackMem m;
    SOLRT_D void put(int k, int v) {
        if (k < m.slots) sts_u32(m.base + (uint32_t)k * m.stride, (uint32_t)v);
        else m.deep[(size_t)((uint32_t)k * m.deep_stride)] = v;
    }
    SOLRT_D int get(int k) {
        if (k < m.slots) return (int)lds_u32(m.base + (uint32_t)k * m.stride);
        return m.deep[(size_t)((uint32_t)k * m.deep_stride)];
    }
};

// The 4 float4 of BVH2 node `node` (64-byte aligned) in two 256-bit loads.
SOLRT_D void load_bvh2_node(const float4* nodes, int node, float4& n0, float4& n1, float4& n2, int4& n3) {
    const float4* np = nodes + 4 * (size_t)node;
    float4 r;
    ldg_2x4(np, n0, n1);
    ldg_2x4(np + 2, n2, r);
    n3 = make_int4(__float_as_int(r.x), __float_as_int(r.y), __float_as_int(r.z), __float_as_int(r.w));
}

// A ray's constants of the slab test: (1/d, -o/d) per axis for FP32 nodes,
// (c/d, (G - o)/d - 2^23 c/d) for BVH2-q16 nodes (q16_ray).
template <bool kQ16>
struct RayBox {
    float ix, iy, iz, nox, noy, noz;
    SOLRT_D void set(const float4* nodes, float ox, float oy, float oz, float dx, float dy, float dz) {
        if constexpr (kQ16) {
            q16_ray(nodes, ox, oy, oz, dx, dy, dz, ix, iy, iz, nox, noy, noz);
        } else {
            ix = box_rcp(box_dir(dx));
            iy = box_rcp(box_dir(dy));
            iz = box_rcp(box_dir(dz));
            nox = -(ox * ix);
            noy = -(oy * iy);
            noz = -(oz * iz);
        }
    }
};

// One node test in either node format (kQ16: 32-byte BVH2-q16 nodes, one
// 256-bit load; else 64-byte FP32 nodes, two).
template <bool kQ16>
SOLRT_D void bvh2_node_step(const float4* nodes, int node, const RayBox<kQ16>& r, float tmin, float tmax, bool& h0,
                            float& t0, bool& h1, float& t1, int& ref0, int& ref1) {
    if constexpr (kQ16) {
        float4 a, b;
        ldg_2x4(nodes + 2 + 2 * (size_t)node, a, b);
        slab2_q16(a, b, r.ix, r.iy, r.iz, r.nox, r.noy, r.noz, tmin, tmax, h0, t0, h1, t1);
        ref0 = __float_as_int(a.x);
        ref1 = __float_as_int(a.y);
    } else {
        float4 n0, n1, n2;
        int4 n3;
        load_bvh2_node(nodes, node, n0, n1, n2, n3);
        slab2_fma(n0, n1, n2, r.ix, r.iy, r.iz, r.nox, r.noy, r.noz, tmin, tmax, h0, t0, h1, t1);
        ref0 = n3.x;
        ref1 = n3.y;
    }
}

template <class IO, bool kCount, bool kQ16 = false>
SOLRT_D void extend_bvh2_ww(IO& io, uint32_t n, unsigned int* work, const StackMem& mem, TraceCounters& cnt,
                            uint32_t& ef) {
    Bvh2Stack stack;
    stack.m = mem;
    const RayMem rm = mem.ray_mem();
    int sp = 0;
    int node = kBvh2Sentinel;  // >= 0 inner node, < 0 leaf ~k, sentinel = nothing left
    int leaf = 0;              // parked leaf (< 0) or none (>= 0)
    bool has = false;
    bool drained = false;      // the queue has no more rays for this warp
    uint32_t budget = 0;
    TravScene ts = io.first_scene();
    RayBox<kQ16> rb{};
    float tmin = 0.0f, best_t = 0.0f;
    for (;;) {
        // no inner node (an index past the last one counts as none) and no leaf
        const bool idle = (unsigned)node >= ts.node_count && node >= 0 && leaf >= 0;
        if (idle && node != kBvh2Sentinel) {
            ef |= SOLRT_EFLAG_INDEX;
            node = kBvh2Sentinel;
        }
        float4 o, d;
        if (warp_feed(io, idle, has, drained, rm, n, work, tmin, best_t, o, d, ts, cnt, ef)) {
            rm.set_ray(o.x, o.y, o.z, d.x, d.y, d.z);
            rm.clear_hit();
            if (ts.tri_count) rb.set(ts.nodes, o.x, o.y, o.z, d.x, d.y, d.z);
            tmin = o.w;
            best_t = d.w;
            budget = 2u * (ts.node_count + ts.tri_count) + 64u;
            stack.put(0, kBvh2Sentinel);
            sp = 1;
            node = ts.tri_count ? 0 : kBvh2Sentinel;
            leaf = 0;
        }
        if (!__any_sync(0xffffffffu, has)) {
            if (drained) break;
            continue;
        }
        // node phase
        for (;;) {
            // two ballots decide the phase: stop when no lane without a
            // parked leaf has inner nodes, or when few lanes still have inner
            // nodes while others hold leaves (test the leaves first; the leaf
            // phase then has work, so this ends)
            const bool inner = (unsigned)node < ts.node_count;
            const uint32_t b_inner = __ballot_sync(0xffffffffu, inner);
            const uint32_t b_leaf = __ballot_sync(0xffffffffu, leaf < 0);
            if ((b_inner & ~b_leaf) == 0u) break;
            if (__popc(b_inner) < IO::kNodeMin && b_leaf) break;
            if (!inner) continue;
            if (--budget == 0u) {
                ef |= SOLRT_EFLAG_INDEX;
                node = kBvh2Sentinel;
                leaf = 0;
                continue;
            }
            constexpr int kUnroll = IO::kNodeUnroll;
#pragma unroll kUnroll
            for (int u = 0; u < IO::kNodeSteps; ++u) {
                if (u > 0 && (unsigned)node >= ts.node_count) break;
                if (kCount) ++cnt.nodes;
                float t0, t1;
                bool h0, h1;
                int c0, c1;
                bvh2_node_step<kQ16>(ts.nodes, node, rb, tmin, best_t, h0, t0, h1, t1, c0, c1);
                // nearer child first; the other one, when hit too, is pushed
                const bool first0 = h0 && (!h1 || !(t1 < t0));
                node = first0 ? c0 : c1;
                if (h0 && h1) {
                    if (sp <= SOLRT_BVH2_STACK) stack.put(sp++, first0 ? c1 : c0);
                    else ef |= SOLRT_EFLAG_STACK;
                } else if (!h0 && !h1) {
                    node = stack.get(--sp);
                }
                if (node < 0 && leaf >= 0) {  // park the leaf, keep descending
                    leaf = node;
                    node = stack.get(--sp);
                }
            }
        }
        // leaf phase
        for (;;) {
            const uint32_t b_leaf = __ballot_sync(0xffffffffu, leaf < 0);
            if (b_leaf == 0u) break;
            // (the node phase then has kNodeMin lanes, most of them without a
            // leaf, and takes a step)
            if (__popc(b_leaf) < IO::kLeafMin &&
                __popc(__ballot_sync(0xffffffffu, (unsigned)node < ts.node_count)) >= IO::kNodeMin)
                break;
            if (leaf < 0) {
                const uint32_t k = (uint32_t)(~leaf);
                if (--budget == 0u || k >= ts.tri_count) {
                    ef |= SOLRT_EFLAG_INDEX;
                    node = kBvh2Sentinel;
                    leaf = 0;
                } else {
                    const float4* tp = ts.tris + 3 * (size_t)k;
                    if (kCount) ++cnt.tris;
                    if (intersect_tri(rm, tmin, __ldg(tp), __ldg(tp + 1), __ldg(tp + 2), best_t, cnt.fallbacks) &&
                        io.any_hit) {  // occlusion query: done at the first hit
                        node = kBvh2Sentinel;
                        leaf = 0;
                    } else {
                        leaf = node;
                        if (node < 0) node = stack.get(--sp);
                    }
                }
            }
        }
    }
}

// One ray, plain depth-first loop (nearer child first): the traversal of the
// per-pixel megakernel.
template <bool kQ16 = false>
SOLRT_D void trace_bvh2_ray(const TravScene& ts, float ox, float oy, float oz, float dx, float dy, float dz,
                            float tmin, float tmax, HitRec& best, TraceCounters& cnt, uint32_t& ef) {
    best = HitRec{tmax, SOLRT_NO_HIT, 0.0f, 0.0f};
    if (ts.tri_count == 0) return;
    const RayWT r = setup_ray(ox, oy, oz, dx, dy, dz, tmin);
    RayBox<kQ16> rb;
    rb.set(ts.nodes, ox, oy, oz, dx, dy, dz);
    int stack[SOLRT_BVH2_STACK + 1];
    stack[0] = kBvh2Sentinel;
    int sp = 1;
    int node = 0;
    uint32_t budget = 2u * (ts.node_count + ts.tri_count) + 64u;
    while (node != kBvh2Sentinel) {
        if (--budget == 0u) {
            ef |= SOLRT_EFLAG_INDEX;
            return;
        }
        if (node >= 0) {
            if ((uint32_t)node >= ts.node_count) {
                ef |= SOLRT_EFLAG_INDEX;
                return;
            }
            float t0, t1;
            bool h0, h1;
            int c0, c1;
            bvh2_node_step<kQ16>(ts.nodes, node, rb, tmin, best.t, h0, t0, h1, t1, c0, c1);
            if (h0 && h1) {
                const bool swap = t1 < t0;
                if (sp <= SOLRT_BVH2_STACK) stack[sp++] = swap ? c0 : c1;
                else ef |= SOLRT_EFLAG_STACK;
                node = swap ? c1 : c0;
                continue;
            }
            if (h0) { node = c0; continue; }
            if (h1) { node = c1; continue; }
        } else {
            const uint32_t k = (uint32_t)(~node);
            if (k >= ts.tri_count) {
                ef |= SOLRT_EFLAG_INDEX;
                return;
            }
            const float4* tp = ts.tris + 3 * (size_t)k;
            cnt.fallbacks += intersect_tri(r, __ldg(tp), __ldg(tp + 1), __ldg(tp + 2), best);
        }
        node = stack[--sp];
    }
}

// The queue loop for small scenes: every lane of a warp traces its ray to the
// end with trace_bvh2_ray, then all of them go on together (warp_feed). A ray
// visits a dozen nodes there and the lanes differ little, so votes and parked
// leaves cost more than they save.
template <class IO>
SOLRT_D void extend_bvh2_plain(IO& io, uint32_t n, unsigned int* work, const StackMem& mem, TraceCounters& cnt,
                               uint32_t& ef) {
    const RayMem rm = mem.ray_mem();
    const TravScene scene = io.first_scene();
    bool has = false, drained = false;
    float tmin = 0.0f, best_t = 0.0f;
    for (;;) {
        float4 o, d;
        TravScene ts = scene;
        const bool fresh = warp_feed(io, true, has, drained, rm, n, work, tmin, best_t, o, d, ts, cnt, ef);
        if (!__any_sync(0xffffffffu, has)) {
            if (drained) break;
            continue;
        }
        if (fresh) {
            HitRec best;
            trace_bvh2_ray(scene, o.x, o.y, o.z, d.x, d.y, d.z, o.w, d.w, best, cnt, ef);
            tmin = o.w;
            best_t = best.t;
            rm.put(kRayPrim, best.prim);
            rm.putf(kRayU, best.u);
            rm.putf(kRayV, best.v);
        }
        __syncwarp();
    }
}

}  // namespace solrt
