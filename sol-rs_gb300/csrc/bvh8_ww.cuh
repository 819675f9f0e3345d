// bvh8_ww.cuh — traversal of the 8-wide quantised BVH (bvh8.cuh) organised
// like bvh2_ww.cuh: a warp keeps 32 rays in flight and every step of its loop
// is warp-uniform.
//   refill  lanes whose ray has finished take new rays from the global queue
//           once enough lanes are free (warp_feed);
//   nodes   lanes visit one 8-wide node per step: the nearest remaining
//           internal child of their current node group (octant order), pushing
//           the rest of the group; the node's hit internal children become the
//           new group and its hit triangles are parked. A lane goes on until it
//           holds the triangles of two nodes. The phase ends when no lane can
//           step, or when fewer than IO::kWideMin lanes can while others hold
//           triangles;
//   leaves  lanes test their parked triangles, one per step, until none has any
//           left, or fewer than IO::kWideTriMin have while kWideMin lanes could
//           step again.
// Every other node visit finds triangles (tunnel scene: 14 nodes and 8 triangles
// per ray), so with one parked node and leaf phases that ran to their end 13 of
// 32 lanes were active on average. A 1366x768 tunnel frame (16 spp): 64.8 ms so,
// 60.7 with the threshold in the leaf phase, 58.0 with a second parked node as
// well, 55.3 at 64 registers a thread (traverse_min_blocks); 4.2M incoherent
// rays 2.79 / 2.66 / 2.77 / 2.56 ms. Once the queue is empty kWideEnd takes the
// place of kWideMin, which few warps reach any more: calls of 20k and 80k rays
// 43.7 -> 42.6 and 24.5 -> 22.9 us (three in flight; 4.2M rays 2.56 -> 2.59 ms).
// The child-box tests are those of trace_bvh8 (bvh8_traverse.cuh: quantised
// or, for SOLRT_BVH8_F32, full-precision nodes), so the closest hit equals
// that of the per-ray loop.
#pragma once

#include "bvh2_ww.cuh"
#include "bvh8_traverse.cuh"

namespace solrt {


// The stack of node groups is in local memory (kept in shared memory it
// was 1-7 % slower: the groups are 8 bytes and rarely popped).
template <class IO, bool kCount, bool kF32 = false>
SOLRT_D void extend_bvh8_ww(IO& io, uint32_t n, unsigned int* work, const StackMem& mem, TraceCounters& cnt,
                            uint32_t& ef) {
    uint2 stack[SOLRT_BVH8_STACK];
    int sp = 0;
    uint2 grp = make_uint2(0u, 0u);   // (child base, hit bits << 24 | internal mask)
    uint2 tgrp = make_uint2(0u, 0u);  // parked triangles: (triangle base, hit bits)
    uint2 tmore = make_uint2(0u, 0u); // those of a second node (only beside the first)
    bool has = false;
    bool drained = false;
    uint32_t budget = 0, oct = 0;
    bool negx = false, negy = false, negz = false;
    const RayMem rm = mem.ray_mem();
    float ox = 0.0f, oy = 0.0f, oz = 0.0f, tmin = 0.0f, best_t = 0.0f;
    TravScene ts = io.first_scene();
    float ix = 0.0f, iy = 0.0f, iz = 0.0f;
    float nox = 0.0f, noy = 0.0f, noz = 0.0f;  // -o / box_dir(d) (FP32 nodes)
    const uint4* nodes = nullptr;
    for (;;) {
        const bool idle = (grp.y >> 24) == 0u && sp == 0 && tgrp.y == 0u;
        float4 o, d;
        if (warp_feed(io, idle, has, drained, rm, n, work, tmin, best_t, o, d, ts, cnt, ef)) {
            rm.set_ray(o.x, o.y, o.z, d.x, d.y, d.z);
            rm.clear_hit();
            ox = o.x;
            oy = o.y;
            oz = o.z;
            tmin = o.w;
            best_t = d.w;
            const float bx = box_dir(d.x), by = box_dir(d.y), bz = box_dir(d.z);
            ix = box_rcp(bx);
            iy = box_rcp(by);
            iz = box_rcp(bz);
            negx = signbit(bx);
            negy = signbit(by);
            negz = signbit(bz);
            nox = -(o.x * ix);
            noy = -(o.y * iy);
            noz = -(o.z * iz);
            oct = (negx ? 1u : 0u) | (negy ? 2u : 0u) | (negz ? 4u : 0u);
            budget = 2u * (ts.node_count + ts.tri_count) + 64u;
            nodes = reinterpret_cast<const uint4*>(ts.nodes);
            sp = 0;
            tgrp = tmore = make_uint2(0u, 0u);
            // the root as a group of one internal child in slot 0
            grp = ts.tri_count ? make_uint2(0u, (1u << (24u + oct)) | 1u) : make_uint2(0u, 0u);
        }
        if (!__any_sync(0xffffffffu, has)) {
            if (drained) break;
            continue;
        }
        const int node_min = drained ? IO::kWideEnd : IO::kWideMin;
        // node phase
        for (;;) {
            const bool want = tmore.y == 0u && ((grp.y >> 24) != 0u || sp > 0);
            const uint32_t wb = __ballot_sync(0xffffffffu, want);
            if (wb == 0u) break;
            if (__popc(wb) < node_min && __any_sync(0xffffffffu, tgrp.y != 0u)) break;
            if (want) {
                if ((grp.y >> 24) == 0u) grp = stack[--sp];
                const uint32_t j = (uint32_t)(__ffs(grp.y >> 24) - 1);
                grp.y &= ~(1u << (24u + j));
                const uint32_t s = j ^ oct;
                const uint32_t node = grp.x + (uint32_t)__popc(grp.y & ((1u << s) - 1u) & 0xffu);
                if (grp.y >> 24) {
                    if (sp < SOLRT_BVH8_STACK) stack[sp++] = grp;
                    else ef |= SOLRT_EFLAG_STACK;
                }
                grp = make_uint2(0u, 0u);
                if (--budget == 0u || node >= ts.node_count) {
                    ef |= SOLRT_EFLAG_INDEX;
                    sp = 0;
                } else {
                    if (kCount) ++cnt.nodes;
                    uint32_t hi = 0, ht = 0, tbase = 0;
                    if constexpr (kF32) {
                        uint32_t cbase = 0, imask = 0;
                        bvh8f_node_test(ts.nodes + 14 * (size_t)node, ix, iy, iz, nox, noy, noz, oct, tmin, best_t,
                                        hi, ht, cbase, tbase, imask);
                        if (hi) grp = make_uint2(cbase, (hi << 24) | imask);
                    } else {
                        const uint4* np = nodes + 5 * (size_t)node;
                        const uint4 w0 = __ldg(np), w1 = __ldg(np + 1), w2 = __ldg(np + 2), w3 = __ldg(np + 3),
                                    w4 = __ldg(np + 4);
                        bvh8_node_test(w0, w1, w2, w3, w4, ox, oy, oz, ix, iy, iz, negx, negy, negz, oct,
                                       tmin, best_t, hi, ht);
                        if (hi) grp = make_uint2(w1.x, (hi << 24) | (w0.w >> 24));
                        tbase = w1.y;
                    }
                    if (ht) {
                        if (tgrp.y) tmore = make_uint2(tbase, ht);
                        else tgrp = make_uint2(tbase, ht);
                    }
                }
            }
        }
        // leaf phase
        for (;;) {
            const uint32_t tb = __ballot_sync(0xffffffffu, tgrp.y != 0u);
            if (tb == 0u) break;
            // (the node phase then has node_min lanes and takes a step)
            if (__popc(tb) < IO::kWideTriMin &&
                __popc(__ballot_sync(0xffffffffu, tmore.y == 0u && ((grp.y >> 24) != 0u || sp > 0))) >= node_min)
                break;
            if (tgrp.y) {
                const uint32_t k = (uint32_t)(__ffs(tgrp.y) - 1);
                tgrp.y &= tgrp.y - 1u;
                const uint32_t ti = tgrp.x + k;
                if (--budget == 0u || ti >= ts.tri_count) {
                    ef |= SOLRT_EFLAG_INDEX;
                    tgrp.y = tmore.y = 0u;
                    grp = make_uint2(0u, 0u);
                    sp = 0;
                } else {
                    const float4* tp = ts.tris + 3 * (size_t)ti;
                    if (kCount) ++cnt.tris;
                    if (intersect_tri(rm, tmin, __ldg(tp), __ldg(tp + 1), __ldg(tp + 2), best_t, cnt.fallbacks) &&
                        io.any_hit) {  // occlusion query: done at the first hit
                        tgrp.y = tmore.y = 0u;
                        grp = make_uint2(0u, 0u);
                        sp = 0;
                    }
                }
                if (tgrp.y == 0u) {
                    tgrp = tmore;
                    tmore.y = 0u;
                }
            }
        }
    }
}

}  // namespace solrt
