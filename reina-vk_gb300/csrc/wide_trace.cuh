// Traversal with eight lanes per ray, for launches of few rays.
//
// What such a launch takes is the longest ray's chain of node visits (66 of them among 128 rays of the 1.3M-triangle
// scene: 52 us cooperative, 40 us here), and a visit is shorter when a lane tests one child box and then one of
// the node's triangles instead of eight boxes.  Up to four rays per warp, each group of eight lanes holding its ray's
// state; the next node is on its way before the current one's triangles are tested.  Bound by the visits' dependent
// instructions (about 180 of a warp, 4 to 5 cycles each) and a load's latency; a prefetch of the other hit
// children changed nothing, a lane testing its own child's triangles one after the other was 5 to 10 % slower.  No
// fetch counter, so no memset before the launch.  Same hits as the other forms: the lowest (t, prim) among the
// triangles hit.
#pragma once

#include <stdint.h>

#include <algorithm>

#include "coop_trace.cuh"
#include "trace_device.cuh"

namespace rt {

constexpr int kWideBlock = 128;

// Rays up to which a cast runs this form: eight lanes per ray until the chip is a few times full of them, two rays per
// warp while that leaves SMs with free slots (a warp takes as long as the longest of its rays).  Cooperative
// against wide with four and with two rays per warp, closest hit, about half of the rays a camera's, us a call:
//                        1,280 triangles   81,920            1,310,720         64 instances of 5,120
//     1,000 rays         22.9  12.1  10.5  35.1  24.7  24.8  61.5  43.3  39.1  63.0  39.1  29.9
//     10,000 rays        24.2  14.4  16.6  49.4  35.0  34.9  67.8  53.5  56.0  78.0  47.2  39.4
//     50,500 rays        33.9  32.1  45.0  73.5  52.1  68.2  86.9  67.1  83.0  90.4  63.8  83.2
//     80,000 rays        35.2  43.3  65.4  82.1  65.8  93.1   101  88.8   119   101  92.1   124
// Where all rays are random the cooperative form gains sooner (from host memory, 1,280 / 246,420 triangles, 20,000
// rays 39.4 / 68 against 37.5 / 62, 50,942 rays 44 / 72 against 50 / 77), which is where the line lies.
inline uint64_t wide_ray_limit(const DeviceScene& s, int sm_count) {
    return (s.inst_trav || s.node_count >= 512 ? 256ull : 192ull) * std::max(1, sm_count);
}
inline uint32_t wide_pair_limit(int sm_count) { return 64u * (uint32_t)std::max(1, sm_count); }
inline int wide_blocks(uint32_t n, uint32_t per_warp) {
    const uint32_t per_block = per_warp * (kWideBlock / 32);
    return (int)((n + per_block - 1) / per_block);
}

// Traces items [0, n), per_warp (1 to 4) at a time in each warp of blocks of kWideBlock threads.  load(i, o, d)
// gives item i's ray (origin and tmin, direction and tmax) and returns its scene; store(i, hit, valid) is
// called by all 32 lanes together (valid marks the lanes holding an item).  `stacks`: kWideBlock / 8 * kTotalStack
// entries of shared memory.  REFINE: hits are refined.  LOOP: the grid may be smaller than the items.  TWO: scenes may
// be two-level.  Returns the device error bits of the lane's rays.
template <bool ANY, bool REFINE, bool TWO, bool LOOP, class Load, class Store>
__device__ __forceinline__ uint32_t wide_trace(uint32_t n, uint32_t per_warp, uint2* stacks, Load load, Store store) {
    constexpr uint32_t kAll = 0xFFFFFFFFu;
    const uint32_t lane = threadIdx.x & 31u, j = lane & 7u, shift = lane & 24u, in_warp = lane >> 3;
    uint2* stack = stacks + (threadIdx.x >> 3) * kTotalStack;
    uint32_t err_all = 0;
    const uint32_t warps = gridDim.x * (kWideBlock / 32);
    uint32_t at_warp = (blockIdx.x * kWideBlock + threadIdx.x) >> 5;
    if ((uint64_t)at_warp * per_warp >= n) return 0u;
    do {
        const uint32_t i = at_warp * per_warp + in_warp;
        const bool valid = in_warp < per_warp && i < n;
        float4 wo, wd;
        const DeviceScene* sc = load(valid ? i : at_warp * per_warp, wo, wd);
        TraceRay r = make_trace_ray(wo.x, wo.y, wo.z, wd.x, wd.y, wd.z, wo.w, wd.w);
        const uint8_t* nodes = reinterpret_cast<const uint8_t*>(sc->nodes);
        const float4* tris = reinterpret_cast<const float4*>(sc->tris);
        const bool empty = sc->node_count == 0;

        uint2 group = make_uint2(0u, valid && !empty ? 0x80000000u : 0u);
        int sp = 0;
        uint32_t err = 0, steps = 0, inst = 0, first = 0, best_inst = 0, best_rec = 0;
        bool in_blas = !TWO || sc->inst_trav == nullptr;
        uint32_t best_prim = kMiss;
        float best_t = wd.w;
        // the node being visited: header, child base and metas, and this lane's child's planes
        uint4 w0 = make_uint4(0u, 0u, 0u, 0u), w1 = w0;
        uint32_t nx = 0, ny = 0, nz = 0, fx = 0, fy = 0, fz = 0, slot = 0;
        bool live = false;

        // (The warp's lanes pop together, with full-mask barriers around the read: with a group's own mask each barrier
        // costs a dozen instructions and a branch, 26.8 us against 24.7 for 1,000 rays.)
        auto push = [&](uint2 g) {
            if (sp < kTotalStack) {
                if (j == 0) stack[sp] = g;
                ++sp;
            } else {
                err |= kErrStackOverflow;
            }
        };
        // The ray's next node, if it has one, on its way to the registers.
        auto advance = [&]() {
            if (TWO) {   // up to a node group, through the ends of instances and into the next ones
                for (;;) {
                    const bool enters = group.y != 0u && group.y <= 0x00FFFFFFu && !err, pops = group.y == 0u && sp != 0 && !err;
                    if (!__any_sync(kAll, enters || pops)) break;
                    if (pops) --sp;
                    __syncwarp();
                    if (pops) group = stack[sp];
                    __syncwarp();
                    if (pops && group.x == kLevelMarker && group.y == 0u) {   // back to the top level
                        r = make_trace_ray(wo.x, wo.y, wo.z, wd.x, wd.y, wd.z, wo.w, wd.w);
                        in_blas = false;
                    }
                    if (enters) {   // the nearest pending instance
                        const uint32_t k = (uint32_t)__ffs(group.y) - 1u, ii = __ldg(sc->tlas_refs + group.x + k);
                        group.y &= group.y - 1u;
                        if (group.y) push(group);
                        group = make_uint2(0u, 0u);
                        const uint4 tail = __ldg(reinterpret_cast<const uint4*>(sc->inst_trav + ii) + 3);
                        if (tail.x != 0xFFFFFFFFu) {   // (a model without triangles has no bottom level)
                            push(make_uint2(kLevelMarker, 0u));
                            r = instance_ray(make_trace_ray(wo.x, wo.y, wo.z, wd.x, wd.y, wd.z, wo.w, wd.w), sc->inst_trav + ii);
                            in_blas = true;
                            inst = ii;
                            first = tail.y;
                            group = make_uint2(tail.x, 0x80000000u);
                        }
                    }
                }
            } else {
                const bool pops = group.y == 0u && sp != 0;
                if (pops) --sp;
                __syncwarp();
                if (pops) group = stack[sp];
                __syncwarp();
            }
            live = group.y > 0x00FFFFFFu && !err;
            if (live && ++steps > kMaxTraversalSteps) {
                err |= kErrStepLimit;
                live = false;
            }
            const uint32_t bit = 31u - __clz(group.y | 1u), child_slot = (bit - 24u) ^ r.oct_inv;
            const uint32_t child = live ? group.x + __popc(group.y & ((1u << (child_slot & 31u)) - 1u)) : 0u;
            group.y &= ~(1u << bit);
            if (live && group.y > 0x00FFFFFFu) push(group);
            slot = j ^ r.oct_inv;   // lane j has the j-th child in the ray's order
            if (empty) return;   // no node to load
            const uint8_t* p = nodes + 80ull * child;
            w0 = __ldg(reinterpret_cast<const uint4*>(p));
            w1 = __ldg(reinterpret_cast<const uint4*>(p) + 1);
            const uint8_t* q = p + 32 + slot;
            const bool bx = r.idx < 0.0f, by = r.idy < 0.0f, bz = r.idz < 0.0f;
            nx = __ldg(q + (bx ? 24 : 0));
            fx = __ldg(q + (bx ? 0 : 24));
            ny = __ldg(q + (by ? 32 : 8));
            fy = __ldg(q + (by ? 8 : 32));
            nz = __ldg(q + (bz ? 40 : 16));
            fz = __ldg(q + (bz ? 16 : 40));
        };

        advance();
        while (__any_sync(kAll, live)) {
            // this lane's child box, with the arithmetic of intersect_children
            const float sx = __uint_as_float(((w0.w & 0xFFu) + 15u) << 23) * r.idx, sy = __uint_as_float((((w0.w >> 8) & 0xFFu) + 15u) << 23) * r.idy,
                        sz = __uint_as_float((((w0.w >> 16) & 0xFFu) + 15u) << 23) * r.idz;
            const float ox = (__uint_as_float(w0.x) - r.ox) * r.idx - sx, oy = (__uint_as_float(w0.y) - r.oy) * r.idy - sy,
                        oz = (__uint_as_float(w0.z) - r.oz) * r.idz - sz;
            auto at = [](uint32_t q, float s, float o) { return fmaf(__uint_as_float(0x3F800000u | (q << 8)), s, o); };
            const float tn = fmaxf(fmaxf(at(nx, sx, ox), at(ny, sy, oy)), fmaxf(at(nz, sz, oz), r.tmin));
            const float tf = fminf(fminf(at(fx, sx, ox), at(fy, sy, oy)), fminf(at(fz, sz, oz), best_t));
            const uint32_t meta = ((slot < 4u ? w1.z : w1.w) >> (8u * (slot & 3u))) & 0xFFu;
            const bool box = live && tn <= tf, inner = (meta & (meta << 1) & 0x10u) != 0u;
            const uint32_t inner_mask = (__ballot_sync(kAll, box && inner) >> shift) & 0xFFu;
            uint32_t entries = box && !inner ? (meta >> 5) << (meta & 31u) : 0u;   // the node's hit leaf entries
            entries |= __shfl_xor_sync(kAll, entries, 1);
            entries |= __shfl_xor_sync(kAll, entries, 2);
            entries |= __shfl_xor_sync(kAll, entries, 4);
            const uint32_t rec = w1.y + j;   // lane j tests entries j, j + 8 and j + 16
            group = inner_mask ? make_uint2(w1.x, inner_mask << 24 | w0.w >> 24) : make_uint2(0u, 0u);
            if (TWO && live && !in_blas && entries) {   // instances first, the rest of the top level below them
                if (group.y > 0x00FFFFFFu) push(group);
                group = make_uint2(w1.y, entries);
                entries = 0u;
            }
            const bool tests = __any_sync(kAll, entries != 0u);
            const TraceRay rt = r;
            const uint32_t tri_inst = inst, tri_first = first;
            const bool was_live = live;
            advance();
            if (tests) {
                uint32_t key = ~0u, prim_mine = 0, rec_mine = 0;   // this lane's closest: ordered t, triangle
                float t_mine = 0.0f;
                auto test = [&](uint32_t k) {
                    if (!(entries >> (j + k) & 1u)) return;
                    const float4* tp = tris + 3ull * (rec + k);
                    const float4 a = __ldg(tp), b = __ldg(tp + 1), c = __ldg(tp + 2);
                    float t, u, v;
                    if (!intersect_triangle(rt, a, b, c, best_t, t, u, v)) return;
                    const uint32_t hk = coop_ordered(t + 0.0f), prim = __float_as_uint(a.w) + tri_first;
                    if (hk < key || (hk == key && prim < prim_mine)) {
                        key = hk;
                        prim_mine = prim;
                        t_mine = t;
                        rec_mine = rec + k;
                    }
                };
                test(0);
                if (__any_sync(kAll, entries >> 8 != 0u)) {
                    test(8);
                    test(16);
                }
                if (__any_sync(kAll, key != ~0u)) {
                    uint32_t low = min(key, __shfl_xor_sync(kAll, key, 1));
                    low = min(low, __shfl_xor_sync(kAll, low, 2));
                    low = min(low, __shfl_xor_sync(kAll, low, 4));
                    uint32_t winners = (__ballot_sync(kAll, key == low) >> shift) & 0xFFu;
                    if (__any_sync(kAll, low != ~0u && (winners & (winners - 1u)) != 0u)) {   // equal t: the lowest triangle
                        uint32_t p = key == low ? prim_mine : ~0u;
#pragma unroll
                        for (int o = 1; o < 8; o <<= 1) p = min(p, __shfl_xor_sync(kAll, p, o));
                        winners = (__ballot_sync(kAll, key == low && prim_mine == p) >> shift) & 0xFFu;
                    }
                    const int from = (int)(shift + (uint32_t)__ffs(winners) - 1u);
                    const float t_low = __shfl_sync(kAll, t_mine, from);
                    const uint32_t rec_low = __shfl_sync(kAll, rec_mine, from), prim_low = __shfl_sync(kAll, prim_mine, from);
                    if (was_live && low != ~0u && (t_low < best_t || prim_low < best_prim)) {   // t <= best_t holds
                        best_t = t_low;
                        best_prim = prim_low;
                        best_rec = rec_low;
                        best_inst = tri_inst;
                        if (ANY) {
                            live = false;
                            sp = 0;
                        }
                    }
                }
            }
        }
        CoopHit c;
        c.h.prim = best_prim;
        c.h.t = best_t;
        c.h.u = 0.0f;
        c.h.v = 0.0f;
        c.inst = best_inst;
        c.pad1 = 0u;
        c.pad2 = 0u;
        const bool stores = valid && j == 0;
        if (REFINE && stores && best_prim != kMiss) {
            TraceRay w = make_trace_ray(wo.x, wo.y, wo.z, wd.x, wd.y, wd.z, wo.w, wd.w);
            if (TWO && sc->inst_trav) w = instance_ray(w, sc->inst_trav + best_inst);
            const float4* tp = tris + 3ull * best_rec;
            const float4 a = __ldg(tp), b = __ldg(tp + 1), v = __ldg(tp + 2);
            if (!refine_hit(w, a, b, v, c.h)) {   // the test's own t, u, v stand (a degenerate determinant)
                w.tmin = -INFINITY;
                intersect_triangle(w, a, b, v, INFINITY, c.h.t, c.h.u, c.h.v);
            }
            c.pad1 = __float_as_uint(b.w);
            c.pad2 = __float_as_uint(v.w);
        }
        __syncwarp();
        store(i, c, stores);
        if (stores) err_all |= err;
        __syncwarp();   // the stacks serve the warp's next rays
        at_warp += warps;
    } while (LOOP && (uint64_t)at_warp * per_warp < n);
    return err_all;
}

}  // namespace rt
