// Warp-cooperative persistent BVH8 traversal, of flat and of two-level scenes: the default launch form.
//
// The per-thread traversal of trace_device.cuh loses most of a warp's issue slots to divergence on
// incoherent rays: lanes whose rays have ended wait for the warp's longest ray, and the triangle tests
// run with the few lanes whose node had leaf children.  Here a warp keeps 32 rays in flight and shares
// the work that diverges:
//   * rays are fetched 32 at a time (a chunk of the global fetch counter, one ray per lane, into shared
//     memory), and idle lanes take the next staged ray once at most `refill_at` lanes still trace (refill: Aila
//     and Laine, "Understanding the Efficiency of Ray Traversal on GPUs", HPG 2009);
//   * node visits: every tracing lane visits its nearest pending child node (box test of the 8 quantized
//     children, near-to-far order by ray octant), VISITS times between two rounds of the warp's bookkeeping
//     (refill, list tests, finishing), so that the bookkeeping is paid once per several visits;
//   * triangle tests: a node's leaf triangles are not tested by the lane that found them; the warp collects
//     them in a shared list, a group per node, and once it holds kFlushGroups groups (or a lane with groups in it
//     has nothing else to do) tests them with one (ray, triangle) pair per lane, the closest (t, prim) per ray
//     kept by a 64-bit atomic minimum in shared memory;
//   * instances (TWO): a lane that reaches a top-level leaf enters its instances one after the other; the
//     lanes that want to enter one do it together, once per round, and the world ray waits in shared memory;
//   * finishing: ended rays go to a shared list that the warp refines (refine_hit) and stores one per
//     lane once it is full, so the hit refinement also runs at full width.
// The closest hit is the lowest (t, prim) over the triangles hit in [tmin, tmax], as in every other form,
// so hits are bit-identical to the per-thread traversal; any-hit rays end at the first triangle found.
#pragma once

#include <stdint.h>

#include <type_traits>

#include "kernels.h"
#include "trace_device.cuh"

namespace rt {

// Items per fetch: one per lane.  Small chunks also interleave the warps over the item list, so the last
// items end together.
constexpr uint32_t kCoopChunk = 32;
// Blocks of 128 threads per SM the cooperative kernels are compiled for: 7 (at most 72 registers, 30.4 KB of shared
// memory each): 0.418 ms against 0.423 ms with 6 and 0.444 ms with 8 (and a 6-entry stack).
#ifndef RT_COOP_MINB
#define RT_COOP_MINB 7
#endif
#ifndef RT_COOP_BLOCK
#define RT_COOP_BLOCK 128
#endif
constexpr int kCoopBlock = RT_COOP_BLOCK;   // threads per block; warps share nothing
constexpr int kCoopMinBlocks = RT_COOP_MINB * 128 / kCoopBlock;
// Blocks per SM of the two-level form, which keeps more state (5 blocks: 5 % slower; 7: the same, with spills).
#ifndef RT_COOP_MINB_TWO
#define RT_COOP_MINB_TWO 6
#endif
constexpr int kCoopMinBlocksTwo = RT_COOP_MINB_TWO * 128 / kCoopBlock;
#ifndef RT_COOP_FLUSH
#define RT_COOP_FLUSH 12
#endif
constexpr uint32_t kFlushGroups = RT_COOP_FLUSH;   // groups (two triangles on average) collected before the test
// Node visits per lane per round of bookkeeping (1.3M-triangle ray cast, closest hit: 1 visit 0.436 ms, 2 visits
// 0.418 ms, 3 visits 0.420 ms; 256 instances: 0.952, 0.930 and 1.127 ms).
#ifndef RT_COOP_VISITS
#define RT_COOP_VISITS 2
#endif
constexpr int kCoopVisits = RT_COOP_VISITS;
#ifndef RT_COOP_VISITS_TWO
#define RT_COOP_VISITS_TWO 1
#endif
constexpr int kCoopVisitsTwo = RT_COOP_VISITS_TWO;
// Shared-memory stack entries per thread (deeper levels spill to local memory): what fits beside the lists.
#ifndef RT_COOP_STACK
#define RT_COOP_STACK 8
#endif
constexpr int kCoopStack = RT_COOP_STACK;
constexpr uint32_t kCoopGroups = 64;   // list capacity: a visit adds at most 32, and a flush comes before the next

// Per-warp shared state of the cooperative traversal.
struct CoopWarpFlat {
    float4 ray_o[32];                 // per lane: origin, tmin of its ray (in its instance's space while in one)
    float4 ray_s[32];                 // per lane: shear constants sx, sy, sz, axes kx | ky << 2 | kz << 4
    float4 ray_d[32];                 // per lane: direction, tmax (world space)
    unsigned long long best[32];      // per lane: ordered(t) << 32 | prim of the closest hit so far
    uint2 best_rec[32];               // per lane: triangle record and t (as tested) of that hit
    uint32_t g_base[kCoopGroups];     // groups: first triangle record of the node
    uint32_t g_meta[2][kCoopGroups];  // groups: meta bytes of the hit leaf children, by child slot
    uint16_t g_prefix[kCoopGroups];   // groups: inclusive prefix of their triangle counts
    uint8_t g_own[kCoopGroups];       // groups: lane of the ray
    float4 fin_o[32];                 // finished rays: origin, t
    float4 fin_d[32];                 // finished rays: direction
    uint4 fin_i[32];                  // finished rays: item, prim, triangle record, instance
    float4 stage_o[32], stage_d[32];  // fetched rays: origin, tmin; direction, tmax
};
struct CoopWarpTwo {
    float4 world_o[32];               // per lane: origin, tmin in world space
    uint32_t inst[32];                // per lane: instance its ray is in
    uint32_t best_inst[32];           // per lane: instance of the closest hit
    uint32_t first[32];               // per lane: first global triangle of that instance
};
struct CoopWarpMixed {
    const DeviceScene* scene[32];     // per lane: its ray's scene
    const DeviceScene* fin_scene[32]; // finished rays: their scene
    const DeviceScene* stage_scene[32];
};
struct CoopNotTwo {};
struct CoopNotMixed {};
template <bool MIXED, bool TWO>
struct CoopWarp : CoopWarpFlat,
                  std::conditional_t<TWO, CoopWarpTwo, CoopNotTwo>,
                  std::conditional_t<MIXED, CoopWarpMixed, CoopNotMixed> {};

// The cooperative kernels' dynamic shared memory: a CoopWarp per warp, then the threads' stacks.  The functions
// below reach it through this symbol, so that they access it as shared memory also where they are not inlined.
extern __shared__ __align__(16) unsigned char coop_shared[];
template <bool MIXED, bool TWO>
__device__ __forceinline__ CoopWarp<MIXED, TWO>& coop_warp() {
    return reinterpret_cast<CoopWarp<MIXED, TWO>*>(coop_shared)[threadIdx.x >> 5];
}
template <bool MIXED, bool TWO>
constexpr size_t coop_shared_bytes() {
    return (kCoopBlock / 32) * sizeof(CoopWarp<MIXED, TWO>) + kCoopBlock * kCoopStack * sizeof(uint2);
}

__device__ __forceinline__ uint32_t coop_ordered(float f) {
    const uint32_t b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float coop_unordered(uint32_t o) {
    return __uint_as_float((o & 0x80000000u) ? (o & 0x7FFFFFFFu) : ~o);
}
__device__ __forceinline__ uint32_t lanemask_lt() {
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// Adds a warp's traversal counts to two u64 device counters (one atomic per warp).
__device__ __forceinline__ void coop_add_counts(const TraceCounters& c, uint32_t* counters, int nodes_at, int tris_at) {
    unsigned long long nv = c.nodes, tv = c.tris;
    for (int o = 16; o > 0; o >>= 1) {
        nv += __shfl_down_sync(0xFFFFFFFFu, nv, o);
        tv += __shfl_down_sync(0xFFFFFFFFu, tv, o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (nv) atomicAdd(reinterpret_cast<unsigned long long*>(counters + nodes_at), nv);
        if (tv) atomicAdd(reinterpret_cast<unsigned long long*>(counters + tris_at), tv);
    }
}

// What a finished ray hands to its caller: the hit, its instance (two-level scenes) and the words that the
// triangle record carries beside its vertices (flat scenes; see TriRecord).
struct CoopHit {
    Hit h;
    uint32_t inst;
    uint32_t pad1, pad2;
};

// Tests the n collected groups, one (ray, triangle) pair per lane per round.  Not inlined, like
// coop_store_finished: both run once per several traversal steps, and kept out of the traversal loop they leave
// it more registers (1.3M-triangle ray cast: 0.566 -> 0.534 ms when they moved out).
template <bool COUNT, bool MIXED, bool TWO>
__device__ __noinline__ uint32_t coop_test_groups(uint32_t n, const float4* tris) {
    CoopWarp<MIXED, TWO>& S = coop_warp<MIXED, TWO>();
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t total = 0, tested = 0;
    for (uint32_t h = 0; h < n; h += 32u) {
        const uint32_t g = h + lane;
        uint32_t c = g < n ? __popc(leaf_bits(S.g_meta[0][g])) + __popc(leaf_bits(S.g_meta[1][g])) : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, c, o);
            if (lane >= (uint32_t)o) c += y;
        }
        c += total;
        if (g < n) S.g_prefix[g] = (uint16_t)c;
        total = __shfl_sync(0xFFFFFFFFu, c, 31);
    }
    __syncwarp();
    for (uint32_t b0 = 0; b0 < total; b0 += 32u) {
        const uint32_t p = b0 + lane;
        bool hit = false;
        uint32_t o = 0, rec = 0;
        unsigned long long key = 0;
        float t = 0.0f;
        if (p < total) {
            uint32_t g = 0;   // the group holding pair p: binary search over the prefix
            if (n > 32u && S.g_prefix[31] <= p) g = 32u;
#pragma unroll
            for (uint32_t s = 16; s; s >>= 1)
                if (g + s - 1 < n && S.g_prefix[g + s - 1] <= p) g += s;
            uint32_t k = p - (g ? S.g_prefix[g - 1] : 0u);   // the k-th triangle of the group
            uint32_t m = S.g_meta[0][g];
            uint32_t bits = leaf_bits(m);
            const uint32_t c0 = (uint32_t)__popc(bits);
            if (k >= c0) {
                k -= c0;
                m = S.g_meta[1][g];
                bits = leaf_bits(m);
            }
            for (; k; --k) bits &= bits - 1u;
            const uint32_t at = (uint32_t)__ffs(bits) - 1u;   // bit of the triangle within its child's byte
            rec = S.g_base[g] + ((m >> (at & 24u)) & 31u) + (at & 7u);
            o = S.g_own[g];
            const float4* tp = tris;
            if constexpr (MIXED) tp = reinterpret_cast<const float4*>(S.scene[o]->tris);
            tp += 3ull * rec;
            const float4 a = __ldg(tp), b = __ldg(tp + 1), c = __ldg(tp + 2);
            const float4 ra = S.ray_o[o], rb = S.ray_s[o];
            TraceRay q;
            q.ox = ra.x; q.oy = ra.y; q.oz = ra.z; q.tmin = ra.w;
            q.sx = rb.x; q.sy = rb.y; q.sz = rb.z;
            const uint32_t kk = __float_as_uint(rb.w);
            q.kx = (int)(kk & 3u); q.ky = (int)((kk >> 2) & 3u); q.kz = (int)((kk >> 4) & 3u);
            if (COUNT) ++tested;
            float u, v;
            if (intersect_triangle(q, a, b, c, coop_unordered((uint32_t)(S.best[o] >> 32)), t, u, v)) {
                hit = true;
                uint32_t prim = __float_as_uint(a.w);
                if constexpr (TWO) prim += S.first[o];
                key = ((unsigned long long)coop_ordered(t + 0.0f) << 32) | prim;
                atomicMin(&S.best[o], key);
            }
        }
        __syncwarp();
        if (hit && S.best[o] == key) {
            S.best_rec[o] = make_uint2(rec, __float_as_uint(t));
            if constexpr (TWO) S.best_inst[o] = S.inst[o];
        }
        __syncwarp();
    }
    return tested;
}

// Refines (REFINE) and stores the finished rays of the list, one per lane; store is called by all lanes.
template <bool REFINE, bool MIXED, bool TWO, class Store>
__device__ __noinline__ void coop_store_finished(uint32_t n_fin, const DeviceScene& uniform, Store& store) {
    CoopWarp<MIXED, TWO>& S = coop_warp<MIXED, TWO>();
    const uint32_t lane = threadIdx.x & 31u;
    __syncwarp();
    const bool valid = lane < n_fin;
    CoopHit c;
    c.h.prim = kMiss; c.h.t = 0.0f; c.h.u = 0.0f; c.h.v = 0.0f;
    c.inst = 0; c.pad1 = 0; c.pad2 = 0;
    uint32_t item = 0;
    if (valid) {
        const float4 o = S.fin_o[lane], d = S.fin_d[lane];
        const uint4 fi = S.fin_i[lane];
        item = fi.x;
        c.h.prim = fi.y;
        c.h.t = o.w;
        c.inst = fi.w;
        if (REFINE && c.h.prim != kMiss) {
            const DeviceScene* sc = &uniform;
            if constexpr (MIXED) sc = S.fin_scene[lane];
            const float4* tp = reinterpret_cast<const float4*>(sc->tris) + 3ull * fi.z;
            const float4 a = __ldg(tp), b = __ldg(tp + 1), v = __ldg(tp + 2);
            TraceRay r;
            r.ox = o.x; r.oy = o.y; r.oz = o.z;
            r.dx = d.x; r.dy = d.y; r.dz = d.z;
            r.tmin = 0.0f; r.tmax = 0.0f;
            if (TWO && sc->inst_trav) r = instance_ray(r, sc->inst_trav + fi.w);
            if (!refine_hit(r, a, b, v, c.h)) {   // the test's own t, u, v stand (a degenerate determinant)
                TraceRay q = make_trace_ray(r.ox, r.oy, r.oz, r.dx, r.dy, r.dz, -INFINITY, INFINITY);
                intersect_triangle(q, a, b, v, INFINITY, c.h.t, c.h.u, c.h.v);
            }
            c.pad1 = __float_as_uint(b.w);
            c.pad2 = __float_as_uint(v.w);
        }
    }
    __syncwarp();
    store(item, c, valid);
}

// Traces items [0, n) of the caller's list.  load(i, o, d) gives item i's ray (origin and tmin, direction and tmax);
// with MIXED it also returns the item's scene (batched waves mix scenes), otherwise every item uses `uniform`.
// store(i, hit, valid) is called by all 32 lanes together with up to 32 finished items (valid marks the lanes
// holding one).  `next` is the global fetch counter (zero at launch); a warp refills its idle lanes once at most
// `refill_at` lanes still trace.  Requires blocks of kCoopBlock threads and coop_shared_bytes() of dynamic shared
// memory.  Returns the device error bits of the warp's rays.  TWO: scenes may be two-level.  VISITS: node visits per
// lane between two rounds of the warp's bookkeeping (the triangles found meanwhile are tested at the next flush, so
// the closest distance a visit culls with may lag by up to VISITS - 1 visits: a few more nodes, same hits).
template <bool ANY, bool COUNT, bool REFINE, bool MIXED, bool TWO, int SS = kCoopStack, uint32_t FLUSH = kFlushGroups,
          int VISITS = TWO ? kCoopVisitsTwo : kCoopVisits, class Load, class Store>
__device__ __forceinline__ uint32_t coop_trace(const DeviceScene& uniform, uint32_t n, uint32_t* next, uint32_t refill_at,
                                               Load load, Store store, TraceCounters& cnt) {
    constexpr uint32_t kAll = 0xFFFFFFFFu;
    constexpr int stride = kCoopBlock;
    CoopWarp<MIXED, TWO>& S = coop_warp<MIXED, TWO>();
    uint2* stack = reinterpret_cast<uint2*>(coop_shared + (kCoopBlock / 32) * sizeof(CoopWarp<MIXED, TWO>)) + threadIdx.x;
    const uint32_t lane = threadIdx.x & 31u;
    uint2 spill[kTotalStack - SS];
    uint32_t err = 0;
    bool has = false;
    TraceRay r;                                     // origin, reciprocal direction, tmin, octant: the box test's part
    uint32_t wlo = 0, whi = 0;                      // octant_weights of the ray
    const uint4* nodes = reinterpret_cast<const uint4*>(uniform.nodes);
    const float4* utris = reinterpret_cast<const float4*>(uniform.tris);
    uint32_t item = 0;
    uint2 group = make_uint2(0u, 0u);
    uint2 entry = make_uint2(0u, 0u);               // TWO: instances to enter (first leaf entry, hits)
    bool in_blas = false;                           // TWO: the ray is in an instance's space (or its scene is flat)
    bool at_marker = false;                         // TWO: popped the end of an instance, waits to leave it
    int sp = 0;
    uint32_t steps = 0;
    float best_t = 0.0f;
    bool pending = false;                           // this lane has groups in the list
    uint32_t n_groups = 0, n_fin = 0;               // warp-uniform list sizes
    uint32_t st_next = 0, st_count = 0, st_base = 0;   // warp-uniform: staged rays not taken yet, item of the first
    bool exhausted = false;

    auto pop = [&]() {
        --sp;
        group = sp < SS ? stack[sp * stride] : spill[sp - SS];
    };
    auto push = [&](uint2 g) {
        if (sp < SS) {
            stack[sp * stride] = g;
            ++sp;
        } else if (sp < kTotalStack) {
            spill[sp - SS] = g;
            ++sp;
        } else {
            err |= kErrStackOverflow;
        }
    };
    // tests the warp's list (all lanes together) and takes each lane's result
    auto flush = [&]() {
        __syncwarp();
        cnt.tris += coop_test_groups<COUNT, MIXED, TWO>(n_groups, utris);
        n_groups = 0;
        if (pending) {
            const unsigned long long key = S.best[lane];
            if (ANY) {
                if ((uint32_t)key != 0xFFFFFFFFu) {
                    group = make_uint2(0u, 0u);
                    sp = 0;
                    if (TWO) { entry.y = 0u; at_marker = false; }
                }
            } else {
                best_t = coop_unordered((uint32_t)(key >> 32));
            }
        }
        pending = false;
    };

    for (;;) {
        // refill idle lanes from the staged rays, staging the next chunk when they run out
        const uint32_t active = __ballot_sync(kAll, has);
        if ((uint32_t)__popc(active) <= refill_at && !(exhausted && st_next >= st_count)) {
            uint32_t idle = ~active;
            while (idle) {
                if (st_next >= st_count) {
                    if (exhausted) break;
                    uint32_t base = 0;
                    if (lane == 0) base = atomicAdd(next, kCoopChunk);
                    base = __shfl_sync(kAll, base, 0);
                    st_next = 0;
                    st_count = base < n ? min(kCoopChunk, n - base) : 0u;
                    st_base = base;
                    if (st_count < kCoopChunk) exhausted = true;
                    if (st_count == 0) break;
                    if (lane < st_count) {
                        float4 o, d;
                        if constexpr (MIXED) S.stage_scene[lane] = load(base + lane, o, d);
                        else load(base + lane, o, d);
                        S.stage_o[lane] = o;
                        S.stage_d[lane] = d;
                    }
                    __syncwarp();
                }
                const uint32_t take = min((uint32_t)__popc(idle), st_count - st_next);
                const uint32_t rank = (uint32_t)__popc(idle & lanemask_lt());
                const bool mine = ((idle >> lane) & 1u) && rank < take;
                if (mine) {
                    const uint32_t e = st_next + rank;
                    const float4 o = S.stage_o[e], d = S.stage_d[e];
                    item = st_base + e;
                    r = make_trace_ray(o.x, o.y, o.z, d.x, d.y, d.z, o.w, d.w);
                    octant_weights(r.oct_inv, wlo, whi);
                    uint32_t node_count = uniform.node_count;
                    bool two = TWO;
                    if constexpr (MIXED) {
                        const DeviceScene* sc = S.stage_scene[e];
                        S.scene[lane] = sc;
                        nodes = reinterpret_cast<const uint4*>(sc->nodes);
                        node_count = sc->node_count;
                        if (TWO) two = sc->inst_trav != nullptr;
                    }
                    if constexpr (TWO) {
                        S.world_o[lane] = o;
                        S.first[lane] = 0;
                        S.inst[lane] = 0;
                        S.best_inst[lane] = 0;
                        in_blas = !two;
                        at_marker = false;
                        entry.y = 0u;
                    }
                    has = true;
                    group = make_uint2(0u, node_count ? 0x80000000u : 0u);
                    sp = 0;
                    steps = 0;
                    best_t = d.w;
                    S.ray_o[lane] = o;
                    S.ray_s[lane] = make_float4(r.sx, r.sy, r.sz,
                                                __uint_as_float((uint32_t)r.kx | ((uint32_t)r.ky << 2) | ((uint32_t)r.kz << 4)));
                    S.ray_d[lane] = d;
                    S.best[lane] = ((unsigned long long)coop_ordered(d.w) << 32) | 0xFFFFFFFFull;
                }
                idle &= ~__ballot_sync(kAll, mine);
                st_next += take;
            }
        }
        if (!__any_sync(kAll, has)) break;   // nothing staged is left either
        // watchdog: a ray's traversal ends with kErrStepLimit after kMaxTraversalSteps visit slots
        if (has) {
            steps += VISITS;
            if (steps > kMaxTraversalSteps) {
                err |= kErrStepLimit;
                group = make_uint2(0u, 0u);
                sp = 0;
                if (TWO) { entry.y = 0u; at_marker = false; }
            }
        }
        // VISITS node visits per tracing lane, each followed by its stack pop; every visit's leaf triangles
        // join the warp's list (tested when a further visit's could overflow it)
#pragma unroll
        for (int v = 0; v < VISITS; ++v) {
            uint32_t tbase = 0;
            uint2 leaf = make_uint2(0u, 0u);   // meta bytes of the hit leaf children
            if (has && group.y > 0x00FFFFFFu && (!TWO || entry.y == 0u)) {
                const uint32_t slot_bit = 31u - __clz(group.y);
                const uint32_t slot = (slot_bit - 24u) ^ r.oct_inv;
                const uint32_t child = group.x + (uint32_t)__popc(group.y & ((1u << slot) - 1u));
                group.y &= ~(1u << slot_bit);
                if (group.y > 0x00FFFFFFu) push(group);
                const uint4* np = nodes + 5ull * child;
                const uint4 w0 = __ldg(np + 0), w1 = __ldg(np + 1), w2 = __ldg(np + 2), w3 = __ldg(np + 3),
                            w4 = __ldg(np + 4);
                if (COUNT) cnt.nodes++;
                uint32_t ordered;
                child_hits(r, wlo, whi, w0, w1, w2, w3, w4, best_t, ordered, leaf);
                group = make_uint2(w1.x, ordered << 24 | (w0.w >> 24));
                tbase = w1.y;
            }
            if constexpr (TWO) {
                if (!in_blas && (leaf.x | leaf.y)) {   // top-level leaves: the lane's instances to enter
                    entry.x = tbase;
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const uint32_t m = ((i < 4 ? leaf.x : leaf.y) >> (8 * (i & 3))) & 0xFFu;
                        entry.y |= (m >> 5) << (m & 31u);
                    }
                    leaf = make_uint2(0u, 0u);
                }
                if (has && !at_marker && entry.y == 0u && group.y <= 0x00FFFFFFu && sp > 0) {
                    pop();
                    if (group.x == kLevelMarker && group.y == 0u) {
                        at_marker = true;
                    } else if (group.y <= 0x00FFFFFFu) {   // instances left of an earlier top-level leaf
                        entry = group;
                        group = make_uint2(0u, 0u);
                    }
                }
            } else {
                if (has && group.y <= 0x00FFFFFFu && sp > 0) pop();
            }
            const bool found = (leaf.x | leaf.y) != 0u;
            const uint32_t app = __ballot_sync(kAll, found);
            if (found) {
                const uint32_t pos = n_groups + (uint32_t)__popc(app & lanemask_lt());
                S.g_base[pos] = tbase;
                S.g_meta[0][pos] = leaf.x;
                S.g_meta[1][pos] = leaf.y;
                S.g_own[pos] = (uint8_t)lane;
                pending = true;
            }
            n_groups += (uint32_t)__popc(app);
            if (v + 1 < VISITS && n_groups > 32u) flush();
        }
        // test the list when it is full enough, could overflow next step, or lanes with groups in it have nothing
        // else to do
        const bool idle_pending = has && pending && group.y <= 0x00FFFFFFu && (TWO ? (at_marker || (sp == 0 && entry.y == 0u)) : sp == 0);
        const bool waiting = __any_sync(kAll, idle_pending);
        if (n_groups && (waiting || n_groups >= FLUSH || n_groups > 32u)) flush();
        if constexpr (TWO) {
            // leave instances: back to the world ray and the entries below the marker
            if (at_marker && !pending) {
                at_marker = false;
                in_blas = false;
                const float4 o = S.world_o[lane], d = S.ray_d[lane];
                r.ox = o.x; r.oy = o.y; r.oz = o.z;
                r.idx = safe_rcp(d.x); r.idy = safe_rcp(d.y); r.idz = safe_rcp(d.z);
                r.oct_inv = 7u - ((d.x < 0.0f ? 1u : 0u) | (d.y < 0.0f ? 2u : 0u) | (d.z < 0.0f ? 4u : 0u));
                octant_weights(r.oct_inv, wlo, whi);
                group = make_uint2(0u, 0u);
                if (sp > 0) {
                    pop();
                    if (group.y <= 0x00FFFFFFu) {
                        entry = group;
                        group = make_uint2(0u, 0u);
                    }
                }
            }
            // enter the next instance; the rest of the top level waits below a marker
            if (entry.y) {
                const DeviceScene* sc = &uniform;
                if constexpr (MIXED) sc = S.scene[lane];
                const uint32_t k = (uint32_t)__ffs(entry.y) - 1u;
                entry.y &= entry.y - 1u;
                const uint32_t ii = __ldg(sc->tlas_refs + entry.x + k);
                const uint4 tail = __ldg(reinterpret_cast<const uint4*>(sc->inst_trav + ii) + 3);
                if (tail.x != 0xFFFFFFFFu) {   // (a model without triangles has no bottom level)
                    if (group.y > 0x00FFFFFFu) push(group);
                    if (entry.y) push(entry);
                    entry.y = 0u;
                    push(make_uint2(kLevelMarker, 0u));
                    const float4 o = S.world_o[lane], d = S.ray_d[lane];
                    TraceRay w;
                    w.ox = o.x; w.oy = o.y; w.oz = o.z;
                    w.dx = d.x; w.dy = d.y; w.dz = d.z;
                    w.tmin = o.w; w.tmax = d.w;
                    r = instance_ray(w, sc->inst_trav + ii);
                    octant_weights(r.oct_inv, wlo, whi);
                    S.ray_o[lane] = make_float4(r.ox, r.oy, r.oz, r.tmin);
                    S.ray_s[lane] = make_float4(r.sx, r.sy, r.sz,
                                                __uint_as_float((uint32_t)r.kx | ((uint32_t)r.ky << 2) | ((uint32_t)r.kz << 4)));
                    S.inst[lane] = ii;
                    S.first[lane] = tail.y;
                    in_blas = true;
                    group = make_uint2(tail.x, 0x80000000u);
                } else if (entry.y == 0u && group.y <= 0x00FFFFFFu && sp > 0) {
                    pop();   // at the top level: nodes or instances, never a marker
                    if (group.y <= 0x00FFFFFFu) {
                        entry = group;
                        group = make_uint2(0u, 0u);
                    }
                }
            }
        }
        // finished rays join the warp's finished list
        const bool done = has && group.y <= 0x00FFFFFFu && sp == 0 && !pending && (!TWO || (entry.y == 0u && !at_marker));
        const uint32_t dm = __ballot_sync(kAll, done);
        if (dm) {
            if (n_fin + (uint32_t)__popc(dm) > 32u) {
                coop_store_finished<REFINE, MIXED, TWO>(n_fin, uniform, store);
                n_fin = 0;
            }
            if (done) {
                const uint32_t pos = n_fin + (uint32_t)__popc(dm & lanemask_lt());
                const unsigned long long key = S.best[lane];
                const bool miss = (uint32_t)key == 0xFFFFFFFFu;
                float4 o;
                uint32_t inst = 0;
                if constexpr (TWO) {
                    o = S.world_o[lane];
                    inst = S.best_inst[lane];
                } else {
                    o = S.ray_o[lane];
                }
                const float4 d = S.ray_d[lane];
                const uint2 rec = S.best_rec[lane];
                S.fin_o[pos] = make_float4(o.x, o.y, o.z, miss ? d.w : __uint_as_float(rec.y));
                S.fin_d[pos] = d;
                S.fin_i[pos] = make_uint4(item, (uint32_t)key, rec.x, inst);
                if constexpr (MIXED) S.fin_scene[pos] = S.scene[lane];
                has = false;
            }
            n_fin += (uint32_t)__popc(dm);
        }
    }
    if (n_fin) coop_store_finished<REFINE, MIXED, TWO>(n_fin, uniform, store);
    return err;
}

}  // namespace rt
