// Ray-cast kernels (closest hit / any hit) over the BVH8, in three launch forms — one thread per ray
// (grid), persistent warps with dynamic ray fetch, and eight lanes per ray — and, for the grid form, in several block sizes
// and shared-memory stack depths (the autotuner's choices; every variant computes the same hits).
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "coop_trace.cuh"
#include "kernels.h"
#include "trace_device.cuh"

namespace rt {

static_assert(kSmemStack == kDefaultTraceStack, "default traversal stack depth");

// Minimum resident blocks per SM requested from the compiler (register cap), when set.
#ifdef RT_TRACE_MINB
#define RT_TRACE_BOUNDS(B) __launch_bounds__(B, RT_TRACE_MINB)
#else
#define RT_TRACE_BOUNDS(B) __launch_bounds__(B)
#endif

template <bool COUNT>
__device__ __forceinline__ void reduce_counters(const TraceCounters& c, unsigned long long* counters) {
    if (COUNT) {
        unsigned long long nodes_v = c.nodes, tris_v = c.tris;
        for (int o = 16; o > 0; o >>= 1) {
            nodes_v += __shfl_down_sync(0xFFFFFFFFu, nodes_v, o);
            tris_v += __shfl_down_sync(0xFFFFFFFFu, tris_v, o);
        }
        if ((threadIdx.x & 31) == 0) {
            atomicAdd(counters + 0, nodes_v);
            atomicAdd(counters + 1, tris_v);
        }
    }
}

// Warp-cooperative persistent form (coop_trace.cuh): warps refill idle lanes once at most `refill_at` of
// their lanes still trace; triangle tests and hit refinement are spread over the warp.
template <bool ANY, bool COUNT, bool TWO>
__global__ void __launch_bounds__(kCoopBlock, TWO ? kCoopMinBlocksTwo : kCoopMinBlocks)
    raycast_kernel(const __grid_constant__ DeviceScene scene, const Ray* __restrict__ rays, uint32_t n, Hit* __restrict__ hits,
                   unsigned long long* counters, uint32_t* err_flag, uint32_t* next, uint32_t refill_at) {
    TraceCounters c{0u, 0u};
    auto load = [&](uint32_t i, float4& o, float4& d) {
        const float4* rp = reinterpret_cast<const float4*>(rays) + 2ull * i;
        o = __ldcs(rp);
        d = __ldcs(rp + 1);
    };
    auto store = [&](uint32_t i, const CoopHit& c, bool valid) {
        const Hit& h = c.h;
        if (valid && hits) __stcs(reinterpret_cast<float4*>(hits) + i, make_float4(__uint_as_float(h.prim), h.t, h.u, h.v));
    };
    const uint32_t e = coop_trace<ANY, COUNT, true, false, TWO>(scene, n, next, refill_at, load, store, c);
    if (e) atomicOr(err_flag, e);
    reduce_counters<COUNT>(c, counters);
}

// One thread per ray (the hardware block scheduler balances the load at block granularity).
template <bool ANY, bool COUNT, int BLOCK, int SS>
__global__ void RT_TRACE_BOUNDS(BLOCK) raycast_kernel_grid(const Bvh8Node* __restrict__ nodes,
                                                          const TriRecord* __restrict__ tris, uint32_t node_count,
                                                          const Ray* __restrict__ rays, uint32_t n,
                                                          Hit* __restrict__ hits, unsigned long long* counters,
                                                          uint32_t* err_flag, const uint32_t* __restrict__ order) {
    __shared__ uint2 stack[SS * BLOCK];
    const uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    TraceCounters c{0u, 0u};
    if (k < n) {
        const uint64_t i = order ? order[k] : k;   // thread k traces the k-th ray of the coherence order
        const float4* rp = reinterpret_cast<const float4*>(rays) + 2ull * i;
        const float4 a = __ldcs(rp), b = __ldcs(rp + 1);
        const TraceRay r = make_trace_ray(a.x, a.y, a.z, b.x, b.y, b.z, a.w, b.w);
        Hit h;
        HitTail tail;
        uint32_t e = 0;
        if (node_count) {
            e = traverse<ANY, COUNT, true, SS>(nodes, tris, r, stack + threadIdx.x, BLOCK, h, c, tail);
        } else {
            h.prim = kMiss; h.t = r.tmax; h.u = 0.0f; h.v = 0.0f;
        }
        if (hits) __stcs(reinterpret_cast<float4*>(hits) + i, make_float4(__uint_as_float(h.prim), h.t, h.u, h.v));
        if (e) atomicOr(err_flag, e);
    }
    reduce_counters<COUNT>(c, counters);
}

// Eight lanes per ray, for casts of few rays: what such a cast takes is the longest ray's chain of node visits (66 of
// them among 128 rays of the 1.3M-triangle scene: 52 us cooperative, 40 us here), and a visit is shorter when a lane
// tests one child box and then one of the node's triangles instead of eight boxes.  Up to four rays per warp, each
// group of eight lanes holding its ray's state; the next node is on its way before the current one's triangles are
// tested.  Bound by the visits' dependent instructions (about 180 of a warp, 4 to 5 cycles each) and a load's latency;
// a prefetch of the other hit children changed nothing, a lane testing its own child's triangles one after the
// other was 5 to 10 % slower.  No fetch counter, so no memset before the launch.  Same hits as the other forms: the
// lowest (t, prim) among the triangles hit.
constexpr int kWideBlock = 128;
template <bool ANY, bool TWO>
__global__ void __launch_bounds__(kWideBlock) raycast_kernel_wide(const __grid_constant__ DeviceScene sc, const Ray* __restrict__ rays,
                                                                 uint32_t n, Hit* __restrict__ hits, uint32_t* err_flag, uint32_t per_warp) {
    constexpr uint32_t kAll = 0xFFFFFFFFu;
    __shared__ uint2 stacks[kWideBlock / 8][kTotalStack];
    const uint32_t lane = threadIdx.x & 31u, j = lane & 7u, shift = lane & 24u;
    uint2* stack = stacks[threadIdx.x >> 3];
    const uint32_t in_warp = lane >> 3, i = ((blockIdx.x * kWideBlock + threadIdx.x) >> 5) * per_warp + in_warp;
    const bool valid = in_warp < per_warp && i < n;
    const float4* rp = reinterpret_cast<const float4*>(rays) + 2ull * (valid ? i : 0u);
    const float4 wo = __ldg(rp), wd = __ldg(rp + 1);
    TraceRay r = make_trace_ray(wo.x, wo.y, wo.z, wd.x, wd.y, wd.z, wo.w, wd.w);
    const uint8_t* nodes = reinterpret_cast<const uint8_t*>(sc.nodes);
    const float4* tris = reinterpret_cast<const float4*>(sc.tris);

    uint2 group = make_uint2(0u, valid && sc.node_count ? 0x80000000u : 0u);
    int sp = 0;
    uint32_t err = 0, steps = 0, inst = 0, first = 0, best_inst = 0, best_rec = 0;
    bool in_blas = !TWO || sc.inst_trav == nullptr;
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
                    const uint32_t k = (uint32_t)__ffs(group.y) - 1u, ii = __ldg(sc.tlas_refs + group.x + k);
                    group.y &= group.y - 1u;
                    if (group.y) push(group);
                    group = make_uint2(0u, 0u);
                    const uint4 tail = __ldg(reinterpret_cast<const uint4*>(sc.inst_trav + ii) + 3);
                    if (tail.x != 0xFFFFFFFFu) {   // (a model without triangles has no bottom level)
                        push(make_uint2(kLevelMarker, 0u));
                        r = instance_ray(make_trace_ray(wo.x, wo.y, wo.z, wd.x, wd.y, wd.z, wo.w, wd.w), sc.inst_trav + ii);
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

    const bool empty = sc.node_count == 0;
    if (!empty) advance();
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
    if (err && valid && j == 0) atomicOr(err_flag, err);
    if (!valid || j != 0 || !hits) return;
    Hit h;
    h.prim = best_prim;
    h.t = best_t;
    h.u = 0.0f;
    h.v = 0.0f;
    if (h.prim != kMiss) {
        TraceRay w = make_trace_ray(wo.x, wo.y, wo.z, wd.x, wd.y, wd.z, wo.w, wd.w);
        if (TWO && sc.inst_trav) w = instance_ray(w, sc.inst_trav + best_inst);
        const float4* tp = tris + 3ull * best_rec;
        const float4 a = __ldg(tp), b = __ldg(tp + 1), c = __ldg(tp + 2);
        if (!refine_hit(w, a, b, c, h)) {   // the test's own t, u, v stand (a degenerate determinant)
            w.tmin = -INFINITY;
            intersect_triangle(w, a, b, c, INFINITY, h.t, h.u, h.v);
        }
    }
    __stcs(reinterpret_cast<float4*>(hits) + i, make_float4(__uint_as_float(h.prim), h.t, h.u, h.v));
}

// The same for two-level scenes (top level over instances, bottom levels per model).  Closest hit is
// held to 64 registers (8 blocks per SM): 4 % faster than the 80 it takes unbounded on 256 instances;
// any hit was 1 % slower when bounded, so it keeps its own allocation.
template <bool ANY, bool COUNT>
__global__ void __launch_bounds__(kTraceBlock, ANY ? 1 : 8) raycast_kernel_two_level(DeviceScene sc, const Ray* __restrict__ rays,
                                                                      uint32_t n, Hit* __restrict__ hits,
                                                                      unsigned long long* counters, uint32_t* err_flag,
                                                                      const uint32_t* __restrict__ order) {
    __shared__ uint2 stack[kSmemStack * kTraceBlock];
    const uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    TraceCounters c{0u, 0u};
    if (k < n) {
        const uint64_t i = order ? order[k] : k;
        const float4* rp = reinterpret_cast<const float4*>(rays) + 2ull * i;
        const float4 a = __ldcs(rp), b = __ldcs(rp + 1);
        const TraceRay r = make_trace_ray(a.x, a.y, a.z, b.x, b.y, b.z, a.w, b.w);
        Hit h;
        HitTail tail;
        uint32_t e = 0;
        if (sc.node_count) {
            e = traverse_two_level<ANY, COUNT, true, kSmemStack>(sc, r, stack + threadIdx.x, kTraceBlock, h, c, tail);
        } else {
            h.prim = kMiss; h.t = r.tmax; h.u = 0.0f; h.v = 0.0f;
        }
        if (hits) __stcs(reinterpret_cast<float4*>(hits) + i, make_float4(__uint_as_float(h.prim), h.t, h.u, h.v));
        if (e) atomicOr(err_flag, e);
    }
    reduce_counters<COUNT>(c, counters);
}

// ------------------------------------------------------------------------------------------------
// Coherence order: rays binned by (direction octant, Morton code of the origin's cell on an 8^3 grid
// over the bounds of the ray origins), bins in Morton order, rays in input order within a bin per warp.
// Threads that trace consecutive rays of this order follow similar paths through the tree; hits are
// written to each ray's own slot, so results do not depend on the order.
constexpr int kBinBits = 12;
constexpr uint32_t kBins = 1u << kBinBits;
constexpr int kBinBlock = 256;

// Float bits mapped to an unsigned key with the same order (min/max by integer atomics).
__device__ __forceinline__ uint32_t ordered_bits(float f) {
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float from_ordered(uint32_t k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k);
}

// bounds[0..2] = ordered min of the origins, bounds[3..5] = ordered max (pre-set to 0xFFFFFFFF / 0).
__global__ void __launch_bounds__(kBinBlock) k_ray_bounds(const Ray* __restrict__ rays, uint32_t n,
                                                          uint32_t* __restrict__ bounds) {
    uint32_t lo[3] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu}, hi[3] = {0u, 0u, 0u};
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const float4 a = __ldg(reinterpret_cast<const float4*>(rays) + 2ull * i);
        const uint32_t k[3] = {ordered_bits(a.x), ordered_bits(a.y), ordered_bits(a.z)};
        for (int c = 0; c < 3; ++c) {
            lo[c] = min(lo[c], k[c]);
            hi[c] = max(hi[c], k[c]);
        }
    }
    for (int c = 0; c < 3; ++c)
        for (int o = 16; o > 0; o >>= 1) {
            lo[c] = min(lo[c], __shfl_xor_sync(0xFFFFFFFFu, lo[c], o));
            hi[c] = max(hi[c], __shfl_xor_sync(0xFFFFFFFFu, hi[c], o));
        }
    if ((threadIdx.x & 31) == 0)
        for (int c = 0; c < 3; ++c) {
            atomicMin(bounds + c, lo[c]);
            atomicMax(bounds + 3 + c, hi[c]);
        }
}

__device__ __forceinline__ uint32_t spread3(uint32_t v) {   // 3 bits -> bits 0, 3, 6
    return (v & 1u) | ((v & 2u) << 2) | ((v & 4u) << 4);
}

__device__ __forceinline__ uint32_t ray_bin(const Ray* rays, uint64_t i, const uint32_t* bounds) {
    const float4* rp = reinterpret_cast<const float4*>(rays) + 2ull * i;
    const float4 a = __ldg(rp), b = __ldg(rp + 1);
    const uint32_t oct = (b.x < 0.0f ? 4u : 0u) | (b.y < 0.0f ? 2u : 0u) | (b.z < 0.0f ? 1u : 0u);
    auto cell = [&](float x, int c) {
        const float lo = from_ordered(bounds[c]), hi = from_ordered(bounds[3 + c]);
        const float t = hi > lo ? (x - lo) / (hi - lo) * 8.0f : 0.0f;
        return t >= 7.0f ? 7u : (t > 0.0f ? (uint32_t)t : 0u);   // NaN -> 0
    };
    return (oct << 9) | (spread3(cell(a.x, 0)) << 2) | (spread3(cell(a.y, 1)) << 1) | spread3(cell(a.z, 2));
}

// Per-block shared histograms, added to the global one with one atomic per non-empty bin and block.
__global__ void __launch_bounds__(kBinBlock) k_ray_bins(const Ray* __restrict__ rays, uint32_t n,
                                                        const uint32_t* __restrict__ bounds, uint32_t* __restrict__ bin_of,
                                                        uint32_t* __restrict__ hist) {
    __shared__ uint32_t h[kBins];
    for (uint32_t b = threadIdx.x; b < kBins; b += blockDim.x) h[b] = 0;
    __syncthreads();
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t b = ray_bin(rays, i, bounds);
        bin_of[i] = b;
        atomicAdd(h + b, 1u);
    }
    __syncthreads();
    for (uint32_t b = threadIdx.x; b < kBins; b += blockDim.x)
        if (h[b]) atomicAdd(hist + b, h[b]);
}

// Exclusive prefix sum of the kBins counts, in place (one block of 1024 threads, 4 bins each).
__global__ void __launch_bounds__(1024) k_bin_offsets(uint32_t* __restrict__ hist) {
    __shared__ uint32_t part[1024];
    constexpr uint32_t per = kBins / 1024;
    uint32_t local[per];
    uint32_t sum = 0;
    for (uint32_t j = 0; j < per; ++j) {
        local[j] = hist[threadIdx.x * per + j];
        sum += local[j];
    }
    part[threadIdx.x] = sum;
    __syncthreads();
    for (uint32_t off = 1; off < 1024; off <<= 1) {   // Hillis-Steele inclusive scan
        const uint32_t v = threadIdx.x >= off ? part[threadIdx.x - off] : 0u;
        __syncthreads();
        part[threadIdx.x] += v;
        __syncthreads();
    }
    uint32_t run = part[threadIdx.x] - sum;
    for (uint32_t j = 0; j < per; ++j) {
        hist[threadIdx.x * per + j] = run;
        run += local[j];
    }
}

__global__ void __launch_bounds__(kBinBlock) k_ray_scatter(const uint32_t* __restrict__ bin_of, uint32_t n,
                                                           uint32_t* __restrict__ cursor, uint32_t* __restrict__ order) {
    for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x; base < n; base += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t i = base + threadIdx.x;
        const bool valid = i < n;
        const uint32_t b = valid ? bin_of[i] : 0xFFFFFFFFu;
        const unsigned same = __match_any_sync(0xFFFFFFFFu, b);
        const int lane = threadIdx.x & 31, leader = __ffs(same) - 1;
        uint32_t pos = 0;
        if (valid && lane == leader) pos = atomicAdd(cursor + b, (uint32_t)__popc(same));
        pos = __shfl_sync(0xFFFFFFFFu, pos, leader);
        if (valid) order[pos + __popc(same & ((1u << lane) - 1u))] = (uint32_t)i;
    }
}

// Builds the coherence order of n rays in `order` (scratch: n bin ids, kBins counters, 6 bound words).
static void ray_order(const Ray* d_rays, uint64_t n, uint32_t* bin_of, uint32_t* hist, uint32_t* bounds,
                      uint32_t* order, int sm_count, cudaStream_t st) {
    const int grid = std::max(1, std::min<int>((int)((n + kBinBlock - 1) / kBinBlock), 2 * std::max(1, sm_count)));
    check_cuda(cudaMemsetAsync(hist, 0, kBins * sizeof(uint32_t), st), "cudaMemsetAsync");
    check_cuda(cudaMemsetAsync(bounds, 0xFF, 3 * sizeof(uint32_t), st), "cudaMemsetAsync");
    check_cuda(cudaMemsetAsync(bounds + 3, 0, 3 * sizeof(uint32_t), st), "cudaMemsetAsync");
    k_ray_bounds<<<grid, kBinBlock, 0, st>>>(d_rays, (uint32_t)n, bounds);
    k_ray_bins<<<grid, kBinBlock, 0, st>>>(d_rays, (uint32_t)n, bounds, bin_of, hist);
    k_bin_offsets<<<1, 1024, 0, st>>>(hist);
    k_ray_scatter<<<grid * 4, kBinBlock, 0, st>>>(bin_of, (uint32_t)n, hist, order);
}

template <bool ANY, bool COUNT, bool TWO>
static int persistent_grid(int sm_count) {
    static const int per_sm = [] {   // initialised once, thread-safely (a function-local static)
        int b = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, raycast_kernel<ANY, COUNT, TWO>, kCoopBlock,
                                                      coop_shared_bytes<false, TWO>());
        return std::max(1, b);
    }();
    return per_sm * std::max(1, sm_count);
}

template <bool ANY, bool COUNT, bool TWO>
static void launch_coop(const DeviceScene& s, const Ray* d_rays, uint64_t n, Hit* d_hits, unsigned long long* d_counters,
                        uint32_t* d_err, uint32_t* d_next, int sm_count, int refill, cudaStream_t st) {
    const uint64_t needed = (n + kCoopBlock - 1) / kCoopBlock;
    check_cuda(cudaMemsetAsync(d_next, 0, sizeof(uint32_t), st), "cudaMemsetAsync");
    const int grid = (int)std::min<uint64_t>(needed, (uint64_t)persistent_grid<ANY, COUNT, TWO>(sm_count));
    raycast_kernel<ANY, COUNT, TWO><<<grid, kCoopBlock, coop_shared_bytes<false, TWO>(), st>>>(
        s, d_rays, (uint32_t)n, d_hits, d_counters, d_err, d_next, (uint32_t)(32 - refill));
}

// Two-level scenes always run the default block size and stack depth.
template <bool ANY, bool COUNT, int BLOCK, int SS>
static void launch_grid(const DeviceScene& s, const Ray* d_rays, uint64_t n, Hit* d_hits,
                        unsigned long long* d_counters, uint32_t* d_err, const uint32_t* order, cudaStream_t st) {
    if (s.inst_trav) {
        const uint64_t blocks = (n + kTraceBlock - 1) / kTraceBlock;
        raycast_kernel_two_level<ANY, COUNT><<<(unsigned)blocks, kTraceBlock, 0, st>>>(s, d_rays, (uint32_t)n, d_hits,
                                                                                     d_counters, d_err, order);
        return;
    }
    const uint64_t blocks = (n + BLOCK - 1) / BLOCK;
    raycast_kernel_grid<ANY, COUNT, BLOCK, SS><<<(unsigned)blocks, BLOCK, 0, st>>>(
        s.nodes, s.tris, s.node_count, d_rays, (uint32_t)n, d_hits, d_counters, d_err, order);
}

template <bool ANY, int BLOCK>
static void launch_grid_stack(int stack, const DeviceScene& s, const Ray* d_rays, uint64_t n, Hit* d_hits,
                              uint32_t* d_err, const uint32_t* order, cudaStream_t st) {
    if (stack == 8) launch_grid<ANY, false, BLOCK, 8>(s, d_rays, n, d_hits, nullptr, d_err, order, st);
    else if (stack == 16) launch_grid<ANY, false, BLOCK, 16>(s, d_rays, n, d_hits, nullptr, d_err, order, st);
    else launch_grid<ANY, false, BLOCK, kSmemStack>(s, d_rays, n, d_hits, nullptr, d_err, order, st);
}

template <bool ANY>
static void launch(const DeviceScene& s, const Ray* d_rays, uint64_t n, Hit* d_hits, uint32_t* d_err, uint32_t* d_next,
                   int sm_count, const TraceConfig& cfg, cudaStream_t st) {
    // grid form (also for more than 2^31 rays, where the persistent form's fetch counter could wrap)
    if (cfg.refill <= 0 || n > (1ull << 31)) {
        uint32_t* scratch = nullptr;
        const uint32_t* order = nullptr;
        if (cfg.sort) {   // stream-ordered scratch: concurrent calls on other streams do not share it
            check_cuda(cudaMallocAsync((void**)&scratch, (2 * n + kBins + 8) * sizeof(uint32_t), st), "cudaMallocAsync");
            ray_order(d_rays, n, scratch, scratch + 2 * n, scratch + 2 * n + kBins, scratch + n, sm_count, st);
            order = scratch + n;
        }
        if (cfg.block == 64) launch_grid_stack<ANY, 64>(cfg.stack, s, d_rays, n, d_hits, d_err, order, st);
        else if (cfg.block == 256) launch_grid_stack<ANY, 256>(cfg.stack, s, d_rays, n, d_hits, d_err, order, st);
        else launch_grid_stack<ANY, kTraceBlock>(cfg.stack, s, d_rays, n, d_hits, d_err, order, st);
        if (scratch) check_cuda(cudaFreeAsync(scratch, st), "cudaFreeAsync");
        return;
    }
    // The default form of few rays: eight lanes per ray until the chip is several times full of them, two rays per warp
    // while that leaves SMs with free slots (a warp takes as long as the longest of its rays).  Cooperative against
    // wide with four and with two rays per warp, closest hit, us a call:
    //                        1,280 triangles   81,920            1,310,720         64 instances of 5,120
    //     1,000 rays         22.9  12.1  10.5  35.1  24.7  24.8  61.5  43.3  39.1  63.0  39.1  29.9
    //     10,000 rays        24.2  14.4  16.6  49.4  35.0  34.9  67.8  53.5  56.0  78.0  47.2  39.4
    //     50,500 rays        33.9  32.1  45.0  73.5  52.1  68.2  86.9  67.1  83.0  90.4  63.8  83.2
    //     80,000 rays        35.2  43.3  65.4  82.1  65.8  93.1   101  88.8   119   101  92.1   124
    const uint64_t sms = (uint64_t)std::max(1, sm_count);
    if (cfg.refill == kDefaultRefill && n <= sms * 352) {
        const uint32_t per_warp = n <= sms * 64 ? 2u : 4u;
        const unsigned blocks = (unsigned)((n + per_warp * (kWideBlock / 32) - 1) / (per_warp * (kWideBlock / 32)));
        if (s.inst_trav) raycast_kernel_wide<ANY, true><<<blocks, kWideBlock, 0, st>>>(s, d_rays, (uint32_t)n, d_hits, d_err, per_warp);
        else raycast_kernel_wide<ANY, false><<<blocks, kWideBlock, 0, st>>>(s, d_rays, (uint32_t)n, d_hits, d_err, per_warp);
        return;
    }
    if (s.inst_trav) launch_coop<ANY, false, true>(s, d_rays, n, d_hits, nullptr, d_err, d_next, sm_count, cfg.refill, st);
    else launch_coop<ANY, false, false>(s, d_rays, n, d_hits, nullptr, d_err, d_next, sm_count, cfg.refill, st);
}

// Writes a flat scene's per-triangle InstanceProperties and instance indices into its triangle records.
__global__ void __launch_bounds__(256) k_tag_triangles(TriRecord* tris, uint32_t n, const uint32_t* __restrict__ prim_props,
                                                       const uint32_t* __restrict__ prim_instance) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t prim = tris[i].prim;
    if (prim >= n) return;
    tris[i].pad1 = __uint_as_float(prim_props[prim]);
    tris[i].pad2 = __uint_as_float(prim_instance[prim]);
}

void tag_triangles(TriRecord* d_tris, uint32_t n, const uint32_t* d_prim_props, const uint32_t* d_prim_instance, cudaStream_t st) {
    if (n == 0) return;
    k_tag_triangles<<<(n + 255u) / 256u, 256, 0, st>>>(d_tris, n, d_prim_props, d_prim_instance);
    check_cuda(cudaGetLastError(), "triangle tagging");
}

bool valid_trace_config(const TraceConfig& c) {
    const bool block_ok = c.block == 0 || c.block == 64 || c.block == 128 || c.block == 256;
    const bool stack_ok = c.stack == 0 || c.stack == 8 || c.stack == 12 || c.stack == 16;
    return block_ok && stack_ok && c.refill >= 0 && c.refill <= 32 && (c.sort == 0 || c.sort == 1);
}

void launch_raycast(const DeviceScene& s, const Ray* d_rays, uint64_t n, Hit* d_hits, bool any, uint32_t* d_err,
                    uint32_t* d_next, int sm_count, const TraceConfig& cfg, cudaStream_t st) {
    if (n == 0) return;
    if (!valid_trace_config(cfg)) fail(REINA_ERR_INVALID, "invalid traversal launch configuration");
    if (any) launch<true>(s, d_rays, n, d_hits, d_err, d_next, sm_count, cfg, st);
    else launch<false>(s, d_rays, n, d_hits, d_err, d_next, sm_count, cfg, st);
}

void launch_raycast_counters(const DeviceScene& s, const Ray* d_rays, uint64_t n, bool any,
                             unsigned long long* d_counters, uint32_t* d_err, uint32_t* d_next, int sm_count,
                             cudaStream_t st) {
    if (n == 0) return;
    // The counting build of the default form, the cooperative one (its deferred triangle tests cull later, so it
    // may visit a few more nodes than the grid form); the grid form for more rays than its fetch counter holds.
    if (n > (1ull << 31)) {
        if (any) launch_grid<true, true, kTraceBlock, kSmemStack>(s, d_rays, n, nullptr, d_counters, d_err, nullptr, st);
        else launch_grid<false, true, kTraceBlock, kSmemStack>(s, d_rays, n, nullptr, d_counters, d_err, nullptr, st);
        return;
    }
    auto go = [&](auto any_c, auto two_c) {
        launch_coop<any_c.value, true, two_c.value>(s, d_rays, n, nullptr, d_counters, d_err, d_next, sm_count, kDefaultRefill, st);
    };
    if (any && s.inst_trav) go(std::true_type{}, std::true_type{});
    else if (any) go(std::true_type{}, std::false_type{});
    else if (s.inst_trav) go(std::false_type{}, std::true_type{});
    else go(std::false_type{}, std::false_type{});
}

}  // namespace rt
