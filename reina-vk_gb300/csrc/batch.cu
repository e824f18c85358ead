// Multi-job wavefront engine.  A wave is a set of path slots, each one (job, pixel, sample); it runs the same
// kernel sequence as the single-frame wavefront (init, extend, per-material shade, shadow, finish), with every
// kernel reading its path's job record for the scene, camera and integrator options.  A job's samples are
// scheduled in order (any number of a pixel's in one wave in NEE+MIS mode, one in the reference's mode) and
// summed in sample order: a job's image does not depend on the jobs it shares waves with.  The per-wave launch
// sequence is captured once per shape (bounces, materials, traversal form) into a CUDA graph and replayed;
// only the wave descriptor (segments + job table) is copied in before each wave.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <type_traits>

#include "batch.h"
#include "coop_trace.cuh"
#include "trace_device.cuh"
#include "wavefront_device.cuh"
#include "wide_trace.cuh"

namespace rt {

// Per-slot records of a path, each one a 32-byte sector that a kernel reads or writes as a whole (one array per
// field cost a sector per field once the queues had shuffled the paths).  Their members are read one by one,
// never as float4: the compiler then forms the same fused multiply-adds from them as from the arrays of
// the pass-by-pass kernels, so that all forms of a render keep the same bits.
struct alignas(16) PathRay {   // the current ray and what follows it from vertex to vertex
    float ox, oy, oz;
    uint32_t tag;              // job | kFlag* << kFlagShift
    float dx, dy, dz;
    uint32_t rng;
};
struct alignas(16) PathHit {   // the closest hit of the current ray
    uint32_t prim;
    float u, v;
    uint32_t props, inst, unused[3];
};
struct alignas(16) PathSum {
    float tr, tg, tb;          // throughput
    float ppdf;                // BSDF pdf of the direction sampled at the previous vertex
    float rr, rg, rb;          // radiance of the current sample
    float acc;                 // accumulatedDistance
};
struct alignas(16) ShadowRay {
    float ox, oy, oz, tmax, dx, dy, dz;
    uint32_t slot;
    float cr, cg, cb;          // contribution if unoccluded
    uint32_t job;
};
constexpr uint32_t kFlagShift = 30;
constexpr uint32_t kJobMask = (1u << kFlagShift) - 1u;

// Queue lengths of one bounce (u32 words of a 64-byte block, zero at the wave's start).
constexpr int kBncActive = 0;          // rays entering the bounce
constexpr int kBncQueue = 1;           // kNumQueues shade queues: miss, then material + 1
constexpr int kBncShadow = 6;
constexpr int kBncFetchExtend = 7;     // ray-fetch counters of the cooperative kernels
constexpr int kBncFetchShadow = 8;
constexpr uint32_t kBncWords = 16;
// Blocks of a wave: bounce b uses block b modulo kBncBlocks; a wave with more bounces clears the half it has
// left behind whenever it enters the other.
constexpr uint32_t kBncBlocks = 1024;

struct BatchLaunch {
    PathRay* ray;
    PathHit* hit;
    PathSum* sum;
    ShadowRay* shadow;
    uint32_t* active[2];     // queues of slots (ping-pong)
    uint32_t* miss;          // shade queues: a path is in one of them, so the materials share two arrays,
    uint32_t* shade[2];      // Lambertian from the front and Disney from the back, metal and dielectric
    uint32_t* totals;        // error word, ray and work counters of the wave (kCnt*)
    uint32_t* bounces;       // kBncBlocks blocks of kBncWords
    const WaveHeader* hdr;
    const WaveSeg* segs;
    const JobGpu* jobs;
    uint32_t P;
};

__device__ __forceinline__ uint32_t* shade_entry(const BatchLaunch& B, int m, uint32_t pos) {
    pos = checked_index(pos, B.P, B.totals + kCntError);
    if (m == kQueueMiss) return B.miss + pos;
    return B.shade[m == 2 || m == 3] + (m >= 3 ? B.P - 1u - pos : pos);
}

// Appends every lane to the queue `m` of its path (-1: none) at counters[m]: one atomic instruction for all
// queues.  All 32 lanes of the warp call it together.
__device__ __forceinline__ uint32_t append_by_queue(uint32_t* counters, int m) {
    const uint32_t same = __match_any_sync(0xFFFFFFFFu, m);
    const int lane = threadIdx.x & 31, leader = __ffs(same) - 1;
    uint32_t base = 0;
    if (lane == leader && m >= 0) base = atomicAdd(counters + m, (uint32_t)__popc(same));
    base = __shfl_sync(0xFFFFFFFFu, base, leader);
    return base + (uint32_t)__popc(same & ((1u << lane) - 1u));
}

// Appends the threads of a block with `pred` set to two queues at once, one atomic per queue and block.
// shared: 2 * (kBlock / 32) words; every thread of the block calls it together.
__device__ __forceinline__ void append_block(uint32_t* counter0, bool pred0, uint32_t& pos0, uint32_t* counter1, bool pred1,
                                             uint32_t& pos1, uint32_t* shared) {
    constexpr int kWarps = kBlock / 32;
    const uint32_t m0 = __ballot_sync(0xFFFFFFFFu, pred0), m1 = __ballot_sync(0xFFFFFFFFu, pred1);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) {
        shared[warp] = (uint32_t)__popc(m0);
        shared[kWarps + warp] = (uint32_t)__popc(m1);
    }
    __syncthreads();
    if (threadIdx.x < 2) {
        uint32_t* c = shared + kWarps * threadIdx.x;
        uint32_t total = 0;
        for (int w = 0; w < kWarps; ++w) {
            const uint32_t k = c[w];
            c[w] = total;
            total += k;
        }
        if (total) {
            const uint32_t base = atomicAdd(threadIdx.x == 0 ? counter0 : counter1, total);
            for (int w = 0; w < kWarps; ++w) c[w] += base;
        }
    }
    __syncthreads();
    const uint32_t lt = (1u << lane) - 1u;
    pos0 = shared[warp] + (uint32_t)__popc(m0 & lt);
    pos1 = shared[kWarps + warp] + (uint32_t)__popc(m1 & lt);
    __syncthreads();   // before the next call's writes
}

// Sets up slot i (job, pixel, sample, camera ray — raytrace.rgen.glsl:250-263); returns whether its job
// traces any segment (paths of jobs with maxBounces = 0 finish with zero radiance).
__device__ __forceinline__ bool init_slot(const BatchLaunch& B, const JobGpu* __restrict__ jobs, uint32_t i) {
    int lo = 0, hi = (int)B.hdr->nseg - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) / 2;
        if (B.segs[mid].wave_start <= i) lo = mid;
        else hi = mid - 1;
    }
    const WaveSeg sg = B.segs[lo];
    const JobGpu& J = jobs[sg.job];
    const uint32_t pixel = sg.pixel_start + (i - sg.wave_start);
    const uint32_t k = sg.sample;
    const uint32_t x = pixel % J.W, y = pixel / J.W;
    uint32_t rng;
    float acc;
    if (J.mode == kModeNeeMis) {
        rng = path_seed(pixel, J.pc.sampleBatch * J.spp + k, J.seed);
        acc = 0.0f;
    } else if (k == 0) {
        rng = (J.pc.sampleBatch * J.H + y) * J.W + x;
        acc = 0.0f;
    } else {
        rng = J.pix_rng[pixel];
        acc = J.pix_acc[pixel];
    }
    if (k == 0) {
        J.sr[pixel] = 0.0f; J.sg[pixel] = 0.0f; J.sb[pixel] = 0.0f;
        J.cnt[pixel] = 0;
    }
    V3 o, d;
    camera_ray(J.pc, J.W, J.H, x, y, rng, o, d);
    B.ray[i] = PathRay{o.x, o.y, o.z, sg.job, d.x, d.y, d.z, rng};
    B.sum[i] = PathSum{1.0f, 1.0f, 1.0f, 0.0f, 0.0f, 0.0f, 0.0f, acc};
    return J.max_bounces > 0;
}

__global__ void __launch_bounds__(kBlock) kb_init(BatchLaunch B, const JobGpu* __restrict__ jobs) {
    const uint32_t n = B.hdr->count;
    for (uint32_t base = blockIdx.x * blockDim.x; base < n; base += gridDim.x * blockDim.x) {
        const uint32_t i = base + threadIdx.x;
        const bool live = i < n && init_slot(B, jobs, i);
        const uint32_t pos = warp_append(B.bounces + kBncActive, live);
        if (live) B.active[0][checked_index(pos, B.P, B.totals + kCntError)] = i;
    }
}

// Records the hit of slot p and returns its shade queue.  `tail` names the instance and, for a flat scene, the
// InstanceProperties index (its triangle record carries both).
__device__ __forceinline__ int store_hit(const BatchLaunch& B, const DeviceScene& s, uint32_t p, const Hit& h, uint32_t inst,
                                         uint32_t pad1, uint32_t pad2) {
    if (h.prim == kMiss) return kQueueMiss;
    uint32_t props = pad1;
    if (s.inst_trav) props = instance_props(s, inst, h.prim);
    else inst = pad2;
    B.hit[p] = PathHit{h.prim, h.u, h.v, props, inst, {0u, 0u, 0u}};
    return 1 + (int)s.props_material[props];
}

// Adds a launch's ray count to a u64 total (one thread per launch; launches of a wave that add to the same
// total run one after the other).
__device__ __forceinline__ void count_rays(uint32_t* total, uint32_t n) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *reinterpret_cast<unsigned long long*>(total) += n;
}

// Grid form.  COUNT: the traversal work (nodes visited, triangles tested) is added to the wave's counters.
template <int BLOCK, int SS, bool TWO, bool COUNT = false>
__global__ void __launch_bounds__(BLOCK, 1024 / BLOCK) kb_extend(BatchLaunch B, const JobGpu* __restrict__ jobs, int cur,
                                                                 uint32_t* bounce) {
    __shared__ uint2 stack[SS * BLOCK];
    const uint32_t n = bounce[kBncActive];
    const uint32_t* q = B.active[cur];
    count_rays(B.totals + kCntRays, n);
    TraceCounters c{0u, 0u};
    for (uint32_t base = blockIdx.x * blockDim.x; base < n; base += gridDim.x * blockDim.x) {
        const uint32_t i = base + threadIdx.x;
        const bool active = i < n;
        int m = -1;
        uint32_t p = 0;
        if (active) {
            p = checked_index(q[i], B.P, B.totals + kCntError);
            const PathRay& w = B.ray[p];
            const DeviceScene& s = jobs[w.tag & kJobMask].s;
            const TraceRay r = make_trace_ray(w.ox, w.oy, w.oz, w.dx, w.dy, w.dz, 0.0f, 10000.0f);
            Hit h;
            HitTail tail;
            uint32_t e = 0;
            if (s.node_count) e = trace_scene<false, COUNT, true, SS, TWO>(s, r, stack + threadIdx.x, BLOCK, h, c, tail);
            else h.prim = kMiss;
            if (e) atomicOr(B.totals + kCntError, e);
            m = store_hit(B, s, p, h, tail.inst, tail.pad1, tail.pad2);
        }
        if (COUNT) warp_count64(reinterpret_cast<unsigned long long*>(B.totals + kCntShaded), active && m != kQueueMiss);
        const uint32_t pos = append_by_queue(bounce + kBncQueue, m);
        if (active) *shade_entry(B, m, pos) = p;
    }
    if (COUNT) coop_add_counts(c, B.totals, kCntNodes, kCntTris);
}

// Cooperative persistent form (coop_trace.cuh).  MIXED: the wave holds several jobs, and each lane's ray uses
// its own job's scene.
template <bool MIXED, bool TWO, bool COUNT>
__global__ void __launch_bounds__(kCoopBlock, TWO ? kCoopMinBlocksTwo : kCoopMinBlocks)
    kb_extend_coop(const __grid_constant__ BatchLaunch B, const JobGpu* __restrict__ jobs, int cur, uint32_t* bounce,
                   uint32_t refill_at) {
    const uint32_t n = bounce[kBncActive];
    const uint32_t* q = B.active[cur];
    count_rays(B.totals + kCntRays, n);
    TraceCounters c{0u, 0u};
    auto load = [&](uint32_t i, float4& o, float4& d) {
        const uint32_t p = checked_index(q[i], B.P, B.totals + kCntError);
        const PathRay& w = B.ray[p];
        o = make_float4(w.ox, w.oy, w.oz, 0.0f);
        d = make_float4(w.dx, w.dy, w.dz, 10000.0f);
        return &jobs[w.tag & kJobMask].s;
    };
    auto store = [&](uint32_t i, const CoopHit& h, bool valid) {   // called by all 32 lanes
        int m = -1;
        uint32_t p = 0;
        if (valid) {
            p = checked_index(q[i], B.P, B.totals + kCntError);
            const DeviceScene& s = jobs[MIXED ? B.ray[p].tag & kJobMask : 0u].s;
            m = store_hit(B, s, p, h.h, h.inst, h.pad1, h.pad2);
        }
        if (COUNT) warp_count64(reinterpret_cast<unsigned long long*>(B.totals + kCntShaded), valid && m != kQueueMiss);
        const uint32_t pos = append_by_queue(bounce + kBncQueue, m);
        if (valid) *shade_entry(B, m, pos) = p;
    };
    const uint32_t e = coop_trace<false, COUNT, true, MIXED, TWO>(jobs[0].s, n, bounce + kBncFetchExtend, refill_at, load, store, c);
    if (e) atomicOr(B.totals + kCntError, e);
    if (COUNT) coop_add_counts(c, B.totals, kCntNodes, kCntTris);
}

// Eight lanes per ray (wide_trace.cuh), for waves of few paths; up to `pairs` rays go two to a warp.
template <bool TWO>
__global__ void __launch_bounds__(kWideBlock) kb_extend_wide(BatchLaunch B, const JobGpu* __restrict__ jobs, int cur, uint32_t* bounce,
                                                            uint32_t pairs) {
    __shared__ uint2 stacks[kWideBlock / 8 * kTotalStack];
    const uint32_t n = bounce[kBncActive];
    const uint32_t* q = B.active[cur];
    count_rays(B.totals + kCntRays, n);
    auto load = [&](uint32_t i, float4& o, float4& d) {
        const uint32_t p = checked_index(q[i], B.P, B.totals + kCntError);
        const PathRay& w = B.ray[p];
        o = make_float4(w.ox, w.oy, w.oz, 0.0f);
        d = make_float4(w.dx, w.dy, w.dz, 10000.0f);
        return &jobs[w.tag & kJobMask].s;
    };
    auto store = [&](uint32_t i, const CoopHit& h, bool valid) {   // called by all 32 lanes
        int m = -1;
        uint32_t p = 0;
        if (valid) {
            p = checked_index(q[i], B.P, B.totals + kCntError);
            m = store_hit(B, jobs[B.ray[p].tag & kJobMask].s, p, h.h, h.inst, h.pad1, h.pad2);
        }
        const uint32_t pos = append_by_queue(bounce + kBncQueue, m);
        if (valid) *shade_entry(B, m, pos) = p;
    };
    const uint32_t e = wide_trace<false, true, TWO, true>(n, n <= pairs ? 2u : 4u, stacks, load, store);
    if (e) atomicOr(B.totals + kCntError, e);
}

// One kernel per material queue (MAT = 1 Lambertian, 2 metal, 3 dielectric, 4 Disney): the closest-hit shader,
// then the raygen loop body (raytrace.rgen.glsl:124-180).  `seg`: the bounce, which is also every path's depth.
template <int MAT>
__global__ void __launch_bounds__(kBlock, MAT == 4 ? kShadeMinBlocks : kShadeMinBlocksLight) kb_shade(BatchLaunch B, const JobGpu* __restrict__ jobs, int cur,
                                                                    uint32_t seg, const uint32_t* bounce, uint32_t* next_bounce,
                                                                    uint32_t* shadow_count) {
    __shared__ uint32_t appends[2 * (kBlock / 32)];
    const uint32_t n = bounce[kBncQueue + MAT];
    for (uint32_t base = blockIdx.x * blockDim.x; base < n; base += gridDim.x * blockDim.x) {
        const uint32_t i = base + threadIdx.x;
        const bool active = i < n;
        bool emit = false, cont = false;
        ShadowRec sh;
        uint32_t p = 0, job = 0;
        if (active) {
            p = checked_index(*shade_entry(B, MAT, i), B.P, B.totals + kCntError);
            const PathRay& w = B.ray[p];
            const PathHit& hit = B.hit[p];
            PathSum& sum = B.sum[p];
            const V3 ro{w.ox, w.oy, w.oz};
            const V3 rd{w.dx, w.dy, w.dz};
            uint32_t rng = w.rng;
            job = w.tag & kJobMask;
            uint32_t flags = w.tag >> kFlagShift;
            const uint32_t prim = hit.prim;
            V3 thr{sum.tr, sum.tg, sum.tb}, rad{sum.rr, sum.rg, sum.rb};
            float ppdf = sum.ppdf, acc = sum.acc;
            const JobGpu& J = jobs[job];
            const bool nee = J.mode == kModeNeeMis;
            const HitInfo h = hit_info<MAT == 4>(J.s, prim, hit.inst, hit.props, hit.u, hit.v, rd);
            const InstanceProperties& pr = J.s.props[h.props];
            const bool inside = (flags & kFlagInside) != 0;
            M3 tbn{};
            if (MAT == 4) tbn = h.tbn;
            Vertex vx;
            if (MAT == 1) vx = shade_lambert(J.s, h, pr, rd, rng, inside, acc);
            else if (MAT == 2) vx = shade_metal(J.s, h, pr, rd, rng, inside, acc);
            else if (MAT == 3) vx = shade_dielectric(J.s, h, pr, ro, rd, rng, inside, acc);
            else vx = shade_disney(J.s, h, tbn, pr, ro, rd, rng, inside, acc);
            if (vx.skip) {
                flags &= ~kFlagPrevNee;
            } else {
                flags = vx.inside ? (flags | kFlagInside) : (flags & ~kFlagInside);
                if (!vx.inside) {
                    V3 contrib = vx.emission;
                    if (nee) {
                        const float tw = J.pc.totalEmissiveWeight;
                        if ((flags & kFlagPrevNee) && (vx.emission.x != 0.0f || vx.emission.y != 0.0f || vx.emission.z != 0.0f))
                            contrib = contrib * power_heuristic(ppdf, light_pdf_sa(J.s, tw, prim, h.inst, h.props, ro, vx.newO));
                        const bool do_nee = (MAT == 1 || MAT == 4) && J.s.emissive_count > 0;
                        if (do_nee) emit = next_event(J.s, tw, rng, MAT == 4, vx.newO, vx.n, vx.albedo, pr, tbn, rd, thr, sh);
                        flags = do_nee ? (flags | kFlagPrevNee) : (flags & ~kFlagPrevNee);
                        ppdf = vx.pdf;
                    }
                    rad = rad + contrib * thr;
                    thr = thr * vx.color;
                } else {
                    flags &= ~kFlagPrevNee;
                }
            }
            sum = PathSum{thr.x, thr.y, thr.z, ppdf, rad.x, rad.y, rad.z, acc};
            B.ray[p] = PathRay{vx.newO.x, vx.newO.y, vx.newO.z, job | (flags << kFlagShift), vx.newD.x, vx.newD.y, vx.newD.z, rng};
            cont = seg + 1u < J.max_bounces;
        }
        uint32_t pos, spos;
        append_block(next_bounce + kBncActive, cont, pos, shadow_count, emit, spos, appends);
        if (cont) B.active[cur ^ 1][checked_index(pos, B.P, B.totals + kCntError)] = p;
        if (emit) {
            ShadowRay& r = B.shadow[checked_index(spos, B.P, B.totals + kCntError)];
            r = ShadowRay{sh.o.x, sh.o.y, sh.o.z, sh.tmax, sh.d.x, sh.d.y, sh.d.z, p, sh.contrib.x, sh.contrib.y, sh.contrib.z, job};
        }
    }
}

__global__ void __launch_bounds__(kBlock) kb_shade_miss(BatchLaunch B, const JobGpu* __restrict__ jobs, const uint32_t* bounce) {
    const uint32_t n = bounce[kBncQueue + kQueueMiss];
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t p = checked_index(*shade_entry(B, kQueueMiss, i), B.P, B.totals + kCntError);
        const PathRay& w = B.ray[p];
        PathSum& sum = B.sum[p];
        const JobGpu& J = jobs[w.tag & kJobMask];
        V3 sky;
        if (J.env_mode == 1) {
            sky = V3{J.env[0], J.env[1], J.env[2]};
        } else {
            const float y = norm3(V3{w.dx, w.dy, w.dz}).y;
            const float t = 0.5f * (y + 1.0f);
            sky = mix3(V3{0.1f, 0.1f, 0.1f}, V3{0.4f, 1.7f, 2.0f}, t) * 0.07f;
        }
        const V3 rad = V3{sum.rr, sum.rg, sum.rb} + sky * V3{sum.tr, sum.tg, sum.tb};
        sum.rr = rad.x; sum.rg = rad.y; sum.rb = rad.z;
    }
}

__device__ __forceinline__ void add_unoccluded(const BatchLaunch& B, uint32_t i) {
    const ShadowRay& s = B.shadow[i];
    PathSum& sum = B.sum[checked_index(s.slot, B.P, B.totals + kCntError)];
    const V3 rad = V3{sum.rr, sum.rg, sum.rb} + V3{s.cr, s.cg, s.cb};
    sum.rr = rad.x; sum.rg = rad.y; sum.rb = rad.z;
}

template <int BLOCK, int SS, bool TWO, bool COUNT = false>
__global__ void __launch_bounds__(BLOCK) kb_shadow(BatchLaunch B, const JobGpu* __restrict__ jobs, uint32_t* bounce) {
    __shared__ uint2 stack[SS * BLOCK];
    const uint32_t n = bounce[kBncShadow];
    count_rays(B.totals + kCntShadowRays, n);
    TraceCounters c{0u, 0u};
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const ShadowRay& w = B.shadow[i];
        const DeviceScene& s = jobs[w.job].s;
        const TraceRay r = make_trace_ray(w.ox, w.oy, w.oz, w.dx, w.dy, w.dz, 0.0f, w.tmax);
        Hit h;
        uint32_t e = 0;
        if (s.node_count) e = trace_scene<true, COUNT, false, SS, TWO>(s, r, stack + threadIdx.x, BLOCK, h, c);
        else h.prim = kMiss;
        if (e) atomicOr(B.totals + kCntError, e);
        if (h.prim == kMiss) add_unoccluded(B, i);
    }
    if (COUNT) {
        __syncwarp();
        coop_add_counts(c, B.totals, kCntShadowNodes, kCntShadowTris);
    }
}

// Cooperative persistent form of the shadow kernel.
template <bool MIXED, bool TWO, bool COUNT>
__global__ void __launch_bounds__(kCoopBlock, TWO ? kCoopMinBlocksTwo : kCoopMinBlocks)
    kb_shadow_coop(const __grid_constant__ BatchLaunch B, const JobGpu* __restrict__ jobs, uint32_t* bounce, uint32_t refill_at) {
    const uint32_t n = bounce[kBncShadow];
    count_rays(B.totals + kCntShadowRays, n);
    TraceCounters c{0u, 0u};
    auto load = [&](uint32_t i, float4& o, float4& d) {
        const ShadowRay& w = B.shadow[i];
        o = make_float4(w.ox, w.oy, w.oz, 0.0f);
        d = make_float4(w.dx, w.dy, w.dz, w.tmax);
        return &jobs[MIXED ? w.job : 0u].s;
    };
    auto store = [&](uint32_t i, const CoopHit& h, bool valid) {
        if (valid && h.h.prim == kMiss) add_unoccluded(B, i);
    };
    const uint32_t e = coop_trace<true, COUNT, false, MIXED, TWO>(jobs[0].s, n, bounce + kBncFetchShadow, refill_at, load, store, c);
    if (e) atomicOr(B.totals + kCntError, e);
    if (COUNT) coop_add_counts(c, B.totals, kCntShadowNodes, kCntShadowTris);
}

// Eight lanes per shadow ray.
template <bool TWO>
__global__ void __launch_bounds__(kWideBlock) kb_shadow_wide(BatchLaunch B, const JobGpu* __restrict__ jobs, uint32_t* bounce,
                                                            uint32_t pairs) {
    __shared__ uint2 stacks[kWideBlock / 8 * kTotalStack];
    const uint32_t n = bounce[kBncShadow];
    count_rays(B.totals + kCntShadowRays, n);
    auto load = [&](uint32_t i, float4& o, float4& d) {
        const ShadowRay& w = B.shadow[i];
        o = make_float4(w.ox, w.oy, w.oz, 0.0f);
        d = make_float4(w.dx, w.dy, w.dz, w.tmax);
        return &jobs[w.job].s;
    };
    auto store = [&](uint32_t i, const CoopHit& h, bool valid) {
        if (valid && h.h.prim == kMiss) add_unoccluded(B, i);
    };
    const uint32_t e = wide_trace<true, false, TWO, true>(n, n <= pairs ? 2u : 4u, stacks, load, store);
    if (e) atomicOr(B.totals + kCntError, e);
}

// raytrace.rgen.glsl:264-275 per pixel of each job in the wave: clamp (NaN kept), sample output, NaN
// drop, sum — over the pixel's samples in this wave in sample order (a job whose samples are independent
// may have several samples of a pixel in one wave) — and carry the RNG state and accumulatedDistance of
// the last one to the pixel's next sample.
__global__ void __launch_bounds__(kBlock) kb_finish(BatchLaunch B, const JobGpu* __restrict__ jobs) {
    const uint32_t n = B.hdr->finish_total;
    const int nj = (int)B.hdr->njobs;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        int lo = 0, hi = nj - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) / 2;
            if (jobs[mid].finish_start <= i) lo = mid;
            else hi = mid - 1;
        }
        const JobGpu& J = jobs[lo];
        const uint64_t px = (uint64_t)J.W * J.H;
        const uint64_t first = J.cursor0 + (i - J.finish_start), end = J.cursor0 + J.take;
        const uint32_t pixel = (uint32_t)(first % px);
        float sr = J.sr[pixel], sg = J.sg[pixel], sb = J.sb[pixel];
        uint32_t cnt = J.cnt[pixel];
        uint32_t slot = 0;
        float acc = 0.0f;
        for (uint64_t idx = first; idx < end; idx += px) {
            slot = J.wave_start + (uint32_t)(idx - J.cursor0);
            const PathSum& sum = B.sum[slot];
            acc = sum.acc;
            const V3 c = clamp_keep_nan(V3{sum.rr, sum.rg, sum.rb}, J.pc.directClamp);
            if (J.samples) {
                float* o = J.samples + 3ull * ((uint64_t)pixel * J.spp + idx / px);
                o[0] = c.x; o[1] = c.y; o[2] = c.z;
            }
            if (!has_nan3(c)) {
                sr += c.x;
                sg += c.y;
                sb += c.z;
                cnt += 1;
            }
        }
        J.sr[pixel] = sr; J.sg[pixel] = sg; J.sb[pixel] = sb;
        J.cnt[pixel] = cnt;
        J.pix_rng[pixel] = B.ray[slot].rng;
        J.pix_acc[pixel] = acc;
    }
}

// raytrace.rgen.glsl:277-284 for one finished job.
__global__ void __launch_bounds__(kBlock) kb_resolve(JobGpu J) {
    const uint32_t n = J.W * J.H;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float k = (float)J.cnt[i];
        V3 fin{J.sr[i] / k, J.sg[i] / k, J.sb[i] / k};
        float4* a = reinterpret_cast<float4*>(J.accum) + i;
        if (J.pc.sampleBatch > 0) {
            const float4 prev = *a;
            fin = div3(V3{prev.x, prev.y, prev.z} * (float)J.pc.sampleBatch + fin, (float)(J.pc.sampleBatch + 1));
        }
        *a = make_float4(fin.x, fin.y, fin.z, 1.0f);
    }
}

// ------------------------------------------------------------------------------------------------
// Host side
static_assert(kBatchPathBytes == sizeof(PathRay) + sizeof(PathHit) + sizeof(PathSum) + sizeof(ShadowRay) + 5 * sizeof(uint32_t),
              "path state and queues of a wave slot");
constexpr size_t kWaveHeadBytes = 256 + kBncBlocks * kBncWords * sizeof(uint32_t);   // totals, bounce blocks
constexpr uint32_t kMaxWaveJobs = kMaxWaveSegments / 2;
static_assert(kMaxWaveJobs <= kJobMask, "a path's job index shares a word with its flags");

static BatchLaunch layout_batch(uint8_t* w, size_t P) {
    BatchLaunch b;
    std::memset(&b, 0, sizeof(b));
    b.totals = reinterpret_cast<uint32_t*>(w);
    b.bounces = reinterpret_cast<uint32_t*>(w + 256);
    w += kWaveHeadBytes;
    auto take = [&](auto*& p) {
        p = reinterpret_cast<std::remove_reference_t<decltype(p)>>(w);
        w += P * sizeof(*p);
    };
    take(b.ray);
    take(b.hit);
    take(b.sum);
    take(b.shadow);
    take(b.active[0]);
    take(b.active[1]);
    take(b.miss);
    take(b.shade[0]);
    take(b.shade[1]);
    b.P = (uint32_t)P;
    return b;
}

static int occupancy(const void* fn, int sm_count) {
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kBlock, 0);
    return std::max(1, per_sm) * std::max(1, sm_count);
}

BatchEngine::BatchEngine(int device, int sm_count, uint32_t wave_capacity, bool use_graphs, const TraceConfig& trace,
                         int lanes)
    : device_(device), sm_count_(sm_count), capacity_(wave_capacity), use_graphs_(use_graphs), trace_(trace) {
    if (wave_capacity == 0) fail(REINA_ERR_INVALID, "wave capacity must be positive");
    if (lanes < 1 || lanes > 16) fail(REINA_ERR_INVALID, "a batch engine has 1 to 16 lanes");
    desc_bytes_ = sizeof(WaveHeader) + kMaxWaveSegments * sizeof(WaveSeg) + kMaxWaveJobs * sizeof(JobGpu);
    lanes_.resize((size_t)lanes);
    try {
        // one block of path state: a part per lane, or all of it one wave's (coop_)
        paths_.alloc(lanes_.size() * lane_bytes());
        check_cuda(cudaEventCreateWithFlags(&caller_, cudaEventDisableTiming), "cudaEventCreate");
        for (size_t k = 0; k < lanes_.size(); ++k) {
            Lane& L = lanes_[k];
            L.index = k;
            L.desc.alloc(desc_bytes_);
            check_cuda(cudaMallocHost(&L.host_desc, desc_bytes_), "cudaMallocHost");
            check_cuda(cudaMallocHost(reinterpret_cast<void**>(&L.host_counters), kNumCounters * sizeof(uint32_t)),
                       "cudaMallocHost");
            check_cuda(cudaStreamCreateWithFlags(&L.stream, cudaStreamNonBlocking), "cudaStreamCreate");
            check_cuda(cudaEventCreateWithFlags(&L.finished, cudaEventDisableTiming), "cudaEventCreate");
            check_cuda(cudaEventCreateWithFlags(&L.done, cudaEventDisableTiming), "cudaEventCreate");
        }
    } catch (...) {   // the destructor does not run for a constructor that throws
        release_lanes();
        throw;
    }
    with_trace_variant(trace_, [&](auto B, auto S) {
        blocks_ext_ = resident_grid((const void*)kb_extend<B.value, S.value, false>, B.value, sm_count);
        blocks_sh_ = resident_grid((const void*)kb_shadow<B.value, S.value, false>, B.value, sm_count);
    });
    blocks_shade_[1] = occupancy((const void*)kb_shade<1>, sm_count);
    blocks_shade_[2] = occupancy((const void*)kb_shade<2>, sm_count);
    blocks_shade_[3] = occupancy((const void*)kb_shade<3>, sm_count);
    blocks_shade_[4] = occupancy((const void*)kb_shade<4>, sm_count);
    blocks_simple_ = occupancy((const void*)kb_finish, sm_count);
}

BatchEngine::~BatchEngine() { release_lanes(); }

void BatchEngine::release_lanes() {
    for (Lane& L : lanes_) {
        if (L.stream) cudaStreamSynchronize(L.stream);
        for (auto& g : L.graphs)
            if (g.exec) cudaGraphExecDestroy(g.exec);
        if (L.finished) cudaEventDestroy(L.finished);
        if (L.done) cudaEventDestroy(L.done);
        if (L.stream) cudaStreamDestroy(L.stream);
        if (L.host_desc) cudaFreeHost(L.host_desc);
        if (L.host_counters) cudaFreeHost(L.host_counters);
    }
    lanes_.clear();
    if (caller_) cudaEventDestroy(caller_);
    caller_ = nullptr;
}

size_t BatchEngine::lane_bytes() const { return kWaveHeadBytes + (kBatchPathBytes * (size_t)capacity_ + 255) / 256 * 256; }

void BatchEngine::prepare(BatchJob& job, cudaMemPool_t pool, cudaStream_t st) {
    const size_t px = (size_t)job.opt.width * job.opt.height;
    job.total = (uint64_t)job.pc.samplesPerPixel * px;
    job.cursor = 0;
    job.resolved = false;
    job.placed.clear();
    if (pool) job.pixel_state.alloc_async(px * 6 * sizeof(uint32_t), pool, st);
    else job.pixel_state.alloc(px * 6 * sizeof(uint32_t));
}

static JobGpu job_record(const BatchJob& j) {
    JobGpu g;
    std::memset(&g, 0, sizeof(g));
    g.s = j.scene;
    g.pc = j.pc;
    g.W = j.opt.width;
    g.H = j.opt.height;
    g.mode = j.opt.mode;
    g.seed = j.opt.seed;
    g.env_mode = j.opt.env_mode;
    for (int k = 0; k < 3; ++k) g.env[k] = j.opt.env_color[k];
    g.spp = j.pc.samplesPerPixel;
    g.max_bounces = j.pc.maxBounces;
    g.accum = j.d_accum;
    g.samples = j.d_samples;
    const size_t px = (size_t)g.W * g.H;
    uint32_t* w = j.pixel_state.as<uint32_t>();
    g.pix_rng = w;
    g.pix_acc = reinterpret_cast<float*>(w + px);
    g.sr = reinterpret_cast<float*>(w + 2 * px);
    g.sg = reinterpret_cast<float*>(w + 3 * px);
    g.sb = reinterpret_cast<float*>(w + 4 * px);
    g.cnt = w + 5 * px;
    return g;
}

// Work of a wave's bounces that may run side by side goes to streams of its own while the wave is captured:
// the graph then holds the kernels as parallel branches.  Without capture all of them are the wave's stream.
namespace {
class Branches {
public:
    Branches(cudaStream_t main, bool fork) : fork_(fork) {
        s_[0] = main;
        for (int k = 1; k < kCount; ++k) {
            s_[k] = main;
            if (fork_) check_cuda(cudaStreamCreateWithFlags(&s_[k], cudaStreamNonBlocking), "cudaStreamCreate");
        }
    }
    ~Branches() {
        for (cudaEvent_t e : events_) cudaEventDestroy(e);
        for (int k = 1; k < kCount && fork_; ++k)
            if (s_[k]) cudaStreamDestroy(s_[k]);
    }
    Branches(const Branches&) = delete;
    Branches& operator=(const Branches&) = delete;
    cudaStream_t operator[](int k) const { return s_[k]; }
    // Branch `to` continues after what branch `from` holds so far.
    void after(int to, int from) {
        if (!fork_) return;
        cudaEvent_t e;
        check_cuda(cudaEventCreateWithFlags(&e, cudaEventDisableTiming), "cudaEventCreate");
        events_.push_back(e);
        check_cuda(cudaEventRecord(e, s_[from]), "cudaEventRecord");
        check_cuda(cudaStreamWaitEvent(s_[to], e, 0), "cudaStreamWaitEvent");
    }
    static constexpr int kCount = 5;

private:
    bool fork_;
    cudaStream_t s_[kCount] = {};
    std::vector<cudaEvent_t> events_;
};
}  // namespace

template <bool MIXED, bool TWO, bool COUNT>
void BatchEngine::launch_coop(const BatchLaunch& B, bool extend, int cur, uint32_t* bounce, cudaStream_t st) {
    constexpr size_t shared = coop_shared_bytes<MIXED, TWO>();
    int& grid = blocks_coop_[extend][MIXED][TWO][COUNT];
    const void* fn = extend ? (const void*)kb_extend_coop<MIXED, TWO, COUNT> : (const void*)kb_shadow_coop<MIXED, TWO, COUNT>;
    if (grid == 0) grid = resident_grid(fn, kCoopBlock, sm_count_, shared);
    const uint32_t refill_at = (uint32_t)(32 - (trace_.refill > 0 ? trace_.refill : kDefaultRefill));
    if (extend) kb_extend_coop<MIXED, TWO, COUNT><<<grid, kCoopBlock, shared, st>>>(B, B.jobs, cur, bounce, refill_at);
    else kb_shadow_coop<MIXED, TWO, COUNT><<<grid, kCoopBlock, shared, st>>>(B, B.jobs, bounce, refill_at);
}

// The form of a call's waves: cooperative traversal or the grid form where it was asked for
// (reina_tuning.wave_refill), else by the jobs' scenes and paths.  A call of few paths waits for each bounce's
// longest ray, so it traces with eight lanes per ray (frames of 8 bounces with 4.6k / 12k / 30k / 46k paths, us,
// grid or cooperative against wide: 3 nodes 268 / 271 / 285 / 303 against 223 / 258 / 322 / 410; zoo of 12 instances
// 962 / 995 / 1061 / 1096 against 656 / 788 / 1036 / 1409; 64 instances 1275 / 1340 / 1428 / 1503 against 749 / 925
// / 1231 / 1692; 82k triangles 743 / 789 / 851 / 894 against 492 / 521 / 601 / 703, and 63k paths 934 against 816).
// (Counting waves without that request run the grid form, whose counts repeat from run to run.)
//
// The cooperative kernels fill every SM until their queue is empty, so waves of that form run one after the other,
// as large as the path state of all lanes allows (the launches' tails are what they lose: a 1920x1080, 16
// spp, 12-bounce frame of 1.3M triangles 75.3 ms in the grid form, 70.8, 53.5, 48.8 ms cooperative in waves
// of 2^21, 2^23, 2^24 paths).  Their bookkeeping pays from some hundred nodes on (frames of 1M paths,
// grid / cooperative: 3 nodes 1.36 / 1.85 ms, 144 nodes 1.75 / 1.87, 894 nodes 2.21 / 2.15, 21,898 nodes 3.14 /
// 2.78), for two-level scenes, whose rays do more per instance than per node, with enough paths (64k paths
// 1.25 / 1.33 ms, 400k 2.06 / 2.17, 1.4M 5.74 / 5.62, 1.6M over 64 instances 11.8 / 10.2).
//
// Grid-form waves overlap: a call of more than a few paths per SM's thread is cut into three waves even where one
// would hold it (1M paths: 1.54 ms as one wave, 1.36 as two, 1.39 as three; 1.4M of a two-level scene 6.40,
// 5.91, 5.74; 64k paths: one is best; 8 samples of the reference's mode, whose next sample of a pixel waits for
// its last, over 360k / 491k / 922k pixels of the zoo 10.9 / 19.8 / 22.9 ms with a wave per sample, 10.8 / 17.6 /
// 19.8 as three).
void BatchEngine::choose_form(const std::vector<BatchJob*>& jobs) {
    constexpr uint32_t kCoopNodes = 512;
    constexpr uint64_t kCoopTwoLevelPaths = kFormPaths;
    constexpr uint64_t kOverlapPaths = 1ull << 18, kOverlapWaves = 3;
    uint64_t paths = 0;   // that waves could hold at once: one sample per pixel of a job in the reference's mode
    uint32_t nodes = 0;
    bool two = false;
    for (const BatchJob* j : jobs) {
        const uint64_t px = (uint64_t)j->opt.width * j->opt.height;
        paths += std::min(j->total - j->cursor, j->opt.mode == kModeNeeMis ? j->total : px);
        nodes = std::max(nodes, j->scene.node_count);
        two = two || j->scene.inst_trav;
    }
    const uint64_t wide_paths = (two ? 192ull : nodes >= kCoopNodes ? 352ull : 96ull) * sm_count_;
    wide_ = trace_.refill == 0 && !count_ && paths <= wide_paths;
    coop_ = trace_.refill > 0 ||
            (trace_.refill == 0 && !count_ && !wide_ && (two ? paths >= kCoopTwoLevelPaths : nodes >= kCoopNodes));
    wave_limit_ = UINT32_MAX;
    if (!coop_ && paths >= kOverlapPaths) {
        const uint64_t waves = std::max<uint64_t>(std::min<uint64_t>(kOverlapWaves, lanes_.size()), (paths + capacity_ - 1) / capacity_);
        wave_limit_ = (uint32_t)((paths + waves - 1) / waves);
    }
}

// One traversal launch of the wave in the form that suits it.
void BatchEngine::launch_trace(const BatchLaunch& B, const Shape& w, bool extend, int cur, uint32_t* bounce, cudaStream_t st) {
    if (w.coop) {
        auto by = [&](auto mixed, auto two) {
            if (w.count) launch_coop<mixed.value, two.value, true>(B, extend, cur, bounce, st);
            else launch_coop<mixed.value, two.value, false>(B, extend, cur, bounce, st);
        };
        if (w.mixed && w.two) by(std::true_type{}, std::true_type{});
        else if (w.mixed) by(std::true_type{}, std::false_type{});
        else if (w.two) by(std::false_type{}, std::true_type{});
        else by(std::false_type{}, std::false_type{});
        return;
    }
    if (w.wide) {
        const uint32_t pairs = wide_pair_limit(sm_count_);
        auto by = [&](auto two) {
            if (extend) kb_extend_wide<two.value><<<w.wide, kWideBlock, 0, st>>>(B, B.jobs, cur, bounce, pairs);
            else kb_shadow_wide<two.value><<<w.wide, kWideBlock, 0, st>>>(B, B.jobs, bounce, pairs);
        };
        if (w.two) by(std::true_type{});
        else by(std::false_type{});
        return;
    }
    // grid form: two-level scenes and counting waves run the default variant
    auto go = [&](auto bs, auto ss, auto two, auto count, int grid) {
        if (extend) kb_extend<bs.value, ss.value, two.value, count.value><<<grid, bs.value, 0, st>>>(B, B.jobs, cur, bounce);
        else kb_shadow<bs.value, ss.value, two.value, count.value><<<grid, bs.value, 0, st>>>(B, B.jobs, bounce);
    };
    auto plain = [&](auto two, auto count) {
        std::integral_constant<int, kTraceBlock> bs;
        std::integral_constant<int, kDefaultTraceStack> ss;
        int& grid = blocks_plain_[extend][two.value][count.value];
        if (grid == 0)
            grid = resident_grid(extend ? (const void*)kb_extend<bs.value, ss.value, two.value, count.value>
                                        : (const void*)kb_shadow<bs.value, ss.value, two.value, count.value>,
                                 kTraceBlock, sm_count_);
        go(bs, ss, two, count, grid);
    };
    if (w.two && w.count) plain(std::true_type{}, std::true_type{});
    else if (w.two) plain(std::true_type{}, std::false_type{});
    else if (w.count) plain(std::false_type{}, std::true_type{});
    else
        with_trace_variant(trace_, [&](auto bs, auto ss) {
            go(bs, ss, std::false_type{}, std::false_type{}, extend ? blocks_ext_ : blocks_sh_);
        });
}

// The kernels of a wave: init, then per bounce extend -> the shade kernels of the materials that the wave's scenes
// have and the miss kernel, side by side -> the next bounce's extend, beside which the shadow rays run (they
// touch the radiance only, which nothing reads before the next bounce's shade and miss kernels).
void BatchEngine::launch_sequence(const BatchLaunch& B, const Shape& w, cudaStream_t main, bool fork) {
    enum { kMain = 0, kMissB = 1, kDisneyB = 2, kSpecularB = 3, kShadowB = 4 };
    const int simple = std::min<int>(blocks_simple_, (int)((B.P + kBlock - 1) / kBlock));
    check_cuda(cudaMemsetAsync(B.totals, 0, kWaveHeadBytes, main), "cudaMemsetAsync");
    kb_init<<<simple, kBlock, 0, main>>>(B, B.jobs);
    Branches br(main, fork);
    auto has = [&](int material) { return (w.materials >> material & 1u) != 0; };
    bool shadows = false;   // a shadow launch is in flight
    for (uint32_t seg = 0; seg < w.bounces; ++seg) {
        const int cur = (int)(seg & 1u);
        constexpr uint32_t kHalf = kBncBlocks / 2;
        if (seg > 0 && seg % kHalf == 0) {   // entering a half: the other one is clear again for its next use
            if (shadows) br.after(kMain, kShadowB);
            const uint32_t other = (seg / kHalf + 1) % 2;
            check_cuda(cudaMemsetAsync(B.bounces + (size_t)other * kHalf * kBncWords, 0, kHalf * kBncWords * sizeof(uint32_t), main),
                       "cudaMemsetAsync");
        }
        uint32_t* bounce = B.bounces + (seg % kBncBlocks) * kBncWords;
        uint32_t* next = B.bounces + ((seg + 1) % kBncBlocks) * kBncWords;
        launch_trace(B, w, true, cur, bounce, br[kMain]);
        const bool specular = has(1) || has(2);
        if (shadows) br.after(kMain, kShadowB);   // the previous bounce's shadow rays have added their radiance
        br.after(kMissB, kMain);
        if (has(3)) br.after(kDisneyB, kMain);
        if (specular) br.after(kSpecularB, kMain);
        kb_shade_miss<<<simple, kBlock, 0, br[kMissB]>>>(B, B.jobs, bounce);
        uint32_t* shadow_count = bounce + kBncShadow;
        if (has(3)) kb_shade<4><<<blocks_shade_[4], kBlock, 0, br[kDisneyB]>>>(B, B.jobs, cur, seg, bounce, next, shadow_count);
        if (has(0)) kb_shade<1><<<blocks_shade_[1], kBlock, 0, br[kMain]>>>(B, B.jobs, cur, seg, bounce, next, shadow_count);
        if (has(2)) kb_shade<3><<<blocks_shade_[3], kBlock, 0, br[kSpecularB]>>>(B, B.jobs, cur, seg, bounce, next, shadow_count);
        if (has(1)) kb_shade<2><<<blocks_shade_[2], kBlock, 0, br[kSpecularB]>>>(B, B.jobs, cur, seg, bounce, next, shadow_count);
        if (has(3)) br.after(kMain, kDisneyB);
        if (w.nee) {
            br.after(kShadowB, kMain);
            launch_trace(B, w, false, cur, bounce, br[kShadowB]);
            shadows = true;
        }
        br.after(kMain, kMissB);
        if (specular) br.after(kMain, kSpecularB);
    }
    if (shadows) br.after(kMain, kShadowB);
}

void BatchEngine::launch_body(Lane& L, const Packed& pk, cudaStream_t st) {
    const WaveHeader& h = pk.hdr;
    uint8_t* d = L.desc.as<uint8_t>();
    const uint8_t* hd = static_cast<const uint8_t*>(L.host_desc);
    check_cuda(cudaMemcpyAsync(d, hd, sizeof(WaveHeader) + h.nseg * sizeof(WaveSeg), cudaMemcpyHostToDevice, st),
               "H2D wave");
    const size_t job_off = sizeof(WaveHeader) + kMaxWaveSegments * sizeof(WaveSeg);
    check_cuda(cudaMemcpyAsync(d + job_off, hd + job_off, h.njobs * sizeof(JobGpu), cudaMemcpyHostToDevice, st),
               "H2D jobs");
    const BatchLaunch B = wave_view(L);
    Shape w = pk.shape;
    w.count = count_;
    w.coop = coop_;
    if (wide_) {   // blocks for the wave's first bounce, as a power of two (a graph is kept per shape)
        w.wide = 1;
        while (w.wide < (uint32_t)wide_blocks(h.count, h.count <= wide_pair_limit(sm_count_) ? 2u : 4u)) w.wide *= 2;
    }
    if (!w.coop) w.mixed = false;   // (the grid form reads the job's scene per path either way)
    if (!use_graphs_) {
        launch_sequence(B, w, st, false);
        check_cuda(cudaGetLastError(), "batch wave launch");
        return;
    }
    GraphSlot* slot = nullptr;
    for (auto& g : L.graphs)
        if (g.shape == w) slot = &g;
    if (!slot) {
        make_room(L, w.bounces);
        cudaStream_t cap;
        check_cuda(cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking), "cudaStreamCreate");
        cudaGraph_t graph = nullptr;
        cudaError_t err = cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal);
        if (err == cudaSuccess) {
            try {
                launch_sequence(B, w, cap, true);
            } catch (...) {   // end the capture before the stream goes
                cudaStreamEndCapture(cap, &graph);
                if (graph) cudaGraphDestroy(graph);
                cudaStreamDestroy(cap);
                throw;
            }
            err = cudaStreamEndCapture(cap, &graph);
        }
        cudaStreamDestroy(cap);
        check_cuda(err, "wave capture");
        GraphSlot g;
        g.shape = w;
        err = cudaGraphInstantiate(&g.exec, graph, 0);
        cudaGraphDestroy(graph);
        check_cuda(err, "cudaGraphInstantiate");
        L.graphs.push_back(g);
        slot = &L.graphs.back();
    }
    slot->used = submissions_;
    check_cuda(cudaGraphLaunch(slot->exec, st), "cudaGraphLaunch");
}

// Destroys the lane's graphs used longest ago until one of `bounces` more fits into kGraphBounces.  The lane is free,
// so none of them is running.
void BatchEngine::make_room(Lane& L, uint32_t bounces) {
    uint64_t held = 0;
    for (const GraphSlot& g : L.graphs) held += g.shape.bounces;
    while (!L.graphs.empty() && held + bounces > kGraphBounces) {
        const auto oldest = std::min_element(L.graphs.begin(), L.graphs.end(),
                                             [](const GraphSlot& a, const GraphSlot& b) { return a.used < b.used; });
        held -= oldest->shape.bounces;
        cudaGraphExecDestroy(oldest->exec);
        L.graphs.erase(oldest);
    }
}

BatchLaunch BatchEngine::wave_view(const Lane& L) const {
    uint8_t* d = L.desc.as<uint8_t>();
    BatchLaunch B = layout_batch(paths_.as<uint8_t>() + L.index * lane_bytes(), wave_slots());
    B.hdr = reinterpret_cast<const WaveHeader*>(d);
    B.segs = reinterpret_cast<const WaveSeg*>(d + sizeof(WaveHeader));
    B.jobs = reinterpret_cast<const JobGpu*>(d + sizeof(WaveHeader) + kMaxWaveSegments * sizeof(WaveSeg));
    return B;
}

void BatchEngine::launch_finish(Lane& L, const Packed& pk, cudaStream_t st) {
    const BatchLaunch B = wave_view(L);
    const int simple = std::min<int>(blocks_simple_, (int)((B.P + kBlock - 1) / kBlock));
    kb_finish<<<simple, kBlock, 0, st>>>(B, B.jobs);
    for (BatchJob* j : pk.completed) {   // resolve the jobs this wave completed
        const JobGpu g = job_record(*j);
        const uint32_t px = g.W * g.H;
        const int blocks = (int)std::min<uint32_t>((px + kBlock - 1) / kBlock, (uint32_t)blocks_simple_);
        kb_resolve<<<blocks, kBlock, 0, st>>>(g);
    }
    check_cuda(cudaGetLastError(), "batch launch");
    check_cuda(cudaEventRecord(L.finished, st), "cudaEventRecord");
    check_cuda(cudaMemcpyAsync(L.host_counters, B.totals, kNumCounters * sizeof(uint32_t), cudaMemcpyDeviceToHost,
                               st), "D2H counters");
    check_cuda(cudaEventRecord(L.done, st), "cudaEventRecord");
    L.pending = true;
}

void BatchEngine::collect(Lane& L) {
    if (!L.pending) return;
    L.pending = false;
    const uint32_t* c = L.host_counters;
    auto u64 = [&](int at) { uint64_t v; std::memcpy(&v, c + at, 8); return v; };
    rays_ += u64(kCntRays);
    shadow_rays_ += u64(kCntShadowRays);
    work_.nodes += u64(kCntNodes);
    work_.tris += u64(kCntTris);
    work_.shadow_nodes += u64(kCntShadowNodes);
    work_.shadow_tris += u64(kCntShadowTris);
    work_.shaded += u64(kCntShaded);
    waves_++;
    if (c[kCntError])
        fail(REINA_ERR_DEVICE, "batch wave kernels raised error flag " + std::to_string(c[kCntError]) +
                                   device_error_text(c[kCntError]));
}

BatchEngine::Packed BatchEngine::pack(const std::vector<BatchJob*>& jobs, bool fifo, Lane& L) {
    Packed pk;
    const uint64_t capacity = std::min(wave_slots(), wave_limit_);
    std::memset(&pk.hdr, 0, sizeof(pk.hdr));
    // active jobs (at most kMaxWaveJobs per wave; the rest wait for a later wave)
    std::vector<BatchJob*> active;
    for (BatchJob* j : jobs)
        if (j->cursor < j->total && active.size() < kMaxWaveJobs) active.push_back(j);
    if (active.empty()) return pk;
    // fair share of the capacity, then leftovers to the oldest jobs (or, first-come first-served, each
    // job in order takes all it can use)
    // A job's samples per pixel in one wave: any number when its samples are independent (NEE+MIS: seeded
    // by (pixel, sample); the finish kernel sums a pixel's samples of the wave in order); one in the
    // reference's mode, where a pixel's next sample starts from the state its previous one left.
    // Where waves are cut to overlap, such a job's do not cross from one sample into the next: with 3 waves a sample,
    // each then waits for the third wave ahead of it, and not for the second.
    auto cap = [&](const BatchJob* j) -> uint64_t {
        if (j->opt.mode == kModeNeeMis) return UINT64_MAX;
        const uint64_t px = (uint64_t)j->opt.width * j->opt.height;
        return wave_limit_ == UINT32_MAX ? px : px - j->cursor % px;
    };
    std::vector<uint64_t> take(active.size(), 0);
    const uint64_t fair = fifo ? capacity : std::max<uint64_t>(1, capacity / active.size());
    uint64_t used = 0;
    for (size_t a = 0; a < active.size(); ++a) {
        const BatchJob* j = active[a];
        take[a] = std::min({fair, cap(j), j->total - j->cursor, capacity - used});
        used += take[a];
    }
    for (size_t a = 0; a < active.size() && used < capacity; ++a) {
        const BatchJob* j = active[a];
        const uint64_t more = std::min(std::min(cap(j), j->total - j->cursor) - take[a], capacity - used);
        take[a] += more;
        used += more;
    }
    uint8_t* h = static_cast<uint8_t*>(L.host_desc);
    WaveHeader* hdr = reinterpret_cast<WaveHeader*>(h);
    WaveSeg* segs = reinterpret_cast<WaveSeg*>(h + sizeof(WaveHeader));
    JobGpu* jt = reinterpret_cast<JobGpu*>(h + sizeof(WaveHeader) + kMaxWaveSegments * sizeof(WaveSeg));
    uint32_t nseg = 0, njobs = 0, wave_pos = 0, bounces = 0, finish = 0;
    for (size_t a = 0; a < active.size(); ++a) {
        if (take[a] == 0) continue;
        if (nseg >= kMaxWaveSegments) break;   // the descriptor is full: later jobs wait for the next wave
        BatchJob* j = active[a];
        const uint64_t px = (uint64_t)j->opt.width * j->opt.height;
        const uint32_t ji = njobs++;
        jt[ji] = job_record(*j);
        pk.members.push_back(j);
        bounces = std::max(bounces, j->pc.maxBounces);
        pk.shape.nee = pk.shape.nee || (j->opt.mode == kModeNeeMis && j->scene.emissive_count > 0);
        pk.shape.two = pk.shape.two || j->scene.inst_trav != nullptr;
        pk.shape.materials |= j->scene.material_mask;
        const uint64_t c0 = j->cursor;
        const uint32_t ws = wave_pos;
        uint64_t m = take[a];
        while (m > 0 && nseg < kMaxWaveSegments) {
            const uint64_t sample = j->cursor / px, pixel = j->cursor % px;
            const uint64_t c = std::min(m, px - pixel);
            WaveSeg& s = segs[nseg++];
            s.job = ji;
            s.wave_start = wave_pos;
            s.pixel_start = (uint32_t)pixel;
            s.count = (uint32_t)c;
            s.sample = (uint32_t)sample;
            wave_pos += (uint32_t)c;
            j->cursor += c;
            m -= c;
        }
        const uint64_t placed = j->cursor - c0;
        jt[ji].cursor0 = c0;
        jt[ji].wave_start = ws;
        jt[ji].take = (uint32_t)placed;
        jt[ji].finish_start = finish;
        finish += (uint32_t)std::min(placed, px);
        // samples after a pixel's first start from the state its previous sample left (reference mode): the wave that
        // holds the previous sample of the last pixel placed here, and with it those of the pixels before, comes first
        if (j->opt.mode != kModeNeeMis && j->pc.samplesPerPixel > 1) {
            const uint64_t end = c0 + placed;
            if (end > px && !j->placed.empty()) {
                size_t k = 0;
                while (k + 1 < j->placed.size() && j->placed[k].first < end - px) ++k;
                pk.after = std::max(pk.after, j->placed[k].second + 1);
                j->placed.erase(j->placed.begin(), j->placed.begin() + (std::ptrdiff_t)k);
            }
            j->placed.emplace_back(end, submitted_);
        }
        if (j->cursor == j->total && !j->resolved) {
            pk.completed.push_back(j);
            j->resolved = true;
        }
    }
    hdr->count = wave_pos;
    hdr->nseg = nseg;
    hdr->njobs = njobs;
    hdr->max_bounces = bounces;
    hdr->finish_total = finish;
    pk.shape.bounces = bounces;
    pk.shape.mixed = njobs > 1;
    pk.hdr = *hdr;
    return pk;
}

bool BatchEngine::submit_wave(const std::vector<BatchJob*>& jobs, bool fifo, std::vector<BatchJob*>* members,
                              std::vector<BatchJob*>* completed) {
    Lane& L = lane_of(submitted_);
    if (L.pending) fail(REINA_ERR_STATE, "batch engine: no free lane");
    Packed pk = pack(jobs, fifo, L);
    if (pk.hdr.count == 0) return false;
    if (!L.ordered) {   // the lane's first wave of a run_all: after the caller's work
        check_cuda(cudaStreamWaitEvent(L.stream, caller_, 0), "cudaStreamWaitEvent");
        L.ordered = true;
    }
    Lane* prev = submitted_ > 0 ? &lane_of(submitted_ - 1) : nullptr;
    if (prev == &L) prev = nullptr;   // one lane: stream order already chains the waves
    if (pk.after > 0) {   // (a wave of this lane is ahead of this one on its stream)
        Lane& D = lane_of(pk.after - 1);
        if (&D != &L) check_cuda(cudaStreamWaitEvent(L.stream, D.finished, 0), "cudaStreamWaitEvent");
    }
    ++submissions_;
    launch_body(L, pk, L.stream);
    if (prev) check_cuda(cudaStreamWaitEvent(L.stream, prev->finished, 0), "cudaStreamWaitEvent");
    launch_finish(L, pk, L.stream);
    ++submitted_;
    if (members) *members = std::move(pk.members);
    if (completed) *completed = std::move(pk.completed);
    return true;
}

void BatchEngine::wait_oldest() {
    if (!pending()) return;
    Lane& L = lane_of(retired_);
    ++retired_;
    check_cuda(cudaEventSynchronize(L.done), "cudaEventSynchronize");
    collect(L);
}

void BatchEngine::drain() {
    for (Lane& L : lanes_) {
        cudaStreamSynchronize(L.stream);
        L.pending = false;
    }
    retired_ = submitted_;
}

void BatchEngine::run_all(const std::vector<BatchJob*>& jobs, cudaStream_t st, bool fifo) {
    try {
        choose_form(jobs);
        if (!pending()) submitted_ = retired_ = 0;   // from lane 0, whose graphs earlier calls have captured
        // each lane's first wave waits for the caller's work, and the caller's next work for the lanes used
        check_cuda(cudaEventRecord(caller_, st), "cudaEventRecord");
        for (Lane& L : lanes_) L.ordered = false;
        for (;;) {
            if (!lane_free()) wait_oldest();   // reuse the lane of the oldest wave
            if (!submit_wave(jobs, fifo)) break;
        }
        while (pending()) wait_oldest();
        for (Lane& L : lanes_)
            if (L.ordered) check_cuda(cudaStreamWaitEvent(st, L.done, 0), "cudaStreamWaitEvent");
        for (Lane& L : lanes_) L.ordered = true;
    } catch (...) {
        drain();   // nothing of this call stays in flight
        for (Lane& L : lanes_) L.ordered = true;
        throw;
    }
}

}  // namespace rt
