// Multi-job wavefront engine: many scenes, resolutions and sample budgets traced together in shared
// waves.  Used by reina_render_batch (all jobs known up front) and by the request server (jobs join
// and leave between waves).
#pragma once

#include <cstdint>
#include <memory>
#include <utility>
#include <vector>

#include <cuda_runtime_api.h>

#include "device_scene.h"
#include "errors.h"
#include "render.h"
#include "../../include/reina/polyglot.h"

namespace rt {

constexpr uint32_t kMaxWaveSegments = 1024;
constexpr size_t kBatchPathBytes = 164;   // path state and queues of a wave slot
// Bounces of the wave graphs that a lane keeps: about 130 KB of device and 20 KB of host memory each (graphs of 10
// to 329 bounces, one of each, took 7 GB and 2.4 GB).  A hundred shapes of ten bounces fit.
constexpr uint64_t kGraphBounces = 1024;
// Paths from which on the form of a call's waves no longer depends on their number (choose_form).
constexpr uint64_t kFormPaths = 1ull << 20;
struct BatchLaunch;                       // the kernels' view of a wave (batch.cu)

// Per-job data the kernels read (one table per wave, holding the jobs present in that wave).
struct JobGpu {
    DeviceScene s;
    RtPushConsts pc;
    uint32_t W, H, mode, seed, env_mode, spp, max_bounces, pad;
    float env[3];
    float pad2;
    float* accum;            // W*H RGBA32F
    float* samples;          // optional W*H*spp*3
    uint32_t* pix_rng;       // per-pixel state: carried RNG, accumulatedDistance, sample sums, count
    float* pix_acc;
    float *sr, *sg, *sb;
    uint32_t* cnt;
    // this wave: the job's slots are [wave_start, wave_start + take), holding its (sample * W*H + pixel)
    // indices [cursor0, cursor0 + take); finish threads [finish_start, finish_start + min(take, W*H)),
    // one per pixel, sum each pixel's samples of the wave in sample order
    uint64_t cursor0;
    uint32_t wave_start;
    uint32_t take;
    uint32_t finish_start;
    uint32_t pad3;
};

// A run of wave slots [wave_start, wave_start + count) holding pixels [pixel_start, ...) of one job's
// sample `sample`.
struct WaveSeg {
    uint32_t job;            // index into the wave's job table
    uint32_t wave_start;
    uint32_t pixel_start;
    uint32_t count;
    uint32_t sample;
    uint32_t pad[3];
};

struct WaveHeader {
    uint32_t count;          // paths in the wave
    uint32_t nseg;
    uint32_t njobs;
    uint32_t max_bounces;    // segments to run (max over the wave's jobs)
    uint32_t finish_total;   // finish threads (sum over jobs of min(take, W*H))
    uint32_t pad[3];         // 32 bytes: the job table after the segments stays 16-byte aligned
};
static_assert(sizeof(WaveHeader) == 32, "WaveHeader must stay 32 bytes");

// Host-side description of one job.
struct BatchJob {
    DeviceScene scene;
    RtPushConsts pc;
    RenderOpts opt;
    float* d_accum = nullptr;
    float* d_samples = nullptr;
    // progress
    uint64_t cursor = 0;     // next (sample * W*H + pixel) to schedule
    uint64_t total = 0;      // spp * W*H
    DeviceBuffer pixel_state;
    bool resolved = false;   // every sample is scheduled (set when the job's last wave is packed)
    std::vector<std::pair<uint64_t, uint64_t>> placed;   // samples that carry state: end cursor and number of recent waves
    void* owner = nullptr;   // the caller's record of the job (the server's request)
};

class BatchEngine {
public:
    // `lanes` path-state buffers (1 to 16) of `wave_capacity` slots each; waves rotate over them so that
    // one wave's last bounces overlap the next waves' first ones.
    BatchEngine(int device, int sm_count, uint32_t wave_capacity, bool use_graphs,
                const TraceConfig& trace = TraceConfig(), int lanes = 1);
    ~BatchEngine();
    BatchEngine(const BatchEngine&) = delete;
    BatchEngine& operator=(const BatchEngine&) = delete;

    // Allocates the job's per-pixel state (24 bytes per pixel); the job must outlive its waves.  With a
    // pool, the allocation is stream-ordered on `st` (DeviceBuffer::alloc_async).
    static void prepare(BatchJob& job, cudaMemPool_t pool = nullptr, cudaStream_t st = nullptr);
    // Waves are packed from `jobs`: an equal share of the capacity per job with samples left, leftovers
    // to the first jobs (or, with `fifo`, each job in list order taking all it can use); a job in the
    // reference's mode places at most one sample of each pixel in a wave, a NEE+MIS job any number (the
    // finish kernel sums each pixel's samples of the wave in sample order).  Wave k runs on lane k mod lanes, on
    // the lane's own stream.  Each wave's finish kernel (the per-pixel sums) runs after the previous wave's, so a
    // pixel's samples are summed in sample order; a wave holding a job whose samples carry state from the
    // pixel's previous sample (the reference's seeding mode) starts only after the finish of the wave that
    // holds that sample.
    //
    // Packs the next wave into the next lane, which must be free (lane_free()), and launches it.
    // Returns false when no job has samples left to schedule.  `members` and `completed` (optional)
    // receive the jobs in the wave and the jobs whose last samples it holds.
    bool submit_wave(const std::vector<BatchJob*>& jobs, bool fifo, std::vector<BatchJob*>* members = nullptr,
                     std::vector<BatchJob*>* completed = nullptr);
    bool lane_free() const { return !lanes_[lane_index(submitted_)].pending; }
    bool pending() const { return retired_ < submitted_; }
    // Waits for the oldest wave in flight and adds its ray counts; throws on a device error flag.
    void wait_oldest();
    // Waits for every wave in flight without reading their results (error and shutdown paths).
    void drain();
    // Runs waves until every job is resolved: waves of the lanes' slots, as many in flight as the engine has
    // lanes, or (cooperative traversal, choose_form) waves of all lanes' slots one after the other.  Ordered
    // after the work queued on `st` before the call; returns with every wave complete and the work
    // queued on `st` afterwards ordered after them.
    void run_all(const std::vector<BatchJob*>& jobs, cudaStream_t st, bool fifo = false);
    uint32_t capacity() const { return capacity_; }
    int lanes() const { return (int)lanes_.size(); }
    const TraceConfig& trace() const { return trace_; }
    uint64_t rays() const { return rays_; }
    uint64_t shadow_rays() const { return shadow_rays_; }
    // traversal work (nodes, triangles of closest and any-hit rays, shaded hits) over the waves collected
    // so far: counted by the cooperative kernels always, and by the grid-form kernels while counting is on
    const RenderStats& work() const { return work_; }
    // Counting on: waves launched from now on run the grid form's counting kernels (default block size and
    // stack depth; the same traversal, so the same images) where they would run the grid form.
    void set_counting(bool on) { count_ = on; }
    uint32_t waves() const { return waves_; }

private:
    // What the kernel sequence of a wave depends on.
    struct Shape {
        uint32_t bounces = 0;
        uint32_t materials = 0;  // bit m: a scene of the wave has material m
        bool nee = false;        // shadow rays may be cast
        bool two = false;        // the wave holds a two-level scene
        bool mixed = false;      // several jobs (cooperative form: each ray looks up its scene)
        bool count = false;      // counting kernels (traversal work)
        bool coop = false;       // cooperative traversal
        uint32_t wide = 0;       // traversal with eight lanes per ray: its blocks
        bool operator==(const Shape& o) const {
            return bounces == o.bounces && materials == o.materials && nee == o.nee && two == o.two && mixed == o.mixed &&
                   count == o.count && coop == o.coop && wide == o.wide;
        }
    };
    struct GraphSlot {
        Shape shape;
        cudaGraphExec_t exec = nullptr;
        uint64_t used = 0;   // submissions_ at its last launch
    };
    struct Lane {
        size_t index = 0;
        DeviceBuffer desc;              // header + segments + job table
        void* host_desc = nullptr;      // pinned staging of the descriptor
        uint32_t* host_counters = nullptr;   // pinned copy of the wave's counters
        cudaStream_t stream = nullptr;  // run_all's stream for this lane
        cudaEvent_t finished = nullptr; // after the lane's last finish kernel and resolves
        cudaEvent_t done = nullptr;     // after the lane's last counter copy
        bool ordered = true;            // ordered after the caller's stream (run_all)
        bool pending = false;           // a wave whose counters are not collected yet
        std::vector<GraphSlot> graphs;  // captured wave bodies (pointers into this lane's buffers)
    };
    struct Packed {
        WaveHeader hdr;
        Shape shape;
        uint64_t after = 0;      // number + 1 of the wave whose finish the wave has to wait for, 0 for none
        std::vector<BatchJob*> members, completed;
    };
    // Packs the next wave into the lane's host descriptor; hdr.count == 0 when nothing is left.
    Packed pack(const std::vector<BatchJob*>& jobs, bool fifo, Lane& L);
    // Descriptor upload + wave body (init and the bounce kernels) on `s`.
    void launch_body(Lane& L, const Packed& pk, cudaStream_t s);
    void make_room(Lane& L, uint32_t bounces);
    void launch_sequence(const BatchLaunch& B, const Shape& w, cudaStream_t main, bool fork);
    void launch_trace(const BatchLaunch& B, const Shape& w, bool extend, int cur, uint32_t* bounce, cudaStream_t st);
    template <bool MIXED, bool TWO, bool COUNT>
    void launch_coop(const BatchLaunch& B, bool extend, int cur, uint32_t* bounce, cudaStream_t st);
    void choose_form(const std::vector<BatchJob*>& jobs);
    size_t lane_index(uint64_t wave) const { return coop_ ? 0 : wave % lanes_.size(); }
    Lane& lane_of(uint64_t wave) { return lanes_[lane_index(wave)]; }
    size_t lane_bytes() const;
    // Slots of one wave: a lane's, or all lanes' in the cooperative form.
    uint32_t wave_slots() const { return coop_ ? capacity_ * (uint32_t)lanes_.size() : capacity_; }
    BatchLaunch wave_view(const Lane& L) const;
    // Finish kernel, resolves of the completed jobs, counter copy on `s`.
    void launch_finish(Lane& L, const Packed& pk, cudaStream_t s);
    // Adds a synchronized lane's counters to the totals; throws on a device error flag.
    void collect(Lane& L);
    // Waits for and releases every lane's streams, events, graphs and buffers.
    void release_lanes();
    int device_, sm_count_;
    uint32_t capacity_;
    bool use_graphs_;
    TraceConfig trace_;           // grid-form traversal variant of the extend and shadow kernels
    size_t desc_bytes_ = 0;
    std::vector<Lane> lanes_;
    uint64_t rays_ = 0, shadow_rays_ = 0;
    RenderStats work_;
    uint32_t waves_ = 0;
    uint64_t submitted_ = 0, retired_ = 0;   // waves launched / waited for
    uint64_t submissions_ = 0;               // waves launched since the engine was made
    int blocks_ext_ = 0, blocks_shade_[5] = {0, 0, 0, 0, 0}, blocks_sh_ = 0, blocks_simple_ = 0;
    int blocks_plain_[2][2][2] = {};       // grids of the default grid-form variant: [extend][two][count]
    int blocks_coop_[2][2][2][2] = {};     // of the cooperative form: [extend][mixed][two][count]
    bool count_ = false;
    DeviceBuffer paths_;                   // path state of all lanes
    cudaEvent_t caller_ = nullptr;         // the caller's stream at run_all
    bool coop_ = false;                    // form of the waves in flight (chosen while none is)
    bool wide_ = false;                    // the waves trace with eight lanes per ray
    uint32_t wave_limit_ = UINT32_MAX;     // paths of one wave, where fewer than its slots are wanted
};

}  // namespace rt
