// Host-callable launchers of the CUDA kernels (implemented in the .cu files).
#pragma once

#include <cstdint>

#include <cuda_runtime_api.h>

#include "device_scene.h"
#include "errors.h"
#include "rt_common.h"

namespace rt {

constexpr int kTraceBlock = 128;
// Traversal launch form: 0 = one thread per ray (grid); 1..32 = the warp-cooperative persistent form
// (coop_trace.cuh), whose warps take new rays once this many of their 32 lanes are idle.  The cooperative form
// is the default: on the 1.3M-triangle ray cast closest hit 0.42 ms against 0.80 ms for the grid form, on 256
// instances of a 20,480-triangle model (two-level) 0.93 against 1.48 ms.
constexpr int kDefaultRefill = 8;
// Launch form of the wavefront extension and shadow kernels (renders, batches, the server): 0, the pass-by-pass
// engine's and the server's grid form, and the batch engine's own choice by scene and paths
// (BatchEngine::choose_form, which holds the measurements).
constexpr int kDefaultWaveRefill = 0;
// Of those kernels only: the grid form whatever the engine would choose (block size and stack depth apply to every
// wave of a flat scene then).
constexpr int kGridAlways = -1;

// Launch configuration of the traversal kernels: block size (64, 128, 256) and shared-memory stack
// entries per thread (8, 12, 16) of the grid form, or the cooperative persistent form with its refill
// threshold (refill > 0; block 128, stack 12).
constexpr int kDefaultTraceStack = 12;
struct TraceConfig {
    int block = kTraceBlock;
    int stack = kDefaultTraceStack;
    int refill = kDefaultRefill;
    int sort = 0;                 // ray casts (grid form): 1 = trace the rays in coherence order
};
bool valid_trace_config(const TraceConfig& c);
bool valid_wave_config(const TraceConfig& c);   // of the wavefront kernels: kGridAlways too

// `d_next` is a device u32 used as the ray-fetch counter (reset by the launcher); n < 2^32.
void launch_raycast(const DeviceScene& s, const Ray* d_rays, uint64_t n, Hit* d_hits, bool any, uint32_t* d_err,
                    uint32_t* d_next, int sm_count, const TraceConfig& cfg, cudaStream_t st);
void launch_raycast_counters(const DeviceScene& s, const Ray* d_rays, uint64_t n, bool any,
                             unsigned long long* d_counters, uint32_t* d_err, uint32_t* d_next, int sm_count,
                             cudaStream_t st);

// Writes a flat scene's per-triangle indices into the padding of its n triangle records (TriRecord).
void tag_triangles(TriRecord* d_tris, uint32_t n, const uint32_t* d_prim_props, const uint32_t* d_prim_instance, cudaStream_t st);

}  // namespace rt
