// csp_kernels.cuh -- launch interface of the CUDA kernels (host side).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "csp_types.cuh"

namespace csp {

struct HostGrid;

// Bounds-check builds (-DCSP_BOUNDS_CHECK): the failed-check sites recorded on the current device by
// the kernels of each translation unit, read and cleared (0 in other builds).
#ifdef CSP_BOUNDS_CHECK
constexpr bool kBoundsCheckBuild = true;
#else
constexpr bool kBoundsCheckBuild = false;
#endif
uint32_t bounds_sites_trace();
uint32_t bounds_sites_batch();
uint32_t bounds_sites_sungrid();

// Every device and pinned-host allocation of the library goes through these (csp_c_api.cpp): the
// allocation-failure injection of csp_debug_fail_allocation lives there.
cudaError_t dev_alloc(void** p, size_t bytes);
cudaError_t host_alloc(void** p, size_t bytes);

// Closest-hit search of a launch: the element list in shared memory (<= 8 elements), the BVH, or
// the field grid (GridDesc).
enum Accel : int { kAccelFlat = 0, kAccelBvh = 1, kAccelGrid = 2 };

struct TraceArgs {
    const Node* nodes;
    const Prim* prims;
    const Optics* optics;
    const SunFrame* sun;
    float4* hits;        // [count * kMaxDepth] for rays ray_begin .. ray_begin + count - 1
    uint32_t* ids;       // [count * kMaxDepth] or nullptr
    uint64_t ray_begin;  // global index of the first ray of this launch
    uint64_t count;      // rays in this launch
    uint64_t seed;
    uint32_t instance;
    int n_prims;         // elements of the scene
    const GridDesc* grid;  // field grid of the scene, nullptr: BVH (or element list) traversal
    const float* h3t12;    // Halton base-3 partial sums after 12 digits (halton3_table), or nullptr
    const SunGrid* sgrid;  // candidate grid of the sun rays (scenes of more than 8 elements)
    // single-scene launches: tiles handed out by this device counter ([0] tiles, [1] CTAs done; zero
    // between launches, the last CTA sees to that) in guided grabs; launches that overlap on the GPU have
    // different ones.  nullptr: static shares
    unsigned int* tile_counter;
};

// Arguments of the single-scene element-list kernel: TraceArgs plus the Philox key schedule of
// `seed` (philox_keys), read as kernel parameters.
struct TraceArgsK : TraceArgs {
    uint32_t keys[20];
};

// Device table of the base-3 Halton fold: its sums after 12 digits, t[m] = the reference loop's sum
// for m < 3^12, and the addends of the next six (2.1 MB, filled once per device by the same loop), or
// nullptr if it could not be
// made.  Thread-safe; the calling thread's current device.
const float* halton3_table();

// Sun-plane distance and parallelogram (lib/geometry_manager.cpp:97-148 with the reductions of
// lib/sun_utils.cu:53-179) plus the per-launch cone frame (cuda/sun.cu:76-79): one block, a cluster of
// eight from 1,024 elements.
cudaError_t launch_prepare_sun(const Aabb* aabbs, int n, float sx, float sy, float sz, float tan_pad, int shape,
                               float param, SunFrame* out, cudaStream_t stream);

// Sun-ray candidate grid of one scene state (SunGrid): device arrays of its build and where its
// descriptor goes.  All of it is written by launch_sungrid_build (nothing needs zeroing).
struct SunGridJob {
    SunGrid* desc;            // the descriptor the trace reads (TraceArgs::sgrid)
    const SunFrame* sun;      // sun frame of the state (prepare_sun output)
    const Aabb* aabbs;        // [n] exact boxes, lo.w = element | type << kTypeShift
    int n;
    int cap_cells;
    uint32_t cap_items;
    int pad;
    uint2* cells;             // [cap_cells]
    uint32_t* alloc;          // items handed out to cells so far
    float4* rect;             // [n] candidate rectangles
    float4* reach_rect;       // [n] reach rectangles (in the space of item_rect)
    uint32_t* reach;          // [kReachRaster^2 / 32]
    // the state's field grid, when the device builds it (cells null: not)
    const Aabb* prune;        // [n] pruning boxes
    uint2* field_cells;       // [field_nx * field_ny]
    uint32_t* field_alloc;
    Aabb* field_items;        // [field_cap]
    float field_x0, field_y0, field_inv;
    int field_nx, field_ny;
    uint32_t field_cap;
    float4* item_rect;        // [cap_items]
    Aabb* item_box;           // [cap_items]
    uint32_t* global_id;      // [n]
};

// Capacities of the sun grid of an n-element scene and the device bytes of its arrays (each array
// 256-byte aligned, in the order of sungrid_place), descriptor included, the raster too or not.
struct SunGridCaps {
    int cap_cells;
    uint32_t cap_items;
};
SunGridCaps sungrid_caps(uint32_t n);
constexpr size_t kReachBytes = kReachRaster * kReachRaster / 8;
size_t sungrid_bytes(uint32_t n, bool raster = true);
// Carve the arrays of an n-element scene's sun grid out of `base` (sungrid_bytes(n, !raster) bytes, 256-byte
// aligned), the reach raster out of `raster` (kReachBytes) if given; fills every SunGridJob field except
// sun and aabbs.
void sungrid_place(unsigned char* base, uint32_t n, SunGridJob& job, unsigned char* raster = nullptr);

// Build the sun grids (and field grids, where the jobs have them) of n_jobs scene states (jobs: device
// array) on `stream`; max_n, max_field_cells = the largest element count and field_nx * field_ny
// among the jobs (0: no field grids).
cudaError_t launch_sungrid_build(const SunGridJob* jobs, int n_jobs, int max_n, int max_field_cells,
                                 cudaStream_t stream);
// Bytes of a device-built field grid of nx * ny cells and cap items (256-byte aligned parts), and its
// place in `base` (256-byte aligned): fills the job's field members.
size_t field_bytes(int nx, int ny, uint32_t cap);
void field_place(unsigned char* base, const HostGrid& g, const Aabb* prune, SunGridJob& job);

// Trace rays [ray_begin, ray_begin + count): generation, closest-hit search, shading, the dense
// hit-record write.  Scenes of up to 8 elements take the shared-memory element list path; larger ones
// need args.sgrid.
cudaError_t launch_trace(const TraceArgs& args, cudaStream_t stream);

// Compact form of a dense hit buffer of n rays (csp_run_to_host_compact): count pass -- per ray the
// sun-plane point (3 floats) and the number of records after slot 0 (uint8) and, in
// block_sums[compact_blocks(n) + 1], the exclusive offsets of the 256-ray blocks with the total at the
// end (and in *host_total, pinned host memory, unless null) -- then the write pass: the records after
// slot 0, in ray order.  points 16-byte aligned.
uint64_t compact_blocks(uint64_t n);
cudaError_t launch_compact_count(const float4* hits, uint64_t n, float* points, uint8_t* counts,
                                 unsigned long long* block_sums, unsigned long long* host_total,
                                 cudaStream_t stream);
cudaError_t launch_compact_write(const float4* hits, uint64_t n, const uint8_t* counts,
                                 const unsigned long long* block_offsets, float4* records, cudaStream_t stream);

// Bin the stage-2 records of a dense hit buffer into F.counts and count records into F.stats[1..3]
// (both zeroed by the caller).
cudaError_t launch_flux_records(const float4* hits, uint64_t n_records, const FluxTarget& F, cudaStream_t stream);

// ---------------------------------------------------------------------- multi-instance launches --
// One instance = one scene state (its own prims, optics, node boxes, sun frame) traced for
// rays [args.ray_begin, args.ray_begin + args.count) with (args.seed, args.instance), its receiver
// records binned into flux.counts.  Instances of one launch are laid out as consecutive tile
// ranges; CTAs take chunks of tiles from a global counter.
struct alignas(16) InstanceDesc {
    TraceArgs args;       // hits = ids = nullptr; args.grid -> grid (grid instances)
    FluxTarget flux;
    GridDesc grid;
    uint64_t tile_begin;  // first tile of this instance in the launch
    int n_prims;
    int pad[3];
};

struct BatchLaunch {
    const InstanceDesc* inst;        // device
    const uint64_t* tile_begin;      // device, [n_inst + 1]; last entry = total_tiles
    int n_inst;
    int chunk;                       // tiles per grab
    uint64_t total_tiles;
    unsigned long long* next_tile;   // device work counter, zero before the launch
};

struct BatchTuning {
    int block;        // CTA size = tile size: 128 or 256
    int ctas_per_sm;  // resident CTAs per SM of the persistent grid (<= occupancy limit)
    int chunk;        // tiles taken per grab
};

// Bottom-up refit of one BVH topology into per-instance node arrays: leaves get the exact element
// AABB, internal nodes the union of the pruning boxes of the leaves below them.
struct RefitJob {
    const Node* topo;   // node links of the topology (boxes ignored)
    const Aabb* aabbs;  // exact element AABBs of the instance
    const Aabb* prune;  // pruning boxes of the instance
    Node* out;          // [n_nodes]
    int n_nodes;
    int pad;
};

struct SunJob {
    const Aabb* aabbs;
    int n;
    float sx, sy, sz, tan_pad;
    int shape;
    float param;
    SunFrame* out;
};

cudaError_t launch_refit(const RefitJob* jobs, int n_jobs, int max_nodes, cudaStream_t stream);
// max_n: the largest element count among the jobs
cudaError_t launch_prepare_sun_batch(const SunJob* jobs, int n_jobs, int max_n, cudaStream_t stream);
// Closest-hit search of a batch group: 0 element list (<= 8 elements), 1 BVH, 2 field grid.
constexpr int kBatchGroups = 3;
// Occupancy limit of the multi-instance kernel for (accel, block); 0 if unsupported.
int batch_occupancy(int accel, int block);
// Fingerprint of the multi-instance kernels of a group as built (registers, shared and local memory
// of both block sizes): part of the autotuner cache key.
uint32_t batch_kernel_build(int accel);
cudaError_t launch_trace_batch(const BatchLaunch& L, int accel, const BatchTuning& t, cudaStream_t stream);

}  // namespace csp
