// csp_system.h -- state behind one csp_handle.
#pragma once

#include <atomic>
#include <cstdint>
#include <string>
#include <vector>

#include <cuda_runtime.h>
#include <nvtx3/nvToolsExt.h>

#include "csp_c_api.h"
#include "csp_kernels.cuh"
#include "csp_pool.h"
#include "csp_scene.h"

namespace csp {

int set_error(int status, const std::string& msg);

// A named range on the NVTX timeline (Nsight Systems, Nsight Compute's range filters) for the
// lifetime of the object: the host stages of the library (setup, update, trace, copies, batch runs,
// server steps).  Without a tool attached the calls do nothing.
struct NvtxRange {
    explicit NvtxRange(const char* name) { nvtxRangePushA(name); }
    ~NvtxRange() { nvtxRangePop(); }
    NvtxRange(const NvtxRange&) = delete;
    NvtxRange& operator=(const NvtxRange&) = delete;
};
int cuda_status(cudaError_t e, const char* what);

// Sun shapes the ABI accepts: pillbox or Gaussian, with or without CSP_SUN_ACCURATE.
inline bool valid_sun_shape(int shape) { return shape >= 0 && shape <= (CSP_SUN_GAUSSIAN | CSP_SUN_ACCURATE); }

// Angle the sun plane is padded by: the pillbox half angle (lib/geometry_manager.cpp:129), or 5
// sigma for the Gaussian sun.
inline double sun_pad_angle(int shape, double param) { return (shape & CSP_SUN_GAUSSIAN) ? 5.0 * param : param; }

// A ray window [first, first + count) whose indices all stay below kRayIndexLimit (checked without
// overflow).
inline bool valid_ray_window(uint64_t first, uint64_t count) {
    return first <= kRayIndexLimit && count <= kRayIndexLimit - first;
}

struct System {
    int device = -1;
    uint64_t num_rays = 0;
    std::vector<csp_element> elements;
    double sun_dir[3] = {0.0, 0.0, 1.0};
    int sun_shape = CSP_SUN_PILLBOX;
    double sun_param = 0.0;
    uint64_t seed = 0;
    uint32_t instance = 0;
    bool record_ids = false;
    bool initialized = false;  // since the last set_accel
    bool loaded = false;       // the device's scene is complete (a set-up that fails half-way leaves it false)

    HostScene scene;       // of the last elements packed (a refused set-up leaves its own here)
    HostGrid grid;         // of the scene on the device
    uint32_t n_scene = 0;  // elements of the scene on the device
    int accel = CSP_ACCEL_AUTO;

    HostPool pool;                  // element records of scenes of kPoolElements or more, in ranges
    bool topology = false;          // scene.nodes are the BVH (or leaf list) of this element count
    Node* d_nodes = nullptr;
    // element records: prims, optics, exact and pruning boxes in one device block, put together in
    // pinned memory and uploaded in one copy
    unsigned char* d_records = nullptr;
    unsigned char* h_records = nullptr;
    size_t cap_records = 0;
    bool records_busy = false;  // an upload from h_records that no synchronisation has followed yet
    Prim* d_prims = nullptr;
    Optics* d_optics = nullptr;
    Aabb* d_aabbs = nullptr;
    Aabb* d_prune = nullptr;
    SunFrame* d_sun = nullptr;
    float4* d_hits = nullptr;
    uint32_t* d_ids = nullptr;
    GridDesc* d_grid = nullptr;
    const float* h3t12 = nullptr;  // Halton table of the device (halton3_table)
    GridDesc grid_host{};  // host copy of the descriptor (source of the async upload)
    // cells, items and global list of a field grid built on the host, or the block of one that the
    // device builds
    uint2* d_cells = nullptr;
    Aabb* d_items = nullptr;
    Aabb* d_global = nullptr;
    size_t cap_cells = 0, cap_items = 0, cap_global = 0;
    unsigned char* d_field = nullptr;
    size_t cap_field = 0;
    // sun-ray candidate grid (scenes of more than kFlatListMax elements): its arrays, and the build
    // job (host copy = source of the async upload)
    unsigned char* d_sgrid = nullptr;
    size_t cap_sgrid = 0;
    SunGridJob* d_sgjob = nullptr;
    // work counters {tiles, CTAs done} of the launches, see next_counter
    static constexpr unsigned kCounters = 64;
    static constexpr size_t kCounterBytes = 2 * kCounters * 2 * sizeof(unsigned int);
    unsigned int* d_counters = nullptr;
    std::atomic<unsigned> next_eager{0}, next_captured{0};
    SunGridJob sgjob_host{};
    // compact records (csp_run_to_host_compact): points, counts, block offsets, records
    float* d_cpoints = nullptr;
    uint8_t* d_ccounts = nullptr;
    unsigned long long* d_csums = nullptr;
    float4* d_crecords = nullptr;
    uint64_t cap_compact_rays = 0, cap_crecords = 0;
    // chunked runs: records of the chunks between their trace and their copy, and those chunks' totals
    // (pinned host memory)
    float4* d_cring = nullptr;
    uint64_t cap_cring = 0;
    unsigned long long* h_ctotal = nullptr;
    unsigned char* d_flux = nullptr;  // csp_flux_map: counters [4], then the map
    unsigned char* h_flux = nullptr;  // pinned: the sun frame, then the map
    size_t cap_flux = 0, cap_hflux = 0;  // bins of the two
    size_t cap_nodes = 0;
    uint64_t cap_rays = 0;
    bool ids_allocated = false;

    cudaStream_t stream = nullptr;
    cudaStream_t copy_stream = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;

    double time_setup = 0.0;
    double time_trace = 0.0;

    ~System();
    void release();
    int ensure_streams();
    bool ready() const { return initialized && loaded; }
    int build_scene(const char* not_planar);
    int load_scene(const char* not_planar, bool first);
    int upload_nodes();
    int upload_grid();
    int prepare_sun();
    int build_sungrid();
    float pad_angle() const;
    int ensure_hit_buffers();
    int initialize();
    int update();
    unsigned int* next_counter(cudaStream_t st);
    TraceArgs args(uint64_t begin, uint64_t count, unsigned int* counter) const;
    int trace_async(cudaStream_t st);
    int run();
    int run_to_host(float* dst, uint32_t* ids);
    int ensure_compact_buffers(uint64_t n);
    int run_compact_chunks(float* points, uint8_t* counts, float* records, uint64_t chunk, uint64_t* n_records);
    int run_to_host_compact(float* points, uint8_t* counts, float* records, uint64_t capacity, uint64_t* n_records);
    int flux_map(uint32_t nx, uint32_t ny, uint32_t* counts, double dni, double* flux, bool staged = false);
};

// |(v1 - v0) x (v3 - v0)| of a sun frame, in double
double sun_plane_area(const SunFrame& f);

// flux = counts * dni * sun area / rays / bin area
void counts_to_flux(const uint32_t* counts, size_t n, double dni, double sun_area, uint64_t rays, double bin_area,
                    double* flux);

}  // namespace csp
