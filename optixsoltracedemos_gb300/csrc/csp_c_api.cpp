// csp_c_api.cpp -- the C ABI (include/csp_c_api.h): handle lifecycle, device buffers, launches.
#include "csp_c_api.h"

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <new>
#include <string>
#include <vector>

#include <cuda_runtime.h>

#include "csp_kernels.cuh"
#include "csp_math.cuh"
#include "csp_scene.h"
#include "csp_system.h"

namespace {

thread_local std::string t_last_error;

int fail(int status, const std::string& msg) {
    t_last_error = msg;
    return status;
}

}  // namespace

namespace csp {

int set_error(int status, const std::string& msg) { return fail(status, msg); }

namespace {

// Allocations left before the injected failure (csp_debug_fail_allocation); -1: none pending.
std::atomic<long long> g_fail_after{-1};

bool injected_failure() {
    long long v = g_fail_after.load();
    while (v >= 0) {
        if (g_fail_after.compare_exchange_weak(v, v == 0 ? -1 : v - 1)) return v == 0;
    }
    return false;
}

}  // namespace

cudaError_t dev_alloc(void** p, size_t bytes) {
    if (injected_failure()) {
        *p = nullptr;
        return cudaErrorMemoryAllocation;
    }
    return cudaMalloc(p, bytes);
}

cudaError_t host_alloc(void** p, size_t bytes) {
    if (injected_failure()) {
        *p = nullptr;
        return cudaErrorMemoryAllocation;
    }
    return cudaHostAlloc(p, bytes, cudaHostAllocDefault);
}

int cuda_status(cudaError_t e, const char* what) {
    if (e == cudaSuccess) return CSP_OK;
    const int st = (e == cudaErrorMemoryAllocation) ? CSP_ERR_OUT_OF_MEMORY : CSP_ERR_CUDA;
    cudaGetLastError();  // clear the sticky-free error state of the runtime API
    return fail(st, std::string(what) + ": " + cudaGetErrorString(e));
}

template <typename T>
static int upload(T*& dptr, size_t& cap, const std::vector<T>& host, cudaStream_t st, const char* what) {
    const size_t n = host.size();
    if (n > cap) {
        if (dptr) cudaFree(dptr);
        dptr = nullptr;
        cap = 0;
        int rc = cuda_status(dev_alloc((void**)&dptr, std::max<size_t>(n, 1) * sizeof(T)), what);
        if (rc) return rc;
        cap = n;
    }
    if (n) return cuda_status(cudaMemcpyAsync(dptr, host.data(), n * sizeof(T), cudaMemcpyHostToDevice, st), what);
    return CSP_OK;
}

System::~System() { release(); }

void System::release() {
    if (device >= 0) cudaSetDevice(device);
    cudaFree(d_nodes);
    cudaFree(d_records);
    if (h_records) cudaFreeHost(h_records);
    d_records = h_records = nullptr;
    cap_records = 0;
    cudaFree(d_field);
    d_field = nullptr;
    cap_field = 0;
    topology = false;
    cudaFree(d_sun);
    cudaFree(d_hits);
    cudaFree(d_ids);
    cudaFree(d_grid);
    cudaFree(d_cells);
    cudaFree(d_items);
    cudaFree(d_global);
    d_grid = nullptr;
    d_cells = nullptr;
    d_items = d_global = nullptr;
    cap_cells = cap_items = cap_global = 0;
    cudaFree(d_sgrid);
    cudaFree(d_sgjob);
    cudaFree(d_counters);
    d_sgrid = nullptr;
    d_sgjob = nullptr;
    d_counters = nullptr;
    cap_sgrid = 0;
    cudaFree(d_cpoints);
    cudaFree(d_ccounts);
    cudaFree(d_csums);
    cudaFree(d_crecords);
    d_cpoints = nullptr;
    d_ccounts = nullptr;
    d_csums = nullptr;
    d_crecords = nullptr;
    cap_compact_rays = cap_crecords = 0;
    cudaFree(d_cring);
    d_cring = nullptr;
    cap_cring = 0;
    if (h_ctotal) cudaFreeHost(h_ctotal);
    h_ctotal = nullptr;
    cudaFree(d_flux);
    if (h_flux) cudaFreeHost(h_flux);
    d_flux = h_flux = nullptr;
    cap_flux = cap_hflux = 0;
    d_nodes = nullptr;
    d_prims = nullptr;
    d_optics = nullptr;
    d_aabbs = d_prune = nullptr;
    d_sun = nullptr;
    d_hits = nullptr;
    d_ids = nullptr;
    cap_nodes = 0;
    cap_rays = 0;
    ids_allocated = false;
    loaded = false;
    if (ev0) cudaEventDestroy(ev0);
    if (ev1) cudaEventDestroy(ev1);
    if (copy_stream) cudaStreamDestroy(copy_stream);
    if (stream) cudaStreamDestroy(stream);
    ev0 = ev1 = nullptr;
    stream = copy_stream = nullptr;
    initialized = false;
}

int System::ensure_streams() {
    if (stream) return CSP_OK;
    int rc = cuda_status(cudaSetDevice(device), "cudaSetDevice");
    if (rc) return rc;
    if ((rc = cuda_status(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking), "cudaStreamCreate"))) return rc;
    if ((rc = cuda_status(cudaStreamCreateWithFlags(&copy_stream, cudaStreamNonBlocking), "cudaStreamCreate")))
        return rc;
    if ((rc = cuda_status(cudaEventCreate(&ev0), "cudaEventCreate"))) return rc;
    return cuda_status(cudaEventCreate(&ev1), "cudaEventCreate");
}

// Element count from which a scene's records are packed on the handle's host threads.  With the threads
// up, a whole update() is as fast with as without them at 700 elements (129 and 134 us; 2,000: 271 and 174,
// 4,000: 495 and 276 on a 16-core host), but they have to pay for their start first.
constexpr uint32_t kPoolElements = 2048;

// Element records of the current elements, packed and put on the device, and the plan of their field
// grid.  An error of the elements or of the plan, whatever their count, leaves the device's scene
// (n_scene, the record buffers, `grid`) as it was and traceable; from there on the scene is not loaded
// until the caller is through.
int System::build_scene(const char* not_planar) {
    const uint32_t n = (uint32_t)elements.size();
    int rc;
    // the last upload from h_records may still be under way if its call failed after it
    if (records_busy && (rc = cuda_status(cudaStreamSynchronize(stream), "element records"))) return rc;
    records_busy = false;
    auto align = [](size_t x) { return (x + 255) & ~(size_t)255; };
    const size_t o_optics = align(n * sizeof(Prim)), o_aabbs = o_optics + align(n * sizeof(Optics));
    const size_t o_prune = o_aabbs + align(n * sizeof(Aabb)), bytes = o_prune + align(n * sizeof(Aabb));
    // larger buffers next to the old ones, which serve the device's scene until the new one is accepted
    struct Grown {
        unsigned char *d = nullptr, *h = nullptr;
        ~Grown() {
            if (d) cudaFree(d);
            if (h) cudaFreeHost(h);
        }
    } grown;
    if (bytes > cap_records) {
        if ((rc = cuda_status(dev_alloc((void**)&grown.d, bytes), "cudaMalloc element records"))) return rc;
        if ((rc = cuda_status(host_alloc((void**)&grown.h, bytes), "cudaHostAlloc element records"))) return rc;
    }
    unsigned char* const staged = grown.h ? grown.h : h_records;
    auto stage = [&](uint32_t b, uint32_t e) {
        std::memcpy(staged + b * sizeof(Prim), &scene.prims[b], (e - b) * sizeof(Prim));
        std::memcpy(staged + o_optics + b * sizeof(Optics), &scene.optics[b], (e - b) * sizeof(Optics));
        std::memcpy(staged + o_aabbs + b * sizeof(Aabb), &scene.aabbs[b], (e - b) * sizeof(Aabb));
        std::memcpy(staged + o_prune + b * sizeof(Aabb), &scene.prune[b], (e - b) * sizeof(Aabb));
    };
    std::string err;
    GridStats stats;
    if (n >= kPoolElements) {
        pool.start(std::min({15u, std::max(2u, std::thread::hardware_concurrency()) - 1, build_ranges(n) - 1}));
        rc = build_elements(
            elements.data(), n, scene, err,
            [this](size_t tasks, const std::function<void(size_t)>& body) { pool.run(tasks, body); }, &stats, stage);
    } else {
        rc = build_elements(elements.data(), n, scene, err, &stats);
        if (!rc) stage(0, n);
    }
    if (rc) return fail(rc, err);
    // the grid holds one set of poses: planned anew for these
    HostGrid plan;
    if (accel != CSP_ACCEL_BVH) plan_grid(scene, stats, plan);
    if (accel == CSP_ACCEL_GRID && !plan.valid && n > kFlatListMax) return fail(CSP_ERR_BAD_SCENE, not_planar);
    loaded = false;
    if (grown.d) {
        std::swap(d_records, grown.d);
        std::swap(h_records, grown.h);
        cap_records = bytes;
    }
    n_scene = n;
    grid = std::move(plan);
    d_prims = reinterpret_cast<Prim*>(d_records);
    d_optics = reinterpret_cast<Optics*>(d_records + o_optics);
    d_aabbs = reinterpret_cast<Aabb*>(d_records + o_aabbs);
    d_prune = reinterpret_cast<Aabb*>(d_records + o_prune);
    records_busy = true;
    return cuda_status(cudaMemcpyAsync(d_records, h_records, bytes, cudaMemcpyHostToDevice, stream), "upload records");
}

int System::upload_nodes() {
    // scenes that trace through the field grid need no BVH
    if (grid.valid) return CSP_OK;
    if (topology) refit_bvh(scene);
    else build_bvh(scene);
    topology = true;
    return upload(d_nodes, cap_nodes, scene.nodes, stream, "upload bvh");
}

// Field grid on the device: its arrays where the host built them, else room for the device's, and the
// descriptor.
int System::upload_grid() {
    if (!grid.valid) return CSP_OK;
    int rc;
    if (grid.on_device) {
        const size_t bytes = field_bytes(grid.nx, grid.ny, grid.cap_items);
        if (bytes > cap_field) {
            cudaFree(d_field);
            d_field = nullptr;
            cap_field = 0;
            if ((rc = cuda_status(dev_alloc((void**)&d_field, bytes), "cudaMalloc field grid"))) return rc;
            cap_field = bytes;
        }
        SunGridJob at{};
        field_place(d_field, grid, d_prune, at);
        grid_host = csp::grid_desc(grid, at.field_cells, at.field_items, d_aabbs + (n_scene - 1));
    } else {
        if ((rc = upload(d_cells, cap_cells, grid.cells, stream, "upload grid cells"))) return rc;
        if ((rc = upload(d_items, cap_items, grid.items, stream, "upload grid items"))) return rc;
        if ((rc = upload(d_global, cap_global, grid.global, stream, "upload grid globals"))) return rc;
        grid_host = csp::grid_desc(grid, d_cells, d_items, d_global);
    }
    if (!d_grid && (rc = cuda_status(dev_alloc((void**)&d_grid, sizeof(GridDesc)), "cudaMalloc grid"))) return rc;
    return cuda_status(cudaMemcpyAsync(d_grid, &grid_host, sizeof(GridDesc), cudaMemcpyHostToDevice, stream),
                       "upload grid");
}

float System::pad_angle() const {
    return (float)sun_pad_angle(sun_shape, sun_param);
}

int System::prepare_sun() {
    float s[3];
    sun_vector_f(sun_dir, s);
    scene.sun[0] = s[0];
    scene.sun[1] = s[1];
    scene.sun[2] = s[2];
    const float tan_pad = tanf(pad_angle());
    return cuda_status(launch_prepare_sun(d_aabbs, (int)n_scene, s[0], s[1], s[2], tan_pad, sun_shape,
                                          (float)sun_param, d_sun, stream),
                       "prepare_sun_kernel");
}

// Sun-ray candidate grid of the current poses and sun frame, built on the device behind the sun
// plane (scenes of more than kFlatListMax elements; the element list needs none).
int System::build_sungrid() {
    const uint32_t n = n_scene;
    if (n <= kFlatListMax) return CSP_OK;
    int rc;
    const size_t bytes = sungrid_bytes(n);
    if (bytes > cap_sgrid) {
        cudaFree(d_sgrid);
        d_sgrid = nullptr;
        cap_sgrid = 0;
        if ((rc = cuda_status(dev_alloc((void**)&d_sgrid, bytes), "cudaMalloc sun grid"))) return rc;
        cap_sgrid = bytes;
    }
    if (!d_sgjob && (rc = cuda_status(dev_alloc((void**)&d_sgjob, sizeof(SunGridJob)), "cudaMalloc sun grid job")))
        return rc;
    sungrid_place(d_sgrid, n, sgjob_host);
    sgjob_host.sun = d_sun;
    sgjob_host.aabbs = d_aabbs;
    const int field_cells = grid.valid && grid.on_device ? grid.nx * grid.ny : 0;
    if (field_cells) field_place(d_field, grid, d_prune, sgjob_host);
    if ((rc = cuda_status(cudaMemcpyAsync(d_sgjob, &sgjob_host, sizeof(SunGridJob), cudaMemcpyHostToDevice, stream),
                          "upload sun grid job")))
        return rc;
    return cuda_status(launch_sungrid_build(d_sgjob, 1, (int)n, field_cells, stream), "sun grid build");
}

int System::ensure_hit_buffers() {
    if (num_rays > cap_rays || (record_ids && !ids_allocated)) {
        cudaFree(d_hits);
        cudaFree(d_ids);
        d_hits = nullptr;
        d_ids = nullptr;
        cap_rays = 0;
        ids_allocated = false;
        const size_t n = std::max<uint64_t>(num_rays, 1);
        int rc = cuda_status(dev_alloc((void**)&d_hits, n * kMaxDepth * sizeof(float4)), "cudaMalloc hit buffer");
        if (rc) return rc;
        if (record_ids) {
            rc = cuda_status(dev_alloc((void**)&d_ids, n * kMaxDepth * sizeof(uint32_t)), "cudaMalloc id buffer");
            if (rc) return rc;
            ids_allocated = true;
        }
        cap_rays = num_rays;
    }
    return CSP_OK;
}

// The current elements and sun on the device, complete when it returns, and room for the records.  After a
// failure past build_scene's checks (device memory) the handle traces nothing until a later update() or
// initialize() gets through; the records and the flux map of its last run stay readable.
int System::load_scene(const char* not_planar, bool first) {
    int rc;
    if ((rc = build_scene(not_planar))) return rc;
    if ((rc = upload_nodes())) return rc;
    if ((rc = upload_grid())) return rc;
    if ((rc = prepare_sun())) return rc;
    if ((rc = build_sungrid())) return rc;
    // the counters are zero before the first launch, and every launch leaves its own so
    if (first && (rc = cuda_status(cudaMemsetAsync(d_counters, 0, kCounterBytes, stream), "memset"))) return rc;
    const int no_hits = ensure_hit_buffers();  // while the device works; the scene is complete without
    if ((rc = cuda_status(cudaStreamSynchronize(stream), "scene set-up"))) return rc;
    records_busy = false;
    loaded = true;
    return no_hits;
}

int System::initialize() {
    NvtxRange nvtx("csp initialize");
    const auto t0 = std::chrono::steady_clock::now();
    int rc = ensure_streams();
    if (rc) return rc;
    if (!d_counters && (rc = cuda_status(dev_alloc((void**)&d_counters, kCounterBytes), "cudaMalloc tile counters")))
        return rc;
    h3t12 = halton3_table();
    topology = false;
    if (!d_sun && (rc = cuda_status(dev_alloc((void**)&d_sun, sizeof(SunFrame)), "cudaMalloc sun"))) return rc;
    if ((rc = load_scene("the scene is not a planar field: no grid (use CSP_ACCEL_AUTO or _BVH)", true))) return rc;
    initialized = true;
    time_setup = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    return CSP_OK;
}

int System::update() {
    NvtxRange nvtx("csp update");
    if (!initialized) return fail(CSP_ERR_STATE, "update() before initialize()");
    if (elements.size() != n_scene)
        return fail(CSP_ERR_STATE, "update() needs the element count of initialize(); call initialize() again");
    return load_scene("the new poses are not a planar field: no grid (use CSP_ACCEL_AUTO or _BVH)", false);
}

// Work counter of a launch on `st`.  A launch hands out its tiles by its counter and leaves it zero, so two
// that overlap on the GPU must not share one, or they and every later launch of it would skip tiles: the
// launches take turns on kCounters of them, captured ones (whose counter stays with the graph) on as many
// others.
unsigned int* System::next_counter(cudaStream_t st) {
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (st != stream && cudaStreamIsCapturing(st, &capture) != cudaSuccess) {
        cudaGetLastError();  // the launch itself reports what is wrong with the stream
        capture = cudaStreamCaptureStatusNone;
    }
    const bool captured = capture != cudaStreamCaptureStatusNone;
    const unsigned k = (captured ? next_captured : next_eager).fetch_add(1u, std::memory_order_relaxed) % kCounters;
    return d_counters + 2 * (captured ? kCounters + k : k);
}

TraceArgs System::args(uint64_t begin, uint64_t count, unsigned int* counter) const {
    TraceArgs a;
    a.nodes = d_nodes;
    a.prims = d_prims;
    a.optics = d_optics;
    a.sun = d_sun;
    a.hits = d_hits + begin * kMaxDepth;
    a.ids = (record_ids && d_ids) ? d_ids + begin * kMaxDepth : nullptr;
    a.ray_begin = begin;
    a.count = count;
    a.seed = seed;
    a.instance = instance;
    a.n_prims = (int)n_scene;
    a.grid = grid.valid ? d_grid : nullptr;
    a.h3t12 = h3t12;
    a.sgrid = n_scene > kFlatListMax && d_sgrid ? sgjob_host.desc : nullptr;
    a.tile_counter = counter;
    return a;
}

int System::trace_async(cudaStream_t st) {
    if (!ready()) return fail(CSP_ERR_STATE, "trace before initialize()");
    int rc = ensure_hit_buffers();
    if (rc) return rc;
    if (!st) st = stream;
    return cuda_status(launch_trace(args(0, num_rays, next_counter(st)), st), "trace_kernel");
}

int System::run() {
    NvtxRange nvtx("csp run");
    if (!ready()) return fail(CSP_ERR_STATE, "run() before initialize()");
    int rc = ensure_hit_buffers();
    if (rc) return rc;
    if ((rc = cuda_status(cudaEventRecord(ev0, stream), "cudaEventRecord"))) return rc;
    if ((rc = cuda_status(launch_trace(args(0, num_rays, next_counter(stream)), stream), "trace_kernel"))) return rc;
    if ((rc = cuda_status(cudaEventRecord(ev1, stream), "cudaEventRecord"))) return rc;
    if ((rc = cuda_status(cudaEventSynchronize(ev1), "trace"))) return rc;
    float ms = 0.f;
    cudaEventElapsedTime(&ms, ev0, ev1);
    time_trace = ms * 1e-3;
    return CSP_OK;
}

int System::run_to_host(float* dst, uint32_t* ids_dst) {
    NvtxRange nvtx("csp run_to_host");
    if (!ready()) return fail(CSP_ERR_STATE, "run() before initialize()");
    int rc = ensure_hit_buffers();
    if (rc) return rc;
    const uint64_t chunk = std::max<uint64_t>(1u << 20, (num_rays + 15) / 16);
    std::vector<cudaEvent_t> done;
    const auto t0 = std::chrono::steady_clock::now();
    for (uint64_t b = 0; b < num_rays; b += chunk) {
        const uint64_t c = std::min(chunk, num_rays - b);
        if ((rc = cuda_status(launch_trace(args(b, c, next_counter(stream)), stream), "trace_kernel"))) break;
        cudaEvent_t ev;
        if ((rc = cuda_status(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming), "cudaEventCreate"))) break;
        done.push_back(ev);
        if ((rc = cuda_status(cudaEventRecord(ev, stream), "cudaEventRecord"))) break;
        if ((rc = cuda_status(cudaStreamWaitEvent(copy_stream, ev, 0), "cudaStreamWaitEvent"))) break;
        rc = cuda_status(cudaMemcpyAsync(dst + b * kMaxDepth * 4, d_hits + b * kMaxDepth, c * kMaxDepth * sizeof(float4),
                                         cudaMemcpyDeviceToHost, copy_stream),
                         "D2H hit records");
        if (rc) break;
        if (ids_dst && record_ids && d_ids) {
            rc = cuda_status(cudaMemcpyAsync(ids_dst + b * kMaxDepth, d_ids + b * kMaxDepth,
                                             c * kMaxDepth * sizeof(uint32_t), cudaMemcpyDeviceToHost, copy_stream),
                             "D2H ids");
            if (rc) break;
        }
    }
    const int sync_rc = cuda_status(cudaStreamSynchronize(copy_stream), "D2H sync");
    const int sync_rc2 = cuda_status(cudaStreamSynchronize(stream), "trace sync");
    for (cudaEvent_t ev : done) cudaEventDestroy(ev);
    if (rc) return rc;
    if (sync_rc) return sync_rc;
    if (sync_rc2) return sync_rc2;
    time_trace = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    return CSP_OK;
}

// Chunks of a compact run: traced and compacted on `stream` while the chunk before is copied on
// `copy_stream`: up to four parts of the run, of at most 2^20 rays (84 MB of rows, still in L2 when they are
// compacted) and at least 327,680.  A copy costs about 2 us besides its bytes (16 B per ray of the single
// parabolic heliostat at the host link's ~190 GB/s), so the counts follow in one copy at the end.  4M rays
// of that heliostat: 577 us in one piece, 445 in eight chunks, 436 in four, 444 to 464 with chunks that
// start at 2^18 or 2^17 and double; the copies alone 349 us.  A part's launches and waits cost about 15 us, and
// field launches gain least from an early copy.  Times in 1 / 2 / 3 / 4 parts, us, of a hillside of 600, the
// parabolic heliostat, and a corridor of 1.5 records a ray: 300,000 rays 103 / 120 / 148 / 183, 87 / 91 / 106 / 125,
// 141 / 129 / 143 / 154; 600,000 154 / 150 / 184 / 205, 123 / 113 / 127 / 142, 230 / 196 / 202 / 208; 2^20 211 / 199 / 217 /
// 242, 173 / 155 / 165 / 173, 369 / 308 / 294 / 289; 2^21 350 / 306 / 314 / 334, 309 / 259 / 251 / 253, 684 / 570 / 535 / 523
// (into pageable memory 20 to 40 us more, alike).
constexpr uint64_t kCompactChunkMin = 327680, kCompactChunkMax = 1u << 20, kCompactParts = 4;
constexpr int kCompactRing = 2;  // chunks whose records wait on the device for their copy

int System::ensure_compact_buffers(uint64_t n) {
    if (n <= cap_compact_rays) return CSP_OK;
    cudaFree(d_cpoints);
    cudaFree(d_ccounts);
    cudaFree(d_csums);
    d_cpoints = nullptr;
    d_ccounts = nullptr;
    d_csums = nullptr;
    cap_compact_rays = 0;
    int rc;
    if ((rc = cuda_status(dev_alloc((void**)&d_cpoints, std::max<uint64_t>(n, 1) * 3 * sizeof(float)), "cudaMalloc")))
        return rc;
    if ((rc = cuda_status(dev_alloc((void**)&d_ccounts, std::max<uint64_t>(n, 1)), "cudaMalloc"))) return rc;
    // the offsets of the whole run, or of the chunks in flight
    const size_t sums = std::max<size_t>(compact_blocks(n) + 1, kCompactRing * (kCompactChunkMax / 256 + 1));
    if ((rc = cuda_status(dev_alloc((void**)&d_csums, sums * sizeof(unsigned long long)), "cudaMalloc"))) return rc;
    cap_compact_rays = n;
    return CSP_OK;
}

// The chunked form of run_to_host_compact, for a host buffer that holds any run's records.
int System::run_compact_chunks(float* points, uint8_t* counts, float* records, uint64_t chunk, uint64_t* n_records) {
    struct Chunk {
        uint64_t begin = 0, count = 0;
    } prev;
    cudaEvent_t done[kCompactRing] = {}, copied[kCompactRing] = {};
    int rc = CSP_OK;
    for (int i = 0; i < kCompactRing && !rc; ++i) {
        rc = cuda_status(cudaEventCreateWithFlags(&done[i], cudaEventDisableTiming), "cudaEventCreate");
        if (!rc) rc = cuda_status(cudaEventCreateWithFlags(&copied[i], cudaEventDisableTiming), "cudaEventCreate");
    }
    const uint64_t n = num_rays;
    uint64_t total = 0, next = 0;
    for (uint64_t k = 0; !rc; ++k) {
        Chunk cur;
        if (next < n) {
            // queue chunk k: it takes the place of chunk k - 2, whose copy was queued a turn ago
            cur = Chunk{next, std::min(chunk, n - next)};
            next += cur.count;
            const int at = (int)(k % kCompactRing);
            unsigned long long* sums = d_csums + (chunk / 256 + 1) * at;
            const float4* rows = d_hits + cur.begin * kMaxDepth;
            rc = cuda_status(launch_trace(args(cur.begin, cur.count, next_counter(stream)), stream), "trace_kernel");
            if (!rc && k >= kCompactRing)
                rc = cuda_status(cudaStreamWaitEvent(stream, copied[at], 0), "cudaStreamWaitEvent");
            if (!rc)
                rc = cuda_status(launch_compact_count(rows, cur.count, d_cpoints + 3 * cur.begin, d_ccounts + cur.begin,
                                                      sums, h_ctotal + at, stream),
                                 "compact_count_kernel");
            if (!rc)
                rc = cuda_status(launch_compact_write(rows, cur.count, d_ccounts + cur.begin, sums,
                                                      d_cring + 4 * chunk * at, stream),
                                 "compact_write_kernel");
            if (!rc) rc = cuda_status(cudaEventRecord(done[at], stream), "cudaEventRecord");
        }
        if (prev.count && !rc) {
            // copy chunk k - 1, whose number of records is known once it is done
            const int at = (int)((k - 1) % kCompactRing);
            if ((rc = cuda_status(cudaEventSynchronize(done[at]), "compact chunk"))) break;
            const uint64_t found = *(volatile unsigned long long*)(h_ctotal + at);
            auto copy = [&](void* dst, const void* src, size_t bytes, const char* what) {
                if (!rc && bytes)
                    rc = cuda_status(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, copy_stream), what);
            };
            copy(points + 3 * prev.begin, d_cpoints + 3 * prev.begin, prev.count * 3 * sizeof(float), "D2H points");
            copy(records + 4 * total, d_cring + 4 * chunk * at, found * sizeof(float4), "D2H records");
            if (!rc) rc = cuda_status(cudaEventRecord(copied[at], copy_stream), "cudaEventRecord");
            total += found;
        }
        prev = cur;
        if (!cur.count) break;
    }
    if (!rc) rc = cuda_status(cudaMemcpyAsync(counts, d_ccounts, n, cudaMemcpyDeviceToHost, copy_stream), "D2H counts");
    const int rc1 = cuda_status(cudaStreamSynchronize(copy_stream), "compact copy");
    const int rc2 = cuda_status(cudaStreamSynchronize(stream), "compact trace");
    for (int i = 0; i < kCompactRing; ++i) {
        if (done[i]) cudaEventDestroy(done[i]);
        if (copied[i]) cudaEventDestroy(copied[i]);
    }
    if (n_records) *n_records = total;
    return rc ? rc : (rc1 ? rc1 : rc2);
}

// Trace, then move the records in compact form: per ray its sun-plane point and the number of its
// further records, and those records in ray order (kernels in csp_kernels.cu).  Nothing is copied
// when the records exceed `capacity`; *n_records then tells how many there are.
int System::run_to_host_compact(float* points, uint8_t* counts, float* records, uint64_t capacity,
                                uint64_t* n_records) {
    NvtxRange nvtx("csp run_to_host_compact");
    if (!ready()) return fail(CSP_ERR_STATE, "run() before initialize()");
    int rc = ensure_hit_buffers();
    if (rc) return rc;
    const uint64_t n = num_rays;
    if ((rc = ensure_compact_buffers(n))) return rc;
    const auto t0 = std::chrono::steady_clock::now();
    auto timed = [&] {
        time_trace = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
        return CSP_OK;
    };
    // in chunks when no number of records can exceed the capacity (else it is known only after the
    // whole trace, and nothing may be copied before) and the run has more than one
    const uint64_t parts = std::max<uint64_t>(1, std::min(kCompactParts, n / kCompactChunkMin));
    const uint64_t chunk = std::min(kCompactChunkMax, ((n + parts - 1) / parts + 255) / 256 * 256);
    if (n > chunk && capacity / 4 >= n) {
        const uint64_t need = 4 * chunk * kCompactRing;
        if (need > cap_cring) {
            cudaFree(d_cring);
            d_cring = nullptr;
            cap_cring = 0;
            if (dev_alloc((void**)&d_cring, need * sizeof(float4)) == cudaSuccess) cap_cring = need;
            else cudaGetLastError();
        }
        if (!h_ctotal &&
            host_alloc((void**)&h_ctotal, kCompactRing * sizeof(unsigned long long)) != cudaSuccess) {
            h_ctotal = nullptr;
            cudaGetLastError();
        }
        if (cap_cring >= need && h_ctotal) {  // else in one piece, which needs less memory
            rc = run_compact_chunks(points, counts, records, chunk, n_records);
            return rc ? rc : timed();
        }
    }
    if ((rc = cuda_status(launch_trace(args(0, n, next_counter(stream)), stream), "trace_kernel"))) return rc;
    if ((rc = cuda_status(launch_compact_count(d_hits, n, d_cpoints, d_ccounts, d_csums, nullptr, stream),
                          "compact_count_kernel")))
        return rc;
    unsigned long long total = 0;
    if (n && (rc = cuda_status(cudaMemcpyAsync(&total, d_csums + compact_blocks(n), sizeof total, cudaMemcpyDeviceToHost,
                                               stream),
                               "D2H record count")))
        return rc;
    if ((rc = cuda_status(cudaStreamSynchronize(stream), "compact count"))) return rc;
    if (n_records) *n_records = total;
    if (total > capacity) return fail(CSP_ERR_INVALID_ARGUMENT, "the run's records exceed the capacity");
    if (total > cap_crecords) {
        cudaFree(d_crecords);
        d_crecords = nullptr;
        cap_crecords = 0;
        if ((rc = cuda_status(dev_alloc((void**)&d_crecords, total * sizeof(float4)), "cudaMalloc compact records")))
            return rc;
        cap_crecords = total;
    }
    if ((rc = cuda_status(launch_compact_write(d_hits, n, d_ccounts, d_csums, d_crecords, stream), "compact_write_kernel")))
        return rc;
    if (n && (rc = cuda_status(cudaMemcpyAsync(points, d_cpoints, n * 3 * sizeof(float), cudaMemcpyDeviceToHost, stream),
                               "D2H points")))
        return rc;
    if (n && (rc = cuda_status(cudaMemcpyAsync(counts, d_ccounts, n, cudaMemcpyDeviceToHost, stream), "D2H counts")))
        return rc;
    if (total && (rc = cuda_status(cudaMemcpyAsync(records, d_crecords, total * sizeof(float4), cudaMemcpyDeviceToHost,
                                                   stream),
                                   "D2H records")))
        return rc;
    if ((rc = cuda_status(cudaStreamSynchronize(stream), "compact copy"))) return rc;
    return timed();
}

double sun_plane_area(const SunFrame& f) {
    const double a[3] = {(double)f.v1.x - f.v0.x, (double)f.v1.y - f.v0.y, (double)f.v1.z - f.v0.z};
    const double b[3] = {(double)f.v3.x - f.v0.x, (double)f.v3.y - f.v0.y, (double)f.v3.z - f.v0.z};
    const double c[3] = {a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]};
    return std::sqrt(c[0] * c[0] + c[1] * c[1] + c[2] * c[2]);
}

void counts_to_flux(const uint32_t* counts, size_t n, double dni, double sun_area, uint64_t rays, double bin_area,
                    double* flux) {
    const double per = (rays > 0 && bin_area > 0) ? dni * sun_area / (double)rays / bin_area : 0.0;
    for (size_t i = 0; i < n; ++i) flux[i] = counts[i] * per;
}

int System::flux_map(uint32_t nx, uint32_t ny, uint32_t* counts, double dni, double* flux, bool staged) {
    NvtxRange nvtx("csp flux_map");
    if (!initialized || !d_hits) return fail(CSP_ERR_STATE, "flux map before initialize()/run()");
    if (nx == 0 || ny == 0 || (uint64_t)nx * ny > (1u << 26)) return fail(CSP_ERR_INVALID_ARGUMENT, "bad flux grid");
    const size_t nb = (size_t)nx * ny;
    // device: counters and map, zeroed in one go; host, pinned where there is memory for it: the sun frame
    // and the map
    constexpr size_t kStats = 4 * sizeof(unsigned long long);
    const size_t map_bytes = nb * sizeof(uint32_t), host_bytes = sizeof(SunFrame) + map_bytes;
    int rc;
    if (nb > cap_flux) {
        cudaFree(d_flux);
        d_flux = nullptr;
        cap_flux = 0;
        if ((rc = cuda_status(dev_alloc((void**)&d_flux, kStats + map_bytes), "cudaMalloc flux map"))) return rc;
        cap_flux = nb;
    }
    if (nb > cap_hflux) {
        if (h_flux) cudaFreeHost(h_flux);
        h_flux = nullptr;
        cap_hflux = 0;
        if (host_alloc((void**)&h_flux, host_bytes) == cudaSuccess) cap_hflux = nb;
        else cudaGetLastError();  // a slower copy
    }
    std::vector<float4> pageable(nb > cap_hflux ? (host_bytes + sizeof(float4) - 1) / sizeof(float4) : 0);
    unsigned char* const block = nb > cap_hflux ? reinterpret_cast<unsigned char*>(pageable.data()) : h_flux;
    FluxTarget F;
    flux_target(elements.back(), nx, ny, F);
    F.stats = reinterpret_cast<unsigned long long*>(d_flux);
    F.counts = reinterpret_cast<uint32_t*>(d_flux + kStats);
    F.staged = staged ? 1 : 0;
    if ((rc = cuda_status(cudaMemsetAsync(d_flux, 0, kStats + map_bytes, stream), "memset flux"))) return rc;
    if ((rc = cuda_status(launch_flux_records(d_hits, num_rays * kMaxDepth, F, stream), "flux_records_kernel")))
        return rc;
    if ((rc = cuda_status(cudaMemcpyAsync(block + sizeof(SunFrame), F.counts, map_bytes, cudaMemcpyDeviceToHost, stream),
                          "D2H flux map")))
        return rc;
    if ((rc = cuda_status(cudaMemcpyAsync(block, d_sun, sizeof(SunFrame), cudaMemcpyDeviceToHost, stream),
                          "D2H sun frame")))
        return rc;
    if ((rc = cuda_status(cudaStreamSynchronize(stream), "flux map"))) return rc;
    const SunFrame& f = *reinterpret_cast<const SunFrame*>(block);
    const uint32_t* host = reinterpret_cast<const uint32_t*>(block + sizeof(SunFrame));
    if (counts) std::copy(host, host + nb, counts);
    if (flux)
        counts_to_flux(host, nb, dni, sun_plane_area(f), num_rays, flux_bin_area(elements.back(), nx, ny), flux);
    return CSP_OK;
}

}  // namespace csp

using csp::System;

#define CSP_GUARD(h)                                                              \
    do {                                                                          \
        if (!(h)) return fail(CSP_ERR_INVALID_ARGUMENT, "null handle");           \
    } while (0)

extern "C" {

const char* csp_last_error(void) { return t_last_error.c_str(); }
int csp_abi_version(void) { return CSP_ABI_VERSION; }

int csp_bounds_check_status(int device, uint32_t* sites) {
    if (!sites) return fail(CSP_ERR_INVALID_ARGUMENT, "null output");
    *sites = 0;
    if (!csp::kBoundsCheckBuild) return fail(CSP_ERR_STATE, "not a bounds-check build (-DCSP_BOUNDS_CHECK)");
    int prev = -1;
    cudaGetDevice(&prev);
    int rc = csp::cuda_status(cudaSetDevice(device), "cudaSetDevice");
    if (rc) return rc;
    if ((rc = csp::cuda_status(cudaDeviceSynchronize(), "cudaDeviceSynchronize"))) return rc;
    *sites = csp::bounds_sites_trace() | csp::bounds_sites_batch() | csp::bounds_sites_sungrid();
    if (prev >= 0 && prev != device) cudaSetDevice(prev);
    return CSP_OK;
}

int csp_debug_fail_allocation(int64_t after) {
    if (after < -1) return fail(CSP_ERR_INVALID_ARGUMENT, "after must be >= -1");
    csp::g_fail_after.store((long long)after);
    return CSP_OK;
}

int csp_create(csp_handle* out, int device, uint64_t num_rays) {
    if (!out) return fail(CSP_ERR_INVALID_ARGUMENT, "null output handle");
    *out = nullptr;
    int count = 0;
    cudaError_t e = cudaGetDeviceCount(&count);
    if (e != cudaSuccess) return csp::cuda_status(e, "cudaGetDeviceCount");
    if (device < 0 || device >= count) return fail(CSP_ERR_INVALID_ARGUMENT, "no such CUDA device");
    if (!csp::valid_ray_window(0, num_rays)) return fail(CSP_ERR_INVALID_ARGUMENT, "num_rays must stay below 2^56");
    System* s = new (std::nothrow) System();
    if (!s) return fail(CSP_ERR_OUT_OF_MEMORY, "host allocation failed");
    s->device = device;
    s->num_rays = num_rays;
    *out = reinterpret_cast<csp_handle>(s);
    return CSP_OK;
}

int csp_destroy(csp_handle h) {
    CSP_GUARD(h);
    delete reinterpret_cast<System*>(h);
    return CSP_OK;
}

int csp_set_num_rays(csp_handle h, uint64_t num_rays) {
    CSP_GUARD(h);
    if (!csp::valid_ray_window(0, num_rays)) return fail(CSP_ERR_INVALID_ARGUMENT, "num_rays must stay below 2^56");
    reinterpret_cast<System*>(h)->num_rays = num_rays;
    return CSP_OK;
}

int csp_add_element(csp_handle h, const csp_element* e) {
    CSP_GUARD(h);
    if (!e) return fail(CSP_ERR_INVALID_ARGUMENT, "null element");
    reinterpret_cast<System*>(h)->elements.push_back(*e);
    return CSP_OK;
}

int csp_set_elements(csp_handle h, const csp_element* e, uint32_t n) {
    CSP_GUARD(h);
    if (!e && n) return fail(CSP_ERR_INVALID_ARGUMENT, "null elements");
    System* s = reinterpret_cast<System*>(h);
    s->elements.assign(e, e + n);
    return CSP_OK;
}

int csp_get_num_elements(csp_handle h, uint32_t* n) {
    CSP_GUARD(h);
    if (!n) return fail(CSP_ERR_INVALID_ARGUMENT, "null output");
    *n = (uint32_t)reinterpret_cast<System*>(h)->elements.size();
    return CSP_OK;
}

int csp_get_elements(csp_handle h, csp_element* out, uint32_t cap) {
    CSP_GUARD(h);
    System* s = reinterpret_cast<System*>(h);
    if (!out || cap < s->elements.size()) return fail(CSP_ERR_INVALID_ARGUMENT, "output too small");
    std::copy(s->elements.begin(), s->elements.end(), out);
    return CSP_OK;
}

int csp_set_sun_vector(csp_handle h, double x, double y, double z) {
    CSP_GUARD(h);
    System* s = reinterpret_cast<System*>(h);
    s->sun_dir[0] = x;
    s->sun_dir[1] = y;
    s->sun_dir[2] = z;
    return CSP_OK;
}

int csp_set_sun_shape(csp_handle h, int shape, double param) {
    CSP_GUARD(h);
    if (!csp::valid_sun_shape(shape)) return fail(CSP_ERR_INVALID_ARGUMENT, "unknown sun shape");
    if (!(param >= 0.0) || param > 0.5) return fail(CSP_ERR_INVALID_ARGUMENT, "sun shape parameter out of range");
    System* s = reinterpret_cast<System*>(h);
    s->sun_shape = shape;
    s->sun_param = param;
    return CSP_OK;
}

int csp_set_seed(csp_handle h, uint64_t seed, uint32_t instance) {
    CSP_GUARD(h);
    System* s = reinterpret_cast<System*>(h);
    s->seed = seed;
    s->instance = instance;
    return CSP_OK;
}

int csp_set_accel(csp_handle h, int mode) {
    CSP_GUARD(h);
    if (mode != CSP_ACCEL_AUTO && mode != CSP_ACCEL_BVH && mode != CSP_ACCEL_GRID)
        return fail(CSP_ERR_INVALID_ARGUMENT, "unknown acceleration mode");
    System* s = reinterpret_cast<System*>(h);
    s->accel = mode;
    s->initialized = false;  // takes effect at the next initialize()
    return CSP_OK;
}

int csp_get_accel(csp_handle h, int* mode) {
    CSP_GUARD(h);
    if (!mode) return fail(CSP_ERR_INVALID_ARGUMENT, "null output");
    const System* s = reinterpret_cast<System*>(h);
    *mode = (s->elements.size() <= csp::kFlatListMax) ? CSP_ACCEL_LIST : (s->grid.valid ? CSP_ACCEL_GRID : CSP_ACCEL_BVH);
    return CSP_OK;
}

int csp_set_record_ids(csp_handle h, int enable) {
    CSP_GUARD(h);
    reinterpret_cast<System*>(h)->record_ids = enable != 0;
    return CSP_OK;
}

int csp_initialize(csp_handle h) {
    CSP_GUARD(h);
    return reinterpret_cast<System*>(h)->initialize();
}

int csp_run(csp_handle h) {
    CSP_GUARD(h);
    return reinterpret_cast<System*>(h)->run();
}

int csp_trace_async(csp_handle h, void* stream) {
    CSP_GUARD(h);
    return reinterpret_cast<System*>(h)->trace_async(reinterpret_cast<cudaStream_t>(stream));
}

int csp_update(csp_handle h) {
    CSP_GUARD(h);
    return reinterpret_cast<System*>(h)->update();
}

int csp_copy_hits(csp_handle h, float* dst, uint32_t* ids, uint64_t first, uint64_t count) {
    CSP_GUARD(h);
    System* s = reinterpret_cast<System*>(h);
    if (!s->initialized || !s->d_hits) return fail(CSP_ERR_STATE, "no hit buffer (initialize first)");
    if (first > s->num_rays || count > s->num_rays - first) return fail(CSP_ERR_INVALID_ARGUMENT, "ray range out of bounds");
    if (!dst && count) return fail(CSP_ERR_INVALID_ARGUMENT, "null destination");
    int rc = csp::cuda_status(cudaStreamSynchronize(s->stream), "sync");
    if (rc) return rc;
    if (count) {
        rc = csp::cuda_status(cudaMemcpy(dst, s->d_hits + first * csp::kMaxDepth, count * csp::kMaxDepth * sizeof(float4),
                                         cudaMemcpyDeviceToHost),
                              "D2H hit records");
        if (rc) return rc;
    }
    if (ids) {
        if (!s->record_ids || !s->d_ids) return fail(CSP_ERR_STATE, "element ids are not being recorded");
        if (count)
            return csp::cuda_status(cudaMemcpy(ids, s->d_ids + first * csp::kMaxDepth,
                                               count * csp::kMaxDepth * sizeof(uint32_t), cudaMemcpyDeviceToHost),
                                    "D2H ids");
    }
    return CSP_OK;
}

int csp_trace_into(csp_handle h, void* hits, void* ids, uint64_t first, uint64_t count, void* stream) {
    CSP_GUARD(h);
    System* s = reinterpret_cast<System*>(h);
    if (!s->ready()) return fail(CSP_ERR_STATE, "trace before initialize()");
    if (!hits && count) return fail(CSP_ERR_INVALID_ARGUMENT, "null hit buffer");
    if (!csp::valid_ray_window(first, count))
        return fail(CSP_ERR_INVALID_ARGUMENT, "ray window [first_ray, first_ray + count) must stay below 2^56");
    cudaStream_t st = stream ? reinterpret_cast<cudaStream_t>(stream) : s->stream;
    // off the handle's stream static shares of the tiles
    csp::TraceArgs a = s->args(0, 0, st == s->stream ? s->next_counter(st) : nullptr);
    a.hits = reinterpret_cast<float4*>(hits);
    a.ids = reinterpret_cast<uint32_t*>(ids);
    a.ray_begin = first;
    a.count = count;
    return csp::cuda_status(csp::launch_trace(a, st), "trace_kernel");
}

int csp_run_to_host_compact(csp_handle h, float* points, uint8_t* counts, float* records, uint64_t capacity,
                            uint64_t* n_records) {
    CSP_GUARD(h);
    System* s = reinterpret_cast<System*>(h);
    if (s->num_rays && (!points || !counts)) return fail(CSP_ERR_INVALID_ARGUMENT, "null output");
    if (capacity && !records) return fail(CSP_ERR_INVALID_ARGUMENT, "null records with a capacity");
    return s->run_to_host_compact(points, counts, records, capacity, n_records);
}

int csp_run_to_host(csp_handle h, float* dst, uint32_t* ids) {
    CSP_GUARD(h);
    if (!dst) return fail(CSP_ERR_INVALID_ARGUMENT, "null destination");
    return reinterpret_cast<System*>(h)->run_to_host(dst, ids);
}

int csp_get_device_buffers(csp_handle h, void** hits, void** ids) {
    CSP_GUARD(h);
    System* s = reinterpret_cast<System*>(h);
    if (hits) *hits = s->d_hits;
    if (ids) *ids = s->record_ids ? s->d_ids : nullptr;
    return CSP_OK;
}

int csp_get_timing(csp_handle h, double* setup_s, double* trace_s) {
    CSP_GUARD(h);
    System* s = reinterpret_cast<System*>(h);
    if (setup_s) *setup_s = s->time_setup;
    if (trace_s) *trace_s = s->time_trace;
    return CSP_OK;
}

int csp_element_frame(const csp_element* e, double* euler, double* g2l, double* aabb_lo, double* aabb_hi) {
    if (!e) return fail(CSP_ERR_INVALID_ARGUMENT, "null element");
    double eu[3], G[9], lo[3], hi[3];
    csp::element_frame(*e, eu, G, lo, hi);
    if (euler) std::memcpy(euler, eu, sizeof eu);
    if (g2l) std::memcpy(g2l, G, sizeof G);
    if (aabb_lo) std::memcpy(aabb_lo, lo, sizeof lo);
    if (aabb_hi) std::memcpy(aabb_hi, hi, sizeof hi);
    return CSP_OK;
}

int csp_flux_map(csp_handle h, uint32_t nx, uint32_t ny, uint32_t* counts, double dni, double* flux) {
    CSP_GUARD(h);
    return reinterpret_cast<System*>(h)->flux_map(nx, ny, counts, dni, flux);
}

int csp_flux_map_ex(csp_handle h, uint32_t nx, uint32_t ny, int flags, uint32_t* counts, double dni, double* flux) {
    CSP_GUARD(h);
    if (flags & ~CSP_OUT_STAGED) return fail(CSP_ERR_INVALID_ARGUMENT, "unknown output flags");
    return reinterpret_cast<System*>(h)->flux_map(nx, ny, counts, dni, flux, (flags & CSP_OUT_STAGED) != 0);
}

int csp_flux_target(const csp_element* rcv, uint32_t nx, uint32_t ny, float* out) {
    if (!rcv || !out) return fail(CSP_ERR_INVALID_ARGUMENT, "null argument");
    if (nx == 0 || ny == 0) return fail(CSP_ERR_INVALID_ARGUMENT, "bad flux grid");
    csp::FluxTarget F;
    csp::flux_target(*rcv, nx, ny, F);
    const float v[20] = {F.o.x, F.o.y, F.o.z, F.x.x, F.x.y, F.x.z, F.y.x, F.y.y, F.y.z, F.z.x,
                         F.z.y, F.z.z, F.hx,  F.hy,  F.kx,  F.ky,  F.keep, (float)F.kind,
                         (float)csp::flux_bin_area(*rcv, nx, ny), 0.f};
    std::memcpy(out, v, sizeof(v));
    return CSP_OK;
}

int csp_get_sun_plane(csp_handle h, float* out) {
    CSP_GUARD(h);
    System* s = reinterpret_cast<System*>(h);
    if (!out) return fail(CSP_ERR_INVALID_ARGUMENT, "null output");
    if (!s->initialized) return fail(CSP_ERR_STATE, "initialize first");
    csp::SunFrame f;
    int rc = csp::cuda_status(cudaMemcpy(&f, s->d_sun, sizeof(f), cudaMemcpyDeviceToHost), "D2H sun frame");
    if (rc) return rc;
    const float v[16] = {f.s_d.x, f.s_d.y, f.s_d.z, f.v0.x, f.v0.y, f.v0.z, f.v1.x, f.v1.y,
                         f.v1.z,  f.v2.x,  f.v2.y,  f.v2.z, f.v3.x, f.v3.y, f.v3.z, f.s_d.w};
    std::memcpy(out, v, sizeof(v));
    return CSP_OK;
}

}  // extern "C"
