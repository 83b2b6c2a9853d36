// csp_kernels.cu -- sm_103a kernels of the single-scene trace path.
//
// Built with -fmad=false (plus IEEE division and square root): every expression rounds exactly as
// written, which is what makes the hit records bit-identical to the host restatement of the
// reference.  Fused multiply-adds appear only as explicit fmaf() calls in csp_math.cuh.
//
// Kernel map (reference counterpart in parentheses, paths inside the reference project):
//   prepare_sun_kernel   sun-plane distance, u/v bounds, parallelogram, cone frame
//                        (lib/sun_utils.cu:53-179, lib/geometry_manager.cpp:97-148, cuda/sun.cu:76-79)
//   trace_kernel         ray generation (cuda/sun.cu:16-38,72-134), closest-hit search over the
//                        elements whose AABB the ray overlaps (OptiX traversal + the intersection
//                        programs of cuda/intersection.cu:47-85,177-296,318-448), shading
//                        (cuda/materials.cu:26-231) and the hit_point_buffer write.
//   flux_records_kernel  receiver flux map from a dense hit buffer
//                        (scripts/post_processing/flux_map_calculator.py:135-179)
// The device functions of the path live in csp_trace.cuh.
#include <algorithm>
#include <atomic>
#include <mutex>

#include "csp_kernels.cuh"
#include "csp_trace.cuh"

namespace csp {
namespace {

constexpr int kTraceBlock = 128;
constexpr int kFluxBlock = 256;

template <int kCluster>
__global__ void __launch_bounds__(kStateBlock) __cluster_dims__(kCluster)
    prepare_sun_kernel(const Aabb* __restrict__ aabbs, int n, float3 s, float tan_pad, int shape, float param,
                       SunFrame* __restrict__ out) {
    __shared__ StateSmem sm;
    sun_frame_state<kCluster>(aabbs, n, s, tan_pad, shape, param, out, sm);
}

template <int kAccel, bool kIds>
using PlainCfg = Cfg<kTraceBlock, kAccel, true, false, kIds>;

template <int kAccel>
struct TraceSmem {
    typename PlainCfg<kAccel, false>::Stage stage;
    typename PlainCfg<kAccel, false>::Core core;
};

// Resident CTAs per SM the register budget is cut for: eight of 128 threads (64 registers, 1,024
// threads), more warps to cover the record stream of the element-list kernel and the dependent loads
// of the candidate and cell lists of the others.  64M rays over 10,000 heliostats: seven / eight / nine 4905 /
// 4656 / 4726 us, four of 256 threads (a tile's barriers over twice the warps) 4691; the single
// parabolic heliostat, 16M rays: four of 256 302 against 287 us, ten of 128 (48 registers, spills) 299, two of 512 322.
constexpr int kTraceBlocksPerSM = 1024 / kTraceBlock;

// Persistent kernel over the tiles of one launch; dense records out.  With a tile counter every CTA
// starts on a share of its own (half of an even share for element lists, a quarter for fields, whose
// tiles differ much in work) and then takes guided grabs (a quarter of an even share of the tiles
// left, shrinking to single tiles at the end), each requested while the last tile of the one before is
// traced; grabs and shares are at most kTraceGrab tiles, so that the CTAs work on the same stretch of
// the sun plane and share its scene data in L2 (64M rays over 10,000 heliostats at caps of 4 / 8 / 16
// tiles: 4679 / 4656 / 4652 us; before rows were written by five lanes 32 / 64: 4992 / 5070 against 4857).  Without a counter: one contiguous even share
// (element lists: the next tile's Halton sums are prefetched) or round robin (fields).  The records
// do not depend on which CTA traces a tile.  Guided grabs measured 27.5 ms per 268M rays of the
// 10,000-heliostat field against 30.3 ms round robin (a CTA's tiles differ much in work, so round robin
// ends in a long tail).
constexpr uint32_t kTraceGrab = 8;

template <int kAccel, bool kIds>
__global__ void __launch_bounds__(kTraceBlock, kTraceBlocksPerSM) trace_kernel(
    const typename PlainCfg<kAccel, kIds>::Args A) {
    using C = PlainCfg<kAccel, kIds>;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    TraceSmem<kAccel>& sm = *reinterpret_cast<TraceSmem<kAccel>*>(smem_raw);
    load_instance_smem<C>(A, sm.core);
    if constexpr (C::kFlat)
        for (int i = threadIdx.x; i < kTraceBlock * kMaxDepth; i += kTraceBlock)
            sm.stage.row[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    // the shared-memory Halton table serves only launches without the device-wide 3^12 table
    if (!A.h3t12)
        for (uint32_t m = threadIdx.x; m < kH3Tab; m += kTraceBlock) sm.core.t6[m] = halton3(m);
    if (threadIdx.x == 0) {
        sm.core.qsize = 0;
        sm.core.gsize = 0;
    }
    __syncthreads();
    const Sink none{nullptr, nullptr};
    // 32-bit tile indices: launch_trace_t takes fewer than 2^31 tiles
    const uint32_t tiles = (uint32_t)((A.count + kTraceBlock - 1) / kTraceBlock);
    __shared__ uint32_t s_grab;
    const bool guided = A.tile_counter != nullptr;
    // this CTA's tiles: g, g + step, ... below g1; the counter hands out those from `base` on
    uint32_t g, g1, step = 1, base = 0;
    if (guided) {
        const uint32_t share = max(1u, min(kTraceGrab, tiles / gridDim.x / (C::kFlat ? 2u : 4u)));
        base = share * gridDim.x;
        g = share * blockIdx.x;
        g1 = g + share;
    } else if (C::kFlat) {
        g = (uint32_t)((uint64_t)tiles * blockIdx.x / gridDim.x);
        g1 = (uint32_t)((uint64_t)tiles * (blockIdx.x + 1) / gridDim.x);
    } else {
        g = blockIdx.x;
        g1 = tiles;
        step = gridDim.x;
    }
    bool flush = false;  // no tiles left: the remaining queued rays
    int qs = 0;          // queue size (see phase_b)
    for (;;) {
        if (phase_b<C>(A, none, sm.core, flush, qs)) continue;
        if (flush) break;
        if (g >= g1) {
            flush = true;
            continue;
        }
        const bool last = guided && g + 1 == g1;
        uint32_t want = 0, at = 0;
        if (last) {
            // tiles left as far as this CTA knows
            const uint32_t left = tiles - min(max(g1, base), tiles);
            want = max(1u, min(kTraceGrab, left / (gridDim.x * 4)));
            if (threadIdx.x == 0) at = atomicAdd(A.tile_counter, want);
        }
        trace_tile<C>(A, none, sm.core, &sm.stage, g, qs);
        g += step;
        if (last) {
            // the tile's barrier lies between the reads of the last grab and this write
            if (threadIdx.x == 0) s_grab = at;
            __syncthreads();
            g = min(base + s_grab, tiles);
            g1 = min(g + want, tiles);
        }
    }
    // the last CTA leaves the counter as it found it
    if (guided && threadIdx.x == 0 && atomicAdd(A.tile_counter + 1, 1u) == gridDim.x - 1) {
        A.tile_counter[0] = 0u;
        A.tile_counter[1] = 0u;
    }
}

// Resident CTA slots of the device for a trace kernel; the first call on a device prepares the kernel.
template <int kAccel, bool kIds>
cudaError_t find_slots(int dev, int& slots) {
    int sms = 0, per_sm = 0;
    cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(trace_kernel<kAccel, kIds>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(TraceSmem<kAccel>));
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, trace_kernel<kAccel, kIds>, kTraceBlock,
                                                          sizeof(TraceSmem<kAccel>));
    slots = std::max(1, sms * std::max(1, per_sm));
    return e;
}

template <int kAccel, bool kIds>
cudaError_t launch_trace_ids(const TraceArgs& args, unsigned grid, cudaStream_t stream) {
    typename PlainCfg<kAccel, kIds>::Args a;
    static_cast<TraceArgs&>(a) = args;
    if constexpr (PlainCfg<kAccel, kIds>::kSched) philox_keys(args.seed, a.keys);
    using Smem = TraceSmem<kAccel>;
    // field launches leave the unused Halton table to L1 (64M rays over 10,000 heliostats 4680 -> 4660 us);
    // element lists gain nothing from it (200,000 rays of the single parabolic heliostat 7.20, 7.64 without)
    const size_t smem = sizeof(Smem) - (kAccel != kAccelFlat && args.h3t12 ? sizeof(Smem::core.t6) : 0);
    trace_kernel<kAccel, kIds><<<grid, kTraceBlock, smem, stream>>>(a);
    return cudaGetLastError();
}

// Launches with and without element ids are kernels of their own: in one kernel the ids' stores cost the
// launches without them registers (64M rays over 10,000 heliostats 4807 us, against 4653 apart).
template <int kAccel>
cudaError_t launch_trace_t(const TraceArgs& args, cudaStream_t stream) {
    // persistent grid: every resident CTA slot of the device (found once per device, for both kernels, so
    // that the first launch of either prepares the other too; devices past 63 each time), never more
    // CTAs than tiles
    static std::atomic<uint64_t> slots_of[64];
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    uint64_t both = dev < 64 ? slots_of[dev].load(std::memory_order_acquire) : 0;
    if (both == 0) {
        int plain = 0, ids = 0;
        e = find_slots<kAccel, false>(dev, plain);
        if (e == cudaSuccess) e = find_slots<kAccel, true>(dev, ids);
        if (e != cudaSuccess) return e;
        both = (uint64_t)ids << 32 | (uint32_t)plain;
        if (dev < 64) slots_of[dev].store(both, std::memory_order_release);
    }
    const uint64_t slots = args.ids ? both >> 32 : (uint32_t)both;
    const uint64_t tiles = (args.count + kTraceBlock - 1) / kTraceBlock;  // CTAs that have work
    if (tiles > 0x7FFFFFFFull) return cudaErrorInvalidValue;  // 22 TB of records
    const unsigned grid = (unsigned)std::min(tiles, slots);
    return args.ids ? launch_trace_ids<kAccel, true>(args, grid, stream)
                    : launch_trace_ids<kAccel, false>(args, grid, stream);
}

// Pass over n_records float4 records {stage, x, y, z}: stage-1 records are counted, stage-2 records
// are counted and binned.  HBM-bound (80 B per ray read).  About one record in fifteen of a field is a
// receiver hit, so binning each where it is found runs the angle of the cylinder on two lanes of a
// warp (170 us for the 335 MB of 4M rays); a warp collects its receiver hits in shared memory and
// bins 32 at a time instead: 57 us, 5.9 TB/s.
constexpr int kFluxLoads = 4;  // coalesced loads in flight per thread
__global__ void __launch_bounds__(kFluxBlock) flux_records_kernel(const float4* __restrict__ hits,
                                                                    uint64_t n_records, const FluxTarget F) {
    __shared__ float queue[3][kFluxBlock / 32][64];  // receiver hits of each warp: up to 31 waiting and 32 new
    __shared__ unsigned long long stat[4];
    if (threadIdx.x < 4) stat[threadIdx.x] = 0;
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t mirror = 0, receiver = 0, binned = 0;
    int qn = 0;
    auto bin = [&](int k) {
        const int b = flux_bin(F, f3(queue[0][warp][k], queue[1][warp][k], queue[2][warp][k]));
        if (b >= 0 && CSP_BOUNDS(3, b < F.nx * F.ny)) {
            atomicAdd(F.counts + b, 1u);
            ++binned;
        }
    };
    constexpr uint64_t kSpan = (uint64_t)kFluxBlock * kFluxLoads;
    for (uint64_t base = blockIdx.x * kSpan; base < n_records; base += gridDim.x * kSpan) {
        float4 r[kFluxLoads];
#pragma unroll
        for (int q = 0; q < kFluxLoads; ++q) {
            const uint64_t i = base + (uint64_t)q * kFluxBlock + threadIdx.x;
            r[q] = i < n_records ? __ldg(hits + i) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int q = 0; q < kFluxLoads; ++q) {
            if (r[q].x == 1.0f) ++mirror;
            bool want = r[q].x == 2.0f;
            // direct sun on the receiver (slot 1) is not a staged result
            if (F.staged && want) want = (base + (uint64_t)q * kFluxBlock + threadIdx.x) % kMaxDepth != 1;
            const unsigned mask = __ballot_sync(0xffffffffu, want);
            if (mask == 0u) continue;
            if (want) {
                const int k = qn + __popc(mask & ((1u << lane) - 1u));
                queue[0][warp][k] = r[q].y;
                queue[1][warp][k] = r[q].z;
                queue[2][warp][k] = r[q].w;
                ++receiver;
            }
            qn += __popc(mask);
            if (qn >= 32) {
                __syncwarp();
                qn -= 32;
                bin(qn + lane);
                __syncwarp();
            }
        }
    }
    __syncwarp();
    if (lane < qn) bin(lane);
    for (int o = 16; o > 0; o >>= 1) {
        mirror += __shfl_xor_sync(0xffffffffu, mirror, o);
        receiver += __shfl_xor_sync(0xffffffffu, receiver, o);
        binned += __shfl_xor_sync(0xffffffffu, binned, o);
    }
    if (lane == 0) {
        atomicAdd(stat + 1, (unsigned long long)mirror);
        atomicAdd(stat + 2, (unsigned long long)receiver);
        atomicAdd(stat + 3, (unsigned long long)binned);
    }
    __syncthreads();
    if (threadIdx.x < 4 && threadIdx.x > 0 && stat[threadIdx.x]) atomicAdd(F.stats + threadIdx.x, stat[threadIdx.x]);
}

// Compact records (csp_run_to_host_compact): a row of the dense buffer is the sun-plane record in
// slot 0, then the ray's further records in slots 1.. (stage 1 or 2, so x != 0), then empty slots.
constexpr int kCompactBlock = 256;

// Block-wide exclusive prefix of v (kCompactBlock threads); `total` receives the block's sum.
__device__ uint32_t block_exclusive(uint32_t v, uint32_t* scratch, uint32_t& total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) scratch[warp] = x;
    __syncthreads();
    uint32_t before = 0;
    total = 0;
    for (int w = 0; w < kCompactBlock / 32; ++w) {
        if (w < warp) before += scratch[w];
        total += scratch[w];
    }
    return before + x - v;
}

// Sun-plane points (3 floats per ray), the number of records beyond slot 0 of every ray, and their sum
// per block: the one pass that reads every row.  A block's 256 rows are read as 1,280 coalesced
// records (five loads in flight per thread); points and counts are put together in shared memory.
__global__ void __launch_bounds__(kCompactBlock) compact_count_kernel(const float4* __restrict__ hits, uint64_t n,
                                                                      float* __restrict__ points,
                                                                      uint8_t* __restrict__ counts,
                                                                      unsigned long long* __restrict__ block_sums) {
    __shared__ uint32_t scratch[kCompactBlock / 32], cnt[kCompactBlock];
    __shared__ alignas(16) float pts[3 * kCompactBlock];
    const uint64_t r0 = (uint64_t)blockIdx.x * kCompactBlock;
    const uint32_t rows = (uint32_t)min((uint64_t)kCompactBlock, n - r0);
    cnt[threadIdx.x] = 0;
    __syncthreads();
    float4 rec[kMaxDepth];
#pragma unroll
    for (int q = 0; q < kMaxDepth; ++q) {
        const uint32_t e = threadIdx.x + q * kCompactBlock;
        rec[q] = e < rows * kMaxDepth ? __ldg(hits + r0 * kMaxDepth + e) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int q = 0; q < kMaxDepth; ++q) {
        const uint32_t e = threadIdx.x + q * kCompactBlock, row = e / kMaxDepth;
        if (e == row * kMaxDepth) {
            pts[3 * row] = rec[q].y;
            pts[3 * row + 1] = rec[q].z;
            pts[3 * row + 2] = rec[q].w;
        } else if (rec[q].x != 0.0f) {
            atomicAdd(&cnt[row], 1u);
        }
    }
    __syncthreads();
    const uint32_t c = cnt[threadIdx.x];
    if (threadIdx.x < rows) counts[r0 + threadIdx.x] = (uint8_t)c;
    float* out = points + 3 * r0;
    if (rows == kCompactBlock && threadIdx.x < 3 * kCompactBlock / 4)
        reinterpret_cast<float4*>(out)[threadIdx.x] = reinterpret_cast<const float4*>(pts)[threadIdx.x];
    else if (rows < kCompactBlock)
        for (uint32_t k = threadIdx.x; k < 3 * rows; k += kCompactBlock) out[k] = pts[k];
    uint32_t total;
    block_exclusive(c, scratch, total);
    if (threadIdx.x == 0) block_sums[blockIdx.x] = total;
}

// In place: block sums -> exclusive block offsets, the grand total after the last block and, when
// given, in pinned host memory (a copy of its own would queue behind the record copies of the chunk
// before).
__global__ void __launch_bounds__(1024) compact_scan_kernel(unsigned long long* __restrict__ sums, uint64_t nb,
                                                            unsigned long long* host_total) {
    __shared__ unsigned long long part[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned long long before = 0;
    for (uint64_t c0 = 0; c0 < nb; c0 += 1024) {
        const uint64_t c = c0 + threadIdx.x;
        const unsigned long long v = c < nb ? sums[c] : 0ull;
        unsigned long long x = v;
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) part[warp] = x;
        __syncthreads();
        unsigned long long w = part[lane];
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        const unsigned long long all = __shfl_sync(0xffffffffu, w, 31);
        const unsigned long long mine = __shfl_sync(0xffffffffu, w, (warp + 31) & 31);
        if (c < nb) sums[c] = before + (warp ? mine : 0ull) + x - v;
        before += all;
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        sums[nb] = before;
        if (host_total) *host_total = before;
    }
}

// The records beyond slot 0, in ray order.
__global__ void __launch_bounds__(kCompactBlock) compact_write_kernel(const float4* __restrict__ hits, uint64_t n,
                                                                      const uint8_t* __restrict__ counts,
                                                                      const unsigned long long* __restrict__ offsets,
                                                                      float4* __restrict__ records) {
    __shared__ uint32_t scratch[kCompactBlock / 32];
    const uint64_t r = (uint64_t)blockIdx.x * kCompactBlock + threadIdx.x;
    const uint32_t c = r < n ? counts[r] : 0u;
    uint32_t total;
    const uint32_t ex = block_exclusive(c, scratch, total);
    const uint64_t o = offsets[blockIdx.x] + ex;
    for (uint32_t s = 0; s < c; ++s) records[o + s] = __ldg(&hits[r * kMaxDepth + 1 + s]);
}

__global__ void __launch_bounds__(256) halton3_table_kernel(float* __restrict__ t) {
    const uint32_t m = blockIdx.x * 256u + threadIdx.x;
    if (m < kH3T12) t[m] = halton3(m);
    if (m < kH3Tail) {
        uint32_t j = m;
        for (uint32_t k = 0; k < 8; ++k) {
            const uint32_t q = j / 3u;
            t[kH3TailAt + 8 * m + k] =
                k < kH3TailDigits ? c_halton3_f[kH3T12Digits + k] * (float)(j - 3u * q) : 0.0f;
            j = q;
        }
    }
}

}  // namespace

const float* halton3_table() {
    constexpr int kMaxDevices = 64;
    static std::mutex mu;
    static float* tables[kMaxDevices] = {};
    static bool tried[kMaxDevices] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
        cudaGetLastError();
        return nullptr;
    }
    std::lock_guard<std::mutex> lk(mu);
    if (!tried[dev]) {
        tried[dev] = true;
        float* t = nullptr;
        if (dev_alloc((void**)&t, (kH3TailAt + 8 * kH3Tail) * sizeof(float)) == cudaSuccess) {
            halton3_table_kernel<<<(kH3T12 + 255) / 256, 256>>>(t);
            if (cudaGetLastError() == cudaSuccess && cudaDeviceSynchronize() == cudaSuccess) tables[dev] = t;
            else cudaFree(t);
        }
        cudaGetLastError();  // a failed table only means the loop path
    }
    return tables[dev];
}

cudaError_t launch_prepare_sun(const Aabb* aabbs, int n, float sx, float sy, float sz, float tan_pad, int shape,
                               float param, SunFrame* out, cudaStream_t stream) {
    const float3 s = make_float3(sx, sy, sz);
    if (n >= kStateClusterMin)
        prepare_sun_kernel<kStateCluster>
            <<<kStateCluster, kStateBlock, 0, stream>>>(aabbs, n, s, tan_pad, shape, param, out);
    else
        prepare_sun_kernel<1><<<1, kStateBlock, 0, stream>>>(aabbs, n, s, tan_pad, shape, param, out);
    return cudaGetLastError();
}

cudaError_t launch_trace(const TraceArgs& args, cudaStream_t stream) {
    if (args.count == 0) return cudaSuccess;
    if (args.n_prims <= kFlatMax) return launch_trace_t<kAccelFlat>(args, stream);
    if (!args.sgrid) return cudaErrorInvalidValue;  // scenes above the element list need their sun grid
    if (args.grid) return launch_trace_t<kAccelGrid>(args, stream);
    return launch_trace_t<kAccelBvh>(args, stream);
}

uint64_t compact_blocks(uint64_t n) { return (n + kCompactBlock - 1) / kCompactBlock; }

cudaError_t launch_compact_count(const float4* hits, uint64_t n, float* points, uint8_t* counts,
                                 unsigned long long* block_sums, unsigned long long* host_total,
                                 cudaStream_t stream) {
    const uint64_t nb = compact_blocks(n);
    if (nb == 0) return cudaSuccess;
    if (nb > 0x7FFFFFFFull) return cudaErrorInvalidValue;
    compact_count_kernel<<<(unsigned)nb, kCompactBlock, 0, stream>>>(hits, n, points, counts, block_sums);
    compact_scan_kernel<<<1, 1024, 0, stream>>>(block_sums, nb, host_total);
    return cudaGetLastError();
}

cudaError_t launch_compact_write(const float4* hits, uint64_t n, const uint8_t* counts,
                                 const unsigned long long* block_offsets, float4* records, cudaStream_t stream) {
    const uint64_t nb = compact_blocks(n);
    if (nb == 0) return cudaSuccess;
    compact_write_kernel<<<(unsigned)nb, kCompactBlock, 0, stream>>>(hits, n, counts, block_offsets, records);
    return cudaGetLastError();
}

cudaError_t launch_flux_records(const float4* hits, uint64_t n_records, const FluxTarget& F, cudaStream_t stream) {
    if (n_records == 0) return cudaSuccess;
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    constexpr uint64_t kSpan = (uint64_t)kFluxBlock * kFluxLoads;
    const uint64_t blocks = std::min<uint64_t>((n_records + kSpan - 1) / kSpan, (uint64_t)sms * 8);
    flux_records_kernel<<<(unsigned)blocks, kFluxBlock, 0, stream>>>(hits, n_records, F);
    return cudaGetLastError();
}

uint32_t bounds_sites_trace() { return take_bounds_sites(); }

}  // namespace csp
