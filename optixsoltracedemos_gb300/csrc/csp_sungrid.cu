// csp_sungrid.cu -- device build of the sun-ray candidate grid (SunGrid, csp_types.cuh) of each
// scene state, after its sun frame.
//
// The reference has no counterpart: OptiX traverses its GAS from the sun plane for every ray
// (cuda/sun.cu:119-133).  Here the sun rays of scenes above 8 elements find their candidates in one
// cell of a grid over the sun plane's Halton coordinates, binned from the elements' candidate
// rectangles (cross_rect, csp_trace.cuh), and rays in a clear cell of the reach raster (reach_rect)
// skip the direction and the search altogether.  Which elements a ray tests changes, never which hit
// it finds: the rectangles bound every ray that can meet an element's AABB, and the closest hit keeps
// the lower element index on equal t whatever the order of the candidates.
//
// Four launches per set of states:
//   size    a block or a cluster of kStateCluster blocks per state (dependent reductions over the elements: the
//           middle of the field and with it the reference plane; every element's rectangles; the grid
//           size from the candidate rectangles' mean extent, shrunk until the registered items fit
//           the capacity), the descriptor, zeroed counts and raster
//   count   kElemLanes threads per element: raster bits, per-cell counts, or a place in the global
//           list for rectangles of more than kSunGridMaxCells cells
//   ranges  one thread per four cells: a warp takes the sum of its cells' counts from the state's
//           item counter
//   fill    kElemLanes threads per element: rectangles and exact boxes into their cells
// The last three also build the field grid (GridDesc) of each state that has one, as blockIdx.z = 1.
// Each is a chain of memory latencies, so the wide ones take the whole device rather than one block
// or cluster per state: 16 + 7 + 4.5 + 6 us for 10,001 elements, against 98 us with the count per
// element and the scan in one block, and 96 us with all phases in one cluster.
// The order of the cells' ranges, of the items within a cell and of the global list follows the
// atomics; nothing that a ray records depends on it.
#include <algorithm>

#include "csp_kernels.cuh"
#include "csp_scene.h"
#include "csp_trace.cuh"

namespace csp {
namespace {

constexpr int kMaxAxisCells = 4096;
constexpr float kCellScale = 0.5f;  // cell width / mean rectangle width
constexpr int kMaxJobsPerLaunch = 65535;  // gridDim.y limit
constexpr int kElemBlock = 256;
constexpr int kWideField = 65536;  // field cells (0.5 MB) from which one block would take long to zero them
constexpr int kElemLanes = 8;  // lanes that share an element's cells and raster words

size_t a256(size_t x) { return (x + 255) & ~(size_t)255; }

// Cells covered by rectangle r, clamped to [0, 1]^2, in an nu x nv grid: a candidate point in r,
// clamped the same way by the lookup, lies in one of them.
__device__ __forceinline__ void sg_range(float4 r, float fnu, float fnv, int nu, int nv, int& iu0, int& iu1, int& iv0,
                                         int& iv1) {
    iu0 = sg_cell(__saturatef(r.x), fnu, nu);
    iu1 = sg_cell(__saturatef(r.y), fnu, nu);
    iv0 = sg_cell(__saturatef(r.z), fnv, nv);
    iv1 = sg_cell(__saturatef(r.w), fnv, nv);
}

// Set the raster bits of reach rectangle r (words w = lane of `lanes`, lane + lanes, ...).
__device__ __forceinline__ void set_reach(uint32_t* __restrict__ raster, float4 r, int lane, int lanes) {
    if (!(r.y >= 0.0f && r.x <= 1.0f && r.w >= 0.0f && r.z <= 1.0f)) return;  // holds no ray
    int iu0, iu1, iv0, iv1;
    sg_range(r, (float)kReachRaster, (float)kReachRaster, kReachRaster, kReachRaster, iu0, iu1, iv0, iv1);
    const int w0 = iu0 >> 5, nw = (iu1 >> 5) - w0 + 1;
    for (int k = lane; k < nw * (iv1 - iv0 + 1); k += lanes) {
        const int row = iv0 + k / nw, word = w0 + k % nw;
        const int b0 = max(iu0 - 32 * word, 0), b1 = min(iu1 - 32 * word, 31);
        const uint32_t bits = (0xFFFFFFFFu >> (31 - b1)) & (0xFFFFFFFFu << b0);
        uint32_t* p = raster + row * (kReachRaster / 32) + word;
        if ((*reinterpret_cast<volatile uint32_t*>(p) & bits) != bits) atomicOr(p, bits);
    }
}

template <int kCluster>
__global__ void __launch_bounds__(kStateBlock) __cluster_dims__(kCluster)
    sungrid_size_kernel(const SunGridJob* __restrict__ jobs) {
    const SunGridJob& J = jobs[blockIdx.x / kCluster];
    const int n = J.n;
    constexpr int kThreads = kCluster * kStateBlock;
    const int tid = (int)(blockIdx.x % kCluster) * kStateBlock + (int)threadIdx.x;
    __shared__ SunFrame S;
    __shared__ StateSmem sm;
    __shared__ unsigned long long upart[kStateBlock / 32], uslot;
    if (threadIdx.x < sizeof(SunFrame) / 4)
        reinterpret_cast<uint32_t*>(&S)[threadIdx.x] = reinterpret_cast<const uint32_t*>(J.sun)[threadIdx.x];
    for (int c = tid; c < kReachRaster * kReachRaster / 128; c += kThreads)
        reinterpret_cast<uint4*>(J.reach)[c] = make_uint4(0u, 0u, 0u, 0u);
    if (tid == 0) *J.alloc = 0u;
    if (J.field_cells) {
        for (int c = tid; c < J.field_nx * J.field_ny; c += kThreads) J.field_cells[c] = make_uint2(0u, 0u);
        if (tid == 0) *J.field_alloc = 0u;
    }
    __syncthreads();
    const float inf = __int_as_float(0x7f800000);
    const float tan_a = cone_tan(S);
    // the reference plane, horizontal or across the sun, through the middle of the elements before
    // the receiver (the last one), whichever the cone can move less from
    float zlo = inf, zhi = -inf, hlo = inf, hhi = -inf;
    for (int e = tid; e + 1 < n; e += kThreads) {
        const Aabb b = J.aabbs[e];
        zlo = fminf(zlo, b.lo.z);
        zhi = fmaxf(zhi, b.hi.z);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const float h = dot(corner(b, k), xyz(S.w));
            hlo = fminf(hlo, h);
            hhi = fmaxf(hhi, h);
        }
    }
    const float4 mid = state_reduce<kCluster>(make_float4(zlo, -zhi, hlo, -hhi), sm.part, &sm.slot, Min4());
    const float dz = fabsf(S.w.z) - tan_a * sqrtf(fmaxf(0.0f, 1.0f - S.w.z * S.w.z));
    const bool level = dz > 0.02f && (-mid.y - mid.x) < dz * (-mid.w - mid.z);
    const float4 plane = level ? make_float4(0.0f, 0.0f, 1.0f, 0.5f * (mid.x - mid.y))
                               : make_float4(S.w.x, S.w.y, S.w.z, 0.5f * (mid.z - mid.w));
    const float den = level ? dz : dot(xyz(S.w), xyz(S.w)) - 1e-3f * tan_a;
    // rectangles; mean extent of the ordinary candidate ones (not whole-plane or oversized)
    float4 ext = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (int e = tid; e < n; e += kThreads) {
        const Aabb b = J.aabbs[e];
        const BoxSpan span = box_span(S, plane, b.lo, b.hi);
        J.reach_rect[e] = reach_rect(S, tan_a, span);
        const float4 r = cross_rect(S, tan_a, den, span);
        J.rect[e] = r;
        const float wu = __saturatef(r.y) - __saturatef(r.x), wv = __saturatef(r.w) - __saturatef(r.z);
        if (wu < 0.25f && wv < 0.25f) ext = Sum()(ext, make_float4(wu, wv, 1.0f, 0.0f));
    }
    ext = state_reduce<kCluster>(ext, sm.part, &sm.slot, Sum());
    // cells half as wide as the mean rectangle: a rectangle covers about 3 x 3 cells
    int nu = 1, nv = 1;
    if (ext.z > 0.0f) {
        const float mu = fmaxf(ext.x / ext.z, 1.0f / kMaxAxisCells), mv = fmaxf(ext.y / ext.z, 1.0f / kMaxAxisCells);
        nu = min(kMaxAxisCells, max(1, (int)ceilf(1.0f / (mu * kCellScale))));
        nv = min(kMaxAxisCells, max(1, (int)ceilf(1.0f / (mv * kCellScale))));
    }
    while ((long long)nu * nv > (long long)J.cap_cells) {
        nu = max(1, nu * 3 / 4);
        nv = max(1, nv * 3 / 4);
    }
    // shrink until the registered items fit (at 1 x 1 every element holds one item)
    unsigned long long total;
    for (;;) {
        unsigned long long items = 0;
        for (int e = tid; e < n; e += kThreads) {
            int iu0, iu1, iv0, iv1;
            sg_range(J.rect[e], (float)nu, (float)nv, nu, nv, iu0, iu1, iv0, iv1);
            const long long cells = (long long)(iu1 - iu0 + 1) * (iv1 - iv0 + 1);
            if (cells <= kSunGridMaxCells) items += (unsigned long long)cells;
        }
        total = state_reduce<kCluster>(items, upart, &uslot, Sum());
        if (total <= J.cap_items || (nu == 1 && nv == 1)) break;
        nu = max(1, nu * 3 / 4);
        nv = max(1, nv * 3 / 4);
    }
    for (int c = tid; c < nu * nv; c += kThreads) J.cells[c] = make_uint2(0u, 0u);
    if (tid == 0) {
        SunGrid d;
        d.nu = nu;
        d.nv = nv;
        d.n_global = 0;
        d.n = n;
        d.fnu = (float)nu;
        d.fnv = (float)nv;
        d.n_items = (int)total;
        d.pad = 0;
        d.plane = plane;
        const float l1 = dot(xyz(S.e1), xyz(S.e1)), l2 = dot(xyz(S.e2), xyz(S.e2));
        const bool ok = l1 > 0.0f && l2 > 0.0f;  // else every rectangle is the whole plane
        d.e1 = ok ? make_float4(S.e1.x / l1, S.e1.y / l1, S.e1.z / l1, 0.0f) : make_float4(0.f, 0.f, 0.f, 0.f);
        d.e2 = ok ? make_float4(S.e2.x / l2, S.e2.y / l2, S.e2.z / l2, 0.0f) : make_float4(0.f, 0.f, 0.f, 0.f);
        d.cells = J.cells;
        d.item_rect = J.item_rect;
        d.item_box = J.item_box;
        d.global_id = J.global_id;
        d.rect = J.rect;
        d.reach = J.reach;
        d.aabbs = J.aabbs;
        *J.desc = d;
    }
    if constexpr (kCluster > 1) cooperative_groups::this_cluster().sync();  // the slots are read
}

// Cells of element e's candidate rectangle, k-th of `cells`.
struct ElemCells {
    int iu0, iv0, w, nu;
    long long cells;
    __device__ ElemCells(float4 r, int nu, int nv) : nu(nu) {
        int iu1, iv1;
        sg_range(r, (float)nu, (float)nv, nu, nv, iu0, iu1, iv0, iv1);
        w = iu1 - iu0 + 1;
        cells = (long long)w * (iv1 - iv0 + 1);
    }
    __device__ int at(int k) const { return (iv0 + k / w) * nu + iu0 + k % w; }
};

// Field-grid cells of element e's registered box (every element but the last has one).  The index is
// the walk's own expression, monotonic in the coordinate, so a point of the box lies in one of them.
template <class F>
__device__ __forceinline__ void field_cells_of(const SunGridJob& J, int e, F&& f) {
    if (!J.field_cells || e + 1 >= J.n) return;
    const Aabb p = J.prune[e];
    const float4 b = grid_box(p.lo, p.hi);
    const int ax = field_index(b.x, J.field_x0, J.field_inv, J.field_nx);
    const int bx = field_index(b.z, J.field_x0, J.field_inv, J.field_nx);
    const int ay = field_index(b.y, J.field_y0, J.field_inv, J.field_ny);
    const int by = field_index(b.w, J.field_y0, J.field_inv, J.field_ny);
    for (int y = ay; y <= by; ++y)
        for (int x = ax; x <= bx; ++x) f(J.field_cells + y * J.field_nx + x);
}

__global__ void __launch_bounds__(kElemBlock) sungrid_count_kernel(const SunGridJob* __restrict__ jobs) {
    const SunGridJob& J = jobs[blockIdx.y];
    if (blockIdx.z == 1) {
        field_cells_of(J, (int)(blockIdx.x * kElemBlock + threadIdx.x), [](uint2* c) { atomicAdd(&c->y, 1u); });
        return;
    }
    const int e = (int)(blockIdx.x * kElemBlock + threadIdx.x) / kElemLanes;
    const int lane = threadIdx.x & (kElemLanes - 1);
    if (e >= J.n) return;
    set_reach(J.reach, J.reach_rect[e], lane, kElemLanes);
    const ElemCells E(J.rect[e], J.desc->nu, J.desc->nv);
    if (E.cells > kSunGridMaxCells) {
        if (lane == 0) {
            const int k = atomicAdd(&J.desc->n_global, 1);
            if (CSP_BOUNDS(6, k < J.n)) J.global_id[k] = (uint32_t)e;
        }
        return;
    }
    for (int k = lane; k < (int)E.cells; k += kElemLanes)
        if (CSP_BOUNDS(6, E.at(k) < J.cap_cells)) atomicAdd(&J.cells[E.at(k)].y, 1u);
}

__global__ void __launch_bounds__(kElemBlock) sungrid_ranges_kernel(const SunGridJob* __restrict__ jobs) {
    const SunGridJob& J = jobs[blockIdx.y];
    const bool field = blockIdx.z == 1;
    if (field && !J.field_cells) return;
    uint2* const cells = field ? J.field_cells : J.cells;
    uint32_t* const alloc = field ? J.field_alloc : J.alloc;
    const int nc = field ? J.field_nx * J.field_ny : J.desc->nu * J.desc->nv;
    const int c = 4 * (int)(blockIdx.x * kElemBlock + threadIdx.x), lane = threadIdx.x & 31;
    if (c - 4 * lane >= nc) return;  // whole warps
    uint32_t k[4], sum = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        k[i] = c + i < nc ? cells[c + i].y : 0u;
        sum += k[i];
    }
    uint32_t incl = sum;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    uint32_t base = 0;
    if (lane == 31 && incl) base = atomicAdd(alloc, incl);
    base = __shfl_sync(0xffffffffu, base, 31) + incl - sum;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if (c + i < nc) cells[c + i] = make_uint2(base, base);
        base += k[i];
    }
}

__global__ void __launch_bounds__(kElemBlock) sungrid_fill_kernel(const SunGridJob* __restrict__ jobs) {
    const SunGridJob& J = jobs[blockIdx.y];
    if (blockIdx.z == 1) {
        const int e = (int)(blockIdx.x * kElemBlock + threadIdx.x);
        field_cells_of(J, e, [&](uint2* c) {
            const uint32_t at = atomicAdd(&c->y, 1u);
            if (CSP_BOUNDS(6, at < J.field_cap)) J.field_items[at] = J.aabbs[e];
        });
        return;
    }
    const int e = (int)(blockIdx.x * kElemBlock + threadIdx.x) / kElemLanes;
    if (e >= J.n) return;
    const float4 r = J.rect[e];
    const ElemCells E(r, J.desc->nu, J.desc->nv);
    if (E.cells > kSunGridMaxCells) return;
    const Aabb b = J.aabbs[e];
    for (int k = threadIdx.x & (kElemLanes - 1); k < (int)E.cells; k += kElemLanes) {
        if (!CSP_BOUNDS(6, E.at(k) < J.cap_cells)) continue;
        const uint32_t at = atomicAdd(&J.cells[E.at(k)].y, 1u);
        if (!CSP_BOUNDS(6, at < J.cap_items)) continue;
        J.item_rect[at] = r;
        J.item_box[at] = b;
    }
}

}  // namespace

uint32_t bounds_sites_sungrid() { return take_bounds_sites(); }

SunGridCaps sungrid_caps(uint32_t n) {
    SunGridCaps c;
    c.cap_cells = (int)std::min<uint64_t>(262144, std::max<uint64_t>(64, 8ull * n));
    c.cap_items = (uint32_t)std::min<uint64_t>(0xFFFFFFF0u, (uint64_t)kSunGridItemsPerElem * n + 64);
    return c;
}

size_t sungrid_bytes(uint32_t n, bool raster) {
    const SunGridCaps c = sungrid_caps(n);
    return a256(sizeof(SunGrid) + sizeof(uint32_t)) + a256((size_t)c.cap_cells * sizeof(uint2)) +
           a256((size_t)n * sizeof(float4)) + (raster ? kReachBytes : 0) + a256((size_t)c.cap_items * sizeof(float4)) +
           a256((size_t)c.cap_items * sizeof(Aabb)) + a256((size_t)std::max<uint32_t>(n, 1) * sizeof(uint32_t));
}

void sungrid_place(unsigned char* base, uint32_t n, SunGridJob& job, unsigned char* raster) {
    const SunGridCaps c = sungrid_caps(n);
    size_t o = 0;
    auto take = [&](size_t bytes) {
        unsigned char* p = base + o;
        o += a256(bytes);
        return p;
    };
    job.desc = reinterpret_cast<SunGrid*>(take(sizeof(SunGrid) + sizeof(uint32_t)));
    job.alloc = reinterpret_cast<uint32_t*>(job.desc + 1);
    job.cells = reinterpret_cast<uint2*>(take((size_t)c.cap_cells * sizeof(uint2)));
    job.rect = reinterpret_cast<float4*>(take((size_t)n * sizeof(float4)));
    job.reach = reinterpret_cast<uint32_t*>(raster ? raster : take(kReachBytes));
    job.item_rect = reinterpret_cast<float4*>(take((size_t)c.cap_items * sizeof(float4)));
    job.reach_rect = job.item_rect;  // read by the count pass, before the fill pass writes items (n <= cap_items)
    job.item_box = reinterpret_cast<Aabb*>(take((size_t)c.cap_items * sizeof(Aabb)));
    job.global_id = reinterpret_cast<uint32_t*>(take((size_t)std::max<uint32_t>(n, 1) * sizeof(uint32_t)));
    job.prune = nullptr;
    job.field_cells = nullptr;
    job.field_alloc = nullptr;
    job.field_items = nullptr;
    job.field_x0 = job.field_y0 = job.field_inv = 0.0f;
    job.field_nx = job.field_ny = 0;
    job.field_cap = 0;
    job.n = (int)n;
    job.cap_cells = c.cap_cells;
    job.cap_items = c.cap_items;
    job.pad = 0;
}

size_t field_bytes(int nx, int ny, uint32_t cap) {
    return a256((size_t)nx * ny * sizeof(uint2)) + a256(sizeof(uint32_t)) + a256((size_t)cap * sizeof(Aabb));
}

void field_place(unsigned char* base, const HostGrid& g, const Aabb* prune, SunGridJob& job) {
    job.prune = prune;
    job.field_cells = reinterpret_cast<uint2*>(base);
    base += a256((size_t)g.nx * g.ny * sizeof(uint2));
    job.field_alloc = reinterpret_cast<uint32_t*>(base);
    base += a256(sizeof(uint32_t));
    job.field_items = reinterpret_cast<Aabb*>(base);
    job.field_x0 = g.x0;
    job.field_y0 = g.y0;
    job.field_inv = g.inv_cell;
    job.field_nx = g.nx;
    job.field_ny = g.ny;
    job.field_cap = g.cap_items;
}

cudaError_t launch_sungrid_build(const SunGridJob* jobs, int n_jobs, int max_n, int max_field_cells,
                                 cudaStream_t stream) {
    if (n_jobs <= 0 || max_n <= 0) return cudaSuccess;
    const unsigned elem_blocks = (unsigned)(((uint64_t)max_n * kElemLanes + kElemBlock - 1) / kElemBlock);
    const int max_cells = std::max(sungrid_caps((uint32_t)max_n).cap_cells, max_field_cells);
    const unsigned cell_blocks = (unsigned)((max_cells / 4 + kElemBlock) / kElemBlock);
    const unsigned parts = max_field_cells > 0 ? 2u : 1u;  // blockIdx.z: the sun grids, the field grids
    for (int j0 = 0; j0 < n_jobs; j0 += kMaxJobsPerLaunch) {
        const unsigned nj = (unsigned)std::min(kMaxJobsPerLaunch, n_jobs - j0);
        const SunGridJob* J = jobs + j0;
        // A block does for few elements and field cells to zero: a cluster for each of 64 states of 101
        // elements is 512 CTAs in two waves, 25.6 us against 9 (one state alone 4.5 against 5).
        if (max_n >= kStateClusterMin || max_field_cells >= kWideField)
            sungrid_size_kernel<kStateCluster><<<nj * kStateCluster, kStateBlock, 0, stream>>>(J);
        else
            sungrid_size_kernel<1><<<nj, kStateBlock, 0, stream>>>(J);
        sungrid_count_kernel<<<dim3(elem_blocks, nj, parts), kElemBlock, 0, stream>>>(J);
        sungrid_ranges_kernel<<<dim3(cell_blocks, nj, parts), kElemBlock, 0, stream>>>(J);
        sungrid_fill_kernel<<<dim3(elem_blocks, nj, parts), kElemBlock, 0, stream>>>(J);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace csp
