// k_grid.cu -- spatial hashing: bounding box, cell keys, stable counting sort
// of the particles by key, cell ranges, surface cells and the surface list.
//
// Reference: NeighborSearch_kernel.cuh:129-186 (calculateHash, calCellRange),
// Thrust.cuh:40-50 (thrust::sort_by_key, a stable radix sort of the 44-byte
// particle AoS), Anisotropic_kernel.cuh:15-155 (estimationOfSurfaceParticles,
// compactationOfParticles), FileData.cpp:240-257 (bounding box on the host).
//
// GB300 design: keys are cell indices < sp_size, so the stable sort is a
// counting sort -- one atomic histogram (which doubles as the cell-count
// array), one scan (which doubles as the cell-start array), one scatter, and a
// placement that restores the input order inside each cell (the order a stable
// sort produces) and writes the payload once into SoA float4 arrays that the
// neighbour loops read with one 16-byte load per particle.
#include "pms_internal.h"
#include "k_common.cuh"

namespace pms {

static constexpr int kThreads = 256;
static constexpr uint32_t kBigCell = 4096;     // most particles a cell may hold

// ---------------------------------------------------------------------------
// bounding box (FileData.cpp:240-257); non-finite positions are flagged
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads) k_bbox(const float* __restrict__ pos, uint32_t n, Counters* __restrict__ cnt,
                                                   uint32_t* __restrict__ mirror) {
    uint32_t mn[3] = {0xffffffffu, 0xffffffffu, 0xffffffffu}, mx[3] = {0u, 0u, 0u};
    bool bad = false;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            float v = pos[3 * (size_t)i + k];
            bad |= !isfinite(v);
            uint32_t o = ordered_bits(v);
            mn[k] = min(mn[k], o);
            mx[k] = max(mx[k], o);
        }
    }
    // one set of atomics per block: a warp's own would queue up on the six words (2M
    // particles: 42 us with 58k atomics, the reads take 6)
    __shared__ uint32_t s_mn[kThreads / 32][3], s_mx[kThreads / 32][3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        mn[k] = __reduce_min_sync(0xffffffffu, mn[k]);
        mx[k] = __reduce_max_sync(0xffffffffu, mx[k]);
        if ((threadIdx.x & 31) == 0) { s_mn[threadIdx.x >> 5][k] = mn[k]; s_mx[threadIdx.x >> 5][k] = mx[k]; }
    }
    const bool any_bad = __syncthreads_or(bad);
    if (threadIdx.x < 3) {
        const int k = threadIdx.x;
        uint32_t lo = s_mn[0][k], hi = s_mx[0][k];
#pragma unroll
        for (int w = 1; w < kThreads / 32; ++w) { lo = min(lo, s_mn[w][k]); hi = max(hi, s_mx[w][k]); }
        atomicMin(&cnt->bbox_min[k], lo);
        atomicMax(&cnt->bbox_max[k], hi);
    }
    if (any_bad && threadIdx.x == 0) atomicOr(&cnt->err, kErrNonFinite);
    if (!mirror) return;
    // the last block publishes: every block's atomics come before its own count
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(&cnt->bbox_blocks, 1u) == gridDim.x - 1u;
    __syncthreads();
    if (!last) return;
    __threadfence();
    publish_counters(cnt, mirror);
}

__global__ void k_counters_init(Counters* cnt, uint32_t n, uint32_t nv, uint32_t nvalid, unsigned long long nmesh) {
    Counters c;
    memset(&c, 0, sizeof(c));
    c.n = n;
    c.nv = nv;
    c.nvalid = nvalid;
    c.nmesh = nmesh;
    for (int k = 0; k < 3; ++k) { c.bbox_min[k] = 0xffffffffu; c.bbox_max[k] = 0u; }
    *cnt = c;
}

// The counters into the context's mapped pinned mirror, stored by a kernel: a
// copy-engine transfer would queue behind a streamed mesh or diffuse copy.
__global__ void k_publish_counters(const uint32_t* __restrict__ src, uint32_t* __restrict__ dst, uint32_t words) {
    for (uint32_t i = threadIdx.x; i < words; i += blockDim.x) dst[i] = src[i];
}

pms_status launch_publish_counters(pms_ctx* ctx) {
    static_assert(sizeof(Counters) % 4 == 0, "counters are copied in 32-bit words");
    k_publish_counters<<<1, 128, 0, ctx->stream>>>(ctx->counters.as<uint32_t>(), ctx->h_counters_dev,
                                                   (uint32_t)(sizeof(Counters) / 4));
    PMS_LAUNCHED(ctx);
    return PMS_OK;
}

pms_status launch_bbox(pms_ctx* ctx, bool publish) {
    Counters* cnt = ctx->counters.as<Counters>();
    // (a grid built again on the same upload: the band and the mesh made before it stay, and what is
    // made from them on demand reads their sizes here)
    const bool kept = publish && ctx->have_mc;
    k_counters_init<<<1, 1, 0, ctx->stream>>>(cnt, ctx->n, kept ? ctx->nv : 0u, kept ? ctx->nvalid : 0u, kept ? ctx->nmesh : 0ull);
    PMS_LAUNCHED(ctx);
    k_bbox<<<grid_for(ctx->n, kThreads, 152 * 4), kThreads, 0, ctx->stream>>>(ctx->in_pos.as<float>(), ctx->n, cnt,
                                                                           publish ? ctx->h_counters_dev : nullptr);
    PMS_LAUNCHED(ctx);
    return PMS_OK;
}

// ---------------------------------------------------------------------------
// keys + histogram (calculateHash, NeighborSearch_kernel.cuh:129-152)
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads) k_hash_count(KGrid g, const float* __restrict__ pos, uint32_t n,
                                                         uint32_t* __restrict__ keys, uint32_t* __restrict__ slot,
                                                         uint32_t* __restrict__ cell_count, Counters* __restrict__ cnt) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        uint3 c = sp_cell(g, pos[3 * (size_t)i], pos[3 * (size_t)i + 1], pos[3 * (size_t)i + 2]);
        uint32_t key = lin3(c.x, c.y, c.z, g.spres);
        if (key >= g.sp_size) { atomicOr(&cnt->err, kErrKeyRange); key = g.sp_size - 1; }
        keys[i] = key;
        slot[i] = atomicAdd(&cell_count[key], 1u);
    }
}

__global__ void __launch_bounds__(kThreads) k_scatter(const uint32_t* __restrict__ keys, const uint32_t* __restrict__ slot,
                                                      const uint32_t* __restrict__ cell_start, uint32_t n,
                                                      uint32_t* __restrict__ order) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        order[cell_start[keys[i]] + slot[i]] = i;
}

// Up to three arrays zeroed in one launch (a frame of a few thousand particles pays the
// launches, not the bytes).
struct ZeroList {
    uint32_t* p[3];
    uint64_t n[3];
};
__global__ void __launch_bounds__(kThreads) k_zero(ZeroList z) {
    const uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x, step = (uint64_t)gridDim.x * blockDim.x;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        // whole 16-byte words, then the rest (the arrays are allocations of their own)
        uint4* q = reinterpret_cast<uint4*>(z.p[k]);
        for (uint64_t i = t; i < z.n[k] / 4; i += step) q[i] = make_uint4(0u, 0u, 0u, 0u);
        for (uint64_t i = z.n[k] / 4 * 4 + t; i < z.n[k]; i += step) z.p[k][i] = 0u;
    }
}

// Ascending input order inside every cell, what a stable sort by key yields, and the payload
// in that order: each particle finds its place by counting the smaller indices among its
// cell's entries (neighbouring threads read the same few).  Of a cell past kBigCell the order
// is left as scattered: the frame fails.  (A thread per cell sorting its entries in place, a
// block-wide sort of large cells and a gather took 35 + 2 + 35 us on 2M particles and
// 13 + 2 + 4 us on 4k, where the serial sort of a cell is the latency; this takes 39 and 5.)
__global__ void __launch_bounds__(kThreads) k_place(const uint32_t* __restrict__ scattered, const uint32_t* __restrict__ keys,
                                                    const uint32_t* __restrict__ cell_start, const float* __restrict__ pos,
                                                    const float* __restrict__ vel, uint32_t n, uint32_t* __restrict__ order,
                                                    uint32_t* __restrict__ skeys, float4* __restrict__ spos,
                                                    float4* __restrict__ svel, Counters* __restrict__ cnt) {
    for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x) {
        const uint32_t i = __ldg(&scattered[s]), key = __ldg(&keys[i]);
        const uint32_t st = __ldg(&cell_start[key]), m = __ldg(&cell_start[key + 1u]) - st;
        uint32_t dest = s;
        if (m <= kBigCell) {
            dest = st;
#pragma unroll 4
            for (uint32_t t = 0; t < m; ++t) dest += __ldg(&scattered[st + t]) < i ? 1u : 0u;
        } else if (s == st) {
            atomicOr(&cnt->err, kErrBigCell);
        }
        order[dest] = i;
        skeys[dest] = key;
        spos[dest] = make_float4(pos[3 * (size_t)i], pos[3 * (size_t)i + 1], pos[3 * (size_t)i + 2], 0.f);
        svel[dest] = make_float4(vel[3 * (size_t)i], vel[3 * (size_t)i + 1], vel[3 * (size_t)i + 2], 0.f);
    }
}

pms_status launch_hash_sort(pms_ctx* ctx) {
    const uint32_t n = ctx->n;
    const KGrid g = kgrid_of(ctx->grid);
    Counters* cnt = ctx->counters.as<Counters>();
    // the cell counts, the support radii the anisotropy pass raises, the band's marks: all start
    // at 0, and a stage run again on the same frame sets the same values
    const ZeroList z = {{ctx->cell_count.as<uint32_t>(), ctx->cell_rad.as<uint32_t>(), ctx->bm0.as<uint32_t>()},
                        {g.sp_size, g.sp_size + (uint64_t)g.spres[1] * g.spres[2] * (1 + rad_segments(g.spres[0])),
                         ((uint64_t)g.sc_size + 31) / 32}};
    k_zero<<<grid_for((z.n[0] + z.n[1] + z.n[2]) / 16 + 1, kThreads, 152 * 8), kThreads, 0, ctx->stream>>>(z);
    PMS_LAUNCHED(ctx);
    const unsigned gb = grid_for(n, kThreads);
    k_hash_count<<<gb, kThreads, 0, ctx->stream>>>(g, ctx->in_pos.as<float>(), n, ctx->keys.as<uint32_t>(),
                                                   ctx->slot.as<uint32_t>(), ctx->cell_count.as<uint32_t>(), cnt);
    PMS_LAUNCHED(ctx);
    // cell_start[c + 1] - cell_start[c] is cell c's count for every c, and cell_start[sp_size] = n,
    // so the cells of a row segment form one contiguous particle range
    pms_status st = scan_u32(ctx, ctx->cell_count.as<uint32_t>(), ctx->cell_start.as<uint32_t>(), g.sp_size,
                             ctx->cell_start.as<uint32_t>() + g.sp_size);
    if (st != PMS_OK) return st;
    // (the surface list's buffer holds the scattered indices until the surface pass)
    k_scatter<<<gb, kThreads, 0, ctx->stream>>>(ctx->keys.as<uint32_t>(), ctx->slot.as<uint32_t>(),
                                                ctx->cell_start.as<uint32_t>(), n, ctx->slist.as<uint32_t>());
    PMS_LAUNCHED(ctx);
    if (ctx->vel_pending) {
        PMS_CUDA(ctx, cudaStreamWaitEvent(ctx->stream, ctx->vel_ready, 0));   // the uploaded velocities
        ctx->vel_pending = false;
    }
    k_place<<<gb, kThreads, 0, ctx->stream>>>(ctx->slist.as<uint32_t>(), ctx->keys.as<uint32_t>(), ctx->cell_start.as<uint32_t>(),
                                              ctx->in_pos.as<float>(), ctx->in_vel.as<float>(), n, ctx->order.as<uint32_t>(),
                                              ctx->skeys.as<uint32_t>(), ctx->spos.as<float4>(), ctx->svel.as<float4>(),
                                              cnt);
    PMS_LAUNCHED(ctx);
    return PMS_OK;
}

// ---------------------------------------------------------------------------
// surface cells (estimationOfSurfaceParticles, Anisotropic_kernel.cuh:15-106):
// a non-empty cell with an empty cell in its clamped 3x3x3 neighbourhood.
// Writes numSurParticleGrid (surf_count) and the packed cell record
// cell_info = {start, count | surface << 31} read by the neighbour loops.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads) k_surface_cells(KGrid g, const uint32_t* __restrict__ cell_count,
                                                            const uint32_t* __restrict__ cell_start,
                                                            uint32_t* __restrict__ surf_count, uint2* __restrict__ cell_info) {
    const uint32_t rx = g.spres[0], ry = g.spres[1], rz = g.spres[2], rxy = rx * ry;
    for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < g.sp_size; c += gridDim.x * blockDim.x) {
        uint32_t m = cell_count[c];
        uint32_t s = cell_start[c];
        if (m == 0) { surf_count[c] = 0; cell_info[c] = make_uint2(s, 0u); continue; }
        uint32_t z = c / rxy, r = c - z * rxy, y = r / rx, x = r - y * rx;
        uint32_t lx = min(max(x - 1u, 0u), rx - 1u), hx = min(x + 1u, rx - 1u);
        uint32_t ly = min(max(y - 1u, 0u), ry - 1u), hy = min(y + 1u, ry - 1u);
        uint32_t lz = min(max(z - 1u, 0u), rz - 1u), hz = min(z + 1u, rz - 1u);
        bool surface = false;
        for (uint32_t cz = lz; cz <= hz && !surface; ++cz)
            for (uint32_t cy = ly; cy <= hy && !surface; ++cy)
                for (uint32_t cx = lx; cx <= hx; ++cx)
                    if (cell_count[cz * rxy + cy * rx + cx] == 0) { surface = true; break; }
        surf_count[c] = surface ? m : 0u;
        cell_info[c] = make_uint2(s, m | (surface ? 0x80000000u : 0u));
    }
}

pms_status launch_surface_cells(pms_ctx* ctx) {
    const KGrid g = kgrid_of(ctx->grid);
    Counters* cnt = ctx->counters.as<Counters>();
    k_surface_cells<<<grid_for(g.sp_size, kThreads), kThreads, 0, ctx->stream>>>(
        g, ctx->cell_count.as<uint32_t>(), ctx->cell_start.as<uint32_t>(), ctx->surf_count.as<uint32_t>(),
        ctx->cell_info.as<uint2>());
    PMS_LAUNCHED(ctx);
    pms_status st = scan_u32(ctx, ctx->surf_count.as<uint32_t>(), ctx->surf_start.as<uint32_t>(), g.sp_size, &cnt->ns);
    ctx->surf_current = st == PMS_OK;
    return st;
}

}  // namespace pms
