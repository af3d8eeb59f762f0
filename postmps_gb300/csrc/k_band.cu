// k_band.cu -- outer narrow band of scalar-grid vertices.
//
// Reference: Anisotropic_kernel.cuh:522-636 (estimationOfSurfaceVertices with
// LOWRES on, USING_GRID off) marks, for every surface particle, each scalar
// vertex v of the box idx +- ceil(h / cell) that lies inside the AABB p +- h
// and satisfies (flag || n . (v - p) > 0), plus the vertices one step along
// +x, +y and +z of it (the LOWRES dilation).  Marks go into a dense uint per
// vertex; thrust then scans all S_sc flags and compactationOfSurfaceVertices
// (Anisotropic_kernel.cuh:639-653) gathers the ascending vertex list.
//
// GB300 design: marks are bits, made tile by tile.  Neighbouring surface
// particles' boxes overlap heavily (each band vertex is marked by ~90 of them
// on a 2M-particle crown), so marking straight into the global bitmap costs a
// global atomic per particle and box row.  Instead a warp owns a tile of
// 32 x 4 x 8 vertices, a lane per tile row (its 32 marks one register), and runs
// over the surface particles around the tile, staged in shared memory with what a
// row needs of them; each tile row then lands in the global bitmap with at most two
// atomics.  The dilation is a pass over the bitmap:
// B = B0 | B0<<1 | B0<<rx | B0<<(rx*ry) in linear bit order (the reference's
// index arithmetic, including its row wrap), which also counts the band.  The bitmap
// (S_sc / 8 bytes) replaces three dense S_sc-sized uint arrays; a list of the band (a
// popcount per 32-bit word, one scan over words and a per-word bit extraction) is made
// only for downloads.
#include <algorithm>

#include "pms_internal.h"
#include "k_common.cuh"

namespace pms {

// Tiles of the scalar grid: 32 vertices along x (one bitmap word) by 4 by 8, a row per lane.
static constexpr int kTileX = 32, kTileY = 4, kTileZ = 8;

struct TileDims {
    uint32_t n[3];            // tiles per axis
};

// The clamped box [lo, hi] of scalar vertices a surface particle tests
// (estimationOfSurfaceVertices: idx +- ceil(h / cell), clamped to the grid).
__device__ __forceinline__ void particle_box(const KGrid& g, int ext, const float p[3], int lo[3], int hi[3]) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int res = (int)g.scres[k];
        const int c = __float2int_rz(__fdiv_rn(__fsub_rn(p[k], g.scmin_pos[k]), g.sc_cs));
        lo[k] = min(max(c - ext, 0), res - 1);
        hi[k] = min(max(c + ext, 0), res - 1);
    }
}

// Spatial cells of the particles whose AABB p +- h can hold a vertex of the tile [t0, t1]:
// range_margin cells, and four units in the last place of the largest coordinate, cover the
// rounding of cell keys, vertex coordinates and p +- h.
struct TileCells {
    int lo[3], hi[3];
};
__device__ __forceinline__ TileCells tile_cells(const KGrid& g, float h, float inv_sp, const int t0[3], const int t1[3]) {
    TileCells c;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float slack = (fabsf(g.min_pos[k]) + (float)g.spres[k] * g.sp_cs) * 0x1p-21f + g.margin * g.sp_cs;
        const float a = sc_coord_i(g, t0[k], k) - h - slack - g.min_pos[k], b = sc_coord_i(g, t1[k], k) + h + slack - g.min_pos[k];
        c.lo[k] = max((int)floorf(a * inv_sp), 0);
        c.hi[k] = min((int)floorf(b * inv_sp), (int)g.spres[k] - 1);
    }
    return c;
}
__device__ __forceinline__ void tile_bounds(const KGrid& g, const TileDims& td, uint32_t t, int t0[3], int t1[3]) {
    const uint32_t tx = t % td.n[0], tyz = t / td.n[0], ty = tyz % td.n[1], tz = tyz / td.n[1];
    t0[0] = (int)tx * kTileX; t0[1] = (int)ty * kTileY; t0[2] = (int)tz * kTileZ;
    t1[0] = min(t0[0] + kTileX, (int)g.scres[0]) - 1;
    t1[1] = min(t0[1] + kTileY, (int)g.scres[1]) - 1;
    t1[2] = min(t0[2] + kTileZ, (int)g.scres[2]) - 1;
}
// a row's surface particles over the cells [c0, c1]: first entry of the surface list, and how
// many (the list is in cell order, surf_start the exclusive scan of the cells' counts)
__device__ __forceinline__ uint32_t row_surface(const uint32_t* __restrict__ surf_start, const uint32_t* __restrict__ surf_count,
                                                uint32_t c0, uint32_t c1, uint32_t& first) {
    first = __ldg(&surf_start[c0]);
    return __ldg(&surf_start[c1]) + __ldg(&surf_count[c1]) - first;
}

// One warp per tile (or per share of a tile's particles, where the grid has fewer tiles than
// the GPU holds warps: marks are an OR, so shares meet in the bitmap).  Lanes read 32 surface particles at a time, work out which of
// the tile's x positions and rows each one's box and AABB p +- h hold (one mask each), and
// stage those that hold any.  Then every lane ORs into its row what each staged particle
// marks: all x of the AABB for a flagged particle, else the side n . (v - p) > 0,
// evaluated as estimationOfSurfaceVertices does (Anisotropic_kernel.cuh:551-606): vertex
// coordinates i * cell + min, each difference, product and sum rounded on its own.  Every one
// of those operations is monotone in the vertex's x, so a row's side is all x from (or up
// to) some position: the position is guessed from the plane and corrected with the exact
// test, about two tests instead of one per x.  A particle that would mark only
// vertices marked already (each is marked by dozens) is skipped.
//
// Bound by instruction issue (2.4 of 4 a cycle, dependent integer work).  A block of 256
// threads per 32 x 8 x 8 tile (particles of a chunk split over four threads per row,
// block-wide barriers around each chunk, a test per x) took 0.54 / 0.38 / 0.45 ms on the crown
// 2M / dam 8M / spray 151k (ratio 3) frames, and listing its tiles by one atomic per particle
// and tile another 0.06 / 0.05 / 0.06; this takes 0.23 / 0.25 / 0.23, list included (an empty
// tile costs its rows' bounds).  Cells cut to the AABB's reach instead of a cell more on each
// side: 0.37 -> 0.24 ms on the crown.  A 4k-particle frame: 16 + 22 -> 10 us with shares.
// Particles whose plane leaves their whole part of the tile on one side, settled before the rows
// look at them: spray 0.23 -> 0.20, dam 0.25 -> 0.23, crown and blocks unchanged.
static constexpr int kBandThreads = 128, kBandStage = 64;

__global__ void __launch_bounds__(kBandThreads, 8) k_band_tiles(KGrid g, float h, int ext, TileDims td,
                                                                uint32_t n_tiles, uint32_t shares, Counters* __restrict__ cnt,
                                                                const uint32_t* __restrict__ surf_start,
                                                                const uint32_t* __restrict__ surf_count,
                                                                const uint32_t* __restrict__ slist,
                                                                const float4* __restrict__ spos, const float4* __restrict__ nrm4,
                                                                uint32_t* __restrict__ bm0) {
    constexpr unsigned kAll = 0xffffffffu;
    if (blockIdx.x == 0 && threadIdx.x == 0) cnt->nv = 0u;     // the dilation counts the band
    __shared__ float4 s_p[kBandThreads / 32][kBandStage];      // p, n.x
    __shared__ float4 s_n[kBandThreads / 32][kBandStage];      // n.y, n.z, flag
    __shared__ uint2 s_m[kBandThreads / 32][kBandStage];       // x positions, tile rows inside box and AABB
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t srx = g.spres[0], sry = g.spres[1], n_work = n_tiles * shares;
    const uint64_t rxy = (uint64_t)g.scres[0] * g.scres[1];
    const float inv_cs = 1.f / g.sc_cs, inv_sp = 1.f / g.sp_cs;
    const int my_y = (int)(lane & 3u), my_z = (int)(lane >> 2);
    const uint32_t ticket = min(max(n_work / (gridDim.x * (kBandThreads / 32u) * 8u), 1u), 4u);
    uint32_t ti = 0u, ti_end = 0u;
    for (;;) {
        if (ti == ti_end) {
            if (lane == 0u) ti = atomicAdd(&cnt->band_next, ticket);
            ti = __shfl_sync(kAll, ti, 0);
            if (ti >= n_work) break;
            ti_end = min(ti + ticket, n_work);
        }
        const uint32_t share = ti % shares;
        int t0[3], t1[3];
        tile_bounds(g, td, ti / shares, t0, t1);
        ++ti;
        const float vy = sc_coord_i(g, t0[1] + my_y, 1), vz = sc_coord_i(g, t0[2] + my_z, 2);
        const TileCells c = tile_cells(g, h, inv_sp, t0, t1);
        const int ny = c.hi[1] - c.lo[1] + 1, nz = c.hi[2] - c.lo[2] + 1;
        const int nrow = ny > 0 && nz > 0 && c.lo[0] <= c.hi[0] ? ny * nz : 0;
        uint32_t acc = 0u;
        int staged = 0;

        auto flush = [&]() {
            __syncwarp();
            for (int i = 0; i < staged; ++i) {
                const uint2 m = s_m[warp][i];
                const uint32_t need = (m.y >> lane) & 1u ? m.x & ~acc : 0u;
                if (!__any_sync(kAll, need != 0u)) continue;
                const float4 p = s_p[warp][i], n = s_n[warp][i];
                if (n.z != 0.f) {                              // flag: the whole AABB part
                    acc |= (m.y >> lane) & 1u ? m.x : 0u;
                } else if (need) {
                    const float by = __fmul_rn(n.x, __fsub_rn(vy, p.y));
                    const float cz = __fmul_rn(n.y, __fsub_rn(vz, p.z));
                    auto out = [&](int x) {
                        const float vx = sc_coord_i(g, t0[0] + x, 0);
                        return __fadd_rn(__fadd_rn(__fmul_rn(p.w, __fsub_rn(vx, p.x)), by), cz) > 0.f;
                    };
                    const int lo = __ffs((int)m.x) - 1, hi = 31 - __clz((int)m.x);   // the x positions are one run
                    const int guess = __float2int_rd((p.x - __fdividef(by + cz, p.w) - g.scmin_pos[0]) * inv_cs) - t0[0];
                    if (p.w >= 0.f) {                          // out from some x on
                        int x = min(max(guess, lo - 1), hi) + 1;
                        while (x > lo && out(x - 1)) --x;
                        while (x <= hi && !out(x)) ++x;
                        acc |= x < 32 ? m.x & (kAll << x) : 0u;
                    } else {                                   // out up to some x
                        int x = min(max(guess, lo - 1), hi);
                        while (x < hi && out(x + 1)) ++x;
                        while (x >= lo && !out(x)) --x;
                        acc |= x >= 0 ? m.x & (kAll >> (31 - x)) : 0u;
                    }
                }
            }
            __syncwarp();
            staged = 0;
        };

        for (int r0 = 0; r0 < nrow; r0 += 32) {
            // a row of cells per lane: its stretch of the surface list
            const int r = r0 + (int)lane;
            uint32_t first = 0u, len = 0u;
            if (r < nrow) {
                const uint32_t row = ((uint32_t)(c.lo[2] + r / ny) * sry + (uint32_t)(c.lo[1] + r % ny)) * srx;
                len = row_surface(surf_start, surf_count, row + (uint32_t)c.lo[0], row + (uint32_t)c.hi[0], first);
            }
            uint32_t incl = len;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t v = __shfl_up_sync(kAll, incl, o);
                if (lane >= (uint32_t)o) incl += v;
            }
            const uint32_t total = __shfl_sync(kAll, incl, 31);
            const uint32_t off = first - (incl - len);
            for (uint32_t q0 = 32u * share; q0 < total; q0 += 32u * shares) {
                const uint32_t q = q0 + lane;
                int row = 0;                                   // the first row whose inclusive count exceeds q
#pragma unroll
                for (int s = 16; s > 0; s >>= 1)
                    if (__shfl_sync(kAll, incl, row + s - 1) <= q) row += s;
                const uint32_t s = __shfl_sync(kAll, off, row) + q;
                uint32_t xin = 0u, rows = 0u;
                float4 p4, n4;
                if (q < total) {
                    const uint32_t j = __ldg(&slist[s]);
                    p4 = __ldg(&spos[j]);
                    n4 = __ldg(&nrm4[j]);
                    const float p[3] = {p4.x, p4.y, p4.z};
                    int blo[3], bhi[3];
                    particle_box(g, ext, p, blo, bhi);
                    uint32_t in[3];
                    const float n[3] = {n4.x, n4.y, n4.z};
                    float near = 0.f, far = 0.f, size = 0.f;   // bounds of n . (v - p) over those vertices
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        // vertices i of [box and tile] with a <= v(i) <= b: v rises with i, so they are
                        // one run; its ends are guessed and corrected with the exact comparison
                        const float a = __fsub_rn(p[k], h), b = __fadd_rn(p[k], h);
                        const int b0 = max(blo[k], t0[k]), b1 = min(bhi[k], t1[k]);
                        int i0 = min(max(__float2int_ru((a - g.scmin_pos[k]) * inv_cs), b0), b1 + 1);
                        int i1 = min(max(__float2int_rd((b - g.scmin_pos[k]) * inv_cs), b0 - 1), b1);
                        while (i0 > b0 && !(sc_coord_i(g, i0 - 1, k) < a)) --i0;
                        while (i0 <= b1 && sc_coord_i(g, i0, k) < a) ++i0;
                        while (i1 < b1 && !(sc_coord_i(g, i1 + 1, k) > b)) ++i1;
                        while (i1 >= b0 && sc_coord_i(g, i1, k) > b) --i1;
                        // at most 32 positions of the tile
                        in[k] = i0 <= i1 ? (kAll >> (31 - (i1 - i0))) << (i0 - t0[k]) : 0u;
                        const float d0 = __fmul_rn(n[k], __fsub_rn(sc_coord_i(g, i0, k), p[k]));
                        const float d1 = __fmul_rn(n[k], __fsub_rn(sc_coord_i(g, i1, k), p[k]));
                        near += fminf(d0, d1);
                        far += fmaxf(d0, d1);
                        size += fmaxf(fabsf(d0), fabsf(d1));
                    }
                    // a plane that leaves the whole part of the tile on one side needs no test per
                    // row: all of it is marked, or none.  (Each rounded product of a vertex between the
                    // ends lies between theirs; sums of three in any order differ by less than 1e-6 of
                    // their sizes.)
                    if (n4.w == 0.f) {
                        if (near > 1e-6f * size) n4.w = 1.f;
                        else if (far < -1e-6f * size) in[0] = 0u;
                    }
                    xin = in[0];
                    // row (y, z) of the tile is lane 4 z + y
#pragma unroll
                    for (int z = 0; z < kTileZ; ++z) rows |= ((in[2] >> z) & 1u ? in[1] : 0u) << (kTileY * z);
                }
                const bool keep = xin != 0u && rows != 0u;
                const uint32_t kept = __ballot_sync(kAll, keep);
                if (!kept) continue;
                if (keep) {
                    const int slot = staged + __popc(kept & ((1u << lane) - 1u));
                    s_p[warp][slot] = make_float4(p4.x, p4.y, p4.z, n4.x);
                    s_n[warp][slot] = make_float4(n4.y, n4.z, n4.w, 0.f);
                    s_m[warp][slot] = make_uint2(xin, rows);
                }
                staged += __popc(kept);
                if (staged > kBandStage - 32) flush();
            }
        }
        if (staged) flush();
        if (acc) {
            const uint64_t bit = (uint64_t)(t0[2] + my_z) * rxy + (uint64_t)(t0[1] + my_y) * g.scres[0] + (uint64_t)t0[0];
            const uint64_t w = bit >> 5;
            const uint32_t sh = (uint32_t)(bit & 31u);
            atomicOr(&bm0[w], acc << sh);
            if (sh && (acc >> (32u - sh))) atomicOr(&bm0[w + 1], acc >> (32u - sh));
        }
    }
}

// bits of `b` shifted up by s positions, as seen by word w
__device__ __forceinline__ uint32_t shifted_word(const uint32_t* __restrict__ b, uint64_t w, uint64_t s) {
    const uint64_t q = s >> 5;
    const uint32_t r = (uint32_t)(s & 31u);
    if (w < q) return 0u;
    uint32_t hi = b[w - q];
    if (r == 0) return hi;
    uint32_t lo = (w >= q + 1) ? b[w - q - 1] : 0u;
    return (hi << r) | (lo >> (32u - r));
}

// LOWRES dilation (Anisotropic_kernel.cuh:610-629) and the band's size (Counters::nv, which the
// marking set to 0)
__global__ void __launch_bounds__(256) k_band_dilate(const uint32_t* __restrict__ bm0, uint32_t* __restrict__ bm,
                                                     uint64_t nwords, uint64_t nbits,
                                                     uint64_t sy, uint64_t sz, Counters* __restrict__ cnt) {
    // the tickets of the next launches that take any start at 0
    if (blockIdx.x == 0 && threadIdx.x == 0) cnt->band_next = cnt->n_items = cnt->field_next = 0u;
    uint32_t mine = 0u;
    for (uint64_t w = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; w < nwords; w += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t v = bm0[w] | shifted_word(bm0, w, 1) | shifted_word(bm0, w, sy) | shifted_word(bm0, w, sz);
        if (w == nwords - 1 && (nbits & 31u)) v &= (1u << (nbits & 31u)) - 1u;
        bm[w] = v;
        mine += (uint32_t)__popc(v);
    }
    const uint32_t tot = __reduce_add_sync(0xffffffffu, mine);
    if ((threadIdx.x & 31u) == 0u && tot) atomicAdd(&cnt->nv, tot);
}

// popcount per word
__global__ void __launch_bounds__(256) k_word_popc(const uint32_t* __restrict__ b, uint32_t* __restrict__ wcount,
                                                   uint64_t nwords) {
    for (uint64_t w = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; w < nwords; w += (uint64_t)gridDim.x * blockDim.x)
        wcount[w] = __popc(b[w]);
}

// ascending vertex list from the bitmap
__global__ void __launch_bounds__(256) k_band_list(const uint32_t* __restrict__ bm, const uint32_t* __restrict__ wprefix,
                                                   uint64_t nwords, uint32_t* __restrict__ vlist) {
    for (uint64_t w = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; w < nwords; w += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t b = bm[w];
        uint32_t o = wprefix[w];
        while (b) {
            uint32_t bit = __ffs(b) - 1;
            vlist[o++] = (uint32_t)(w * 32u + bit);
            b &= b - 1u;
        }
    }
}

static TileDims tile_dims(const KGrid& g) {
    TileDims td;
    td.n[0] = (g.scres[0] + kTileX - 1) / kTileX;
    td.n[1] = (g.scres[1] + kTileY - 1) / kTileY;
    td.n[2] = (g.scres[2] + kTileZ - 1) / kTileZ;
    return td;
}

pms_status launch_band(pms_ctx* ctx) {
    const KGrid g = kgrid_of(ctx->grid);
    Counters* cnt = ctx->counters.as<Counters>();
    const uint64_t nbits = g.sc_size, nwords = (nbits + 31) / 32;
    const TileDims td = tile_dims(g);
    const uint64_t ntiles = (uint64_t)td.n[0] * td.n[1] * td.n[2];
    // (the marks and the ticket are 0: the frame's start and the dilation leave them so, and a
    // second band of the same frame sets the same bits)
    // extent = ceil(maxdistance / scGridSize) (Anisotropic_kernel.cuh:551), a correctly rounded float quotient
    const int ext_dev = (int)(uint32_t)ceilf(ctx->prm.h / g.sc_cs);
    const uint64_t warps = 152u * 8u * (kBandThreads / 32);
    const uint32_t shares = (uint32_t)std::min<uint64_t>(std::max<uint64_t>(warps / ntiles, 1u), 8u);
    k_band_tiles<<<grid_for(ntiles * shares * 32, kBandThreads, 152u * 8u), kBandThreads, 0, ctx->stream>>>(
        g, ctx->prm.h, ext_dev, td, (uint32_t)ntiles, shares, cnt, ctx->surf_start.as<uint32_t>(),
        ctx->surf_count.as<uint32_t>(), ctx->slist.as<uint32_t>(), ctx->spos.as<float4>(), ctx->nrm4.as<float4>(),
        ctx->bm0.as<uint32_t>());
    PMS_LAUNCHED(ctx);
    const uint64_t sy = g.scres[0], sz = (uint64_t)g.scres[0] * g.scres[1];
    k_band_dilate<<<grid_for(nwords, 256, 152u * 8u), 256, 0, ctx->stream>>>(ctx->bm0.as<uint32_t>(), ctx->bm.as<uint32_t>(), nwords,
                                                                            nbits, sy, sz, cnt);
    PMS_LAUNCHED(ctx);
    ctx->field_tickets_zero = true;
    return PMS_OK;
}

pms_status launch_bits_list(pms_ctx* ctx, const uint32_t* bm, const uint32_t* wprefix, uint32_t* vlist) {
    const uint64_t nwords = ((uint64_t)ctx->grid.sc_size + 31) / 32;
    k_band_list<<<grid_for(nwords, 256), 256, 0, ctx->stream>>>(bm, wprefix, nwords, vlist);
    PMS_LAUNCHED(ctx);
    return PMS_OK;
}

pms_status launch_band_list(pms_ctx* ctx) {
    const uint64_t nwords = ((uint64_t)ctx->grid.sc_size + 31) / 32;
    PMS_CUDA(ctx, ctx->wcount.ensure(4 * (nwords + 1)));
    PMS_CUDA(ctx, ctx->wprefix.ensure(4 * (nwords + 1)));
    k_word_popc<<<grid_for(nwords, 256), 256, 0, ctx->stream>>>(ctx->bm.as<uint32_t>(), ctx->wcount.as<uint32_t>(), nwords);
    PMS_LAUNCHED(ctx);
    pms_status st = scan_u32(ctx, ctx->wcount.as<uint32_t>(), ctx->wprefix.as<uint32_t>(), nwords, nullptr);
    if (st != PMS_OK) return st;
    return launch_bits_list(ctx, ctx->bm.as<uint32_t>(), ctx->wprefix.as<uint32_t>(), ctx->vlist.as<uint32_t>());
}

}  // namespace pms
