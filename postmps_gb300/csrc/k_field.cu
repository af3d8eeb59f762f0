// k_field.cu -- narrow-band scalar field.
//
// Reference: computationOfScalarFieldGrid, Anisotropic_kernel.cuh:656-777 with
// anisotropicW / anisotropicWOpt (myCuda.cuh:151-191).  For band vertex v at
// position x_v (float32 i*cell + min) in spatial cell c it sums, over cells
// z, y, x in the HALF-OPEN box [c - 2e, c + 2e) (clamped), in that order:
//   surface cell:  (m / rho_j) * sigma * det(G_j) * (1 - |G_j r|^2)^3
//                  if |r| < maxvalue_j * h and |G_j r|^2 < 1, r = x_j - x_v
//   other cell:    (m / rho_j) * sigma / h^3 * (1 - |r|^2 / h^2)^3   if |r| < h
// skipping particles with rho == 0, and after each CELL tests
// sum > 2 * iso, which breaks only the innermost (x) loop: once the sum has
// crossed the threshold, every later row adds exactly its first cell.
//
// GB300 design: a warp per tile of scalar vertices (k_field_tiles).  The vertices of a
// tile share nearly all of the particles they sum, so the warp reads each particle
// once, keeps it in shared memory if its support can reach the tile, and all lanes
// evaluate it together.  Every particle carries its kernel in one packed form --
// M = G^T G, the weight (m / rho) sigma det(G), and the extents of its support's box,
// with G = I / h for particles of non-surface cells -- so one branch-free formula
// serves both kinds.  Cells are sorted by key, so the cells x in [xa, xb) of a row are
// the contiguous particle range [cell_start[row + xa], cell_start[row + xb]).
// Adding a zero contribution leaves the sum unchanged, so leaving out particles that
// cannot reach a vertex changes neither the reference's sum nor its early exit.
//
// Sign certification (the learned band's exact fallback; no reference
// counterpart).  Every term of the sum is >= 0 and float addition of a
// non-negative term never decreases a sum, so a vertex is certainly above the
// iso-value -- marching-cubes corner bit clear, whatever the rest of its walk
// would add -- as soon as a part of its sum exceeds iso.  In this mode a vertex
// (1) first sums the particles of the 2 x 2 x 2 spatial cells nearest to it (in
// any order; the test then asks for iso * (1 + 2^-9), which covers the rounding
// of two float sums in different orders of up to ~30,000 non-zero terms each);
// (2) failing that, walks in the reference's order and stops as soon as its
// running sum exceeds iso -- that prefix is the reference's own, since the
// reference's early exit (2 * iso) cannot have fired before.  A vertex stopped
// either way gets a placeholder above iso (its partial sum) and a bit in
// `cert`; a vertex whose walk ran to the end has exactly the reference's value
// (no early exit fired, the sum never exceeded iso).
#include <algorithm>

#include "pms_internal.h"
#include "k_common.cuh"

namespace pms {

struct FieldParams {
    float h;                  // isotropic support, the smallest culling radius of a cell
    float thr;                // 2 * iso: the early-exit threshold (certification: iso)
    float grow;               // relative margin on culling radii
    float quick;              // certification: iso * (1 + 2^-9), the nearest-cells test
    float ext_unit;           // step of the packed support extents
};

__device__ __forceinline__ float gap2_axis(float p, float lo, float cs, float pad) {
    float a = lo - pad, b = lo + cs + pad;
    float d = fmaxf(a - p, p - b);
    return d > 0.f ? d * d : 0.f;
}

// A particle adds sigma det(G) (m/rho) (1 - |G r|^2)^3 when |G r|^2 < 1
// (anisotropicW, myCuda.cuh:151-191); every other particle adds exactly 0.
// The reference also tests |r| < maxvalue * h first, which |G r| < 1 already
// implies (maxvalue * h = 1 / smallest singular value of G); at the very edge
// the two can differ only by rounding, where the contribution is ~0.  |G r|^2
// is evaluated as r^T M r with the packed M = G^T G (off-diagonals doubled)
// and the weight w = (m/rho) sigma det(G) stored per particle.
// The certification walks runs (k_field_cert), which visit only what their vertices
// reach before they stop.  A work item is a run of up to K vertices that are neighbours along x
// (ids id0, id0 + 1, ...; one row of the scalar grid): item = first band index
// t0 | (count - 1) << 29.  The run shares the slabs and rows of its walk (same
// y and z), each cell's bounds and record loads and each particle's loads;
// every vertex keeps its own window, x range, sum and early exit, and adds its
// contributions in the reference's order, so each value is the one a walk of
// that vertex alone gives.
static constexpr uint32_t kItemShift = 29;
static_assert(kMaxBand == 1u << kItemShift, "an item holds a band index and a count");

// BT threads per block, K vertices per item.  cell_rad holds sp_size per-cell support radii followed by
// one radius per row (z, y): the largest maxvalue * h of the row's particles
// (0 where none is anisotropic).  The z and y ranges are cut from the largest
// support of the frame, each row's x range from the row's own radius, and each
// non-empty cell by its record: the bounding box of its particles and its
// largest support.  The value, or the placeholder of a vertex stopped above iso, goes
// to fdense[id] (the whole scalar grid); cert receives a bit per vertex stopped, n_cert
// their count.
template <int BT, int K>
__global__ void __launch_bounds__(BT, (K == 1 ? 1280 : 1024) / BT)
k_field_cert(KGrid g, FieldParams fp, const Counters* __restrict__ cnt, const uint32_t* __restrict__ n_items_dev,
        const uint32_t* __restrict__ items, const uint32_t* __restrict__ vlist, const uint32_t* __restrict__ cell_start,
        const float* __restrict__ cell_rad, const float4* __restrict__ rec, const float4* __restrict__ spos,
        const float4* __restrict__ aniso, float* __restrict__ fdense,
        uint32_t* __restrict__ cert, uint32_t* __restrict__ n_cert, Counters* __restrict__ cnt_w) {
    const uint32_t n_items = *n_items_dev;
    uint32_t my_cert = 0;
    unsigned long long my_pairs = 0;         // (vertex, particle) pairs evaluated
    const uint32_t rx = g.scres[0], rxy = g.scres[0] * g.scres[1];
    const uint32_t srx = g.spres[0], sry = g.spres[1];
    const uint32_t e2 = 2u * (uint32_t)g.spexpand;
    const float pad = g.pad, inv_cs = 1.f / g.sp_cs;
    const float* __restrict__ row_rad = cell_rad + g.sp_size;
    // largest support of any particle this frame
    const float rmax = fmaxf(__uint_as_float(cnt->rad_max_bits), fp.h) * fp.grow;
    const float rmax2 = rmax * rmax;
    for (uint32_t it = blockIdx.x * blockDim.x + threadIdx.x; it < n_items; it += gridDim.x * blockDim.x) {
        const uint32_t item = items[it];
        const uint32_t t0 = item & ((1u << kItemShift) - 1u);
        const int m = (int)(item >> kItemShift) + 1;
        const uint32_t id = vlist[t0];
        const uint32_t iz = id / rxy, rem = id - iz * rxy, iy = rem / rx, ix = rem - iy * rx;
        const float vy = sc_coord(g, iy, 1), vz = sc_coord(g, iz, 2);
        float vx[K], ux[K], sum[K];
        int wlo[K], whi[K];                          // the vertices' x windows [c - 2e, c + 2e) (clamped)
        uint3 lo, hi;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            vx[k] = sc_coord(g, ix + (uint32_t)k, 0);
            const uint3 c = sp_cell(g, vx[k], vy, vz);
            box_clamp(g, c, e2, lo, hi);             // y and z bounds agree for all vertices of the run
            wlo[k] = (int)lo.x;
            whi[k] = k < m ? (int)hi.x : (int)lo.x;  // vertices past the run: empty windows
            ux[k] = (vx[k] - g.min_pos[0]) * inv_cs;
            sum[k] = 0.f;
        }
        const float uy = (vy - g.min_pos[1]) * inv_cs, uz = (vz - g.min_pos[2]) * inv_cs;
        bool done[K];
#pragma unroll
        for (int k = 0; k < K; ++k) done[k] = false;
        {
            // the 2 x 2 x 2 cells nearest to each vertex (inside its window): the run
            // shares the two slabs and two rows, each vertex takes its own two x cells
            const int cz = (int)floorf(uz), cy = (int)floorf(uy);
            const int z2 = uz - (float)cz >= 0.5f ? cz + 1 : cz - 1, y2 = uy - (float)cy >= 0.5f ? cy + 1 : cy - 1;
            int qa[K], qb[K];
            int XA = 0x7fffffff, XB = -1;
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const int cx = (int)floorf(ux[k]);
                const int x2 = ux[k] - (float)cx >= 0.5f ? cx + 1 : cx - 1;
                qa[k] = max(min(cx, x2), wlo[k]);
                qb[k] = min(max(cx, x2) + 1, whi[k]);
                if (qa[k] < qb[k]) { XA = min(XA, qa[k]); XB = max(XB, qb[k]); }
            }
#pragma unroll
            for (int s2 = 0; s2 < 4; ++s2) {
                const int z = (s2 >> 1) ? z2 : cz, y = (s2 & 1) ? y2 : cy;
                if (z < (int)lo.z || z >= (int)hi.z || y < (int)lo.y || y >= (int)hi.y) continue;
                const uint32_t row = ((uint32_t)z * sry + (uint32_t)y) * srx;
                for (int x = XA; x < XB; ++x) {
                    bool use[K];
#pragma unroll
                    for (int k = 0; k < K; ++k) use[k] = x >= qa[k] && x < qb[k];
                    const uint32_t j0 = __ldg(&cell_start[row + (uint32_t)x]), j1 = __ldg(&cell_start[row + (uint32_t)x + 1u]);
                    {
                        uint32_t nu = 0u;
#pragma unroll
                        for (int k = 0; k < K; ++k) nu += use[k] ? 1u : 0u;
                        my_pairs += (unsigned long long)(j1 - j0) * nu;
                    }
                    for (uint32_t j = j0; j < j1; ++j) {
                        const float4 q = __ldg(&spos[j]);
                        const float4 a0 = __ldg(&aniso[2 * (size_t)j]);
                        const float4 a1 = __ldg(&aniso[2 * (size_t)j + 1]);
                        const float ry = __fsub_rn(q.y, vy), rz = __fsub_rn(q.z, vz);
                        const float pyz = __fmaf_rn(rz, __fmul_rn(a1.z, rz), __fmul_rn(ry, __fmaf_rn(a1.x, ry, __fmul_rn(a1.y, rz))));
                        const float cyz = __fmaf_rn(a0.y, ry, __fmul_rn(a0.z, rz));
#pragma unroll
                        for (int k = 0; k < K; ++k) {
                            const float rxk = __fsub_rn(q.x, vx[k]);
                            const float d2 = __fmaf_rn(rxk, __fmaf_rn(a0.x, rxk, cyz), pyz);
                            const float xx = __fsub_rn(1.f, d2);
                            const float w = (d2 < 1.f) ? __fmul_rn(a1.w, __fmul_rn(__fmul_rn(xx, xx), xx)) : 0.f;
                            if (use[k]) sum[k] = __fadd_rn(sum[k], w);
                        }
                    }
                }
            }
            bool all = true;
#pragma unroll
            for (int k = 0; k < K; ++k) {
                if (k < m && sum[k] > fp.quick) {
                    done[k] = true;
                    whi[k] = wlo[k];                 // nothing left to walk
                } else {
                    sum[k] = 0.f;                    // the walk starts over in the reference's order
                    all = all && !(k < m);
                }
            }
            if (all) {
                uint32_t mask = 0u;
#pragma unroll
                for (int k = 0; k < K; ++k)
                    if (k < m) { fdense[id + k] = sum[k]; mask |= 1u << k; }
                const uint32_t w = id >> 5, sh = id & 31u;
                atomicOr(&cert[w], mask << sh);
                if (sh && (mask >> (32u - sh))) atomicOr(&cert[w + 1], mask >> (32u - sh));
                my_cert += (uint32_t)m;
                continue;
            }
        }
        int za, zb;
        cell_range(uz, rmax * inv_cs + g.margin, lo.z, hi.z, za, zb);
        for (int z = za; z < zb; ++z) {
            const float gz = gap2_axis(vz, g.min_pos[2] + (float)z * g.sp_cs, g.sp_cs, pad);
            if (gz >= rmax2) continue;
            int ya, yb;
            cell_range(uy, sqrtf(rmax2 - gz) * inv_cs + g.margin, lo.y, hi.y, ya, yb);
            for (int y = ya; y < yb; ++y) {
                const float gyz = gz + gap2_axis(vy, g.min_pos[1] + (float)y * g.sp_cs, g.sp_cs, pad);
                const uint32_t rowi = (uint32_t)z * sry + (uint32_t)y;
                const float rr = fmaxf(__ldg(&row_rad[rowi]), fp.h) * fp.grow;
                const float rr2 = rr * rr;
                if (gyz >= rr2) continue;           // every cell of the row adds 0
                const uint32_t row = rowi * srx;
                // each vertex's cells of this row: those the row's largest support reaches
                const float rxc = sqrtf(rr2 - gyz) * inv_cs + g.margin;
                int xs[K], xe[K];
                bool live[K];
                int X0 = 0x7fffffff, X1 = -1;
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    cell_range(ux[k], rxc, (uint32_t)wlo[k], (uint32_t)whi[k], xs[k], xe[k]);
                    live[k] = xs[k] < xe[k];
                    if (live[k]) { X0 = min(X0, xs[k]); X1 = max(X1, xe[k]); }
                }
                for (int x0 = X0; x0 < X1; x0 += 32) {
                    const int nx = min(X1 - x0, 32);
                    // cells of the chunk inside some live vertex's range
                    uint32_t need = 0u;
#pragma unroll
                    for (int k = 0; k < K; ++k) {
                        const int a = max(xs[k] - x0, 0), b = min(xe[k] - x0, nx);
                        if (live[k] && a < b) need |= (b - a == 32 ? ~0u : ((1u << (b - a)) - 1u)) << a;
                    }
                    // cells whose record each vertex reaches (independent loads)
                    uint32_t reach[K];
#pragma unroll
                    for (int k = 0; k < K; ++k) reach[k] = 0u;
                    for (uint32_t todo = need; todo; todo &= todo - 1u) {
                        const int i = __ffs(todo) - 1;
                        const int x = x0 + i;
                        const uint32_t c = row + (uint32_t)x;
                        const float4 b0 = __ldg(&rec[2 * (size_t)c]), b1 = __ldg(&rec[2 * (size_t)c + 1]);
                        const float dy = fmaxf(fmaxf(b0.y - vy, vy - b1.y), 0.f);
                        const float dz = fmaxf(fmaxf(b0.z - vz, vz - b1.z), 0.f);
                        const float dyz = dy * dy + dz * dz;
#pragma unroll
                        for (int k = 0; k < K; ++k) {
                            const float dx = fmaxf(fmaxf(b0.x - vx[k], vx[k] - b1.x), 0.f);
                            const bool in = live[k] && x >= xs[k] && x < xe[k] && dx * dx + dyz < b0.w;
                            reach[k] |= (in ? 1u : 0u) << i;
                        }
                    }
                    uint32_t any = 0u;
#pragma unroll
                    for (int k = 0; k < K; ++k) any |= reach[k];
                    // the reached cells in x order; a vertex stops once its sum passes the
                    // threshold after one of its cells
                    while (any) {
                        const int i = __ffs(any) - 1;
                        const uint32_t bit = 1u << i;
                        const uint32_t c = row + (uint32_t)(x0 + i);
                        bool use[K];
#pragma unroll
                        for (int k = 0; k < K; ++k) use[k] = (reach[k] & bit) != 0u;
                        const uint32_t j0 = __ldg(&cell_start[c]), j1 = __ldg(&cell_start[c + 1u]);
                        {
                            uint32_t nu = 0u;
#pragma unroll
                            for (int k = 0; k < K; ++k) nu += use[k] ? 1u : 0u;
                            my_pairs += (unsigned long long)(j1 - j0) * nu;
                        }
#pragma unroll 1
                        for (uint32_t j = j0; j < j1; ++j) {
                            const float4 q = __ldg(&spos[j]);
                            const float4 a0 = __ldg(&aniso[2 * (size_t)j]);      // {m00, 2 m01, 2 m02, extents}
                            const float4 a1 = __ldg(&aniso[2 * (size_t)j + 1]);  // {m11, 2 m12, m22, w}
                            // r^T M r with every rounding spelled out, so that the value does
                            // not depend on how many vertices share the loads
                            const float ry = __fsub_rn(q.y, vy), rz = __fsub_rn(q.z, vz);
                            const float pyz = __fmaf_rn(rz, __fmul_rn(a1.z, rz), __fmul_rn(ry, __fmaf_rn(a1.x, ry, __fmul_rn(a1.y, rz))));
                            const float cyz = __fmaf_rn(a0.y, ry, __fmul_rn(a0.z, rz));
#pragma unroll
                            for (int k = 0; k < K; ++k) {
                                const float rxk = __fsub_rn(q.x, vx[k]);
                                const float d2 = __fmaf_rn(rxk, __fmaf_rn(a0.x, rxk, cyz), pyz);
                                const float xx = __fsub_rn(1.f, d2);
                                const float w = (d2 < 1.f) ? __fmul_rn(a1.w, __fmul_rn(__fmul_rn(xx, xx), xx)) : 0.f;
                                if (use[k]) sum[k] = __fadd_rn(sum[k], w);
                            }
                        }
                        uint32_t still = 0u;
#pragma unroll
                        for (int k = 0; k < K; ++k) {
                            if (use[k] && sum[k] > fp.thr) {
                                reach[k] = 0u;
                                live[k] = false;
                                done[k] = true;
                                whi[k] = wlo[k];         // certified: stop for good
                            }
                            still |= reach[k];
                        }
                        any = still & ~((bit << 1) - 1u);   // i = 31: bit << 1 = 0, nothing left
                    }
                    bool more = false;
#pragma unroll
                    for (int k = 0; k < K; ++k) more |= live[k] && xe[k] > x0 + nx;
                    if (!more) break;
                }
            }
        }
        uint32_t mask = 0u;
#pragma unroll
        for (int k = 0; k < K; ++k)
            if (k < m) {
                fdense[id + k] = sum[k];
                if (done[k]) mask |= 1u << k;
            }
        if (mask) {
            const uint32_t w = id >> 5, sh = id & 31u;
            atomicOr(&cert[w], mask << sh);
            if (sh && (mask >> (32u - sh))) atomicOr(&cert[w + 1], mask >> (32u - sh));
            my_cert += (uint32_t)__popc(mask);
        }
    }
    const uint32_t tot = __reduce_add_sync(0xffffffffu, my_cert);
    if ((threadIdx.x & 31u) == 0 && tot) atomicAdd(n_cert, tot);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) my_pairs += __shfl_xor_sync(0xffffffffu, my_pairs, o);
    if ((threadIdx.x & 31u) == 0 && my_pairs) atomicAdd(&cnt_w->n_pairs, my_pairs);
}

// ---------------------------------------------------------------------------
// Exact field, tile by tile.  One warp evaluates a tile of 32 K scalar vertices
// (4 x 4 x 2 for K = 1, 4 x 4 x 4 for K = 2, 8 x 4 x 4 for K = 4; a lane owns K
// x-neighbours).  The warp reads the particles that can reach the tile's band
// vertices once, 32 at a time, in the reference's order -- ascending sorted index
// -- keeps those whose support box meets the vertices' box, stages them in shared
// memory, and every lane then runs over the staged particles, all lanes on the
// same one.  A vertex adds every staged particle's contribution in that order, so
// its sum is the one a walk of its own gives (particles left out add exactly 0).
//
// The early exit, restated per cell: a cell adds to a vertex when the vertex's sum
// is not past 2 iso before it, or when it is the first cell of the vertex's window
// in its row (the reference adds it, then breaks).  The sum never decreases, so
// this is the reference's rule whatever was skipped in between.  Windows matter
// only for cells that are not inside every vertex's window (or are some vertex's
// first cell): a chunk with such a particle takes the general path, which tests
// each vertex's own window.
//
// Bound by instruction issue.  A walk per run of vertices (18 of 32 lanes active, its
// rows, records and cell bounds costing more than the pairs) took 2.89 / 2.56 / 7.24 ms
// for the field stage of the crown 2M / dam 8M / spray 151k (ratio 3) frames; tiles take
// 0.91 / 1.01 / 0.65 ms (28 of 32 lanes active, 3.0 instructions a cycle on the dam; the spray
// 0.77 with K = 2, as in the figures here).  Of that:
// - support boxes and the separating plane leave 41, 66 and 28 staged particles per tile of
//   about 52 band vertices; the boxes alone left 60, 99 and 42 (1.29 / 1.64 / 1.22 ms);
// - rows are cut by the largest support of their stretch of 8 cells, tiles listed with their
//   coordinates, and the general path taken per cell (with rows cut by their own largest
//   support and whole chunks taken generally: 1.03 / 1.23 / 0.96 ms with the clearing of
//   the dense field, 0.05 ms);
// - a lane's x-neighbours go through the packed two-float operations, rounded as the
//   scalar ones, and the early exit is a limit on |G r|^2 rather than a flag.  Staging the
//   packed operands twice, as pairs, cost more than the moves it saves (1.07 / 1.09 / 0.81).
// K trades what a tile shares for what its vertices add in vain (pick_k has the rule).
// ---------------------------------------------------------------------------
template <int K> struct FieldTile {
    static constexpr int X = K == 4 ? 8 : 4, Y = 4, Z = K == 1 ? 2 : 4;
};
static constexpr uint32_t kTileTicket = 4;      // consecutive listed tiles a warp takes at once
// Resident warps per SM the registers are capped for.  Crown 2M / dam 8M field stage, before the
// row cuts: 20 warps (96 registers, no spills) 1.03 / 1.23 ms, 24 1.04 / 1.25, 16 1.15 / 1.36.
static constexpr int kFieldWarps = 20;

// How many vertices a lane takes, from the number of vertices to evaluate (a device count: the
// host does not know the band's size yet).  Both launches decide alike.
// - Below 160,000 vertices tiles of 64 do not fill the GPU: tiles of 32.  Field stage with 1 / 2:
//   block 4k 22 / 25 us, 10k 29 / 33, one scalar cell per spacing (3k to 60k) 33 to 39 / 45 to
//   51; the sides meet near 180,000 (crown 10k 31 / 33, 30k 49 / 47; block 30k 45 / 43).
// - Tiles of 128 where many vertices share the same particles.  With 2 / 4: from three scalar
//   cells per spacing on and 500,000 vertices, block 200k 213 / 178 us, crown 400k 723 / 590, dam
//   1M 913 / 768, spray 100k 537 / 393 (338,000 vertices: 39 / 41); at two cells, from h = 4
//   spacings on, dam 1M 2.18 / 2.02 ms, crown 400k 1.60 / 1.48, block 200k 0.54 / 0.46, and for
//   sparse frames (droplets: particles fill less than a tenth of their box, a tile meets few of
//   them), spray 151k (h = 3) 0.76 / 0.65 ms, 30k 0.23 / 0.17.  Elsewhere they lose: h = 2 and two
//   cells, dam 1M 424 / 449 us, block 200k 104 / 119; one cell 1.3 to 2 times.
struct FieldPick {
    uint32_t few, many;                    // below: 1, from here on: 4
    const uint32_t* __restrict__ count;
};
__device__ __forceinline__ uint32_t pick_k(const FieldPick& p) {
    const uint32_t v = *p.count;
    return v < p.few ? 1u : (v >= p.many ? 4u : 2u);
}

// The tiles holding a set bit of a bitmap over the scalar grid, 3 + K words each: the
// first vertex's x, y, z, then for k < K the lanes whose vertex k is set.
template <int K>
__device__ __forceinline__ void field_tile_list(const KGrid& g, const uint32_t* __restrict__ bm,
                                                uint32_t* __restrict__ n_tiles, uint32_t* __restrict__ list) {
    using T = FieldTile<K>;
    const uint3 td = make_uint3((g.scres[0] + T::X - 1) / T::X, (g.scres[1] + T::Y - 1) / T::Y, (g.scres[2] + T::Z - 1) / T::Z);
    const uint32_t ntiles = td.x * td.y * td.z;
    const uint32_t rx = g.scres[0], ry = g.scres[1], rz = g.scres[2];
    // whole warps stay in the loop together (the append is a warp vote)
    for (uint32_t t0 = blockIdx.x * blockDim.x; t0 < ntiles; t0 += gridDim.x * blockDim.x) {
        const uint32_t t = t0 + threadIdx.x;
        uint32_t m[K];
#pragma unroll
        for (int k = 0; k < K; ++k) m[k] = 0u;
        const uint32_t tx = t % td.x, tyz = t / td.x, ty = tyz % td.y, tz = tyz / td.y, x0 = tx * T::X;
        if (t < ntiles) {
            const uint32_t in = rx - x0 >= (uint32_t)T::X ? (1u << T::X) - 1u : (1u << (rx - x0)) - 1u;
#pragma unroll
            for (int z = 0; z < T::Z; ++z)
#pragma unroll
                for (int y = 0; y < T::Y; ++y) {
                    const uint32_t vy = ty * T::Y + (uint32_t)y, vz = tz * T::Z + (uint32_t)z;
                    if (vy >= ry || vz >= rz) continue;
                    const uint64_t bit = ((uint64_t)vz * ry + vy) * rx + x0;
                    const uint64_t w = bit >> 5;
                    const uint32_t sh = (uint32_t)(bit & 31u);
                    uint32_t b = __ldg(&bm[w]) >> sh;
                    if (sh > 32u - (uint32_t)T::X) b |= __ldg(&bm[w + 1]) << (32u - sh);   // bitmaps hold a word more
                    b &= in;
#pragma unroll
                    for (int i = 0; i < T::X; ++i)
                        m[i % K] |= ((b >> i) & 1u) << (z * (32 / T::Z) + y * (T::X / K) + i / K);
                }
        }
        uint32_t any = 0u;
#pragma unroll
        for (int k = 0; k < K; ++k) any |= m[k];
        const uint32_t vote = __ballot_sync(0xffffffffu, any != 0u);
        if (!vote) continue;
        const uint32_t lane = threadIdx.x & 31u;
        uint32_t base = 0u;
        if (lane == 0u) base = atomicAdd(n_tiles, (uint32_t)__popc(vote));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (any) {
            uint32_t* e = list + (size_t)(3 + K) * (base + (uint32_t)__popc(vote & ((1u << lane) - 1u)));
            e[0] = x0; e[1] = ty * T::Y; e[2] = tz * T::Z;
#pragma unroll
            for (int k = 0; k < K; ++k) e[3 + k] = m[k];
        }
    }
}

// K = 0: by the rule (a launch whose K the host knows saves the look at the count: 6 us of the
// dam's 980)
template <int K>
__global__ void __launch_bounds__(256) k_field_tile_list(KGrid g, FieldPick pick, const uint32_t* __restrict__ bm,
                                                         uint32_t* __restrict__ n_tiles, uint32_t* __restrict__ list) {
    const uint32_t k = K ? (uint32_t)K : pick_k(pick);
    if (k == 1u) field_tile_list<1>(g, bm, n_tiles, list);
    else if (k == 4u) field_tile_list<4>(g, bm, n_tiles, list);
    else field_tile_list<2>(g, bm, n_tiles, list);
}

// A staged particle: position and packed kernel, its cell's x, and its row of cells with
// two flags: the first particle of a cell, a cell that needs the general path.
struct FieldStage {
    float4 a;     // x, y, z, m00
    float4 b;     // 2 m01, 2 m02, m11, 2 m12
    float4 c;     // m22, w, x bits, row bits | flags
};
static constexpr int kFieldStage = 64;
static constexpr uint32_t kFresh = 1u << 31, kOdd = 1u << 30;   // (a row of cells is below 2^30: a grid is 4 cells wide at least)
static constexpr float kNever = -1.0e30f;       // below any |G r|^2

template <int BT, int K>
__device__ __forceinline__ void
field_tiles(const KGrid& g, const FieldParams& fp, FieldStage* stage, const Counters* __restrict__ cnt,
            const uint32_t* __restrict__ n_tiles_dev, uint32_t* __restrict__ next, const uint32_t* __restrict__ list,
            const uint32_t* __restrict__ cell_start, const float* __restrict__ cell_rad,
            const uint32_t* __restrict__ skeys, const float4* __restrict__ spos, const float4* __restrict__ aniso,
            float* __restrict__ fdense, Counters* __restrict__ cnt_w) {
    constexpr unsigned kAll = 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t n_tiles = *n_tiles_dev;
    const uint32_t rx = g.scres[0], rxy = g.scres[0] * g.scres[1];
    const int srx = (int)g.spres[0], sry = (int)g.spres[1], srz = (int)g.spres[2];
    const int e2 = 2 * g.spexpand;
    const float pad = g.pad, cs = g.sp_cs, inv_cs = 1.f / g.sp_cs;
    // largest support per stretch of kRadSeg cells of a row
    const float* __restrict__ seg_rad = cell_rad + g.sp_size + g.spres[1] * g.spres[2];
    const uint32_t nseg = rad_segments(g.spres[0]);
    const float rmax = fmaxf(__uint_as_float(cnt->rad_max_bits), fp.h) * fp.grow;
    const float rmax2 = rmax * rmax;
    // the lane's place in a tile
    const uint32_t lx = K == 1 ? lane & 3u : (lane & 1u) * K, ly = K == 1 ? (lane >> 2) & 3u : (lane >> 1) & 3u,
                   lz = K == 1 ? lane >> 4 : lane >> 3;
    // few tiles are spread over all warps; many are taken in stretches, whose rows of cells
    // stay in the SM's cache from tile to tile
    const uint32_t ticket = min(max(n_tiles / (gridDim.x * (BT / 32u) * 4u), 1u), kTileTicket);
    unsigned long long my_pairs = 0;
    for (;;) {
        uint32_t first = 0u;
        if (lane == 0u) first = atomicAdd(next, ticket);
        first = __shfl_sync(kAll, first, 0);
        if (first >= n_tiles) break;
        const uint32_t last = min(first + ticket, n_tiles);
        for (uint32_t e = first; e < last; ++e) {
            const uint32_t* tile = list + (size_t)(3 + K) * e;
            uint32_t m[K];
#pragma unroll
            for (int k = 0; k < K; ++k) m[k] = __ldg(&tile[3 + k]);
            const uint32_t ix = __ldg(&tile[0]) + lx, iy = __ldg(&tile[1]) + ly, iz = __ldg(&tile[2]) + lz;
            const float vy = sc_coord(g, iy, 1), vz = sc_coord(g, iz, 2);
            float vx[K], sum[K];
            float lim[K];                            // |G r|^2 below which a particle adds: 1, or never
            bool have[K];
            uint32_t nvert = 0u, x_lo = 0xffffffffu, x_hi = 0u;
            bool some = false;
#pragma unroll
            for (int k = 0; k < K; ++k) {
                vx[k] = sc_coord(g, ix + (uint32_t)k, 0);
                have[k] = (m[k] >> lane) & 1u;
                lim[k] = have[k] ? 1.f : kNever;
                sum[k] = have[k] ? 0.f : INFINITY;   // no vertex: past the threshold from the start
                nvert += (uint32_t)__popc(m[k]);
                if (have[k]) { x_lo = min(x_lo, ix + (uint32_t)k); x_hi = max(x_hi, ix + (uint32_t)k); some = true; }
            }
            // the box of the tile's band vertices
            x_lo = __reduce_min_sync(kAll, x_lo);
            x_hi = __reduce_max_sync(kAll, x_hi);
            const uint32_t y_lo = __reduce_min_sync(kAll, some ? iy : 0xffffffffu), y_hi = __reduce_max_sync(kAll, some ? iy : 0u);
            const uint32_t z_lo = __reduce_min_sync(kAll, some ? iz : 0xffffffffu), z_hi = __reduce_max_sync(kAll, some ? iz : 0u);
            const float bx0 = sc_coord(g, x_lo, 0), bx1 = sc_coord(g, x_hi, 0);
            const float by0 = sc_coord(g, y_lo, 1), by1 = sc_coord(g, y_hi, 1);
            const float bz0 = sc_coord(g, z_lo, 2), bz1 = sc_coord(g, z_hi, 2);
            const float ux0 = (bx0 - g.min_pos[0]) * inv_cs, ux1 = (bx1 - g.min_pos[0]) * inv_cs;
            const float uy0 = (by0 - g.min_pos[1]) * inv_cs, uy1 = (by1 - g.min_pos[1]) * inv_cs;
            const float uz0 = (bz0 - g.min_pos[2]) * inv_cs, uz1 = (bz1 - g.min_pos[2]) * inv_cs;
            // cells some vertex's window holds [u.., u..), and cells that every window holds past
            // its first column [i.., i..), from the corners' cells taken a margin apart (the
            // vertices' own cells lie between); near the grid's low side, where the reference's
            // unsigned window wraps, every cell takes the general path
            const int cx0 = (int)floorf(ux0 - g.margin), cx1 = (int)floorf(ux1 + g.margin);
            const int cy0 = (int)floorf(uy0 - g.margin), cy1 = (int)floorf(uy1 + g.margin);
            const int cz0 = (int)floorf(uz0 - g.margin), cz1 = (int)floorf(uz1 + g.margin);
            const bool regular = min(cx0, min(cy0, cz0)) >= e2;
            const int ulx = regular ? cx0 - e2 : 0, uhx = regular ? min(cx1 + e2, srx - 1) : srx;
            const int uly = regular ? cy0 - e2 : 0, uhy = regular ? min(cy1 + e2, sry - 1) : sry;
            const int ulz = regular ? cz0 - e2 : 0, uhz = regular ? min(cz1 + e2, srz - 1) : srz;
            const int ilx = cx1 - e2 + 1, ihx = regular ? min(cx0 + e2, srx - 1) : 0;
            const int ily = cy1 - e2, ihy = min(cy0 + e2, sry - 1);
            const int ilz = cz1 - e2, ihz = min(cz0 + e2, srz - 1);
            // rows (z, y) within the frame's largest support of the box
            const float rc = rmax * inv_cs + g.margin;
            const int za = max((int)floorf(uz0 - rc), ulz), zb = min((int)floorf(uz1 + rc) + 1, uhz);
            const int ya = max((int)floorf(uy0 - rc), uly), yb = min((int)floorf(uy1 + rc) + 1, uhy);
            const int ny = yb - ya, nrow = ny > 0 && zb > za ? ny * (zb - za) : 0;
            const int xa0 = max((int)floorf(ux0 - rc), ulx), xb0 = min((int)floorf(ux1 + rc) + 1, uhx);

            int staged = 0;
            bool odd = false;                        // a staged particle needs the general path
            uint32_t key_before = 0xffffffffu;       // cell of the last staged particle

            // every lane over the staged particles
            auto run = [&](auto general) {
                constexpr bool G = decltype(general)::value;
                int wx0[K], wx1[K], wy0 = 0, wy1 = 0, wz0 = 0, wz1 = 0;
                if constexpr (G) {
                    uint3 lo, hi;
#pragma unroll
                    for (int k = 0; k < K; ++k) {
                        const uint3 c = sp_cell(g, vx[k], vy, vz);
                        box_clamp(g, c, (uint32_t)e2, lo, hi);
                        wx0[k] = (int)lo.x;
                        wx1[k] = (int)hi.x;
                    }
                    wy0 = (int)lo.y; wy1 = (int)hi.y; wz0 = (int)lo.z; wz1 = (int)hi.z;
                }
#pragma unroll 2
                for (int i = 0; i < staged; ++i) {
                    const float4 a = stage[i].a, b = stage[i].b, c = stage[i].c;
                    const uint32_t cw = __float_as_uint(c.w);
                    const bool fresh = (cw & kFresh) != 0u;
                    if constexpr (G) {
                        if (fresh && !(cw & kOdd)) {
#pragma unroll
                            for (int k = 0; k < K; ++k) lim[k] = sum[k] > fp.thr ? kNever : 1.f;
                        } else if (fresh) {
                            const int row = (int)(cw & (kOdd - 1u)), x = __float_as_int(c.z);
                            const int z = row / sry, y = row - z * sry;
                            const bool in = y >= wy0 && y < wy1 && z >= wz0 && z < wz1;
#pragma unroll
                            for (int k = 0; k < K; ++k)
                                lim[k] = have[k] && in && x >= wx0[k] && x < wx1[k] && (x == wx0[k] || !(sum[k] > fp.thr)) ? 1.f : kNever;
                        }
                    } else {
                        // (a cell inside every window: a vertex past the threshold takes no more of them)
#pragma unroll
                        for (int k = 0; k < K; ++k)
                            if (fresh) lim[k] = sum[k] > fp.thr ? kNever : 1.f;
                    }
                    // r^T M r with every rounding spelled out (as in the run walk above); the
                    // x-neighbours' parts two at a time
                    const float ry = __fsub_rn(a.y, vy), rz = __fsub_rn(a.z, vz);
                    const float pyz = __fmaf_rn(rz, __fmul_rn(c.x, rz), __fmul_rn(ry, __fmaf_rn(b.z, ry, __fmul_rn(b.w, rz))));
                    const float cyz = __fmaf_rn(b.x, ry, __fmul_rn(b.y, rz));
                    if constexpr (K == 1) {
                        const float rxk = __fsub_rn(a.x, vx[0]);
                        const float d2 = __fmaf_rn(rxk, __fmaf_rn(a.w, rxk, cyz), pyz);
                        const float xx = __fsub_rn(1.f, d2);
                        const float w = __fmul_rn(c.y, __fmul_rn(__fmul_rn(xx, xx), xx));
                        if (d2 < lim[0]) sum[0] = __fadd_rn(sum[0], w);
                    } else {
#pragma unroll
                        for (int k = 0; k < K; k += 2) {
                            const float2 rr = __fadd2_rn(make_float2(a.x, a.x), make_float2(-vx[k], -vx[k + 1]));
                            const float2 d2 = __ffma2_rn(rr, __ffma2_rn(make_float2(a.w, a.w), rr, make_float2(cyz, cyz)),
                                                         make_float2(pyz, pyz));
                            const float2 xx = __ffma2_rn(d2, make_float2(-1.f, -1.f), make_float2(1.f, 1.f));   // 1 - d2
                            const float2 w = __fmul2_rn(make_float2(c.y, c.y), __fmul2_rn(__fmul2_rn(xx, xx), xx));
                            if (d2.x < lim[k]) sum[k] = __fadd_rn(sum[k], w.x);
                            if (d2.y < lim[k + 1]) sum[k + 1] = __fadd_rn(sum[k + 1], w.y);
                        }
                    }
                }
                my_pairs += (unsigned long long)(nvert * (uint32_t)staged);
            };
            auto flush = [&]() {
                __syncwarp();
                if (odd) run(std::true_type());
                else run(std::false_type());
                __syncwarp();
                staged = 0;
                odd = false;
            };

            for (int r0 = 0; r0 < nrow; r0 += 32) {
                // a row per lane: its cells within the row's largest support of the box
                const int r = r0 + (int)lane;
                uint32_t ja = 0u, n = 0u, rowi = 0u;
                bool inner = false;
                if (r < nrow) {
                    const int z = za + r / ny, y = ya + r % ny;
                    rowi = (uint32_t)z * (uint32_t)sry + (uint32_t)y;
                    const float z0 = g.min_pos[2] + (float)z * cs, y0 = g.min_pos[1] + (float)y * cs;
                    const float gz = fmaxf(fmaxf(z0 - pad - bz1, bz0 - (z0 + cs + pad)), 0.f);
                    const float gy = fmaxf(fmaxf(y0 - pad - by1, by0 - (y0 + cs + pad)), 0.f);
                    const float gyz = gz * gz + gy * gy;
                    float rr = fp.h;                 // the row's largest support where the tile can reach it
                    if (gyz < rmax2)
                        for (int s = xa0 / kRadSeg; s * kRadSeg < xb0; ++s) rr = fmaxf(rr, __ldg(&seg_rad[rowi * nseg + (uint32_t)s]));
                    rr *= fp.grow;
                    const float rr2 = rr * rr;
                    if (gyz < rr2) {
                        const float rxc = sqrtf(rr2 - gyz) * inv_cs + g.margin;
                        const int xa = max((int)floorf(ux0 - rxc), ulx), xb = min((int)floorf(ux1 + rxc) + 1, uhx);
                        if (xa < xb) {
                            const uint32_t row = rowi * (uint32_t)srx;
                            ja = __ldg(&cell_start[row + (uint32_t)xa]);
                            n = __ldg(&cell_start[row + (uint32_t)xb]) - ja;
                        }
                    }
                    inner = z >= ilz && z < ihz && y >= ily && y < ihy;
                }
                // (the row's index, with the flag of a row outside some vertex's window)
                const uint32_t row_tag = rowi | (inner ? 0u : kOdd);
                const WarpRows rows = warp_rows(ja, n);
                for (uint32_t p0 = 0u; p0 < rows.total; p0 += 32u) {
                    const uint32_t p = p0 + lane;
                    const int row = warp_row_of(rows, p);
                    const uint32_t j = __shfl_sync(kAll, rows.off, row) + p;
                    const uint32_t tag = __shfl_sync(kAll, row_tag, row);
                    bool keep = false;
                    float4 q, a0, a1;
                    uint32_t key = 0u;
                    if (p < rows.total) {
                        q = __ldg(&spos[j]);
                        a0 = __ldg(&aniso[2 * (size_t)j]);
                        key = __ldg(&skeys[j]);
                        float ex, ey, ez;
                        unpack_extents(__float_as_uint(a0.w), fp.ext_unit, ex, ey, ez);
                        a1 = __ldg(&aniso[2 * (size_t)j + 1]);
                        const float x0 = bx0 - q.x, x1 = bx1 - q.x, y0 = by0 - q.y, y1 = by1 - q.y, z0 = bz0 - q.z, z1 = bz1 - q.z;
                        keep = !(x1 < -ex || x0 > ex || y1 < -ey || y0 > ey || z1 < -ez || z0 > ez);
                        if (keep) {
                            // a plane between the support and the box: its normal n = M r for the box's
                            // nearest point r, the support's reach along it sqrt(n M^-1 n) = sqrt(r M r),
                            // the box's lowest point along it (exact for a ball; never cuts a contribution)
                            const float r0 = fminf(fmaxf(0.f, x0), x1), r1 = fminf(fmaxf(0.f, y0), y1), r2 = fminf(fmaxf(0.f, z0), z1);
                            const float m01 = 0.5f * a0.y, m02 = 0.5f * a0.z, m12 = 0.5f * a1.y;
                            const float n0 = a0.x * r0 + m01 * r1 + m02 * r2, n1 = m01 * r0 + a1.x * r1 + m12 * r2,
                                        n2 = m02 * r0 + m12 * r1 + a1.z * r2;
                            const float s = n0 * r0 + n1 * r1 + n2 * r2;
                            const float low = fminf(n0 * x0, n0 * x1) + fminf(n1 * y0, n1 * y1) + fminf(n2 * z0, n2 * z1);
                            keep = !(low > 0.f && low * low > 1.002f * s);
                        }
                    }
                    const uint32_t kept = __ballot_sync(kAll, keep);
                    if (!kept) continue;
                    // a kept particle opens a cell when the kept one before it lies in another
                    const uint32_t below = kept & ((1u << lane) - 1u);
                    const uint32_t prev = __shfl_sync(kAll, key, below ? 31 - __clz(below) : 0);
                    const uint32_t key_last = __shfl_sync(kAll, key, 31 - __clz(kept));
                    bool my_odd = false;
                    if (keep) {
                        const bool fresh = key != (below ? prev : key_before);
                        const int x = (int)(key - (tag & (kOdd - 1u)) * (uint32_t)srx);
                        my_odd = (tag & kOdd) || x < ilx || x >= ihx;
                        FieldStage& s = stage[staged + __popc(below)];
                        s.a = make_float4(q.x, q.y, q.z, a0.x);
                        s.b = make_float4(a0.y, a0.z, a1.x, a1.y);
                        s.c = make_float4(a1.z, a1.w, __int_as_float(x),
                                          __uint_as_float((tag & (kOdd - 1u)) | (my_odd ? kOdd : 0u) | (fresh ? kFresh : 0u)));
                    }
                    odd |= __any_sync(kAll, my_odd);
                    key_before = key_last;
                    staged += __popc(kept);
                    if (staged > kFieldStage - 32) flush();
                }
            }
            if (staged) flush();
            const uint32_t id = iz * rxy + iy * rx + ix;
#pragma unroll
            for (int k = 0; k < K; ++k)
                if (have[k]) fdense[id + (uint32_t)k] = sum[k];
        }
    }
    if (lane == 0u && my_pairs) atomicAdd(&cnt_w->n_pairs, my_pairs);
}

template <int BT, int K>
__global__ void __launch_bounds__(BT, kFieldWarps * 32 / BT)
k_field_tiles(KGrid g, FieldParams fp, FieldPick pick, const Counters* __restrict__ cnt, const uint32_t* __restrict__ n_tiles_dev,
              uint32_t* __restrict__ next, const uint32_t* __restrict__ list,
              const uint32_t* __restrict__ cell_start, const float* __restrict__ cell_rad,
              const uint32_t* __restrict__ skeys, const float4* __restrict__ spos, const float4* __restrict__ aniso,
              float* __restrict__ fdense, Counters* __restrict__ cnt_w) {
    __shared__ FieldStage stage_all[BT / 32][kFieldStage];
    FieldStage* stage = stage_all[threadIdx.x >> 5];
    const uint32_t k = K ? (uint32_t)K : pick_k(pick);
    if (k == 1u)
        field_tiles<BT, 1>(g, fp, stage, cnt, n_tiles_dev, next, list, cell_start, cell_rad, skeys, spos, aniso, fdense, cnt_w);
    else if (k == 4u)
        field_tiles<BT, 4>(g, fp, stage, cnt, n_tiles_dev, next, list, cell_start, cell_rad, skeys, spos, aniso, fdense, cnt_w);
    else
        field_tiles<BT, 2>(g, fp, stage, cnt, n_tiles_dev, next, list, cell_start, cell_rad, skeys, spos, aniso, fdense, cnt_w);
}

// the listed tiles of a bitmap of at most nv set bits
template <int K>
static uint64_t field_tile_most(const pms_grid& g, uint64_t nv) {
    using T = FieldTile<K>;
    const uint64_t n = (uint64_t)((g.scres[0] + T::X - 1) / T::X) * ((g.scres[1] + T::Y - 1) / T::Y) * ((g.scres[2] + T::Z - 1) / T::Z);
    return std::min<uint64_t>(n, nv);
}
template <int K>
static size_t field_tile_bytes_of(const pms_grid& g, uint64_t nv) {
    return 4 * (size_t)(3 + K) * (field_tile_most<K>(g, nv) + 1);
}
// (room for any choice: the number of vertices is the device's)
size_t field_tile_bytes(const pms_grid& g, uint64_t nv) {
    return std::max(field_tile_bytes_of<1>(g, nv), std::max(field_tile_bytes_of<2>(g, nv), field_tile_bytes_of<4>(g, nv)));
}

// pick_k's lines for this frame, and the choice itself where the host knows it (else 0): a shape
// that was set, or the middle one where nothing asks for 4 and even a block of so many particles
// has a band above `few`: at two cells 24,389 have 171,000 vertices at h = 2, 200,000 at h = 3; at
// h = 1 24,389 have 94,000 and 64,000 have 214,000.  (Field stage there, the middle one / by the
// device's count: 27,000 particles 26.6 / 24.6 us, 39,304 and 64,000 equal.)
static int field_pick(const pms_ctx* ctx, FieldPick& p) {
    p.few = 160000u;
    p.many = 0xffffffffu;
    if (ctx->tune.field_vpt) return ctx->tune.field_vpt;
    const pms_params& P = ctx->prm;
    const pms_grid& g = ctx->grid;
    // the particles' share of their bounding box (the scalar grid has 2 h around it)
    double box = 1.0;
    for (int k = 0; k < 3; ++k)
        box *= std::max((double)g.scmax_pos[k] - (double)g.scmin_pos[k] - 4.0 * P.h, (double)P.particle_spacing);
    const double sp = P.particle_spacing;
    const bool sparse = (double)ctx->n * sp * sp * sp < 0.1 * box;
    if (P.sc_scale >= 3) p.many = 500000u;
    else if (P.sc_scale == 2 && (P.smoothing_radius_ratio >= 4 || sparse)) p.many = 1000000u;
    return p.many == 0xffffffffu && P.sc_scale == 2 && ctx->n >= (P.smoothing_radius_ratio >= 2 ? 24576u : 65536u) ? 2 : 0;
}

template <int K>
static pms_status field_tiles_of(pms_ctx* ctx, const FieldPick& pick, const uint32_t* bm, uint64_t n_host) {
    const KGrid g = kgrid_of(ctx->grid);
    const pms_params& P = ctx->prm;
    FieldParams fp;
    fp.h = P.h;
    fp.thr = 2.f * P.iso_value;
    fp.grow = kSupportGrow;
    fp.quick = 0.f;
    fp.ext_unit = extent_unit(P.h);
    Counters* cnt = ctx->counters.as<Counters>();
    constexpr int kGrid = K ? K : 2;            // what sizes the launches (both loop over what there is)
    PMS_CUDA(ctx, ctx->ftiles.ensure_grow(field_tile_bytes(ctx->grid, n_host)));
    uint32_t* list = ctx->ftiles.as<uint32_t>();
    // the list's length and the next ticket start at 0: the band left them so, for one launch
    if (!ctx->field_tickets_zero) PMS_CUDA(ctx, cudaMemsetAsync(&cnt->n_items, 0, 2 * sizeof(uint32_t), ctx->stream));
    ctx->field_tickets_zero = false;
    k_field_tile_list<K><<<grid_for(field_tile_most<kGrid>(ctx->grid, ~0ull), 256), 256, 0, ctx->stream>>>(g, pick, bm, &cnt->n_items, list);
    PMS_LAUNCHED(ctx);
    const int bt = ctx->tune.field_threads;
    const unsigned per_sm = kFieldWarps * 32u / (unsigned)bt;
    const unsigned blocks = grid_for(field_tile_most<kGrid>(ctx->grid, n_host), (unsigned)bt / 32u, 152u * per_sm);
    auto go = [&](auto kern) {
        kern<<<blocks, bt, 0, ctx->stream>>>(g, fp, pick, cnt, &cnt->n_items, &cnt->field_next, list,
                                             ctx->cell_start.as<uint32_t>(), ctx->cell_rad.as<float>(),
                                             ctx->skeys.as<uint32_t>(), ctx->spos.as<float4>(), ctx->aniso.as<float4>(),
                                             ctx->fdense.as<float>(), cnt);
    };
    if (bt == 64) go(k_field_tiles<64, K>);
    else if (bt == 256) go(k_field_tiles<256, K>);
    else go(k_field_tiles<128, K>);
    PMS_LAUNCHED(ctx);
    return PMS_OK;
}

pms_status launch_field_bits(pms_ctx* ctx, const uint32_t* bm, uint64_t n_host, const uint32_t* n_dev) {
    FieldPick pick = {0u, 0u, n_dev};
    switch (field_pick(ctx, pick)) {
        case 1: return field_tiles_of<1>(ctx, pick, bm, n_host);
        case 2: return field_tiles_of<2>(ctx, pick, bm, n_host);
        case 4: return field_tiles_of<4>(ctx, pick, bm, n_host);
        default: return field_tiles_of<0>(ctx, pick, bm, n_host);
    }
}

// ---------------------------------------------------------------------------
// per-cell culling record for the certification: the bounding box of the cell's
// particles and the square of the largest support among them (h, or the
// cell's largest maxvalue * h), grown by kSupportGrow.  A vertex farther than
// that from the box gets exactly 0 from every particle of the cell.  An empty
// cell gets r^2 = -1, which no vertex reaches.
// rec[2c] = {min x, min y, min z, r^2}, rec[2c + 1] = {max x, max y, max z, 0}.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(128) k_cell_records(const uint32_t* __restrict__ cell_start,
                                                           const float4* __restrict__ spos,
                                                           const float* __restrict__ cell_rad, float h, uint32_t S,
                                                           float4* __restrict__ rec) {
    for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < S; c += gridDim.x * blockDim.x) {
        const uint32_t j0 = cell_start[c], j1 = cell_start[c + 1];
        if (j0 == j1) {
            rec[2 * (size_t)c] = make_float4(0.f, 0.f, 0.f, -1.f);
            continue;
        }
        const float4 q = spos[j0];
        float lx = q.x, ly = q.y, lz = q.z, hx = q.x, hy = q.y, hz = q.z;
        for (uint32_t j = j0 + 1; j < j1; ++j) {
            const float4 p = spos[j];
            lx = fminf(lx, p.x); ly = fminf(ly, p.y); lz = fminf(lz, p.z);
            hx = fmaxf(hx, p.x); hy = fmaxf(hy, p.y); hz = fmaxf(hz, p.z);
        }
        const float r = fmaxf(cell_rad[c], h) * kSupportGrow;
        rec[2 * (size_t)c] = make_float4(lx, ly, lz, r * r);
        rec[2 * (size_t)c + 1] = make_float4(hx, hy, hz, 0.f);
    }
}

// Work items over vlist[0 .. *n_dev): group g = entries [g K, g K + K) splits
// into its runs of x-neighbours (id + 1 in the same row); count, then write.
__global__ void __launch_bounds__(256) k_field_items(const uint32_t* __restrict__ vlist, const uint32_t* __restrict__ n_dev,
                                                     uint32_t ngroups, uint32_t K, uint32_t rx,
                                                     const uint32_t* __restrict__ offs, uint32_t* __restrict__ out) {
    const uint32_t n = *n_dev;
    for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < ngroups; g += gridDim.x * blockDim.x) {
        const uint32_t t0 = g * K, t1 = min(t0 + K, n);
        uint32_t runs = 0, start = t0, o = offs ? offs[g] : 0u;
        for (uint32_t t = t0; t < t1; ++t) {
            const uint32_t id = __ldg(&vlist[t]);
            const bool join = t > t0 && id == __ldg(&vlist[t - 1]) + 1u && id % rx != 0u;
            if (t > t0 && !join) {
                if (offs) out[o + runs] = start | ((t - start - 1u) << kItemShift);
                ++runs;
                start = t;
            }
        }
        if (t0 < t1) {
            if (offs) out[o + runs] = start | ((t1 - start - 1u) << kItemShift);
            ++runs;
        }
        if (!offs) out[g] = runs;
    }
}

// The certification's launch shape, which the field's tuned shape says nothing about: runs of two,
// 128 threads, 8 waves of blocks.  Crown 2M: 0.81 ms; 64 or 256 threads 0.80 / 0.83, 2, 4 or 16 waves
// 0.89 / 0.84 / 0.81.
static constexpr uint32_t kCertRun = 2u;
static constexpr unsigned kCertThreads = 128u, kCertWaves = 8u;

pms_status launch_field_cert(pms_ctx* ctx, const uint32_t* vlist, const uint32_t* n_dev, uint32_t n_host, uint32_t* cert,
                             uint32_t* n_cert) {
    const KGrid g = kgrid_of(ctx->grid);
    const pms_params& P = ctx->prm;
    FieldParams fp;
    fp.h = P.h;
    fp.thr = P.iso_value;
    fp.grow = kSupportGrow;
    fp.quick = P.iso_value * (1.f + 1.f / 512.f);
    fp.ext_unit = 0.f;
    Counters* cnt = ctx->counters.as<Counters>();
    if (n_host >= kMaxBand) return pms_fail(ctx, PMS_ERR_UNSUPPORTED, "band above 2^29 vertices");
    constexpr uint32_t K = kCertRun;
    const uint32_t ngroups = (n_host + K - 1u) / K;
    PMS_CUDA(ctx, ctx->fitem_cnt.ensure(4 * ((size_t)ngroups + 1)));
    PMS_CUDA(ctx, ctx->fitem_off.ensure(4 * ((size_t)ngroups + 1)));
    PMS_CUDA(ctx, ctx->fitems.ensure(4 * ((size_t)n_host + 1)));
    k_cell_records<<<grid_for(g.sp_size, 128), 128, 0, ctx->stream>>>(ctx->cell_start.as<uint32_t>(), ctx->spos.as<float4>(),
                                                                      ctx->cell_rad.as<float>(), P.h, g.sp_size,
                                                                      ctx->cell_rec.as<float4>());
    PMS_LAUNCHED(ctx);
    const unsigned gb = grid_for(ngroups, 256);
    k_field_items<<<gb, 256, 0, ctx->stream>>>(vlist, n_dev, ngroups, K, g.scres[0], nullptr, ctx->fitem_cnt.as<uint32_t>());
    PMS_LAUNCHED(ctx);
    pms_status st = scan_u32(ctx, ctx->fitem_cnt.as<uint32_t>(), ctx->fitem_off.as<uint32_t>(), ngroups, &cnt->n_items);
    if (st != PMS_OK) return st;
    k_field_items<<<gb, 256, 0, ctx->stream>>>(vlist, n_dev, ngroups, K, g.scres[0], ctx->fitem_off.as<uint32_t>(),
                                               ctx->fitems.as<uint32_t>());
    PMS_LAUNCHED(ctx);
    const unsigned blocks = grid_for(n_host, kCertThreads, 152u * kCertWaves * (1024u / kCertThreads));
    k_field_cert<kCertThreads, (int)kCertRun><<<blocks, kCertThreads, 0, ctx->stream>>>(
        g, fp, cnt, &cnt->n_items, ctx->fitems.as<uint32_t>(), vlist, ctx->cell_start.as<uint32_t>(), ctx->cell_rad.as<float>(),
        ctx->cell_rec.as<float4>(), ctx->spos.as<float4>(), ctx->aniso.as<float4>(), ctx->fdense.as<float>(), cert, n_cert, cnt);
    PMS_LAUNCHED(ctx);
    return PMS_OK;
}

pms_status launch_field(pms_ctx* ctx) {
    return launch_field_bits(ctx, ctx->bm.as<uint32_t>(), ctx->nv_pending ? ctx->grid.sc_size : ctx->nv,
                             &ctx->counters.as<Counters>()->nv);
}

// field[t] = fdense[vlist[t]]: the band-order field of a vertex list whose values are all computed
__global__ void __launch_bounds__(256) k_field_gather(const uint32_t* __restrict__ vlist, const uint32_t* __restrict__ n_dev,
                                                      const float* __restrict__ fdense, float* __restrict__ field) {
    const uint32_t n = *n_dev;
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x)
        field[t] = __ldg(&fdense[__ldg(&vlist[t])]);
}

pms_status launch_field_gather(pms_ctx* ctx, const uint32_t* vlist, const uint32_t* n_dev, uint32_t n_host, float* out) {
    k_field_gather<<<grid_for(n_host, 256), 256, 0, ctx->stream>>>(vlist, n_dev, ctx->fdense.as<float>(), out);
    PMS_LAUNCHED(ctx);
    return PMS_OK;
}

}  // namespace pms
