// k_common.cuh -- device helpers shared by the libpms kernels.
#pragma once
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>
#include "pms_internal.h"

namespace pms {

// Grid parameters passed to kernels by value (lives in the kernel's constant bank).
struct KGrid {
    float min_pos[3], scmin_pos[3];
    float sp_cs, sc_cs;
    uint32_t spres[3], scres[3];
    int32_t spexpand, scexpand, spexpand_diffuse;
    uint32_t sp_size, sc_size;
    float margin, pad;        // range_margin in cells; what a cell's box is widened by, a length
};

// Margin, in cells, added to every range that the neighbour walks cut from a
// support radius, and to the cells that a tile's windows are taken from.  The
// ranges are computed from the point's position in cell units, u = (p - min) / cell:
// the difference, the reciprocal, the product and the sum with the radius are each
// rounded by up to 2^-24 of u, as are the difference and the quotient of a
// particle's key, so a cell is up to 6 x 2^-24 of the longest axis off.  0.01 cells
// cover that up to 20,971 cells per axis, 2^-21 of the axis beyond.  A cell left out
// by a cut therefore holds no particle within the support, and the cut changes no sum.
// (0.01 on every grid gave a sheet 262,144 cells from a stray particle field values
// that were up to 2 % off.)
inline float range_margin(const uint32_t res[3]) {
    return std::max(0.01f, 0x1p-21f * (float)std::max(res[0], std::max(res[1], res[2])));
}

inline KGrid kgrid_of(const pms_grid& g) {
    KGrid k;
    for (int i = 0; i < 3; ++i) {
        k.min_pos[i] = g.min_pos[i];
        k.scmin_pos[i] = g.scmin_pos[i];
        k.spres[i] = g.spres[i];
        k.scres[i] = g.scres[i];
    }
    k.sp_cs = g.sp_grid_size;
    k.sc_cs = g.sc_grid_size;
    k.spexpand = g.spexpand;
    k.scexpand = g.scexpand;
    k.spexpand_diffuse = g.spexpand_diffuse;
    k.sp_size = g.sp_size;
    k.sc_size = g.sc_size;
    k.margin = range_margin(g.spres);
    k.pad = (k.margin > 0.01f ? k.margin : 1e-4f) * g.sp_grid_size;
    return k;
}

// float -> uint with the GPU's saturating conversion (cvt.rzi.u32.f32)
__device__ __forceinline__ uint32_t f2u(float x) { return __float2uint_rz(x); }

// Spatial cell of a position: uint((p - min) / cell) per axis, each operation
// rounded separately (getIndex3D, myCuda.cuh:55-59).
__device__ __forceinline__ uint3 sp_cell(const KGrid& g, float x, float y, float z) {
    return make_uint3(f2u(__fdiv_rn(__fsub_rn(x, g.min_pos[0]), g.sp_cs)),
                      f2u(__fdiv_rn(__fsub_rn(y, g.min_pos[1]), g.sp_cs)),
                      f2u(__fdiv_rn(__fsub_rn(z, g.min_pos[2]), g.sp_cs)));
}

__device__ __forceinline__ uint32_t lin3(uint32_t x, uint32_t y, uint32_t z, const uint32_t* res) {
    return z * res[0] * res[1] + y * res[0] + x;   // uint32 arithmetic as the reference
}

// Scalar-grid vertex position (float)i * cell + min, two roundings
// (getVertexPos, myCuda.cuh:121-131).
__device__ __forceinline__ float sc_coord(const KGrid& g, uint32_t i, int axis) {
    return __fadd_rn(__fmul_rn((float)i, g.sc_cs), g.scmin_pos[axis]);
}
__device__ __forceinline__ float sc_coord_i(const KGrid& g, int i, int axis) {
    return __fadd_rn(__fmul_rn((float)i, g.sc_cs), g.scmin_pos[axis]);
}

// [c - e, c + e] with uint wrap-around then clamp to [0, res-1]: the
// reference's neighbourhood bounds (Anisotropic_kernel.cuh:176-184).
__device__ __forceinline__ void box_clamp(const KGrid& g, uint3 c, uint32_t e, uint3& lo, uint3& hi) {
    lo.x = min(max(c.x - e, 0u), g.spres[0] - 1u);
    lo.y = min(max(c.y - e, 0u), g.spres[1] - 1u);
    lo.z = min(max(c.z - e, 0u), g.spres[2] - 1u);
    hi.x = min(max(c.x + e, 0u), g.spres[0] - 1u);
    hi.y = min(max(c.y + e, 0u), g.spres[1] - 1u);
    hi.z = min(max(c.z + e, 0u), g.spres[2] - 1u);
}

// Distance^2 from a point to the axis-aligned box of spatial cell index i along one axis
// (0 inside).  The box is widened by `pad` to cover rounding of the cell keys.
__device__ __forceinline__ float axis_gap(float p, float lo, float hi) {
    float d = fmaxf(lo - p, p - hi);
    return d > 0.f ? d : 0.f;
}

__device__ __forceinline__ uint32_t ordered_bits(float f) {
    uint32_t b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float from_ordered_bits(uint32_t u) {
    uint32_t b = (u & 0x80000000u) ? (u & 0x7fffffffu) : ~u;
    return __uint_as_float(b);
}

// The frame's counters into the context's mapped pinned mirror, by one block: the last work of a
// kernel whose results the host waits for (a launch of its own costs 2.6 us).
__device__ __forceinline__ void publish_counters(const Counters* cnt, uint32_t* mirror) {
    const uint32_t* src = reinterpret_cast<const uint32_t*>(cnt);
    for (uint32_t i = threadIdx.x; i < sizeof(Counters) / 4; i += blockDim.x) mirror[i] = __ldcg(&src[i]);
}

// Cells per stretch of a row that keeps its particles' largest support (the row's own largest
// is often a lone particle's far along it).
constexpr int kRadSeg = 8;
__host__ __device__ __forceinline__ uint32_t rad_segments(uint32_t res_x) { return (res_x + kRadSeg - 1u) / kRadSeg; }

// Relative margin on support radii used for culling: a particle's kernel is
// non-zero only within its support (|G r| < 1 implies |r| < maxvalue * h), and
// float rounding of |G r|^2 moves that edge by ~1e-6 relative at most.
constexpr float kSupportGrow = 1.0001f;

// The half extents of the box around a particle's support {r : |G r| < 1}, per axis,
// packed into the low 24 bits of a word as multiples of extent_unit(h), rounded up and
// grown; bit 24 marks extents past the coded range (no culling).  The largest support is
// 4^(2/3) h (the eigenvalue clamp), so steps of 2.6 h / 255 cover every particle.
constexpr float kExtentRange = 2.6f;
__host__ __device__ __forceinline__ float extent_unit(float h) { return h * (kExtentRange / 255.f); }
__device__ __forceinline__ uint32_t pack_extents(float ex, float ey, float ez, float h) {
    const float s = 1.002f * (255.f / kExtentRange) / h;
    const float a = ceilf(ex * s), b = ceilf(ey * s), c = ceilf(ez * s);
    if (!(a <= 255.f && b <= 255.f && c <= 255.f)) return 1u << 24;
    return (uint32_t)a | (uint32_t)b << 8 | (uint32_t)c << 16;
}
__device__ __forceinline__ void unpack_extents(uint32_t p, float unit, float& ex, float& ey, float& ez) {
    ex = (float)(p & 0xffu) * unit;
    ey = (float)((p >> 8) & 0xffu) * unit;
    ez = (float)((p >> 16) & 0xffu) * unit;
    if (p >> 24) ex = ey = ez = __int_as_float(0x7f800000);
}

// First and one-past-last cell of [u - rc, u + rc] along one axis, clipped to [lo, hi).
__device__ __forceinline__ void cell_range(float u, float rc, uint32_t lo, uint32_t hi, int& a, int& b) {
    a = max((int)floorf(u - rc), (int)lo);
    b = min((int)floorf(u + rc) + 1, (int)hi);
}

// Row-segment neighbour walk of one point.  Cells are sorted by key and key =
// (z * res_y + y) * res_x + x, so the cells x in [xa, xb) of one row hold the
// contiguous particle range [cell_start[row + xa], cell_start[row + xb]).  The
// walk visits only the slabs z and rows y of the window [lo, hi) (hi
// exclusive) that come within sqrt(r2) of p, each row cut to the cells the
// sphere reaches, and body(j) runs over the particle ranges in the reference's
// z, y, x, particle order.  cell_start must have sp_size + 1 entries.
template <class Body>
__device__ __forceinline__ void row_walk(const KGrid& g, float3 p, uint3 lo, uint3 hi, float r2, float pad,
                                         const uint32_t* __restrict__ cell_start, Body&& body) {
    const uint32_t srx = g.spres[0], srxy = g.spres[0] * g.spres[1];
    const float cs = g.sp_cs, inv = 1.f / g.sp_cs;
    const float ux = (p.x - g.min_pos[0]) * inv, uy = (p.y - g.min_pos[1]) * inv, uz = (p.z - g.min_pos[2]) * inv;
    int za, zb;
    cell_range(uz, sqrtf(r2) * inv + g.margin, lo.z, hi.z, za, zb);
    for (int z = za; z < zb; ++z) {
        const float z0 = g.min_pos[2] + (float)z * cs;
        const float gz0 = axis_gap(p.z, z0 - pad, z0 + cs + pad);
        const float gz = gz0 * gz0;
        if (gz >= r2) continue;
        int ya, yb;
        cell_range(uy, sqrtf(r2 - gz) * inv + g.margin, lo.y, hi.y, ya, yb);
        for (int y = ya; y < yb; ++y) {
            const float y0 = g.min_pos[1] + (float)y * cs;
            const float gy0 = axis_gap(p.y, y0 - pad, y0 + cs + pad);
            const float gyz = gz + gy0 * gy0;
            if (gyz >= r2) continue;
            int xa, xb;
            cell_range(ux, sqrtf(r2 - gyz) * inv + g.margin, lo.x, hi.x, xa, xb);
            if (xa >= xb) continue;
            const uint32_t row = (uint32_t)z * srxy + (uint32_t)y * srx;
            const uint32_t ja = __ldg(&cell_start[row + (uint32_t)xa]), jb = __ldg(&cell_start[row + (uint32_t)xb]);
#pragma unroll 2
            for (uint32_t j = ja; j < jb; ++j) body(j);
        }
    }
}

// A warp's list of up to 32 index ranges, one per lane, as one sequence: `off` + position is
// the index in the range that holds the position.
struct WarpRows {
    uint32_t incl, off, total;
};
__device__ __forceinline__ WarpRows warp_rows(uint32_t first, uint32_t n) {
    uint32_t incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
        if ((threadIdx.x & 31u) >= (uint32_t)o) incl += v;
    }
    return {incl, first - (incl - n), __shfl_sync(0xffffffffu, incl, 31)};
}
// the range (lane) holding position p: the first whose inclusive count exceeds it
__device__ __forceinline__ int warp_row_of(const WarpRows& w, uint32_t p) {
    int row = 0;
#pragma unroll
    for (int s = 16; s > 0; s >>= 1)
        if (__shfl_sync(0xffffffffu, w.incl, row + s - 1) <= p) row += s;
    return row;
}

// The particles of row `row` (z, y) of the slabs [za, ..) x [ya, ya + ny) whose cells come
// within sqrt(r2) of the box [b0, b1] (a point when they are equal), x cells clipped to
// [xlo, xhi): first index and count.  `pad` as in row_walk.
__device__ __forceinline__ uint32_t box_row(const KGrid& g, float3 b0, float3 b1, float r2, float pad, int z, int y, int xlo,
                                            int xhi, const uint32_t* __restrict__ cell_start, uint32_t& first) {
    const float cs = g.sp_cs, inv = 1.f / g.sp_cs;
    const float z0 = g.min_pos[2] + (float)z * cs, y0 = g.min_pos[1] + (float)y * cs;
    const float gz = fmaxf(fmaxf(z0 - pad - b1.z, b0.z - (z0 + cs + pad)), 0.f);
    const float gy = fmaxf(fmaxf(y0 - pad - b1.y, b0.y - (y0 + cs + pad)), 0.f);
    const float gap = gz * gz + gy * gy;
    if (gap >= r2) return 0u;
    const float rc = sqrtf(r2 - gap) * inv + g.margin;
    const int xa = max((int)floorf((b0.x - g.min_pos[0]) * inv - rc), xlo);
    const int xb = min((int)floorf((b1.x - g.min_pos[0]) * inv + rc) + 1, xhi);
    if (xa >= xb) return 0u;
    const uint32_t row = ((uint32_t)z * g.spres[1] + (uint32_t)y) * g.spres[0];
    first = __ldg(&cell_start[row + (uint32_t)xa]);
    return __ldg(&cell_start[row + (uint32_t)xb]) - first;
}

// Every particle in the window [lo, hi) (hi exclusive) whose cell comes within sqrt(r2) of p,
// 32 at a time, one per lane: body(valid, j) for all lanes together, in ascending order.
template <class Body>
__device__ __forceinline__ void warp_walk(const KGrid& g, float3 p, uint3 lo, uint3 hi, float r2, float pad,
                                          const uint32_t* __restrict__ cell_start, Body&& body) {
    const uint32_t lane = threadIdx.x & 31u;
    const float inv = 1.f / g.sp_cs, rc = sqrtf(r2) * inv + g.margin;
    int za, zb, ya, yb;
    cell_range((p.z - g.min_pos[2]) * inv, rc, lo.z, hi.z, za, zb);
    cell_range((p.y - g.min_pos[1]) * inv, rc, lo.y, hi.y, ya, yb);
    const int ny = yb - ya, nrow = ny > 0 && zb > za ? ny * (zb - za) : 0;
    for (int r0 = 0; r0 < nrow; r0 += 32) {
        const int r = r0 + (int)lane;
        uint32_t first = 0u, n = 0u;
        if (r < nrow) n = box_row(g, p, p, r2, pad, za + r / ny, ya + r % ny, (int)lo.x, (int)hi.x, cell_start, first);
        const WarpRows rows = warp_rows(first, n);
        for (uint32_t q0 = 0u; q0 < rows.total; q0 += 32u) {
            const uint32_t q = q0 + lane;
            const int row = warp_row_of(rows, q);
            body(q < rows.total, __shfl_sync(0xffffffffu, rows.off, row) + q);
        }
    }
}

__device__ __forceinline__ bool bit_get(const uint32_t* bm, uint64_t nbits, uint64_t id) {
    return id < nbits && ((bm[id >> 5] >> (id & 31u)) & 1u);
}

}  // namespace pms
