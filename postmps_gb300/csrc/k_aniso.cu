// k_aniso.cu -- density of every particle and the anisotropy of every surface
// particle (weighted mean, covariance, eigen decomposition, eigenvalue clamp,
// G matrix, oriented normal, thin-feature flag).
//
// Reference: Anisotropic_kernel.cuh:158-213 (calculationOfDensity),
// 216-281 (calculationOfSmoothed), 350-519 (calculationOfTransformMatrices),
// myCuda.cuh:84-119, 193-203, 403-415 (wij, matrixMul, determinant,
// wij_density), SVD3.cuh (a float32 3x3 SVD).
//
// GB300 design: a thread, a warp or a warp per block of cells (by frame size; the sums
// are the same) walks the sorted cells around a particle; cells whose box lies beyond
// the kernel support are skipped (their contributions are exactly zero), so the
// (4e+1)^3 box shrinks to the cells that can matter, and a surface reconstruction
// leaves out the densities that nothing after it reads.  The covariance is symmetric positive definite (it is seeded
// with h^2 I), so its SVD is its eigen decomposition: a cyclic Jacobi solver
// with exact rotations runs in float32, and covariances whose condition
// number exceeds cfg.fp64_svd_cond are re-solved in float64.  Sums are
// accumulated relative to the particle's own position for accuracy.
#include <algorithm>
#include <cmath>

#include "pms_internal.h"
#include "k_common.cuh"

namespace pms {

static constexpr int kThreads = 128;
// frames of up to this many particles take a warp per particle for the density
static constexpr uint32_t kDensityWarp = 16384;
// frames from this many particles on leave out the densities that no band vertex reads (the two
// launches that find the blocks cost 3 to 8 us; frames: block 110k 478 -> 464 us, block 262k
// 418 -> 411, crown 2M 3.79 -> 3.75 ms, dam 8M 3.65 -> 2.92; a batch of 110k to 300k tanks 5.90 -> 5.93)
static constexpr uint32_t kDensityNear = 65536;
static constexpr float kSigma = 1.56668147f;      // Define.h:11, 315/(64 pi)

struct AnisoParams {
    float h, h_sq, h_inv, r2h, mass, kdens, inv_h2;
    float nn_d2;     // |u| <= h      <=>  |u|^2 <= nn_d2  (|u| = sqrt of |u|^2, rounded)
    float w_d2;      // |u| < 2h      <=>  |u|^2 <= w_d2
    int min_nn;
    uint32_t sp_size, sp_rows, spres_x;   // cells, rows of cells, cells per row
    double cond_limit;
};

// max(1 - |r|^2 / h^2, 0), every rounding spelled out: 0 beyond h
__device__ __forceinline__ float density_term(float dx, float dy, float dz, float inv_h2) {
    const float d2 = __fmaf_rn(dz, dz, __fmaf_rn(dx, dx, __fmul_rn(dy, dy)));
    return __saturatef(__fmaf_rn(-d2, inv_h2, 1.f));         // (never above 1)
}

// m / rho, 0 for rho == 0
__device__ __forceinline__ float mass_over(float mass, float r) { return r == 0.f ? 0.f : mass / r; }

// ---------------------------------------------------------------------------
// density (calculationOfDensity): rho_i = sum_j sigma/h^3 (1 - (d/h)^2)^3, d < h,
// over cells [c - e, c + e].  Also the isotropic kernel of every particle in the field's
// packed form: M = G^T G with G = I / h (off-diagonals doubled), the support's packed
// extents, and the weight (m / rho) sigma det(G) = (m / rho) sigma / h^3, 0 for rho == 0
// (the field skips such particles); the anisotropy pass overwrites the surface
// particles' entries.
//
// Three forms, chosen by the launcher:
// - k_density_tiles: a warp per block of 2 x 2 x 2 cells.  Its particles (27 at rest, one per
//   lane) share their neighbours: the warp reads each once, keeps those within h of the
//   particles' box in shared memory, and all lanes add them.  Used where every particle's
//   window [c - e, c + e] surely holds its support (e cells exceed h by the margin: the
//   sum then does not depend on the window).
// - k_density: a thread per particle over its own window, else.
// - k_density_warp: a warp per particle for frames too small to fill the GPU with
//   either, where one particle's serial walk is the pass's time.
// All add the same contributions in the same order (ascending sorted index; what lies
// beyond h adds exactly 0).  Bound by L1 (93 %: each lane loading its own neighbours)
// before, by instruction issue now: dam 8M 1.47 -> 1.17 ms, crown 2M 0.36 -> 0.28, block 4k 23 -> 7 us;
// without the blocks far from the surface dam 8M 0.45, crown 2M 0.20.
// ---------------------------------------------------------------------------
//
// The pass also writes the surface list (compactationOfParticles, Anisotropic_kernel.cuh:127-155):
// a particle of a surface cell takes the cell's place in the scan of the surface counts plus
// its own in the cell (a launch of its own took 30 us on 8M particles).
struct SurfaceList {
    const uint2* __restrict__ cell_info;      // {first particle, count | surface << 31}
    const uint32_t* __restrict__ surf_start;
    uint32_t* __restrict__ list;
};
__device__ __forceinline__ void put_density(const AnisoParams& ap, const SurfaceList& sl, uint32_t i, uint32_t key, float w,
                                            uint32_t ext, float* __restrict__ rho, float4* __restrict__ aniso) {
    const uint2 ci = __ldg(&sl.cell_info[key]);
    if (ci.y & 0x80000000u) sl.list[__ldg(&sl.surf_start[key]) + (i - ci.x)] = i;
    const float r = ap.kdens * w, inv_h2 = ap.h_inv * ap.h_inv;
    rho[i] = r;
    aniso[2 * (size_t)i + 0] = make_float4(inv_h2, 0.f, 0.f, __uint_as_float(ext));
    aniso[2 * (size_t)i + 1] = make_float4(inv_h2, 0.f, inv_h2, mass_over(ap.mass, r) * ap.kdens);
}

template <int BT>
__global__ void __launch_bounds__(BT, 1024 / BT) k_density(KGrid g, AnisoParams ap, SurfaceList sl,
                                                      const uint32_t* __restrict__ skeys,
                                                      const uint32_t* __restrict__ cell_start, const float4* __restrict__ spos,
                                                      float* __restrict__ rho, float4* __restrict__ aniso, uint32_t n) {
    const uint32_t rx = g.spres[0], rxy = g.spres[0] * g.spres[1];
    const float pad = g.pad;
    const uint32_t ext = pack_extents(ap.h, ap.h, ap.h, ap.h);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4 pi4 = spos[i];
        const float3 p = make_float3(pi4.x, pi4.y, pi4.z);
        const uint32_t key = skeys[i];
        const uint3 c = make_uint3(key % rx, (key / rx) % g.spres[1], key / rxy);
        uint3 lo, hi;
        box_clamp(g, c, (uint32_t)g.spexpand, lo, hi);
        hi = make_uint3(hi.x + 1, hi.y + 1, hi.z + 1);
        // sum of max(1 - d^2/h^2, 0)^3, times sigma / h^3 once at the end
        float w = 0.f;
        row_walk(g, p, lo, hi, ap.h_sq, pad, cell_start, [&](uint32_t j) {
            const float4 q = __ldg(&spos[j]);
            const float s = density_term(p.x - q.x, p.y - q.y, p.z - q.z, ap.inv_h2);
            w = fmaf(s * s, s, w);
        });
        put_density(ap, sl, i, key, w, ext, rho, aniso);
    }
}

// a warp per particle: the lanes work out 32 neighbours' terms, then add the non-zero ones in
// their order
__global__ void __launch_bounds__(kThreads) k_density_warp(KGrid g, AnisoParams ap, SurfaceList sl,
                                                           const uint32_t* __restrict__ skeys,
                                                           const uint32_t* __restrict__ cell_start,
                                                           const float4* __restrict__ spos, float* __restrict__ rho,
                                                           float4* __restrict__ aniso, uint32_t n) {
    const uint32_t rx = g.spres[0], rxy = g.spres[0] * g.spres[1], lane = threadIdx.x & 31u;
    const float pad = g.pad;
    const uint32_t ext = pack_extents(ap.h, ap.h, ap.h, ap.h);
    for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += (gridDim.x * blockDim.x) >> 5) {
        const float4 pi4 = spos[i];
        const float3 p = make_float3(pi4.x, pi4.y, pi4.z);
        const uint32_t key = skeys[i];
        const uint3 c = make_uint3(key % rx, (key / rx) % g.spres[1], key / rxy);
        uint3 lo, hi;
        box_clamp(g, c, (uint32_t)g.spexpand, lo, hi);
        hi = make_uint3(hi.x + 1, hi.y + 1, hi.z + 1);
        float w = 0.f;
        warp_walk(g, p, lo, hi, ap.h_sq, pad, cell_start, [&](bool valid, uint32_t j) {
            float s = 0.f;
            if (valid) {
                const float4 q = __ldg(&spos[j]);
                s = density_term(p.x - q.x, p.y - q.y, p.z - q.z, ap.inv_h2);
            }
            const float ss = s * s;
            for (uint32_t m = __ballot_sync(0xffffffffu, s > 0.f); m; m &= m - 1u) {
                const int l = __ffs((int)m) - 1;
                w = fmaf(__shfl_sync(0xffffffffu, ss, l), __shfl_sync(0xffffffffu, s, l), w);
            }
        });
        if (lane == 0u) put_density(ap, sl, i, key, w, ext, rho, aniso);
    }
}

static constexpr int kDensX = 2, kDensY = 2, kDensZ = 2;      // cells of a block
static constexpr int kDensStage = 64;
static constexpr uint32_t kDensEntry = 64;                     // most particles of an entry of the pass's list

// Which blocks of cells a density pass works on.  A frame whose fields are asked for only at
// its band needs the densities near the surface: a band vertex lies within h per axis of a
// surface particle, or one scalar cell further (the dilation), and a particle counts at a
// vertex, or at a mesh vertex's scalar values, within h of it.  Blocks further than
// 2 h + one scalar cell from every surface cell are "far": kNear writes density 0, whose
// contribution nothing reads, for their particles; kFar makes theirs alone (launch_density_rest).
enum class DensBlocks { kAll, kNear, kFar };
static constexpr uint32_t kFarBlock = 1u << 31;               // (a grid holds less than 2^32 / 8 blocks)

// a bit per block with a surface cell, the blocks of a row along x in whole words: a warp a word
__global__ void __launch_bounds__(256) k_density_surface(KGrid g, uint3 bd, uint32_t wx, const uint2* __restrict__ cell_info,
                                                         uint32_t* __restrict__ bits) {
    const uint32_t nw = wx * bd.y * bd.z, lane = threadIdx.x & 31u;
    for (uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < nw; w += (gridDim.x * blockDim.x) >> 5) {
        const uint32_t bx = (w % wx) * 32u + lane, y0 = w / wx % bd.y * kDensY, z0 = w / wx / bd.y * kDensZ;
        uint32_t any = 0u;
        if (bx < bd.x) {
            const uint32_t x0 = bx * kDensX, x1 = min(x0 + kDensX, g.spres[0]);
            for (uint32_t z = z0; z < min(z0 + kDensZ, g.spres[2]); ++z)
                for (uint32_t y = y0; y < min(y0 + kDensY, g.spres[1]); ++y)
                    for (uint32_t x = x0; x < x1; ++x) any |= __ldg(&cell_info[(z * g.spres[1] + y) * g.spres[0] + x].y);
        }
        const uint32_t vote = __ballot_sync(0xffffffffu, (any >> 31) != 0u);
        if (lane == 0u) bits[w] = vote;
    }
}

// the work of the pass, an entry {block, which kDensEntry of its particles} each: the blocks that hold
// particles (and, for kNear, whether they are far), a warp per 32 blocks along x.  A block at rest is
// one entry; a frame of crowded cells has few blocks, and a warp per block then leaves the GPU idle
// (anisotropy stage of 300,000 particles, 200 or 1000 to a cell: 25 / 268 ms with a warp per block,
// 6.7 / 26 with a thread per particle, 5.7 / 22 so; entries of 32: 5.5 / 21, but crown and dam frames
// 0.2 to 0.5 % slower).
__global__ void __launch_bounds__(256) k_density_list(KGrid g, uint3 bd, uint32_t wx, DensBlocks which, int reach,
                                                      const uint32_t* __restrict__ bits, const uint32_t* __restrict__ cell_start,
                                                      uint32_t* __restrict__ n_entries, uint2* __restrict__ list) {
    constexpr unsigned kAll = 0xffffffffu;
    const uint32_t nw = wx * bd.y * bd.z, lane = threadIdx.x & 31u;
    for (uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < nw; w += (gridDim.x * blockDim.x) >> 5) {
        const uint32_t wi = w % wx, bx = wi * 32u + lane, by = w / wx % bd.y, bz = w / wx / bd.y;
        const uint32_t t = (bz * bd.y + by) * bd.x + bx;
        uint32_t m = 0u;
        if (bx < bd.x) {
            const uint32_t x0 = bx * kDensX, y0 = by * kDensY, z0 = bz * kDensZ, x1 = min(x0 + kDensX, g.spres[0]);
#pragma unroll
            for (int k = 0; k < kDensY * kDensZ; ++k) {
                const uint32_t y = y0 + k % kDensY, z = z0 + k / kDensY;
                if (y >= g.spres[1] || z >= g.spres[2]) continue;
                const uint32_t row = (z * g.spres[1] + y) * g.spres[0];
                m += __ldg(&cell_start[row + x1]) - __ldg(&cell_start[row + x0]);
            }
        }
        uint32_t vote = __ballot_sync(kAll, m != 0u), near = kAll;
        if (which != DensBlocks::kAll && vote) {
            // the surface bits of the (2 reach + 1)^2 rows of blocks around, spread by reach along x
            const int side = 2 * reach + 1;
            near = 0u;
            for (int r = (int)lane; r < side * side; r += 32) {
                const int y = (int)by + r % side - reach, z = (int)bz + r / side - reach;
                if (y < 0 || z < 0 || y >= (int)bd.y || z >= (int)bd.z) continue;
                const uint32_t* row = bits + ((uint32_t)z * bd.y + (uint32_t)y) * wx;
                const uint32_t c = __ldg(&row[wi]), lo = wi ? __ldg(&row[wi - 1u]) : 0u, hi = wi + 1u < wx ? __ldg(&row[wi + 1u]) : 0u;
                near |= c;
                for (int s = 1; s <= reach; ++s)
                    near |= __funnelshift_l(lo, c, s) | __funnelshift_r(c, hi, s);
            }
            near = __reduce_or_sync(kAll, near);
            if (which == DensBlocks::kFar) vote &= ~near;
        }
        if (!vote) continue;
        const uint32_t parts = (vote >> lane) & 1u ? (m + kDensEntry - 1u) / kDensEntry : 0u;
        const WarpRows at = warp_rows(0u, parts);
        uint32_t base = 0u;
        if (lane == 0u) base = atomicAdd(n_entries, at.total);
        base = __shfl_sync(kAll, base, 0) + at.incl - parts;
        const uint32_t tag = t | (which == DensBlocks::kNear && !((near >> lane) & 1u) ? kFarBlock : 0u);
        for (uint32_t k = 0u; k < parts; ++k) list[base + k] = make_uint2(tag, k);
    }
}

__device__ __forceinline__ float warp_min(float v) { return from_ordered_bits(__reduce_min_sync(0xffffffffu, ordered_bits(v))); }
__device__ __forceinline__ float warp_max(float v) { return from_ordered_bits(__reduce_max_sync(0xffffffffu, ordered_bits(v))); }

template <int BT>
__global__ void __launch_bounds__(BT, 1024 / BT) k_density_tiles(KGrid g, AnisoParams ap, SurfaceList sl, uint3 bd,
                                                                 const uint32_t* __restrict__ skeys,
                                                                 const uint32_t* __restrict__ n_entries_dev,
                                                                 uint32_t* __restrict__ next, const uint2* __restrict__ list,
                                                                 const uint32_t* __restrict__ cell_start,
                                                                 const float4* __restrict__ spos, float* __restrict__ rho,
                                                                 float4* __restrict__ aniso) {
    constexpr unsigned kAll = 0xffffffffu;
    __shared__ float4 stage_all[BT / 32][kDensStage];
    float4* stage = stage_all[threadIdx.x >> 5];
    const uint32_t lane = threadIdx.x & 31u, n_entries = *n_entries_dev;
    const float pad = g.pad, inv_cs = 1.f / g.sp_cs;
    const float rc = ap.h * inv_cs + g.margin, reach2 = ap.h_sq * 1.001f;
    const uint32_t ext = pack_extents(ap.h, ap.h, ap.h, ap.h);
    for (;;) {
        uint32_t bi = 0u;
        if (lane == 0u) bi = atomicAdd(next, 1u);
        bi = __shfl_sync(kAll, bi, 0);
        if (bi >= n_entries) break;
        const uint2 entry = __ldg(&list[bi]);
        const uint32_t t = entry.x & ~kFarBlock;
        // the block's particles: a contiguous range per row of cells
        const uint32_t x0 = t % bd.x * kDensX, y0 = t / bd.x % bd.y * kDensY, z0 = t / bd.x / bd.y * kDensZ;
        uint32_t first = 0u, n = 0u;
        if (lane < kDensY * kDensZ) {
            const uint32_t y = y0 + lane % kDensY, z = z0 + lane / kDensY;
            if (y < g.spres[1] && z < g.spres[2]) {
                const uint32_t row = (z * g.spres[1] + y) * g.spres[0];
                first = __ldg(&cell_start[row + x0]);
                n = __ldg(&cell_start[row + min(x0 + kDensX, g.spres[0])]) - first;
            }
        }
        const WarpRows mine = warp_rows(first, n);
        const uint32_t end = min((entry.y + 1u) * kDensEntry, mine.total);
        for (uint32_t t0 = entry.y * kDensEntry; t0 < end; t0 += 32u) {
            // lanes past the block's particles repeat its last one
            const uint32_t own = min(t0 + lane, mine.total - 1u);
            const int own_row = warp_row_of(mine, own);
            const uint32_t id = __shfl_sync(kAll, mine.off, own_row) + own;
            if (entry.x != t) {                                // a far block
                if (t0 + lane < mine.total) put_density(ap, sl, id, __ldg(&skeys[id]), 0.f, ext, rho, aniso);
                continue;
            }
            const float4 pi4 = __ldg(&spos[id]);
            const float3 b0 = make_float3(warp_min(pi4.x), warp_min(pi4.y), warp_min(pi4.z));
            const float3 b1 = make_float3(warp_max(pi4.x), warp_max(pi4.y), warp_max(pi4.z));
            float w = 0.f;
            int staged = 0;
            auto flush = [&]() {
                __syncwarp();
#pragma unroll 4
                for (int i = 0; i < staged; ++i) {
                    const float4 q = stage[i];
                    const float s = density_term(pi4.x - q.x, pi4.y - q.y, pi4.z - q.z, ap.inv_h2);
                    w = __fmaf_rn(__fmul_rn(s, s), s, w);
                }
                __syncwarp();
                staged = 0;
            };
            const int za = max((int)floorf((b0.z - g.min_pos[2]) * inv_cs - rc), 0);
            const int zb = min((int)floorf((b1.z - g.min_pos[2]) * inv_cs + rc) + 1, (int)g.spres[2]);
            const int ya = max((int)floorf((b0.y - g.min_pos[1]) * inv_cs - rc), 0);
            const int yb = min((int)floorf((b1.y - g.min_pos[1]) * inv_cs + rc) + 1, (int)g.spres[1]);
            const int ny = yb - ya, nrow = ny > 0 && zb > za ? ny * (zb - za) : 0;
            for (int r0 = 0; r0 < nrow; r0 += 32) {
                const int r = r0 + (int)lane;
                uint32_t ja = 0u, m = 0u;
                if (r < nrow) m = box_row(g, b0, b1, ap.h_sq, pad, za + r / ny, ya + r % ny, 0, (int)g.spres[0], cell_start, ja);
                const WarpRows rows = warp_rows(ja, m);
                for (uint32_t p0 = 0u; p0 < rows.total; p0 += 32u) {
                    const uint32_t p = p0 + lane;
                    const int row = warp_row_of(rows, p);
                    const uint32_t j = __shfl_sync(kAll, rows.off, row) + p;
                    float4 q;
                    bool keep = false;
                    if (p < rows.total) {
                        q = __ldg(&spos[j]);
                        const float ex = fmaxf(fmaxf(b0.x - q.x, q.x - b1.x), 0.f), ey = fmaxf(fmaxf(b0.y - q.y, q.y - b1.y), 0.f),
                                    ez = fmaxf(fmaxf(b0.z - q.z, q.z - b1.z), 0.f);
                        keep = ex * ex + ey * ey + ez * ez < reach2;
                    }
                    const uint32_t kept = __ballot_sync(kAll, keep);
                    if (keep) stage[staged + __popc(kept & ((1u << lane) - 1u))] = q;
                    staged += __popc(kept);
                    if (staged > kDensStage - 32) flush();
                }
            }
            if (staged) flush();
            if (t0 + lane < mine.total) put_density(ap, sl, id, __ldg(&skeys[id]), w, ext, rho, aniso);
        }
    }
}

// ---------------------------------------------------------------------------
// symmetric 3x3 eigen decomposition, cyclic Jacobi with exact rotations
// (Golub & Van Loan, Algorithm 8.4.2 / the classical Jacobi method)
// ---------------------------------------------------------------------------
template <class T>
__device__ __forceinline__ void jacobi_rotate(T a[3][3], T v[3][3], int p, int q) {
    T apq = a[p][q];
    if (apq == T(0)) return;
    T theta = (a[q][q] - a[p][p]) / (T(2) * apq);
    T t = (theta >= T(0) ? T(1) : T(-1)) / (fabs(theta) + sqrt(theta * theta + T(1)));
    T c = T(1) / sqrt(t * t + T(1)), s = t * c;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        T akp = a[k][p], akq = a[k][q];
        a[k][p] = c * akp - s * akq;
        a[k][q] = s * akp + c * akq;
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        T apk = a[p][k], aqk = a[q][k];
        a[p][k] = c * apk - s * aqk;
        a[q][k] = s * apk + c * aqk;
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        T vkp = v[k][p], vkq = v[k][q];
        v[k][p] = c * vkp - s * vkq;
        v[k][q] = s * vkp + c * vkq;
    }
}

// On return e[0..2] are eigenvalues sorted by decreasing magnitude and
// column k of v the matching unit eigenvector.
template <class T>
__device__ __forceinline__ void eig_sym3(T a[3][3], T e[3], T v[3][3], T tol) {
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) v[i][j] = (i == j) ? T(1) : T(0);
    for (int sweep = 0; sweep < 12; ++sweep) {
        T off = fabs(a[0][1]) + fabs(a[0][2]) + fabs(a[1][2]);
        T dia = fabs(a[0][0]) + fabs(a[1][1]) + fabs(a[2][2]);
        if (off <= tol * dia) break;
        jacobi_rotate<T>(a, v, 0, 1);
        jacobi_rotate<T>(a, v, 0, 2);
        jacobi_rotate<T>(a, v, 1, 2);
    }
    T d[3] = {a[0][0], a[1][1], a[2][2]};
    int i0 = 0, i1 = 1, i2 = 2;
    if (fabs(d[i1]) > fabs(d[i0])) { int t = i0; i0 = i1; i1 = t; }
    if (fabs(d[i2]) > fabs(d[i0])) { int t = i0; i0 = i2; i2 = t; }
    if (fabs(d[i2]) > fabs(d[i1])) { int t = i1; i1 = i2; i2 = t; }
    int idx[3] = {i0, i1, i2};
    T w[3][3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        e[k] = d[idx[k]];
#pragma unroll
        for (int r = 0; r < 3; ++r) w[r][k] = v[r][idx[k]];
    }
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int k = 0; k < 3; ++k) v[r][k] = w[r][k];
}

// ---------------------------------------------------------------------------
// anisotropy, pass 1: weighted moments of the neighbourhood, one surface
// particle per thread, ONE walk over the cells.  With u = x_j - x_i and
// w = 1 - (|u| / 2h)^3 (wij with support 2h):
//   S0 = sum w, S1 = sum w u, S2 = sum w u u^T, J = #{|u| <= h}.
// The reference's two passes (mean, then covariance about the mean) follow
// from these: mean = x_i + S1/S0 and sum w (u - o)(u - o)^T = S2 - S1 S1^T / S0.
// The count and the support test compare |u|^2 with the exact bounds of the
// rounded square root (the same decisions as comparing |u|); the weight uses
// the hardware reciprocal square root (a few ulp, inside the weight's rounding).
// ---------------------------------------------------------------------------
// w = 1 - (|u| / 2h)^3 within the support, 0 beyond, 1 at the particle itself
__device__ __forceinline__ float moment_weight(float d2, float w_d2, float inv_r2h) {
    const float t = d2 * rsqrtf(d2) * inv_r2h;                       // d2 = 0 gives NaN, selected away
    return (d2 <= w_d2 && d2 > 0.f) ? __fmaf_rn(-(t * t), t, 1.f) : (d2 > 0.f ? 0.f : 1.f);
}

// Few surface particles leave the GPU idle, and the pass then takes as long as one particle's
// serial walk (about 80 us whatever the count).  So up to kMomentsWarp of them get a warp
// each: the lanes work out 32 neighbours' weights, those within the support are staged in
// shared memory in their order, and ten lanes run the ten sums over them.  Every product and
// sum is the thread-per-particle form's.  Block 4k (1353 surface particles) 79 -> 12 us; the
// two forms meet near 45,000.
static constexpr uint32_t kMomentsWarp = 32768;

template <int BT>
__device__ __forceinline__ void moments_warp(const KGrid& g, const AnisoParams& ap, const uint32_t* __restrict__ slist, uint32_t ns,
                                             const uint32_t* __restrict__ skeys, const uint32_t* __restrict__ cell_start,
                                             const float4* __restrict__ spos, float4* __restrict__ mom) {
    constexpr unsigned kAll = 0xffffffffu;
    // eight columns of staged neighbours {w, w ux, w uy, w uz, 1, ux, uy, uz}, padded so that the
    // ten lanes' 16-byte reads fall on different banks (the products made by all lanes as they
    // stage, not by the ten as they add: block 262k 64 -> 60 us)
    constexpr int kCol = 68;
    __shared__ __align__(16) float hits_all[BT / 32][8 * kCol];
    float* hits = hits_all[threadIdx.x >> 5];
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t k = lane; k < 64u; k += 32u) hits[4 * kCol + k] = 1.f;
    __syncwarp();
    const uint32_t rx = g.spres[0], rxy = g.spres[0] * g.spres[1];
    const float pad = g.pad, r2h_sq = ap.r2h * ap.r2h, inv_r2h = 1.f / ap.r2h;
    // lane q's sum adds (w f1) f2: s0 | sx sy sz | sxx sxy sxz syy syz szz
    const int f1 = lane < 4u ? (int)lane : (lane < 7u ? 1 : (lane < 9u ? 2 : 3));
    const int f2 = lane < 4u ? 4 : (lane < 7u ? (int)lane + 1 : (lane < 9u ? (int)lane - 1 : 7));
    for (uint32_t s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < ns; s += (gridDim.x * blockDim.x) >> 5) {
        const uint32_t i = slist[s];
        const float4 pi4 = spos[i];
        const float3 p = make_float3(pi4.x, pi4.y, pi4.z);
        const uint32_t key = skeys[i];
        const uint3 c = make_uint3(key % rx, (key / rx) % g.spres[1], key / rxy);
        uint3 lo, hi;
        box_clamp(g, c, 2u * (uint32_t)g.spexpand, lo, hi);
        hi = make_uint3(hi.x + 1, hi.y + 1, hi.z + 1);
        uint32_t nn = 0u;
        int staged = 0;
        float acc = 0.f;
        auto flush = [&]() {
            __syncwarp();
            if (lane < 10u) {
                const float *A = hits + kCol * f1, *B = hits + kCol * f2;
                int k = 0;
                for (; k + 4 <= staged; k += 4) {
                    const float4 a = *reinterpret_cast<const float4*>(A + k), b = *reinterpret_cast<const float4*>(B + k);
                    acc = __fmaf_rn(a.x, b.x, acc);
                    acc = __fmaf_rn(a.y, b.y, acc);
                    acc = __fmaf_rn(a.z, b.z, acc);
                    acc = __fmaf_rn(a.w, b.w, acc);
                }
                for (; k < staged; ++k) acc = __fmaf_rn(A[k], B[k], acc);
            }
            __syncwarp();
            staged = 0;
        };
        warp_walk(g, p, lo, hi, r2h_sq, pad, cell_start, [&](bool valid, uint32_t j) {
            float ux = 0.f, uy = 0.f, uz = 0.f, w = 0.f;
            bool keep = false;
            if (valid) {
                const float4 q = __ldg(&spos[j]);
                ux = __fsub_rn(q.x, p.x); uy = __fsub_rn(q.y, p.y); uz = __fsub_rn(q.z, p.z);
                const float d2 = __fadd_rn(__fadd_rn(__fmul_rn(ux, ux), __fmul_rn(uy, uy)), __fmul_rn(uz, uz));
                keep = d2 <= ap.w_d2;                        // beyond the support everything adds exactly 0
                nn += d2 <= ap.nn_d2 ? 1u : 0u;
                w = moment_weight(d2, ap.w_d2, inv_r2h);
            }
            const uint32_t kept = __ballot_sync(kAll, keep);
            if (keep) {
                float* h = hits + staged + __popc(kept & ((1u << lane) - 1u));
                h[0] = w; h[kCol] = __fmul_rn(w, ux); h[2 * kCol] = __fmul_rn(w, uy); h[3 * kCol] = __fmul_rn(w, uz);
                h[5 * kCol] = ux; h[6 * kCol] = uy; h[7 * kCol] = uz;
            }
            staged += __popc(kept);
            if (staged > 32) flush();
        });
        if (staged) flush();
        nn = __reduce_add_sync(kAll, nn);
        float v[10];
#pragma unroll
        for (int k = 0; k < 10; ++k) v[k] = __shfl_sync(kAll, acc, k);
        if (lane == 0u) {
            mom[3 * (size_t)s + 0] = make_float4(v[0], v[1], v[2], v[3]);
            mom[3 * (size_t)s + 1] = make_float4(v[4], v[5], v[6], v[7]);
            mom[3 * (size_t)s + 2] = make_float4(v[8], v[9], __uint_as_float(nn), 0.f);
        }
    }
}

template <int BT>
__global__ void __launch_bounds__(BT, 1024 / BT) k_moments(KGrid g, AnisoParams ap, const uint32_t* __restrict__ slist,
                                                      const Counters* __restrict__ cnt, const uint32_t* __restrict__ skeys,
                                                      const uint32_t* __restrict__ cell_start, const float4* __restrict__ spos,
                                                      float4* __restrict__ mom) {
    const uint32_t ns = cnt->ns;
    const uint32_t rx = g.spres[0], rxy = g.spres[0] * g.spres[1];
    const float pad = g.pad;
    const float r2h_sq = ap.r2h * ap.r2h;
    const float inv_r2h = 1.f / ap.r2h;
    if (ns <= kMomentsWarp) {
        moments_warp<BT>(g, ap, slist, ns, skeys, cell_start, spos, mom);
        return;
    }
    for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < ns; s += gridDim.x * blockDim.x) {
        const uint32_t i = slist[s];
        const float4 pi4 = spos[i];
        const float3 p = make_float3(pi4.x, pi4.y, pi4.z);
        const uint32_t key = skeys[i];
        const uint3 c = make_uint3(key % rx, (key / rx) % g.spres[1], key / rxy);
        uint3 lo, hi;
        box_clamp(g, c, 2u * (uint32_t)g.spexpand, lo, hi);
        hi = make_uint3(hi.x + 1, hi.y + 1, hi.z + 1);
        float s0 = 0.f, sx = 0.f, sy = 0.f, sz = 0.f;
        float sxx = 0.f, sxy = 0.f, sxz = 0.f, syy = 0.f, syz = 0.f, szz = 0.f;
        uint32_t nn = 0;
        row_walk(g, p, lo, hi, r2h_sq, pad, cell_start, [&](uint32_t j) {
            const float4 q = __ldg(&spos[j]);
            // |u| rounded operation by operation, as the reference's neighbour count sees it
            const float ux = __fsub_rn(q.x, p.x), uy = __fsub_rn(q.y, p.y), uz = __fsub_rn(q.z, p.z);
            const float d2 = __fadd_rn(__fadd_rn(__fmul_rn(ux, ux), __fmul_rn(uy, uy)), __fmul_rn(uz, uz));
            nn += (d2 <= ap.nn_d2) ? 1u : 0u;
            const float w = moment_weight(d2, ap.w_d2, inv_r2h);
            const float wx = __fmul_rn(w, ux), wy = __fmul_rn(w, uy), wz = __fmul_rn(w, uz);
            s0 += w; sx += wx; sy += wy; sz += wz;
            sxx = __fmaf_rn(wx, ux, sxx); sxy = __fmaf_rn(wx, uy, sxy); sxz = __fmaf_rn(wx, uz, sxz);
            syy = __fmaf_rn(wy, uy, syy); syz = __fmaf_rn(wy, uz, syz); szz = __fmaf_rn(wz, uz, szz);
        });
        mom[3 * (size_t)s + 0] = make_float4(s0, sx, sy, sz);
        mom[3 * (size_t)s + 1] = make_float4(sxx, sxy, sxz, syy);
        mom[3 * (size_t)s + 2] = make_float4(syz, szz, __uint_as_float(nn), 0.f);
    }
}

// ---------------------------------------------------------------------------
// anisotropy, pass 2: covariance, eigen decomposition, clamp, G, normal, flag
// (Anisotropic_kernel.cuh:431-518) from the moments; also the per-cell
// and per-row support radius max(maxvalue * h) that lets the field skip far
// rows and cells.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads) k_eigen(AnisoParams ap, const uint32_t* __restrict__ slist,
                                                    const Counters* __restrict__ cnt, const uint32_t* __restrict__ skeys,
                                                    const float4* __restrict__ spos, const float* __restrict__ rho,
                                                    const float4* __restrict__ mom, float4* __restrict__ aniso, float4* __restrict__ nrm4,
                                                    float4* __restrict__ mean4, float* __restrict__ gdebug,
                                                    uint32_t* __restrict__ nnb, float* __restrict__ cell_rad,
                                                    Counters* __restrict__ cnt_w) {
    const uint32_t ns = cnt->ns;
    if (blockIdx.x == 0 && threadIdx.x == 0) cnt_w->dens_entries = cnt_w->dens_next = 0u;   // the next density pass's tickets
    for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < ns; s += gridDim.x * blockDim.x) {
        const uint32_t i = slist[s];
        const float4 pi4 = spos[i];
        const float4 m0 = mom[3 * (size_t)s + 0], m1 = mom[3 * (size_t)s + 1], m2 = mom[3 * (size_t)s + 2];
        const float ws = m0.x;                               // >= 1: the particle itself
        const float ox = m0.y / ws, oy = m0.z / ws, oz = m0.w / ws;   // mean - p
        const uint32_t nn = __float_as_uint(m2.z);
        float G[3][3], nv[3], maxv, flag;
        float ext[3] = {ap.h, ap.h, ap.h};                   // half extents of the support's box
        if ((int)nn < ap.min_nn) {
            // isolated particle: isotropic kernel (Anisotropic_kernel.cuh:435-443)
#pragma unroll
            for (int a = 0; a < 3; ++a)
#pragma unroll
                for (int b = 0; b < 3; ++b) G[a][b] = (a == b) ? ap.h_inv : 0.f;
            maxv = 1.f; flag = 1.f; nv[0] = 1.f; nv[1] = 0.f; nv[2] = 0.f;
        } else {
            // (h^2 I + S2 - S1 S1^T / S0) / S0
            const float inv = 1.f / ws;
            const float c00 = (ap.h_sq + (m1.x - m0.y * ox)) * inv, c01 = (m1.y - m0.y * oy) * inv;
            const float c02 = (m1.z - m0.y * oz) * inv, c11 = (ap.h_sq + (m1.w - m0.z * oy)) * inv;
            const float c12 = (m2.x - m0.z * oz) * inv, c22 = (ap.h_sq + (m2.y - m0.w * oz)) * inv;
            float A[3][3] = {{c00, c01, c02}, {c01, c11, c12}, {c02, c12, c22}};
            float e[3], U[3][3];
            eig_sym3<float>(A, e, U, 1e-7f);
            float sv0 = fabsf(e[0]), sv1 = fabsf(e[1]), sv2 = fabsf(e[2]);
            if ((double)sv0 > ap.cond_limit * (double)sv2) {
                // ill-conditioned covariance: solve again in float64
                double Ad[3][3] = {{c00, c01, c02}, {c01, c11, c12}, {c02, c12, c22}};
                double ed[3], Ud[3][3];
                eig_sym3<double>(Ad, ed, Ud, 1e-15);
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    e[k] = (float)ed[k];
#pragma unroll
                    for (int r = 0; r < 3; ++r) U[r][k] = (float)Ud[r][k];
                }
                sv0 = fabsf(e[0]); sv1 = fabsf(e[1]); sv2 = fabsf(e[2]);
                atomicAdd(&cnt_w->n_fp64, 1u);
            }
            // clamp and scale (Anisotropic_kernel.cuh:459-509)
            const float smax = fmaxf(sv0, fmaxf(sv1, sv2)), smin = fminf(sv0, fminf(sv1, sv2));
            flag = (smin <= smax * 0.25f) ? 1.f : 0.f;
            const float lim = smax / 4.0f;
            sv0 = fmaxf(sv0, lim); sv1 = fmaxf(sv1, lim); sv2 = fmaxf(sv2, lim);
            const float scale = cbrtf(sv0 * sv1 * sv2);
            const float cof = ap.h_inv * scale;
            const float k0 = cof / sv0, k1 = cof / sv1, k2 = cof / sv2;
#pragma unroll
            for (int a = 0; a < 3; ++a)
#pragma unroll
                for (int b = 0; b < 3; ++b)
                    G[a][b] = U[a][0] * k0 * U[b][0] + U[a][1] * k1 * U[b][1] + U[a][2] * k2 * U[b][2];
            nv[0] = U[0][2]; nv[1] = U[1][2]; nv[2] = U[2][2];
            maxv = sv0 / scale;
            // the support is the ellipsoid with semi-axes 1 / k along U's columns
            const float r0 = sv0 / cof, r1 = sv1 / cof, r2 = sv2 / cof;
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const float u0 = U[a][0] * r0, u1 = U[a][1] * r1, u2 = U[a][2] * r2;
                ext[a] = sqrtf(u0 * u0 + u1 * u1 + u2 * u2);
            }
        }
        // orient the normal away from the mean (Anisotropic_kernel.cuh:512-515)
        if (nv[0] * (-ox) + nv[1] * (-oy) + nv[2] * (-oz) < 0.f) { nv[0] = -nv[0]; nv[1] = -nv[1]; nv[2] = -nv[2]; }
        // determinant as the reference evaluates it (myCuda.cuh:193-203)
        const float det = G[0][0] * G[1][1] * G[2][2] + G[0][1] * G[1][2] * G[2][0] + G[0][2] * G[1][0] * G[2][1]
                        - G[0][0] * G[1][2] * G[2][1] - G[0][1] * G[1][0] * G[2][2] - G[0][2] * G[1][1] * G[2][0];
        const float hs = maxv * ap.h;
        // the field's packed form: M = G^T G = G G (G is symmetric), off-diagonals doubled,
        // so |G r|^2 = r^T M r costs 9 multiply-adds; w = (m / rho) sigma det(G)
        float M[3][3];
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < 3; ++b) M[a][b] = G[a][0] * G[0][b] + G[a][1] * G[1][b] + G[a][2] * G[2][b];
        aniso[2 * (size_t)i + 0] = make_float4(M[0][0], 2.f * M[0][1], 2.f * M[0][2],
                                                __uint_as_float(pack_extents(ext[0], ext[1], ext[2], ap.h)));
        aniso[2 * (size_t)i + 1] = make_float4(M[1][1], 2.f * M[1][2], M[2][2],
                                                mass_over(ap.mass, rho[i]) * (kSigma * det));
        nrm4[i] = make_float4(nv[0], nv[1], nv[2], flag);
        mean4[s] = make_float4(pi4.x + ox, pi4.y + oy, pi4.z + oz, ws);
        float* gd = gdebug + 10 * (size_t)s;
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < 3; ++b) gd[3 * a + b] = G[a][b];
        gd[9] = maxv;
        nnb[s] = nn;
        // per-cell, per-row, per-stretch and global support radius (positive floats order like their bits)
        const uint32_t key = skeys[i];
        atomicMax(reinterpret_cast<unsigned int*>(&cell_rad[key]), __float_as_uint(hs));
        const uint32_t row = key / ap.spres_x, x = key - row * ap.spres_x;
        atomicMax(reinterpret_cast<unsigned int*>(&cell_rad[ap.sp_size + row]), __float_as_uint(hs));
        atomicMax(reinterpret_cast<unsigned int*>(&cell_rad[ap.sp_size + ap.sp_rows + row * rad_segments(ap.spres_x) + x / kRadSeg]),
                  __float_as_uint(hs));
        atomicMax(&cnt_w->rad_max_bits, __float_as_uint(hs));
    }
}

// Largest float x >= 0 with sqrt(x) <= r (inclusive) or sqrt(x) < r (strict),
// sqrt correctly rounded: the rounded square root is non-decreasing, so
// sqrt(x) <= r exactly when x <= that bound.
static float sqrt_bound(float r, bool inclusive) {
    auto ok = [&](float x) { const float s = std::sqrt(x); return inclusive ? s <= r : s < r; };
    float x = r * r;
    while (x > 0.f && !ok(x)) x = std::nextafter(x, 0.f);
    while (ok(std::nextafter(x, INFINITY))) x = std::nextafter(x, INFINITY);
    return x;
}

static AnisoParams aniso_params(const pms_ctx* ctx, const KGrid& g) {
    const pms_params& P = ctx->prm;
    AnisoParams ap;
    ap.h = P.h; ap.h_sq = P.h_sq; ap.h_inv = P.h_inv; ap.r2h = P.aniso_radius; ap.mass = P.mass;
    ap.kdens = kSigma / (P.h * P.h * P.h);
    ap.inv_h2 = 1.f / (P.h * P.h);
    ap.min_nn = P.min_num_neighbors;
    ap.cond_limit = ctx->cfg.fp64_svd_cond;
    ap.nn_d2 = sqrt_bound(P.h, true);
    ap.w_d2 = sqrt_bound(P.aniso_radius, false);
    ap.sp_size = g.sp_size;
    ap.sp_rows = g.spres[1] * g.spres[2];
    ap.spres_x = g.spres[0];
    return ap;
}

// Blocks of cells between a surface cell and the first far block: cells whose indices
// differ by k are (k - 1) cells apart at least.
static int density_reach(const KGrid& g, float h) {
    const float cells = 1.001f * (2.f * h + g.sc_cs) / g.sp_cs + 2.f * g.margin;
    return ((int)floorf(cells) + 2) / 2;
}

// the block form of the density over the blocks `which` names
static pms_status density_blocks(pms_ctx* ctx, const KGrid& g, const AnisoParams& ap, const SurfaceList& sl, DensBlocks which) {
    Counters* cnt = ctx->counters.as<Counters>();
    const int bd_threads = ctx->tune.density_threads;
    const uint3 bd = make_uint3((g.spres[0] + kDensX - 1) / kDensX, (g.spres[1] + kDensY - 1) / kDensY,
                                (g.spres[2] + kDensZ - 1) / kDensZ);
    const uint32_t wx = (bd.x + 31u) / 32u;
    const uint64_t words = (uint64_t)wx * bd.y * bd.z;
    // (the moments' buffer holds the list until the moments are made: at most an entry per particle;
    // the certification's cell records, made after the band, hold the bits: a word per cell is plenty)
    uint2* list = ctx->moments.as<uint2>();
    uint32_t* bits = ctx->cell_rec.as<uint32_t>();
    if (which != DensBlocks::kAll) {
        k_density_surface<<<grid_for(words * 32, 256), 256, 0, ctx->stream>>>(g, bd, wx, ctx->cell_info.as<uint2>(), bits);
        PMS_LAUNCHED(ctx);
    }
    k_density_list<<<grid_for(words * 32, 256), 256, 0, ctx->stream>>>(
        g, bd, wx, which, density_reach(g, ap.h), bits, ctx->cell_start.as<uint32_t>(), &cnt->dens_entries, list);
    PMS_LAUNCHED(ctx);
    auto tiles = [&](auto kern) {
        kern<<<152u * (1024u / (unsigned)bd_threads), bd_threads, 0, ctx->stream>>>(
            g, ap, sl, bd, ctx->skeys.as<uint32_t>(), &cnt->dens_entries, &cnt->dens_next, list, ctx->cell_start.as<uint32_t>(), ctx->spos.as<float4>(),
            ctx->rho.as<float>(), ctx->aniso.as<float4>());
    };
    if (bd_threads == 64) tiles(k_density_tiles<64>);
    else if (bd_threads == 256) tiles(k_density_tiles<256>);
    else tiles(k_density_tiles<128>);
    PMS_LAUNCHED(ctx);
    return PMS_OK;
}

// The densities of the far blocks that a frame left out (downloads of all densities).
pms_status launch_density_rest(pms_ctx* ctx) {
    if (!ctx->dens_far) return PMS_OK;
    const KGrid g = kgrid_of(ctx->grid);
    Counters* cnt = ctx->counters.as<Counters>();
    const SurfaceList sl = {ctx->cell_info.as<uint2>(), ctx->surf_start.as<uint32_t>(), ctx->slist.as<uint32_t>()};
    pms_status st = density_blocks(ctx, g, aniso_params(ctx, g), sl, DensBlocks::kFar);
    if (st) return st;
    // (between frames the tickets are zero: the anisotropy pass resets them)
    PMS_CUDA(ctx, cudaMemsetAsync(&cnt->dens_entries, 0, sizeof(uint32_t), ctx->stream));
    PMS_CUDA(ctx, cudaMemsetAsync(&cnt->dens_next, 0, sizeof(uint32_t), ctx->stream));
    ctx->dens_far = false;
    return PMS_OK;
}

pms_status launch_density_aniso(pms_ctx* ctx) {
    const KGrid g = kgrid_of(ctx->grid);
    const pms_params& P = ctx->prm;
    const AnisoParams ap = aniso_params(ctx, g);
    Counters* cnt = ctx->counters.as<Counters>();
    // block sizes of the neighbour walks are autotuned (64, 128 or 256 threads)
    const int bd_threads = ctx->tune.density_threads, bm = ctx->tune.moments_threads;
    const uint32_t n = ctx->n;
    const SurfaceList sl = {ctx->cell_info.as<uint2>(), ctx->surf_start.as<uint32_t>(), ctx->slist.as<uint32_t>()};
    pms_status st;
    ctx->dens_far = false;
    if (n <= kDensityWarp) {
        k_density_warp<<<grid_for((uint64_t)n * 32, kThreads, 152u * 16u), kThreads, 0, ctx->stream>>>(
            g, ap, sl, ctx->skeys.as<uint32_t>(), ctx->cell_start.as<uint32_t>(), ctx->spos.as<float4>(), ctx->rho.as<float>(),
            ctx->aniso.as<float4>(), n);
        PMS_LAUNCHED(ctx);
    } else if ((float)g.spexpand * g.sp_cs - P.h >= g.margin * g.sp_cs) {
        // (a scalar cell above h would let the dilation wrap past the grid's margin of 2 h)
        ctx->dens_far = ctx->dens_near && n >= kDensityNear && 2.f * g.sc_cs <= P.h && density_reach(g, P.h) < 32;
        if ((st = density_blocks(ctx, g, ap, sl, ctx->dens_far ? DensBlocks::kNear : DensBlocks::kAll))) return st;
    } else {
        auto dens = [&](auto kern) {
            kern<<<grid_for(n, (unsigned)bd_threads), bd_threads, 0, ctx->stream>>>(
                g, ap, sl, ctx->skeys.as<uint32_t>(), ctx->cell_start.as<uint32_t>(), ctx->spos.as<float4>(),
                ctx->rho.as<float>(), ctx->aniso.as<float4>(), n);
        };
        if (bd_threads == 64) dens(k_density<64>);
        else if (bd_threads == 256) dens(k_density<256>);
        else dens(k_density<128>);
        PMS_LAUNCHED(ctx);
    }
    // ns is on the device; grids are sized by the particle count (an upper bound)
    // (a thread per surface particle, or a warp where there are few: enough warps for both)
    const unsigned mom_blocks = std::max(grid_for(n, (unsigned)bm), grid_for((uint64_t)n * 32, (unsigned)bm, 152u * (2048u / (unsigned)bm)));
    auto mom = [&](auto kern) {
        kern<<<mom_blocks, bm, 0, ctx->stream>>>(g, ap, ctx->slist.as<uint32_t>(), cnt,
                                                                    ctx->skeys.as<uint32_t>(), ctx->cell_start.as<uint32_t>(),
                                                                    ctx->spos.as<float4>(), ctx->moments.as<float4>());
    };
    if (bm == 64) mom(k_moments<64>);
    else if (bm == 256) mom(k_moments<256>);
    else mom(k_moments<128>);
    PMS_LAUNCHED(ctx);
    k_eigen<<<grid_for(ctx->n, kThreads), kThreads, 0, ctx->stream>>>(
        ap, ctx->slist.as<uint32_t>(), cnt, ctx->skeys.as<uint32_t>(), ctx->spos.as<float4>(), ctx->rho.as<float>(),
        ctx->moments.as<float4>(), ctx->aniso.as<float4>(), ctx->nrm4.as<float4>(), ctx->mean4.as<float4>(), ctx->gdebug.as<float>(),
        ctx->nnb.as<uint32_t>(), ctx->cell_rad.as<float>(), cnt);
    PMS_LAUNCHED(ctx);
    return PMS_OK;
}

}  // namespace pms
