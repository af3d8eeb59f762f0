// scan.cu -- device-wide exclusive prefix sums (replaces the reference's
// thrust::exclusive_scan wrapper, Thrust.cuh:17-38, which also copied the
// total back to the host; here the total stays on the device).
//
// Two forms, by size.
// - Up to kClusterMax elements: one launch of one thread-block cluster.  Every warp keeps
//   its stretch in registers, the blocks exchange their totals through distributed shared
//   memory.  A frame of a few thousand particles runs six scans of this size, and their
//   launches, not their bytes, are what they cost: three launches of about 3.3 us each
//   (reduce, partials, down) before, one now.
// - Above: reduce, then down.  Each block owns one contiguous chunk, each of its warps a
//   contiguous part of it, read in rows of 32 lanes x 16 bytes with no shared memory on the
//   way; the down pass adds up the blocks' sums before its own itself (at most kMaxBlocks
//   values), so no third launch does.
// With a device count the chunks divide that count, so a bound far above it idles no block.
#include <cooperative_groups.h>

#include <algorithm>

#include "pms_internal.h"
#include "k_common.cuh"

namespace pms {

namespace cg = cooperative_groups;

static constexpr int kScanThreads = 256;
static constexpr int kScanWarps = kScanThreads / 32;
static constexpr int kMaxBlocks = 1024;
// the one-launch form: kCluster blocks of kClusterThreads, kRows rows of 32 per warp
static constexpr int kCluster = 8, kClusterThreads = 1024, kRows = 16;
static constexpr uint64_t kClusterMax = (uint64_t)kCluster * kClusterThreads * kRows;   // 131072

// scratch: a sum per block, then one per warp
size_t scan_scratch_bytes() { return sizeof(unsigned long long) * kMaxBlocks * (1 + kScanWarps); }

template <class T>
__device__ __forceinline__ T warp_incl_scan(T v) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const T t = __shfl_up_sync(0xffffffffu, v, o);
        if ((threadIdx.x & 31) >= o) v += t;
    }
    return v;
}
template <class T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

template <class T>
__global__ void __launch_bounds__(kClusterThreads) k_scan_cluster(const T* __restrict__ in, T* __restrict__ out, uint32_t n,
                                                                  T* total_out, const uint32_t* __restrict__ n_dev,
                                                                  const Counters* cnt, uint32_t* mirror) {
    __shared__ T warp_tot[kClusterThreads / 32];
    __shared__ T block_tot;
    const cg::cluster_group cluster = cg::this_cluster();
    const uint32_t nn = n_dev ? min(*n_dev, n) : n;          // elements past nn count as 0
    const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    // rows of 32 per warp, the least that covers nn
    const uint32_t warps = gridDim.x * (kClusterThreads / 32);
    const uint32_t rows = min((nn + warps * 32u - 1u) / (warps * 32u), (uint32_t)kRows);
    const uint32_t base = (blockIdx.x * (kClusterThreads / 32) + wid) * rows * 32u + lane;
    T v[kRows], run = 0;
#pragma unroll
    for (int r = 0; r < kRows; ++r) v[r] = (uint32_t)r < rows && base + 32u * r < nn ? in[base + 32u * r] : T(0);
#pragma unroll
    for (int r = 0; r < kRows; ++r)
        if ((uint32_t)r < rows) {
            const T x = v[r], inc = warp_incl_scan(x);
            v[r] = run + inc - x;
            run += __shfl_sync(0xffffffffu, inc, 31);
        }
    if (lane == 0u) warp_tot[wid] = run;
    __syncthreads();
    if (wid == 0u) {
        const T x = warp_tot[lane], inc = warp_incl_scan(x);
        warp_tot[lane] = inc - x;
        if (lane == 31u) block_tot = inc;
    }
    T before = 0;
    if (gridDim.x > 1u) {
        cluster.sync();
        for (uint32_t b = 0; b < cluster.block_rank(); ++b) before += *cluster.map_shared_rank(&block_tot, b);
        cluster.sync();                                     // no block leaves while its total may be read
    } else {
        __syncthreads();
    }
    if (total_out && blockIdx.x == gridDim.x - 1u && threadIdx.x == 0u) *total_out = before + block_tot;
    if (mirror && blockIdx.x == gridDim.x - 1u) {
        __syncthreads();
        publish_counters(cnt, mirror);
    }
    before += warp_tot[wid];
#pragma unroll
    for (int r = 0; r < kRows; ++r)
        if ((uint32_t)r < rows && base + 32u * r < nn) out[base + 32u * r] = before + v[r];
}

// one block's and one warp's stretch of nn elements, in whole rows of 32 lanes x V elements
struct Stretch { uint64_t begin, end; };
template <int V>
__device__ __forceinline__ Stretch scan_stretch(uint64_t nn) {
    const uint64_t row = 32u * V, rows = (nn + row - 1) / row;
    const uint64_t parts = (uint64_t)gridDim.x * kScanWarps, per = (rows + parts - 1) / parts;
    const uint64_t w = (uint64_t)blockIdx.x * kScanWarps + (threadIdx.x >> 5);
    const uint64_t b = w * per * row, e = b + per * row;
    return {b < nn ? b : nn, e < nn ? e : nn};
}

// V consecutive elements, 16 bytes in one access when V > 1 (the launcher checks the alignment)
template <class T, int V>
__device__ __forceinline__ void load_row(const T* __restrict__ p, uint64_t i, uint64_t end, T (&x)[V]) {
    if (V > 1 && i + V <= end) {
        const uint4 q = __ldg(reinterpret_cast<const uint4*>(p + i));
        memcpy(x, &q, sizeof(x));
    } else {
#pragma unroll
        for (int k = 0; k < V; ++k) x[k] = i + k < end ? p[i + k] : T(0);
    }
}

template <class T, int V>
__global__ void __launch_bounds__(kScanThreads) k_scan_reduce(const T* __restrict__ in, uint64_t n, T* __restrict__ block_sum,
                                                              T* __restrict__ warp_sums, const uint32_t* __restrict__ n_dev) {
    __shared__ T ws[kScanWarps];
    const uint64_t nn = n_dev && (uint64_t)*n_dev < n ? (uint64_t)*n_dev : n;
    const Stretch s = scan_stretch<V>(nn);
    const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    T acc = 0;
#pragma unroll 4
    for (uint64_t i = s.begin + lane * V; i < s.end; i += 32u * V) {
        T x[V];
        load_row<T, V>(in, i, s.end, x);
#pragma unroll
        for (int k = 0; k < V; ++k) acc += x[k];
    }
    acc = warp_sum(acc);
    if (lane == 0u) {
        ws[wid] = acc;
        warp_sums[(size_t)blockIdx.x * kScanWarps + wid] = acc;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        T t = 0;
#pragma unroll
        for (int w = 0; w < kScanWarps; ++w) t += ws[w];
        block_sum[blockIdx.x] = t;
    }
}

template <class T, int V>
__global__ void __launch_bounds__(kScanThreads) k_scan_down(const T* __restrict__ in, T* __restrict__ out, uint64_t n,
                                                            const T* __restrict__ block_sum, const T* __restrict__ warp_sums,
                                                            T* total_out, const uint32_t* __restrict__ n_dev,
                                                            const Counters* cnt, uint32_t* mirror) {
    __shared__ T ws[kScanWarps];
    const uint64_t nn = n_dev && (uint64_t)*n_dev < n ? (uint64_t)*n_dev : n;
    const Stretch s = scan_stretch<V>(nn);
    const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    // the blocks before this one, summed here
    T acc = 0;
    for (uint32_t b = threadIdx.x; b < blockIdx.x; b += kScanThreads) acc += block_sum[b];
    acc = warp_sum(acc);
    if (lane == 0u) ws[wid] = acc;
    __syncthreads();
    T run = 0;
#pragma unroll
    for (int w = 0; w < kScanWarps; ++w) run += ws[w];
    if (total_out && blockIdx.x == gridDim.x - 1u && threadIdx.x == 0u) *total_out = run + block_sum[blockIdx.x];
    if (mirror && blockIdx.x == gridDim.x - 1u) {
        __syncthreads();
        publish_counters(cnt, mirror);
    }
    for (uint32_t w = 0; w < wid; ++w) run += warp_sums[(size_t)blockIdx.x * kScanWarps + w];
#pragma unroll 2
    for (uint64_t r = s.begin; r < s.end; r += 32u * V) {
        const uint64_t i = r + lane * V;
        T x[V], sum = 0;
        load_row<T, V>(in, i, s.end, x);
#pragma unroll
        for (int k = 0; k < V; ++k) { const T t = x[k]; x[k] = sum; sum += t; }
        const T inc = warp_incl_scan(sum);
        const T before = run + inc - sum;
        run += __shfl_sync(0xffffffffu, inc, 31);
#pragma unroll
        for (int k = 0; k < V; ++k) x[k] += before;
        if (V > 1 && i + V <= s.end) {
            uint4 q;
            memcpy(&q, x, sizeof(q));
            *reinterpret_cast<uint4*>(out + i) = q;
        } else {
#pragma unroll
            for (int k = 0; k < V; ++k)
                if (i + k < s.end) out[i + k] = x[k];
        }
    }
}

template <class T, int V>
static pms_status scan_two(pms_ctx* ctx, const T* in, T* out, uint64_t n, T* total_dev, const uint32_t* n_dev,
                            uint32_t* mirror) {
    const uint64_t per = 4u * 32u * V * kScanWarps;          // at least four rows for each warp
    const unsigned nb = (unsigned)std::min<uint64_t>((n + per - 1) / per, kMaxBlocks);
    T *block_sum = ctx->scan.partial.as<T>(), *warp_sums = block_sum + kMaxBlocks;
    k_scan_reduce<T, V><<<nb, kScanThreads, 0, ctx->stream>>>(in, n, block_sum, warp_sums, n_dev);
    PMS_LAUNCHED(ctx);
    k_scan_down<T, V><<<nb, kScanThreads, 0, ctx->stream>>>(in, out, n, block_sum, warp_sums, total_dev, n_dev,
                                                       ctx->counters.as<Counters>(), mirror);
    PMS_LAUNCHED(ctx);
    return PMS_OK;
}

template <class T>
static pms_status scan_impl(pms_ctx* ctx, const T* in, T* out, uint64_t n, T* total_dev, const uint32_t* n_dev,
                            uint32_t* mirror) {
    if (n == 0) {
        if (total_dev) PMS_CUDA(ctx, cudaMemsetAsync(total_dev, 0, sizeof(T), ctx->stream));
        return PMS_OK;
    }
    if (n <= kClusterMax) {
        // one block while it has few rows per warp, else the cluster
        cudaLaunchConfig_t cfg = {};
        const unsigned nb = n <= 4u * kClusterThreads ? 1u : (unsigned)kCluster;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = nb;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cfg.gridDim = dim3(nb);
        cfg.blockDim = dim3(kClusterThreads);
        cfg.stream = ctx->stream;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        PMS_CUDA(ctx, cudaLaunchKernelEx(&cfg, k_scan_cluster<T>, in, out, (uint32_t)n, total_dev, n_dev,
                                         (const Counters*)ctx->counters.as<Counters>(), mirror));
        PMS_LAUNCHED(ctx);
        return PMS_OK;
    }
    PMS_CUDA(ctx, ctx->scan.partial.ensure(scan_scratch_bytes()));
    constexpr int V = 16 / (int)sizeof(T);
    // 16-byte accesses where both arrays start on a 16-byte boundary
    if (((uintptr_t)in | (uintptr_t)out) & 15u) return scan_two<T, 1>(ctx, in, out, n, total_dev, n_dev, mirror);
    return scan_two<T, V>(ctx, in, out, n, total_dev, n_dev, mirror);
}

pms_status scan_u32(pms_ctx* ctx, const uint32_t* in, uint32_t* out, uint64_t n, uint32_t* total_dev,
                    const uint32_t* n_dev) {
    return scan_impl<uint32_t>(ctx, in, out, n, total_dev, n_dev, nullptr);
}
pms_status scan_u64(pms_ctx* ctx, const unsigned long long* in, unsigned long long* out, uint64_t n,
                    unsigned long long* total_dev, const uint32_t* n_dev, bool publish) {
    return scan_impl<unsigned long long>(ctx, in, out, n, total_dev, n_dev, publish ? ctx->h_counters_dev : nullptr);
}

}  // namespace pms

// The scans on device arrays of 4- or 8-byte elements, for tests (exported, not part of
// pms.h's stable surface): n elements or the first *d_n of them; the sum comes back by way
// of the context's counters, for 8-byte elements as the scan itself publishes them.
extern "C" pms_status pms_debug_scan(pms_ctx* ctx, int elem_bytes, const void* d_in, void* d_out, uint64_t n,
                                     const uint32_t* d_n, uint64_t* total) {
    using namespace pms;
    if (!ctx || !total || (elem_bytes != 4 && elem_bytes != 8)) return PMS_ERR_INVALID_ARGUMENT;
    cudaSetDevice(ctx->device);
    Counters* cnt = ctx->counters.as<Counters>();
    if (elem_bytes == 8) {
        PMS_CHECK(scan_u64(ctx, static_cast<const unsigned long long*>(d_in), static_cast<unsigned long long*>(d_out), n,
                           &cnt->mc_total, d_n, true));
        PMS_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        *total = ctx->h_counters->mc_total;
    } else {
        PMS_CHECK(scan_u32(ctx, static_cast<const uint32_t*>(d_in), static_cast<uint32_t*>(d_out), n, &cnt->n_weld, d_n));
        PMS_CHECK(sync_counters(ctx));
        *total = ctx->h_counters->n_weld;
    }
    return PMS_OK;
}
