// scan.cuh — exclusive prefix sums of the regrid and the table build, with
// their totals and a few other words sent to the host in the same launch.
#pragma once
#include <cub/device/device_scan.cuh>

#include "handle.cuh"

namespace fdm {

// A prefix sum of a mesh's counts is a few microseconds of work that a regrid
// waits for: what it costs is launches, copies and the wait.  One cluster of
// up to eight blocks does all of it: every block sums its part, the sums are
// exchanged through distributed shared memory, and every block scans its part
// from there.  The total, the prefix at one index and words that earlier
// kernels left are stored where the caller wants them, pinned host memory
// included.  Against five operations (a scan in two launches, three copies):
// a 3.8k-leaf run with 20 regrids 23.3 -> 21.1 ms, a 45k-leaf one with four
// 8.8 -> 8.4.  A part that is one tile is read once (vector loads, one lane per
// block of the cluster for the exchange): 45k leaves 8.0 -> 7.8, 16k 6.6 -> 6.5.
template <class U>
struct ScanArgs {
    const U *in;
    U *out;
    int64_t n;
    U *total, *total2;    // device or pinned; total2 may be null
    int64_t at;           // -1: none
    U *at_val;
    const int32_t *words; // nwords of them (at most 64) to words_out
    int32_t *words_out;
    int nwords;
};
constexpr int SCAN_TB = 1024, SCAN_ITEMS = 8, SCAN_CTAS = 8, SCAN_TILE = SCAN_TB * SCAN_ITEMS;

// inclusive scan of v over the block; sum: the block's total
template <class U>
__device__ __forceinline__ U block_scan(U v, U (&sw)[33], U &sum) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const U x = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += x;
    }
    __syncthreads();   // sw of the last call is read
    if (lane == 31) sw[wid] = v;
    __syncthreads();
    if (wid == 0) {
        U x = sw[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const U y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        sw[lane] = x;
    }
    __syncthreads();
    sum = sw[31];
    return wid == 0 ? v : v + sw[wid - 1];
}
// items i .. i + 7 (in is 16-byte aligned and i a multiple of 8), zero past the end
template <class U>
__device__ __forceinline__ void scan_load(const ScanArgs<U> &a, int64_t i, U (&v)[SCAN_ITEMS]) {
    if (i + SCAN_ITEMS <= a.n) {
        constexpr int PER = 16 / sizeof(U);
        union {
            uint4 w[SCAN_ITEMS / PER];
            U u[SCAN_ITEMS];
        } x;
#pragma unroll
        for (int q = 0; q < SCAN_ITEMS / PER; ++q) x.w[q] = reinterpret_cast<const uint4 *>(a.in + i)[q];
#pragma unroll
        for (int q = 0; q < SCAN_ITEMS; ++q) v[q] = x.u[q];
        return;
    }
#pragma unroll
    for (int q = 0; q < SCAN_ITEMS; ++q) v[q] = i + q < a.n ? a.in[i + q] : U(0);
}
// the sum of the parts of the cluster's blocks before this one
template <class U>
__device__ __forceinline__ U cluster_prefix(U mine, U &part, U &base) {
    if (threadIdx.x == 0) part = mine;
    cluster_barrier();
    if (threadIdx.x < 32) {   // a lane per block
        U x = 0;
        if (threadIdx.x < blockIdx.x) {
            uint32_t his;
            asm("mapa.shared::cluster.u32 %0, %1, %2;"
                : "=r"(his)
                : "r"((uint32_t)__cvta_generic_to_shared(&part)), "r"(threadIdx.x));
            if constexpr (sizeof(U) == 8) asm volatile("ld.shared::cluster.b64 %0, [%1];" : "=l"(x) : "r"(his) : "memory");
            else asm volatile("ld.shared::cluster.b32 %0, [%1];" : "=r"(x) : "r"(his) : "memory");
        }
#pragma unroll
        for (int o = 4; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);   // eight blocks at most
        if (threadIdx.x == 0) base = x;
    }
    // base is set, and a block's part stays until every block has read it
    cluster_barrier();
    return base;
}
template <class U>
__global__ void __launch_bounds__(SCAN_TB) k_scan(ScanArgs<U> a) {
    __shared__ U sw[33];
    __shared__ U part, base;
    const int64_t tiles = (a.n + SCAN_TILE - 1) / SCAN_TILE, per = (tiles + gridDim.x - 1) / gridDim.x;
    const int64_t t0 = blockIdx.x * per, t1 = t0 + per < tiles ? t0 + per : tiles;
    U v[SCAN_ITEMS], carry = 0, sum;
    if (per > 1) {
        U s = 0;
        for (int64_t t = t0; t < t1; ++t) {
            scan_load(a, t * SCAN_TILE + threadIdx.x * SCAN_ITEMS, v);
#pragma unroll
            for (int q = 0; q < SCAN_ITEMS; ++q) s += v[q];
        }
        block_scan(s, sw, sum);
        carry = cluster_prefix(sum, part, base);
    }
    for (int64_t t = t0; t < t0 + per; ++t) {   // the same number for every block; past the end all zero
        const int64_t i = t * SCAN_TILE + threadIdx.x * SCAN_ITEMS;
        scan_load(a, i, v);
        U s = 0;
#pragma unroll
        for (int q = 0; q < SCAN_ITEMS; ++q) s += v[q];
        U x = block_scan(s, sw, sum) - s;
        if (per == 1 && gridDim.x > 1) carry = cluster_prefix(sum, part, base);
        x += carry;
#pragma unroll
        for (int q = 0; q < SCAN_ITEMS; ++q) {
            if (i + q < a.n) a.out[i + q] = x;
            if (i + q == a.at) *a.at_val = x;
            x += v[q];
        }
        carry += sum;
    }
    if (t1 != tiles || t0 >= t1) return;
    // the block of the last tile; a total among the words overwrites its copy
    if ((int)threadIdx.x < a.nwords) a.words_out[threadIdx.x] = a.words[threadIdx.x];
    __syncthreads();
    if (threadIdx.x == 0) {
        *a.total = carry;
        if (a.total2) *a.total2 = carry;
    }
}

// what cub's scan leaves undone
template <class U>
__global__ void k_scan_rest(ScanArgs<U> a) {
    const int i = threadIdx.x;
    if (i < a.nwords) a.words_out[i] = a.words[i];
    __syncthreads();
    if (i) return;
    *a.total = a.in[a.n - 1] + a.out[a.n - 1];
    if (a.total2) *a.total2 = *a.total;
    if (a.at >= 0 && a.at < a.n) *a.at_val = a.out[a.at];
}

// n > 0; queued on h's stream, without a wait.  One cluster is too few blocks
// for large arrays: at 614k flags (77k leaves) cub's scan is 0.1 ms of two
// regrids faster than the cluster, at 0.5M and below the cluster is ahead (a
// line at 131k costs the same runs 0.2 ms).
constexpr int64_t SCAN_CLUSTER_MAX = 1 << 19;
template <class U>
inline cudaError_t launch_scan(fdm_handle *h, const ScanArgs<U> &a) {
    if (a.n <= SCAN_CLUSTER_MAX) {
        const int64_t tiles = (a.n + SCAN_TILE - 1) / SCAN_TILE;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)(tiles < SCAN_CTAS ? tiles : SCAN_CTAS));
        cfg.blockDim = dim3(SCAN_TB);
        cfg.stream = h->s;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = cfg.gridDim.x;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        return cudaLaunchKernelEx(&cfg, k_scan<U>, a);
    }
    size_t bytes = 0;
    cudaError_t e = cub::DeviceScan::ExclusiveSum(nullptr, bytes, a.in, a.out, (int)a.n, h->s);
    if (e == cudaSuccess) e = h->cub_tmp.ensure(bytes);
    if (e == cudaSuccess) e = cub::DeviceScan::ExclusiveSum(h->cub_tmp.p, bytes, a.in, a.out, (int)a.n, h->s);
    if (e != cudaSuccess) return e;
    k_scan_rest<U><<<1, 64, 0, h->s>>>(a);
    return cudaGetLastError();
}

}  // namespace fdm
