// One SSSP expansion step on a taken batch of (dist << 32 | vertex) keys:
// the caller pattern of applications/sssp_longfei_new/sssp.cu:19-132 (skip
// stale keys, relax every edge of the rest with atomicMin, insert the
// improved keys).  Shared by the standalone SSSP kernel and the served
// queries.
//
// The block scans the degrees of the current keys, then relaxes the batch's
// edges in rounds of kRelaxEdges edges per thread (a binary search over the
// scanned degrees finds each edge's vertex), appends improved keys to `emit`
// and inserts full batches as they form; the remainder, *cnt keys, stays in
// `emit` and its count is returned.  A round is a chain of dependent loads (the search in shared memory,
// the edge, the distance, the atomic), so its time hardly depends on how many
// edges a thread carries through it side by side.
#pragma once
#include "gpuheap_device.cuh"
#include "worklist.cuh"

namespace gh {
namespace app {

constexpr int kRelaxEdges = 4;

// pre: batchSize + 1 long longs; first: batchSize long longs; wsum: 32 long
// longs; emit: batchSize + kRelaxEdges * blockDim.x keys; *cnt (shared) is 0
// on entry.
template <typename H>
__device__ __forceinline__ int sssp_relax_batch(const H& heap, const unsigned long long* batch, int size,
                                                 long long* pre, long long* first, long long* wsum,
                                                 unsigned long long* emit, int* cnt,
                                                 const long long* __restrict__ rowptr, const int* __restrict__ col,
                                                 const unsigned* __restrict__ wt, unsigned* dist, int heapOff,
                                                 unsigned long long& edges, unsigned long long& inserted) {
    using u64 = unsigned long long;
    const int B = heap.batchSize, T = blockDim.x, tid = threadIdx.x;
    // degrees of the keys that are still current (stale keys expand nothing)
    for (int i = tid; i < size; i += T) {
        const u64 key = batch[i];
        const unsigned d = static_cast<unsigned>(key >> 32);
        const int v = static_cast<int>(key & 0xffffffffu);
        const long long r0 = rowptr[v], r1 = rowptr[v + 1];
        pre[i + 1] = d <= __ldcg(dist + v) ? r1 - r0 : 0;
        first[i] = r0;
    }
    __syncthreads();
    // exclusive scan of the degrees over the block (a chunk per thread)
    const int per = (size + T - 1) / T;
    long long local = 0;
    for (int j = 0; j < per; ++j) {
        const int i = tid * per + j;
        if (i < size) local += pre[i + 1];
    }
    long long incl = local;
    const int lane = tid & 31, warp = tid >> 5;
    for (int o = 1; o < 32; o <<= 1) {
        const long long y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        long long x = lane < (T >> 5) ? wsum[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            const long long y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        wsum[lane] = x;
    }
    __syncthreads();
    long long run = incl - local + (warp ? wsum[warp - 1] : 0);
    for (int j = 0; j < per; ++j) {
        const int i = tid * per + j;
        if (i < size) { run += pre[i + 1]; pre[i + 1] = run; }
    }
    if (tid == 0) pre[0] = 0;
    __syncthreads();
    const long long total = pre[size];
    edges += total;
    int top = 1;  // the largest power of two below size (1 for size 1: the probe then finds pre[1] > every edge)
    while (2 * top < size) top <<= 1;
    // relax in rounds; full batches go to the heap
    for (long long base = 0; base < total; base += static_cast<long long>(kRelaxEdges) * T) {
        int lo[kRelaxEdges];  // largest lo with pre[lo] <= edge
        u64 key[kRelaxEdges];
        unsigned nd[kRelaxEdges];
        int u[kRelaxEdges];
#pragma unroll
        for (int j = 0; j < kRelaxEdges; ++j) lo[j] = 0;
        for (int step = top; step > 0; step >>= 1) {
#pragma unroll
            for (int j = 0; j < kRelaxEdges; ++j) {
                const int m = lo[j] + step;
                if (m < size && pre[m] <= base + j * T + tid) lo[j] = m;
            }
        }
#pragma unroll
        for (int j = 0; j < kRelaxEdges; ++j) {
            const long long ei = base + j * T + tid;
            u[j] = -1;
            if (ei < total) {
                const long long e = first[lo[j]] + (ei - pre[lo[j]]);
                key[j] = batch[lo[j]];
                u[j] = col[e];
                nd[j] = wt[e];
            }
        }
        unsigned cur[kRelaxEdges];
#pragma unroll
        for (int j = 0; j < kRelaxEdges; ++j)
            if (u[j] >= 0) {
                const u64 nd64 = (key[j] >> 32) + nd[j];
                nd[j] = nd64 >= 0xffffffffULL ? 0xfffffffeu : static_cast<unsigned>(nd64);
                cur[j] = __ldcg(dist + u[j]);
            }
#pragma unroll
        for (int j = 0; j < kRelaxEdges; ++j)
            if (u[j] >= 0 && nd[j] < cur[j]) cur[j] = atomicMin(dist + u[j], nd[j]);
#pragma unroll
        for (int j = 0; j < kRelaxEdges; ++j)
            if (u[j] >= 0 && nd[j] < cur[j]) emit[atomicAdd(cnt, 1)] = (static_cast<u64>(nd[j]) << 32) | static_cast<unsigned>(u[j]);
        __syncthreads();
        const int c = *cnt;
        if (c >= B) {
            int off = 0;
            for (; c - off >= B; off += B) insert_keys(heap, emit + off, B, heapOff);
            // fewer than B keys are left, behind at least one batch: the move does not overlap
            for (int i = tid; i < c - off; i += T) emit[i] = emit[off + i];
            __syncthreads();
            if (tid == 0) *cnt = c - off;
            inserted += off;
        }
        __syncthreads();
    }
    return *cnt;
}

}  // namespace app
}  // namespace gh
