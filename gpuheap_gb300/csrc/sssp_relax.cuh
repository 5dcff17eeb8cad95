// One SSSP expansion step on a taken batch of (dist << 32 | vertex) keys:
// the caller pattern of applications/sssp_longfei_new/sssp.cu:19-132 (skip
// stale keys, relax every edge of the rest with atomicMin, insert the
// improved keys).  Shared by the standalone SSSP kernel and the served
// queries.
//
// The block compacts the keys that are current and have edges and scans
// their degrees, then relaxes the edges in rounds.  A warp takes kRelaxEdges
// x 32 consecutive edges a round: a ballot search over the scanned degrees
// finds the vertex of the first one, and from there the vertices' first
// edges among the next 32, as a bit mask, give every lane its vertex (a
// binary search per edge was two thirds of the round's instructions, which
// bound it: 7.4 us for 4096 edges).  The loads and atomics of a lane's edges
// are in flight together.  Improved keys go to `emit`, full batches are
// inserted as they form; the remainder, *cnt keys, stays in `emit` and its
// count is returned.
#pragma once
#include "gpuheap_device.cuh"
#include "worklist.cuh"

namespace gh {
namespace app {

// Edges of a thread that are in flight together.  The heap sees a batch's
// improved keys at the end of a round, so that longer rounds have other blocks
// take keys that are farther from the minimum.  SSSP, batch 2048 on 24 blocks,
// 1 / 2 / 4 edges: 10^5 random vertices of degree 8 4.2 / 4.0 / 4.6 ms, 10^6
// of degree 4 14.4 / 14.6 / 16.1, R-MAT 18 9.0 / 8.5 / 8.4; a served burst of
// 16 queries 14.2 / 13.0 / 13.2.
constexpr int kRelaxEdges = 2;

// Shared memory of the step's tables, in bytes.
__host__ __device__ constexpr size_t relax_bytes(int B) {
    return 20 * static_cast<size_t>(B) + 8 + 32 * 8 + 4;
}

// tables: relax_bytes(batchSize) bytes (8-byte aligned); emit: batchSize +
// kRelaxEdges * blockDim.x keys; *cnt (shared) is 0 on entry.
template <typename H>
__device__ __forceinline__ int sssp_relax_batch(const H& heap, const unsigned long long* batch, int size, void* tables,
                                                 unsigned long long* emit, int* cnt,
                                                 const long long* __restrict__ rowptr, const int* __restrict__ col,
                                                 const unsigned* __restrict__ wt, unsigned* dist, int heapOff,
                                                 unsigned long long& edges, unsigned long long& inserted) {
    using u64 = unsigned long long;
    const int B = heap.batchSize, T = blockDim.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    u64* pre = static_cast<u64*>(tables);                        // k-th kept key: its first edge of the batch
    long long* shift = reinterpret_cast<long long*>(pre + B + 1);  // ... its first edge in the graph less that
    u64* wsum = reinterpret_cast<u64*>(shift + B);
    unsigned* base32 = reinterpret_cast<unsigned*>(wsum + 32);   // ... its distance
    // degrees of the keys that are still current (stale keys expand nothing);
    // the scan carries the number of keys with edges in the top 16 bits
    constexpr int kCntShift = 48;
    constexpr u64 kEdgeMask = (u64{1} << kCntShift) - 1;
    u64 run = 0;
    for (int i0 = 0; i0 < size; i0 += T) {
        const int i = i0 + tid;
        u64 x = 0;
        long long r0 = 0;
        unsigned d = 0;
        if (i < size) {
            const u64 key = batch[i];
            d = static_cast<unsigned>(key >> 32);
            const int v = static_cast<int>(key & 0xffffffffu);
            r0 = rowptr[v];
            const long long deg = rowptr[v + 1] - r0;
            if (deg > 0 && d <= __ldcg(dist + v)) x = (u64{1} << kCntShift) | static_cast<u64>(deg);
        }
        u64 incl = x;
        for (int o = 1; o < 32; o <<= 1) {
            const u64 y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) wsum[warp] = incl;
        __syncthreads();
        if (warp == 0) {
            u64 w = lane < (T >> 5) ? wsum[lane] : 0;
            for (int o = 1; o < 32; o <<= 1) {
                const u64 y = __shfl_up_sync(0xffffffffu, w, o);
                if (lane >= o) w += y;
            }
            wsum[lane] = w;
        }
        __syncthreads();
        if (x) {
            const u64 before = run + incl - x + (warp ? wsum[warp - 1] : 0);
            const int k = static_cast<int>(before >> kCntShift);
            pre[k] = before & kEdgeMask;
            shift[k] = r0 - static_cast<long long>(before & kEdgeMask);
            base32[k] = d;
        }
        run += wsum[(T >> 5) - 1];
        __syncthreads();
    }
    const int kept = static_cast<int>(run >> kCntShift);
    const u64 total = run & kEdgeMask;
    edges += total;
    if (tid == 0) pre[kept] = total;
    __syncthreads();
    // relax in rounds; full batches go to the heap
    for (u64 base = 0; base < total; base += static_cast<u64>(kRelaxEdges) * T) {
        const u64 e0 = base + static_cast<u64>(warp) * (32 * kRelaxEdges);  // the warp's first edge
        unsigned nd[kRelaxEdges], cur[kRelaxEdges];
        int u[kRelaxEdges];
#pragma unroll
        for (int j = 0; j < kRelaxEdges; ++j) u[j] = -1;
        if (e0 < total) {
            // the key of edge e0: the last k with pre[k] <= e0
            int lo = 0, hi = kept;
            while (hi - lo > 1) {
                const int step = (hi - lo + 31) >> 5, p = lo + lane * step;
                const int c = __popc(__ballot_sync(0xffffffffu, p < hi && pre[p] <= e0));
                lo += (c - 1) * step;
                hi = lo + step < hi ? lo + step : hi;
            }
#pragma unroll
            for (int j = 0; j < kRelaxEdges; ++j) {
                const u64 ej = e0 + 32 * j;
                // keys that start at edges ej + 1 .. ej + 31, and at ej + 32 for the next 32
                const u64 p = lo + 1 + lane < kept ? pre[lo + 1 + lane] : ~u64{0};
                const unsigned starts = p - ej < 32 ? 1u << static_cast<int>(p - ej) : 0u;
                const unsigned mask = __reduce_or_sync(0xffffffffu, starts);
                const int k = lo + __popc(mask & (0xffffffffu >> (31 - lane)));
                const u64 e = ej + lane;
                if (e < total) {
                    const long long at = shift[k] + static_cast<long long>(e);
                    u[j] = col[at];
                    const u64 nd64 = static_cast<u64>(base32[k]) + wt[at];
                    nd[j] = nd64 >= 0xffffffffULL ? 0xfffffffeu : static_cast<unsigned>(nd64);
                }
                // the key of edge ej + 32
                lo += __popc(mask) + (__any_sync(0xffffffffu, p == ej + 32) ? 1 : 0);
            }
        }
#pragma unroll
        for (int j = 0; j < kRelaxEdges; ++j)
            if (u[j] >= 0) cur[j] = __ldcg(dist + u[j]);
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
