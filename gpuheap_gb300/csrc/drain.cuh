// Bulk delete of a whole heap as one sort.
//
// A bulk delete that empties the heap (deleteKernel, test/heap_test.cu:60-77,
// until nothing is left) writes every key it holds in ascending order,
// whatever the order of the steps in between, and leaves the nodes at
// init_limits.  Made delete by delete it is a chain: each delete's root
// depends on the one before (4.4 us for 2048 keys, 1.3 % of HBM bandwidth).
// k_drain makes the same output with a least-significant-digit radix sort of
// the heap's keys, 8 bits a pass, between the node array and the output
// buffer, so it needs no memory of the heap's size:
//
//   * one cooperative launch; the blocks meet at grid barriers (bounded);
//   * each block owns a contiguous run of tiles of the keys.  A pass counts
//     the run's digits, scans the counts over digits and blocks, and
//     scatters tile by tile: warps rank their keys by ballots (a stable
//     order within the tile that takes the same time for any distribution),
//     the tile is put in digit order in shared memory and leaves from there
//     in runs of consecutive addresses;
//   * digits that all keys share (found with the first count) take no pass;
//   * at the end the keys are in the output and the nodes hold init_limits
//     again.  Every lock word is held meanwhile; one that is not free when
//     the kernel starts leaves the work to the delete loops.
//
// A bulk delete that takes many batches and leaves the rest sorts the same
// way between the node array and a scratch array: the smallest keys go to
// the output, the rest goes back in order, which is a heap (a node's parent
// has a smaller index in both layouts) of the node count and partial-buffer
// size that the deletes would have left.
//
// Measured on GB300: 2^28 u32 keys 6.7 ms (611 ms in owner mode), 2^27 u64
// 8.1 ms, 2^20 u32 154 us (3.8 ms), 2^16 u32 100 us.  Bound by issue slots:
// 2^26 u32 take 1.9 IPC at 28 % of DRAM bandwidth, most of it the ranking's
// eight ballots a key; below 2^20 keys by the three grid barriers a pass.
#pragma once
#include <climits>
#include <cstdint>

#include "owner_delete.cuh"

namespace gh {
namespace impl {

constexpr int kDrainThreads = 512;
constexpr int kDrainWarps = kDrainThreads / 32;
constexpr int kDrainBlocksPerSM = 2;

// Keys of one tile: 16 four-byte or 8 eight-byte keys a thread, 32 KiB.
__host__ __device__ constexpr int drain_ipt(int keyBytes) { return 64 / keyBytes; }
__host__ __device__ constexpr int drain_tile(int keyBytes) { return kDrainThreads * drain_ipt(keyBytes); }

// Device words of one heap's drains; `cnt` (256 x blocks) follows.
struct alignas(128) DrainCtl {
    int arrive;  // grid barrier: arrivals
    int bad;     // a lock word was taken: nothing is done
    int pad0[30];
    unsigned long long orAll, andNot;  // or of the keys, or of their complements
    unsigned long long probe[4];       // DeleteProbe
    int pad1[20];
    unsigned total[256];  // keys per digit of the current pass
};
constexpr int kDrainWords = 64;  // ints ahead of `total`, zero when a drain starts (k_set_output)

struct alignas(16) DrainSmem {
    unsigned warpCnt[kDrainWarps][256];
    unsigned delta[256];  // of a digit: its place in the destination less its place in the tile
    unsigned scan[kDrainWarps];
    int bc, ps, dc, lim, err, ok, bad;
};

inline size_t drain_smem(int keyBytes) { return sizeof(DrainSmem) + static_cast<size_t>(drain_tile(keyBytes)) * keyBytes; }
// Blocks a drain of a heap with room for `keys` keys may use.
inline int drain_blocks(long long keys, int keyBytes, int numSMs) {
    const long long tiles = (keys + drain_tile(keyBytes) - 1) / drain_tile(keyBytes);
    const long long most = static_cast<long long>(kDrainBlocksPerSM) * numSMs;
    return static_cast<int>(tiles < 1 ? 1 : tiles < most ? tiles : most);
}
inline size_t drain_bytes(int blocks) { return sizeof(DrainCtl) + sizeof(unsigned) * 256 * static_cast<size_t>(blocks); }

// Fewest full nodes a drain takes on.  Four nodes of 256 keys take 100 us,
// about what four plain deletes and their launch take.  With the owner mode
// a delete costs 4.4 us and 256 of them 1.1 ms, so the lines cross far below
// 256 nodes (154 us for 1024 nodes of 1024 keys); up to there the owner mode
// stays because its counters (gh_heap_owner_stats) describe such deletes.
constexpr int kDrainNodes = 4;         // heaps without the owner mode
constexpr int kDrainNodesOwner = 256;  // heaps with it
inline int drain_nodes(const Desc& d) { return d.mbox ? kDrainNodesOwner : kDrainNodes; }

namespace dr {

// The key's bits in unsigned order.
template <typename K>
__device__ __forceinline__ unsigned long long ordered(K k) {
    if constexpr (sizeof(K) == 8) return static_cast<unsigned long long>(k);
    else if constexpr (static_cast<K>(-1) < static_cast<K>(0)) return static_cast<unsigned>(k) ^ 0x80000000u;
    else return static_cast<unsigned>(k);
}
template <typename K>
__device__ __forceinline__ unsigned digit(K k, int shift) {
    if constexpr (sizeof(K) == 8) return static_cast<unsigned>(k >> shift) & 255u;
    else return (static_cast<unsigned>(ordered(k)) >> shift) & 255u;
}

// Block-wide: every block of the grid arrives; false (block-uniform) when the
// wait ran out or the heap has an error.
template <typename H>
__device__ __forceinline__ bool grid_sync(const H& h, DrainCtl* ctl, DrainSmem* sm, int& target) {
    target += static_cast<int>(gridDim.x);
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(&ctl->arrive, 1);
        bool ok = true;
        unsigned long long t0 = 0;
        for (unsigned it = 0; detail::ld_acquire(&ctl->arrive) < target; ++it)
            if (!h.keep_waiting(t0, it, kSiteHandOff, -1, target)) { ok = false; break; }
        sm->ok = ok;
    }
    __syncthreads();
    return sm->ok != 0;
}

// Exclusive scan over the first 256 threads (the others take part in the
// barriers).
__device__ __forceinline__ unsigned scan256(unsigned v, unsigned* tmp) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    unsigned x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) tmp[warp] = x;
    __syncthreads();
    unsigned before = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w)
        if (w < warp) before += tmp[w];
    return before + x - v;
}

}  // namespace dr

// tmp == null: everything, if the heap has at least minNodes full nodes and
// the output limit allows it.  Otherwise the `take` smallest of the `expect`
// keys the heap must hold, tmp having room for them all.
template <typename H, typename K>
__global__ void __launch_bounds__(kDrainThreads, kDrainBlocksPerSM) k_drain(H h, K* out, K* tmp, unsigned take,
                                                                             unsigned expect, DrainCtl* ctl,
                                                                             unsigned* cnt, int minNodes) {
    constexpr int IPT = drain_ipt(sizeof(K)), TILE = drain_tile(sizeof(K));
    extern __shared__ __align__(16) unsigned char gh_dyn_smem[];
    DrainSmem* sm = reinterpret_cast<DrainSmem*>(gh_dyn_smem);
    K* tile = reinterpret_cast<K*>(gh_dyn_smem + sizeof(DrainSmem));
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int G = static_cast<int>(gridDim.x), blk = static_cast<int>(blockIdx.x);
    if (tid == 0) {
        sm->bc = detail::ld_relaxed(&h.state->batchCount);
        sm->ps = H::kHasPartialBuffer ? detail::ld_relaxed(&h.state->partialBufferSize) : 0;
        sm->dc = detail::ld_relaxed(&h.state->deleteCount);
        sm->lim = detail::ld_relaxed(&h.state->outLimit);
        sm->err = detail::ld_relaxed(&h.state->err);
    }
    __syncthreads();
    const int bc = sm->bc, ps = sm->ps, dc = sm->dc, B = h.batchSize;
    const long long total = static_cast<long long>(bc) * B + ps;
    // the same in every block: the counters change only after the last barrier
    if (sm->err || (tmp ? total != expect : bc < minNodes || dc + total > sm->lim)) return;
    const unsigned n = static_cast<unsigned>(total);
    if (!tmp) take = n;
    K* A = h.heapItems;
    K* O = out + dc;
    K* T = tmp ? tmp : O;
    int target = 0;

    // this block's run of tiles
    const unsigned tiles = (n + TILE - 1) / TILE;
    const unsigned t0 = static_cast<unsigned>(static_cast<unsigned long long>(tiles) * blk / G);
    const unsigned t1 = static_cast<unsigned>(static_cast<unsigned long long>(tiles) * (blk + 1) / G);
    const unsigned k0 = t0 * TILE, k1 = t1 * TILE < n ? t1 * TILE : n;

    // Take every lock word.  An operation still in flight holds one at any
    // time (it locks the next node before it frees the last), so it makes
    // this fail or waits until the end.  A thread stops at its first failure:
    // the first `mine` of its words are its own.
    const int stride = G * kDrainThreads;
    int mine = 0;
    for (int i = blk * kDrainThreads + tid; i <= bc; i += stride, ++mine)
        if (detail::cas_acquire(h.status + i, 0, H::lockedState()) != 0) {
            atomicOr(&ctl->bad, 1);
            break;
        }

    // key i of the sort is A[i < ps ? i : i + gap] before the first pass
    // (the partial buffer, then the nodes)
    const unsigned gap0 = static_cast<unsigned>(B - ps);
    const K* src = A;
    unsigned gap = gap0;
    bool first = true;
    int passes = 0;
    unsigned long long varies = 0;
    for (int shift = 0; shift < 8 * static_cast<int>(sizeof(K)); shift += 8) {
        if (!first && ((varies >> shift) & 255u) == 0) continue;  // one digit for all keys
        // ---- count the run's digits
        for (int q = tid; q < kDrainWarps * 256; q += kDrainThreads) (&sm->warpCnt[0][0])[q] = 0;
        __syncthreads();
        unsigned long long vOr = 0, vNot = 0;
        const unsigned cut = gap ? static_cast<unsigned>(ps) : 0u;
#pragma unroll 1
        for (unsigned i0 = k0; i0 < k1; i0 += 8 * kDrainThreads) {
            K v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const unsigned i = i0 + j * kDrainThreads + tid;
                if (i < k1) v[j] = __ldcg(src + (i < cut ? i : i + gap));
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const unsigned i = i0 + j * kDrainThreads + tid;
                if (i < k1) {
                    atomicAdd(&sm->warpCnt[warp][dr::digit(v[j], shift)], 1u);
                    if (first) {
                        const unsigned long long x = dr::ordered(v[j]);
                        vOr |= x;
                        vNot |= ~x;
                    }
                }
            }
        }
        if (first) {
            const unsigned lo = __reduce_or_sync(0xffffffffu, static_cast<unsigned>(vOr));
            const unsigned hi = __reduce_or_sync(0xffffffffu, static_cast<unsigned>(vOr >> 32));
            const unsigned nlo = __reduce_or_sync(0xffffffffu, static_cast<unsigned>(vNot));
            const unsigned nhi = __reduce_or_sync(0xffffffffu, static_cast<unsigned>(vNot >> 32));
            if (lane == 0) {
                atomicOr(&ctl->orAll, (static_cast<unsigned long long>(hi) << 32) | lo);
                atomicOr(&ctl->andNot, (static_cast<unsigned long long>(nhi) << 32) | nlo);
            }
        }
        __syncthreads();
        if (tid < 256) {
            unsigned c = 0;
#pragma unroll
            for (int w = 0; w < kDrainWarps; ++w) c += sm->warpCnt[w][tid];
            cnt[static_cast<size_t>(tid) * G + blk] = c;
        }
        if (!dr::grid_sync(h, ctl, sm, target)) return;
        if (first) {
            if (tid == 0) sm->bad = detail::ld_relaxed(&ctl->bad);
            varies = __ldcg(&ctl->orAll) & __ldcg(&ctl->andNot);
            __syncthreads();
            if (sm->bad) {
                for (int i = blk * kDrainThreads + tid; mine > 0; i += stride, --mine) detail::st_release(h.status + i, 0);
                return;
            }
            first = false;
            if (((varies >> shift) & 255u) == 0) continue;
        }
        // ---- scan: per digit over the blocks (one warp), then over the digits
        for (int d = blk * kDrainWarps + warp; d < 256; d += G * kDrainWarps) {
            unsigned run = 0;
            for (int g = 0; g < G; g += 32) {
                unsigned* p = cnt + static_cast<size_t>(d) * G + g + lane;
                const unsigned c = g + lane < G ? __ldcg(p) : 0;
                unsigned x = c;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
                    if (lane >= o) x += y;
                }
                if (g + lane < G) *p = run + x - c;
                run += __shfl_sync(0xffffffffu, x, 31);
            }
            if (lane == 0) ctl->total[d] = run;
        }
        if (!dr::grid_sync(h, ctl, sm, target)) return;
        unsigned off = 0;  // thread d: where the block's next key of digit d goes
        {
            const unsigned c = tid < 256 ? __ldcg(&ctl->total[tid]) : 0;
            const unsigned b = dr::scan256(c, sm->scan);
            if (tid < 256) off = b + __ldcg(&cnt[static_cast<size_t>(tid) * G + blk]);
        }
        // ---- scatter, tile by tile
        K* dst = (passes & 1) ? A : T;
#pragma unroll 1
        for (unsigned base = k0; base < k1; base += TILE) {
            for (int q = tid; q < kDrainWarps * 256; q += kDrainThreads) (&sm->warpCnt[0][0])[q] = 0;
            K v[IPT];
            unsigned rank[IPT / 2];  // two 16-bit ranks within the warp's keys of the digit
            const unsigned w0 = base + warp * (32 * IPT) + lane;
#pragma unroll
            for (int j = 0; j < IPT; ++j) {
                const unsigned i = w0 + j * 32;
                // past the end: the largest digit, ranked behind every key
                v[j] = i < n ? __ldcg(src + (i < cut ? i : i + gap)) : ow::key_max<K>();
            }
            __syncthreads();
#pragma unroll
            for (int j = 0; j < IPT; ++j) {
                const unsigned d = dr::digit(v[j], shift);
                // the lanes with the same digit, a ballot per bit (match.any took 1.3 times as long)
                unsigned same = 0xffffffffu;
#pragma unroll
                for (int b = 0; b < 8; ++b) {
                    const bool bit = (d >> b) & 1u;
                    const unsigned m = __ballot_sync(0xffffffffu, bit);
                    same &= m ^ (bit ? 0u : 0xffffffffu);
                }
                const unsigned before = __popc(same & ((1u << lane) - 1u));
                const unsigned old = sm->warpCnt[warp][d];
                __syncwarp();
                if (before == 0) sm->warpCnt[warp][d] = old + __popc(same);
                __syncwarp();
                if (j & 1) rank[j / 2] |= (old + before) << 16;
                else rank[j / 2] = old + before;
            }
            __syncthreads();
            unsigned run = 0;
            if (tid < 256) {
#pragma unroll
                for (int w = 0; w < kDrainWarps; ++w) run += sm->warpCnt[w][tid];
            }
            unsigned at = dr::scan256(run, sm->scan);
            if (tid < 256) {
                // a digit's place in the tile, warp by warp, and from there to its place in dst
                sm->delta[tid] = off - at;
                off += run;
#pragma unroll
                for (int w = 0; w < kDrainWarps; ++w) {
                    const unsigned c = sm->warpCnt[w][tid];
                    sm->warpCnt[w][tid] = at;
                    at += c;
                }
            }
            __syncthreads();
#pragma unroll
            for (int j = 0; j < IPT; ++j) {
                const unsigned d = dr::digit(v[j], shift);
                tile[sm->warpCnt[warp][d] + ((rank[j / 2] >> (16 * (j & 1))) & 0xffffu)] = v[j];
            }
            __syncthreads();
            const unsigned len = n - base < static_cast<unsigned>(TILE) ? n - base : static_cast<unsigned>(TILE);
#pragma unroll
            for (int j = 0; j < IPT; ++j) {
                const unsigned i = j * kDrainThreads + tid;
                if (i < len) {
                    const K k = tile[i];
                    dst[sm->delta[dr::digit(k, shift)] + i] = k;
                }
            }
            __syncthreads();
        }
        if (!dr::grid_sync(h, ctl, sm, target)) return;
        src = dst;
        gap = 0;
        ++passes;
    }
    // ---- the sorted keys are in T or (an even number of passes) in the node array
    const size_t slots = static_cast<size_t>(bc + 1) * B;
    const int left = bc - static_cast<int>(take / B);  // full nodes that stay (take is a multiple of B or everything)
    const size_t at = static_cast<size_t>(blk) * kDrainThreads + tid, step = static_cast<size_t>(G) * kDrainThreads;
    constexpr int V = 16 / sizeof(K);
    const uint4 pat = detail::splat16<K>(h.init_limits);
    uint4* A4 = reinterpret_cast<uint4*>(A);
    if (passes == 0 || (tmp && (passes & 1) == 0)) {  // equal keys, or keys that cannot move within the node array
        for (size_t i = at; i < n; i += step) T[i] = __ldcg(src + (gap && i < static_cast<unsigned>(ps) ? i : i + gap));
        if (!dr::grid_sync(h, ctl, sm, target)) return;
        src = T;
    }
    if (tmp) {
        // the smallest `take` to the output, the rest to nodes 1.. and the partial buffer
        for (size_t i = at; i < take; i += step) O[i] = __ldcg(T + i);
        const size_t full = static_cast<size_t>(left) * B;
        for (size_t i = at; i < slots; i += step) {
            const size_t k = i < static_cast<size_t>(B) ? full + i : i - B;  // of the keys that stay
            const bool has = i < static_cast<size_t>(B) ? i < static_cast<size_t>(take < n ? ps : 0) : k < full;
            A[i] = has ? __ldcg(T + take + k) : h.init_limits;
        }
    } else {
        const bool copy = src == A;
        const bool vec = (reinterpret_cast<uintptr_t>(O) & 15) == 0;
        for (size_t q = at; q < slots / V; q += step) {
            const size_t i = q * V;
            if (copy && i < n) {
                const uint4 x = __ldcg(A4 + q);
                if (vec && i + V <= n) {
                    reinterpret_cast<uint4*>(O)[q] = x;
                } else {
                    const K* xs = reinterpret_cast<const K*>(&x);
#pragma unroll
                    for (int e = 0; e < V; ++e)
                        if (i + e < n) O[i + e] = xs[e];
                }
            }
            A4[q] = pat;
        }
    }
    // the block that finishes last publishes the counters and frees the lock words
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        sm->ok = atomicAdd(&ctl->arrive, 1) + 1 == target + G;
        if (sm->ok) {
            detail::st_relaxed(&h.state->batchCount, left);
            if (take == n) detail::st_relaxed(&h.state->partialBufferSize, 0);
            detail::st_relaxed(&h.state->deleteCount, dc + static_cast<int>(take));
            __threadfence();
        }
    }
    __syncthreads();
    if (sm->ok)
        for (int i = tid; i <= bc; i += kDrainThreads) detail::st_release(h.status + i, 0);
}

// Keys below `threshold` in the heap (a prefix of each node), counted by a
// warp per node, and the counters a bulk delete plans with.
struct DeleteProbe {
    int bc, ps, err, pad;
    unsigned long long below;
};
template <typename K>
__global__ void __launch_bounds__(256) k_count_below(const K* __restrict__ items, const HeapState* st, int B, K threshold,
                                                     DeleteProbe* probe) {
    const int bc = st->batchCount, ps = st->partialBufferSize;
    const int lane = threadIdx.x & 31;
    unsigned long long sum = 0;
    for (int i = blockIdx.x * 8 + (threadIdx.x >> 5); i <= bc; i += gridDim.x * 8) {
        const K* nd = items + static_cast<size_t>(i) * B;
        int lo = 0, hi = i == 0 ? ps : B;  // nd[lo - 1] < threshold <= nd[hi]
        while (lo < hi) {
            const int stp = (hi - lo + 31) / 32, p = lo + lane * stp;
            const int c = __popc(__ballot_sync(0xffffffffu, p < hi && __ldcg(nd + p) < threshold));
            if (c == 0) break;
            const int nl = lo + (c - 1) * stp + 1;
            hi = min(hi, lo + c * stp);
            lo = nl;
        }
        sum += lo;
    }
    if (lane == 0 && sum) atomicAdd(&probe->below, sum);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        probe->bc = bc;
        probe->ps = ps;
        probe->err = st->err;
    }
}

}  // namespace impl
}  // namespace gh
