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
//     the run's digits, adds up the blocks' counts and scatters tile by
//     tile: warps rank their keys by ballots (a stable
//     order within the tile that takes the same time for any distribution),
//     the tile is put in digit order in shared memory and leaves from there
//     in runs of consecutive addresses;
//   * digits that all keys share (found with the first count) take no pass;
//   * at the end the keys are in the output and the nodes hold init_limits
//     again.  Every lock word is held meanwhile; one that is not free when
//     the kernel starts leaves the work to the delete loops (no other
//     operation may use the heap during a bulk delete).
//
// A bulk delete that takes many batches and leaves the rest sorts the same
// way between the node array and a scratch array: the smallest keys go to
// the output, the rest goes back in order, which is a heap (a node's parent
// has a smaller index in both layouts) of the node count and partial-buffer
// size that the deletes would have left.
//
// Measured on GB300: 2^28 u32 keys 6.7 ms (611 ms in owner mode), 2^27 u64
// 8.3 ms, 2^20 u32 82 us (3.8 ms), one tile about 20 us.  Bound by issue
// slots: 2^26 u32 take 1.96 IPC at 30 % of DRAM bandwidth, most of it the
// ranking's eight ballots a key (64 registers a thread, 112 bytes spilled, 80
// for 8-byte keys); below 2^20 keys by the two grid barriers a
// pass (a third one, with the counts' scan spread over the grid, took 105 us
// at 2^20 and gained nothing at any size).
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
    int arrive;  // arrivals at the grid barriers
    int bad;     // a lock word was taken: nothing is done
    int pad0[30];
    unsigned long long orAll, andNot;  // or of the keys, or of their complements
    unsigned long long below;          // k_count_below
    int pad1[26];
};
// Its words are zero between bulk deletes: every drain and count leaves them
// so, the heap's reset after a failed wait does.
constexpr int kDrainWords = sizeof(DrainCtl) / sizeof(int);
static_assert(kDrainWords == 64, "DrainCtl layout");

struct alignas(16) DrainSmem {
    unsigned warpCnt[kDrainWarps][256];
    unsigned delta[256];  // of a digit: its place in the destination less its place in the tile
    unsigned half[256];
    unsigned scan[kDrainWarps];
    unsigned long long orAll, andNot;
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

// Fewest full nodes a drain takes on.  A single tile takes about as long as
// four plain deletes and their launch; 1024 nodes of 1024 keys take 82 us,
// and the owner mode 4.4 us for each delete, so the owner mode is never the
// faster way to empty a heap.  Up to 256 nodes it stays for the first bulk
// operation on a restored heap, whose deletes are replayed one by one: its
// counters (gh_heap_owner_stats) are read to see which sift steps that very
// heap takes.  A program that restores a snapshot and goes on pays for that
// once (200 nodes of 1024 keys 0.86 ms, 0.07 as a sort).
constexpr int kDrainNodes = 4;
constexpr int kDrainNodesRestored = 256;
inline int drain_nodes(const Desc& d) { return d.mbox && d.restored ? kDrainNodesRestored : kDrainNodes; }

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

// The words a drain uses, zero again; no other block touches them any more.
__device__ __forceinline__ void clear(DrainCtl* ctl) {
    ctl->arrive = 0;
    ctl->bad = 0;
    ctl->orAll = ctl->andNot = 0;
}

// Block-wide: every one of the G working blocks arrives; false
// (block-uniform) when the wait ran out or the heap has an error.
template <typename H>
__device__ __forceinline__ bool grid_sync(const H& h, DrainCtl* ctl, DrainSmem* sm, int G, int& target) {
    target += G;
    __syncthreads();
    if (threadIdx.x == 0) {
        H::fence();
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
// barrier).
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

__device__ __forceinline__ void clear_counts(DrainSmem* sm) {
    for (int q = threadIdx.x; q < kDrainWarps * 256; q += kDrainThreads) (&sm->warpCnt[0][0])[q] = 0;
    __syncthreads();
}
__device__ __forceinline__ unsigned sum_counts(const DrainSmem* sm) {
    unsigned c = 0;
    if (threadIdx.x < 256) {
#pragma unroll
        for (int w = 0; w < kDrainWarps; ++w) c += sm->warpCnt[w][threadIdx.x];
    }
    return c;
}

// A warp's keys lie at w0 + 32 j (w0 holds the lane); past the end it takes
// the largest key, which ranks behind every key of the tile.
template <typename K, int IPT>
__device__ __forceinline__ void load_tile(K (&v)[IPT], const K* src, unsigned w0, unsigned n, unsigned cut, unsigned gap) {
#pragma unroll
    for (int j = 0; j < IPT; ++j) {
        const unsigned i = w0 + j * 32;
        v[j] = i < n ? __ldcg(src + (i < cut ? i : i + gap)) : ow::key_max<K>();
    }
}

// Ranks of the tile's keys among the keys of their digit in their warp, in
// index order, two to a word; the warps' digit counts are left in warpCnt.
// Returns the tile's count of digit threadIdx.x (threads below 256).
template <typename K, int IPT>
__device__ __forceinline__ unsigned rank_tile(const K (&v)[IPT], unsigned (&rank)[IPT / 2], DrainSmem* sm, int shift) {
    const int lane = threadIdx.x & 31;
    unsigned* cnt = sm->warpCnt[threadIdx.x >> 5];
    clear_counts(sm);
#pragma unroll
    for (int j = 0; j < IPT; ++j) {
        const unsigned d = digit(v[j], shift);
        // the lanes with the same digit, a ballot per bit (match.any took 1.3 times as long)
        unsigned same = 0xffffffffu;
#pragma unroll
        for (int b = 0; b < 8; ++b) {
            const bool bit = (d >> b) & 1u;
            const unsigned m = __ballot_sync(0xffffffffu, bit);
            same &= m ^ (bit ? 0u : 0xffffffffu);
        }
        const unsigned before = __popc(same & ((1u << lane) - 1u));
        const unsigned old = cnt[d];
        __syncwarp();
        if (before == 0) cnt[d] = old + __popc(same);
        __syncwarp();
        if (j & 1) rank[j / 2] |= (old + before) << 16;
        else rank[j / 2] = old + before;
    }
    __syncthreads();
    return sum_counts(sm);
}

// Puts the tile in digit order in shared memory: `run` is rank_tile's
// return, `off` where the block's next key of digit threadIdx.x goes (moved
// on past the tile's); sm->delta then leads from a place in the tile to the
// place in the destination.
template <typename K, int IPT>
__device__ __forceinline__ void place_tile(const K (&v)[IPT], const unsigned (&rank)[IPT / 2], K* tile, DrainSmem* sm,
                                           int shift, unsigned run, unsigned& off) {
    const int tid = threadIdx.x, warp = tid >> 5;
    unsigned at = scan256(run, sm->scan);
    if (tid < 256) {
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
    for (int j = 0; j < IPT; ++j)
        tile[sm->warpCnt[warp][digit(v[j], shift)] + ((rank[j / 2] >> (16 * (j & 1))) & 0xffffu)] = v[j];
    __syncthreads();
}

// The tile's `len` keys to their places.
template <typename K, int IPT>
__device__ __forceinline__ void write_tile(K* dst, const K* tile, const DrainSmem* sm, int shift, unsigned len) {
#pragma unroll
    for (int j = 0; j < IPT; ++j) {
        const unsigned i = j * kDrainThreads + threadIdx.x;
        if (i < len) {
            const K k = tile[i];
            dst[sm->delta[digit(k, shift)] + i] = k;
        }
    }
    __syncthreads();
}

// The varying bits of the block's keys, or-ed into the two words (global or
// shared): the or of the keys and of their complements.
__device__ __forceinline__ void or_bits(unsigned long long vOr, unsigned long long vNot, unsigned long long* orAll,
                                        unsigned long long* andNot) {
    const unsigned lo = __reduce_or_sync(0xffffffffu, static_cast<unsigned>(vOr));
    const unsigned hi = __reduce_or_sync(0xffffffffu, static_cast<unsigned>(vOr >> 32));
    const unsigned nlo = __reduce_or_sync(0xffffffffu, static_cast<unsigned>(vNot));
    const unsigned nhi = __reduce_or_sync(0xffffffffu, static_cast<unsigned>(vNot >> 32));
    if ((threadIdx.x & 31) == 0) {
        atomicOr(orAll, (static_cast<unsigned long long>(hi) << 32) | lo);
        atomicOr(andNot, (static_cast<unsigned long long>(nhi) << 32) | nlo);
    }
}

// A single tile: every pass stays in registers and shared memory; the sorted
// keys end up in `tile`.
template <typename K, int IPT>
__device__ __forceinline__ void sort_alone(const K* A, K* tile, DrainSmem* sm, unsigned n, unsigned ps, unsigned gap) {
    const unsigned w0 = (threadIdx.x >> 5) * (32 * IPT) + (threadIdx.x & 31);
    K v[IPT];
    load_tile<K, IPT>(v, A, w0, n, ps, gap);
    unsigned long long vOr = 0, vNot = 0;
#pragma unroll
    for (int j = 0; j < IPT; ++j) {
        tile[w0 + j * 32] = v[j];
        if (w0 + j * 32 < n) {
            vOr |= ordered(v[j]);
            vNot |= ~ordered(v[j]);
        }
    }
    or_bits(vOr, vNot, &sm->orAll, &sm->andNot);
    __syncthreads();
    const unsigned long long varies = sm->orAll & sm->andNot;
#pragma unroll 1
    for (int shift = 0; shift < 8 * static_cast<int>(sizeof(K)); shift += 8) {
        if (((varies >> shift) & 255u) == 0) continue;
        unsigned rank[IPT / 2];
        unsigned off = 0;
        const unsigned run = rank_tile<K, IPT>(v, rank, sm, shift);
        place_tile<K, IPT>(v, rank, tile, sm, shift, run, off);
#pragma unroll
        for (int j = 0; j < IPT; ++j) v[j] = tile[w0 + j * 32];
    }
}

// The passes of a drain over its blocks' tiles (ONE: one tile a block, whose
// keys stay in registers from the count to the scatter).  Returns how many
// were made, -1 on a failed wait; sm->bad tells whether a lock word was taken
// (then nothing was).
template <typename H, typename K, bool ONE>
__device__ __forceinline__ int passes(const H& h, DrainCtl* ctl, unsigned* cnt, DrainSmem* sm, K* tile, K* A, K* T,
                                      unsigned n, unsigned k0, unsigned k1, unsigned ps, unsigned gap, int G, int& target) {
    constexpr int IPT = drain_ipt(sizeof(K));
    constexpr unsigned TILE = drain_tile(sizeof(K));
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, blk = blockIdx.x;
    const K* src = A;
    bool first = true;
    int passes = 0;
    unsigned long long varies = 0;
#pragma unroll 1
    for (int shift = 0; shift < 8 * static_cast<int>(sizeof(K)); shift += 8) {
        if (!first && ((varies >> shift) & 255u) == 0) continue;  // one digit for all keys
        K v[IPT];
        const unsigned cut = gap ? static_cast<unsigned>(ps) : 0u;
        const unsigned w0 = k0 + warp * (32 * IPT) + lane;
        unsigned rank[IPT / 2];
        unsigned run = 0;  // thread d: the block's keys of digit d
        unsigned long long vOr = 0, vNot = 0;
        if constexpr (ONE) {
            load_tile<K, IPT>(v, src, w0, n, cut, gap);
            if (first) {
#pragma unroll
                for (int j = 0; j < IPT; ++j)
                    if (w0 + j * 32 < n) {
                        vOr |= ordered(v[j]);
                        vNot |= ~ordered(v[j]);
                    }
            }
            run = rank_tile<K, IPT>(v, rank, sm, shift);
        } else {
            clear_counts(sm);
#pragma unroll 1
            for (unsigned i0 = k0; i0 < k1; i0 += 8 * kDrainThreads) {
                K x[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const unsigned i = i0 + j * kDrainThreads + tid;
                    if (i < k1) x[j] = __ldcg(src + (i < cut ? i : i + gap));
                }
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const unsigned i = i0 + j * kDrainThreads + tid;
                    if (i < k1) {
                        atomicAdd(&sm->warpCnt[warp][digit(x[j], shift)], 1u);
                        if (first) {
                            vOr |= ordered(x[j]);
                            vNot |= ~ordered(x[j]);
                        }
                    }
                }
            }
            __syncthreads();
            run = sum_counts(sm);
        }
        unsigned off = 0;  // thread d: where the block's next key of digit d goes
        if (first) or_bits(vOr, vNot, &ctl->orAll, &ctl->andNot);
        if (tid < 256) cnt[static_cast<size_t>(blk) * 256 + tid] = run;
        if (!grid_sync(h, ctl, sm, G, target)) return -1;
        if (first) {
            if (tid == 0) sm->bad = detail::ld_relaxed(&ctl->bad);
            varies = __ldcg(&ctl->orAll) & __ldcg(&ctl->andNot);
            __syncthreads();
            if (sm->bad) return 0;
            first = false;
            if (((varies >> shift) & 255u) == 0) continue;
        }
        {
            // each block adds up all blocks' counts, two threads a digit
            const int d = tid & 255;
            unsigned all = 0, before = 0;
#pragma unroll 8
            for (int g = tid >> 8; g < G; g += 2) {
                const unsigned c = __ldcg(&cnt[static_cast<size_t>(g) * 256 + d]);
                all += c;
                before += g < blk ? c : 0;
            }
            if (tid >= 256) {
                sm->delta[d] = all;
                sm->half[d] = before;
            }
            __syncthreads();
            if (tid < 256) {
                all += sm->delta[d];
                before += sm->half[d];
            }
            const unsigned b = scan256(all, sm->scan);
            off = b + before;
        }
        __syncthreads();  // sm->scan is free again
        K* dst = (passes & 1) ? A : T;
        if constexpr (ONE) {
            place_tile<K, IPT>(v, rank, tile, sm, shift, run, off);
            write_tile<K, IPT>(dst, tile, sm, shift, k1 - k0);
        } else {
#pragma unroll 1
            for (unsigned base = k0; base < k1; base += TILE) {
                load_tile<K, IPT>(v, src, base + warp * (32 * IPT) + lane, n, cut, gap);
                run = rank_tile<K, IPT>(v, rank, sm, shift);
                place_tile<K, IPT>(v, rank, tile, sm, shift, run, off);
                write_tile<K, IPT>(dst, tile, sm, shift, k1 - base < TILE ? k1 - base : TILE);
            }
        }
        if (!grid_sync(h, ctl, sm, G, target)) return -1;
        src = dst;
        gap = 0;
        ++passes;
    }
    return passes;
}

}  // namespace dr

// tmp == null: everything, if the heap has at least minNodes full nodes and
// the output limit allows it: `lim` keys from out on or, if it is negative,
// the heap's own limit and output cursor (k_set_output).  Otherwise the `take`
// smallest of the `expect` keys the heap must hold, tmp having room for them
// all.  `must`: the caller neither runs the loops after it nor looks whether
// it started, so that giving way is recorded as the heap's error.
template <typename H, typename K>
__global__ void __launch_bounds__(kDrainThreads, kDrainBlocksPerSM) k_drain(H h, K* out, K* tmp, unsigned take,
                                                                             unsigned expect, DrainCtl* ctl,
                                                                             unsigned* cnt, int minNodes, int lim,
                                                                             HostWords* words, int must) {
    constexpr int IPT = drain_ipt(sizeof(K)), TILE = drain_tile(sizeof(K));
    extern __shared__ __align__(16) unsigned char gh_dyn_smem[];
    DrainSmem* sm = reinterpret_cast<DrainSmem*>(gh_dyn_smem);
    K* tile = reinterpret_cast<K*>(gh_dyn_smem + sizeof(DrainSmem));
    const int tid = threadIdx.x, blk = blockIdx.x;
    if (tid == 0) {
        sm->bc = detail::ld_relaxed(&h.state->batchCount);
        sm->ps = H::kHasPartialBuffer ? detail::ld_relaxed(&h.state->partialBufferSize) : 0;
        sm->dc = lim < 0 ? detail::ld_relaxed(&h.state->deleteCount) : 0;
        sm->lim = lim < 0 ? detail::ld_relaxed(&h.state->outLimit) : lim;
        sm->err = detail::ld_relaxed(&h.state->err);
        sm->orAll = sm->andNot = 0;
        sm->bad = 0;
    }
    __syncthreads();
    const int bc = sm->bc, ps = sm->ps, dc = sm->dc, B = h.batchSize;
    const long long total = static_cast<long long>(bc) * B + ps;
    // the same in every block: the counters change only after the last barrier
    if (sm->err) return;
    if (tmp ? total != expect : bc < minNodes || dc + total > sm->lim) {
        if (must && blk == 0 && tid == 0) h.raise(kErrInvalid, kSiteCapacity, bc, ps);
        return;
    }
    const unsigned n = static_cast<unsigned>(total);
    if (!tmp) take = n;
    K* A = h.heapItems;
    K* O = out + dc;
    K* T = tmp ? tmp : O;
    int target = 0;

    // this block's run of tiles; blocks without one are done
    const unsigned tiles = (n + TILE - 1) / TILE;
    const int G = tiles < gridDim.x ? static_cast<int>(tiles) : static_cast<int>(gridDim.x);
    if (blk >= G) return;
    const unsigned t0 = static_cast<unsigned>(static_cast<unsigned long long>(tiles) * blk / G);
    const unsigned t1 = static_cast<unsigned>(static_cast<unsigned long long>(tiles) * (blk + 1) / G);
    const unsigned k0 = t0 * TILE, k1 = t1 * TILE < n ? t1 * TILE : n;
    // one tile a block: its keys stay in registers between count and scatter,
    // and ranking them counts them; a single tile stays on chip throughout
    // (sort_alone)
    const bool one = G == static_cast<int>(tiles), alone = tiles == 1;

    // Take every lock word.  This finds words that are left taken; it does not
    // make the sort safe beside another operation, which no bulk delete allows:
    // counters and keys are read without waiting for all the words, so that an
    // operation that ends meanwhile could leave its keys unseen.  A thread
    // stops at its first failure: the first `mine` of its words are its own.
    const int stride = G * kDrainThreads;
    int mine = 0;
    for (int i = blk * kDrainThreads + tid; i <= bc; i += stride, ++mine)
        if (const int held = detail::cas_acquire(h.status + i, 0, H::lockedState()); held != 0) {
            if (must) h.raise(kErrTimeout, kSiteLockPath, i, held);
            if (alone) sm->bad = 1;
            else atomicOr(&ctl->bad, 1);
            break;
        }

    // key i of the sort is A[i < ps ? i : i + gap] before the first pass
    // (the partial buffer, then the nodes)
    const K* src = A;
    unsigned gap = static_cast<unsigned>(B - ps);
    int passes = 0;
    if (alone) dr::sort_alone<K, IPT>(A, tile, sm, n, ps, gap);
    if (!alone) {
        const unsigned gap0 = gap;
        passes = one ? dr::passes<H, K, true>(h, ctl, cnt, sm, tile, A, T, n, k0, k1, ps, gap0, G, target)
                     : dr::passes<H, K, false>(h, ctl, cnt, sm, tile, A, T, n, k0, k1, ps, gap0, G, target);
        if (passes < 0) return;
        if (passes > 0) {
            src = (passes & 1) ? T : A;
            gap = 0;
        }
    }
    if (sm->bad) {  // give the lock words back; the loops take over
        for (int i = blk * kDrainThreads + tid; mine > 0; i += stride, --mine) detail::st_release(h.status + i, 0);
        if (tid == 0 && !alone && atomicAdd(&ctl->arrive, 1) + 1 == target + G) dr::clear(ctl);
        return;
    }
    // ---- the sorted keys are in `tile` (a single one), in T or, after an
    // even number of passes, in the node array
    const size_t slots = static_cast<size_t>(bc + 1) * B;
    const int left = bc - static_cast<int>(take / B);  // full nodes that stay (take is a multiple of B or everything)
    const size_t at = static_cast<size_t>(blk) * kDrainThreads + tid, step = static_cast<size_t>(G) * kDrainThreads;
    const unsigned full = static_cast<unsigned>(left) * B, pbLeft = take < n ? ps : 0;
    if (alone) {
        for (unsigned i = tid; i < take; i += kDrainThreads) O[i] = tile[i];
        for (unsigned i = tid; i < slots; i += kDrainThreads) {
            const unsigned k = i < static_cast<unsigned>(B) ? full + i : i - B;  // of the keys that stay
            A[i] = (i < static_cast<unsigned>(B) ? i < pbLeft : k < full) ? tile[take + k] : h.init_limits;
        }
    } else {
        constexpr int V = 16 / sizeof(K);
        const uint4 pat = detail::splat16<K>(h.init_limits);
        uint4* A4 = reinterpret_cast<uint4*>(A);
        if (passes == 0 || (tmp && (passes & 1) == 0)) {  // equal keys, or keys that cannot move within the node array
            for (size_t i = at; i < n; i += step) T[i] = __ldcg(src + (gap && i < static_cast<unsigned>(ps) ? i : i + gap));
            if (!dr::grid_sync(h, ctl, sm, G, target)) return;
            src = T;
        }
        if (tmp) {
            // the smallest `take` to the output, the rest to nodes 1.. and the partial buffer
            for (size_t i = at; i < take; i += step) O[i] = __ldcg(T + i);
            for (size_t i = at; i < slots; i += step) {
                const size_t k = i < static_cast<size_t>(B) ? full + i : i - B;  // of the keys that stay
                const bool has = i < static_cast<size_t>(B) ? i < pbLeft : k < full;
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
    }
    // the block that finishes last publishes the counters and frees the lock words
    __syncthreads();
    if (tid == 0) {
        H::fence();
        sm->ok = alone || atomicAdd(&ctl->arrive, 1) + 1 == target + G;
        if (sm->ok) {
            H::fence();
            detail::st_relaxed(&h.state->batchCount, left);
            if (take == n) detail::st_relaxed(&h.state->partialBufferSize, 0);
            detail::st_relaxed(&h.state->deleteCount, dc + static_cast<int>(take));
            detail::st_relaxed(&h.state->outLimit, INT_MAX);
            if (words) {
                volatile HostWords* w = words;
                w->err = 0;
                w->bc = left;
                w->ps = take == n ? 0 : ps;
                w->dc = dc + static_cast<int>(take);
            }
            if (!alone) dr::clear(ctl);
            H::fence();
        }
    }
    __syncthreads();
    if (sm->ok)
        for (int i = tid; i <= bc; i += kDrainThreads) detail::st_release(h.status + i, 0);
}

// Keys below `threshold` in the heap (a prefix of each node), counted by a
// warp per node into *below (zero before).
template <typename K>
__global__ void __launch_bounds__(256) k_count_below(const K* __restrict__ items, const HeapState* st, int B, K threshold,
                                                     unsigned long long* below) {
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
    if (lane == 0 && sum) atomicAdd(below, sum);
}
// The count and the counters to the host, the count back to zero.
static __global__ void k_report_below(const HeapState* st, unsigned long long* below, HostWords* words) {
    static_cast<volatile HostWords*>(words)->below = *below;
    *below = 0;
    report(words, st, 0);
}

}  // namespace impl
}  // namespace gh
