// Termination protocol for searches whose blocks share one heap (SSSP, grid
// A*, knapsack branch-and-bound).
//
// A block takes a batch (deleteRoot/deleteUpdate), expands it and inserts
// what it generates.  HeapState::busy counts the blocks between deciding to
// take a batch and finishing their inserts.  The search is over when the
// heap is empty while busy is 0: no block holds keys that could still be
// inserted.  A block that finds the heap empty only reads busy, so waiting
// blocks cannot keep each other alive; the block that takes a batch counts
// itself before it can empty the heap.  A block may stay counted over many
// rounds (exchange_batch) and may win the race for node 0 many times in a
// row, so the blocks stamp what they finish (HeapState::progressNs): a wait
// times out when the search stands still for the time limit, not when this
// block does.  The reference's applications stop on a count of active blocks in
// the same way (applications/sssp_longfei_new/
// sssp.cu:19-132, artifacts/knapsack/models_pq.cuh:52-137 activeCount).
#pragma once
#include <type_traits>

#include "gpuheap_device.cuh"

namespace gh {
namespace app {

// A block has inserted or taken keys: waits count their time limit from here.
__device__ __forceinline__ void stamp(HeapState* st) {
    if (threadIdx.x == 0) detail::st_relaxed(&st->progressNs, detail::globaltimer());
}

// Heap calls of the search loops, kept out of line.  Inlined into a search
// loop, insertion and deleteMin (with their merges) compete for registers
// with the loop's own state, and the compiler spills inside the merge
// loops; as calls, the heap code has the registers to itself and a call
// saves and restores a few of the caller's.
template <typename H>
__device__ __noinline__ void insert_keys(H heap, const unsigned long long* keys, int n, int heapOff) {
    heap.insertion(reinterpret_cast<const typename H::key_type*>(keys), n, heapOff, true);
    stamp(heap.state);
}

// Inserts keys[0, n) (0 < n <= batchSize) and takes a batch, in one hold of
// the heap's top (Heap::exchangeMin); returns the number of keys taken.  A
// block that comes out of a round with keys to insert goes into the next one
// like this: it stays counted busy meanwhile, and the heap's serial part, which
// bounds searches of several blocks, is passed once a round instead of twice.
// While all keys fit one batch (a chain, a corridor) no other block sees any
// and `busy` stands still.
template <typename H>
__device__ __noinline__ int exchange_batch(H heap, const unsigned long long* keys, int n, unsigned long long* out,
                                           typename H::key_type threshold, bool check, int heapOff) {
    int size = 0;
    heap.exchangeMin(reinterpret_cast<const typename H::key_type*>(keys), n, reinterpret_cast<typename H::key_type*>(out),
                     size, threshold, check, heapOff);
    stamp(heap.state);
    return size;
}

// deleteRoot with a prune threshold (keys at or above it stay); returns the
// number of keys taken.
template <typename H>
__device__ __noinline__ int take_batch(H heap, unsigned long long* out, typename H::key_type threshold, int heapOff) {
    int size = 0;
    heap.deleteMin(reinterpret_cast<typename H::key_type*>(out), size, threshold, heapOff);
    if (size > 0) stamp(heap.state);
    return size;
}

template <typename H>
__device__ __noinline__ int take_batch(H heap, unsigned long long* out, int heapOff) {
    int size = 0;
    heap.deleteMin(reinterpret_cast<typename H::key_type*>(out), size, heapOff);
    if (size > 0) stamp(heap.state);
    return size;
}

// No prune threshold: every key is worth taking.
struct NoThreshold {
    template <typename H>
    __device__ __forceinline__ typename H::key_type operator()(const H& heap) const { return heap.init_limits; }
};

// Thread 0 waits until the heap holds keys below the prune threshold (then
// this block is counted busy and the call returns false: take a batch) or
// the search is over, `stop` (may be NULL) is set, or the heap has an error
// (returns true).  Every thread calls it; the result is block-uniform.
// `word` is a shared int.  `threshold(heap)` gives the current threshold
// (deleteRoot(items, size, app_t_val), artifacts/astar/BGPQ_B/heap.cuh:
// 260-289): keys at or above it are left in the heap, and the search is over
// once none below it is left and no block is busy.  A block that finds only
// such keys waits like one that finds the heap empty: it reads busy and
// never counts itself, so waiting blocks cannot keep each other alive.  The
// smallest key is read without locks; while blocks are busy it is a hint
// (a wrong one costs one empty deleteRoot or one early exit of this block,
// while busy blocks carry on), and the last block to finish reads it with
// no other block left inside the heap.  A wait with no change of busy and no
// stamp of a working block for longer than the heap's time limit records a
// timeout and stops.
template <typename H, typename Threshold = NoThreshold>
__device__ __forceinline__ bool wait_for_keys(const H& heap, int* word, const int* stop, int& lastBusy,
                                              unsigned long long& waitStart, Threshold threshold = {}) {
    HeapState* st = heap.state;
    // with no threshold every key is worth taking, padding keys included
    auto below = [&](int bc) {
        if constexpr (std::is_same<Threshold, NoThreshold>::value) return true;
        else return heap.minKeyHint(bc) < threshold(heap);
    };
    if (threadIdx.x == 0) {
        int verdict = 0;
        for (;;) {
            if (stop && detail::ld_relaxed(stop) != 0) { verdict = 1; break; }
            const int bc = detail::ld_relaxed(&st->batchCount);
            const int ps = detail::ld_relaxed(&st->partialBufferSize);
            if ((bc || ps) && below(bc)) break;
            const int b = atomicAdd(&st->busy, 0);
            __threadfence();  // the counters below are read after busy
            if (b == 0) {
                const int bc2 = detail::ld_relaxed(&st->batchCount);
                const int ps2 = detail::ld_relaxed(&st->partialBufferSize);
                if ((bc2 == 0 && ps2 == 0) || !below(bc2)) { verdict = 1; break; }
            }
            if (detail::ld_relaxed(&st->err) != 0) { verdict = 1; break; }
            const unsigned long long now = detail::globaltimer();
            if (b != lastBusy || waitStart == 0) { lastBusy = b; waitStart = now; }
            if (heap.standsStill(waitStart, now)) {
                heap.raise(kErrTimeout, kSiteLockPartial, 0, b);
                verdict = 1;
                break;
            }
            __nanosleep(200);
        }
        if (!verdict) {
            atomicAdd(&st->busy, 1);
            __threadfence();  // busy counts this block before it can empty the heap
        }
        *word = verdict;
    }
    __syncthreads();
    const bool r = *word != 0;
    __syncthreads();
    if (!r) lastBusy = -1;
    return r;
}

// Every thread calls it, block-uniform (`word`: a shared int): a busy block
// that holds `kept` keys should put them into the heap and stop being busy
// instead of exchanging them.  With fewer full nodes than busy blocks there is
// no batch for each of them: the frontier is spread over the blocks, and all
// go on expanding vertices whose distances are still far from final.  Put
// together again, the keys make fewer and nearer batches.  A handful of keys
// (a chain) stays with its block, as every hand-over costs a wait.  SSSP,
// batch 2048 on 24 blocks, exchanging always / with this rule: grid of
// 2000 x 2000 vertices 1313 / 547 ms (163 / 57 M keys taken), 1000 x 1000
// 338 / 205; a chain of 20000 158 / 152; R-MAT 18 8.2 / 8.4; four served
// searches on the 1000 x 1000 grid 188 / 159.
template <typename H>
__device__ __forceinline__ bool crowded(const H& heap, int* word, int kept) {
    if (kept <= 8) return false;
    if (threadIdx.x == 0) {
        const int busy = detail::ld_relaxed(&heap.state->busy);
        *word = busy > 1 && detail::ld_relaxed(&heap.state->batchCount) < busy;
    }
    __syncthreads();
    const bool r = *word != 0;
    __syncthreads();
    return r;
}

// Every thread calls it, block-uniform: the heap has an error or `stop` (may
// be NULL) is set.
template <typename H>
__device__ __forceinline__ bool halted(const H& heap, const int* stop) {
    return __syncthreads_or(threadIdx.x == 0 &&
                            (detail::ld_relaxed(&heap.state->err) != 0 || (stop && detail::ld_relaxed(stop) != 0))) != 0;
}

// The block has inserted everything it generated from its batch.
__device__ __forceinline__ void batch_done(HeapState* st) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicSub(&st->busy, 1);
    }
    __syncthreads();
}

}  // namespace app
}  // namespace gh
