// How a bulk delete runs, decided on the host (no CUDA in here).
#pragma once
#include <climits>

namespace gh {
namespace impl {

// The device chooses between one sort of the whole heap and the delete loops
// (kAuto), the loops, one sort of the whole heap, or one sort that leaves the
// larger keys in the heap.
enum class DeletePlan { kAuto, kLoops, kWhole, kPart };

// Whether one sort (k_drain) empties a heap of `keys` keys in `nodes` full
// nodes.  A bulk delete's output limit and cursor are ints, and the sort
// counts its keys in 32 bits: from 2^31 keys on the heap is emptied in
// pieces, by the loops.  minNodes: drain_nodes().
inline bool drains_whole(long long keys, long long nodes, int minNodes) { return keys <= INT_MAX && nodes >= minNodes; }

// Keys of each bulk delete that empties a sorted heap of n keys into host
// memory: all of them, or pieces of whole batches that an int can count.
inline long long out_piece(long long n, long long piece, int batchSize, bool whole) {
    const long long most = INT_MAX / batchSize * static_cast<long long>(batchSize);
    return whole ? n : piece < most ? piece : most;
}

}  // namespace impl
}  // namespace gh
