// A user program that drives Heap::exchangeMin, deleteMin and insertion(...,
// apart) from its own kernels.  One block: every batch taken equals the
// smallest keys of a host multiset (whole batches, the rest once fewer are
// left; nothing when the smallest is not below the threshold).  Several
// blocks at once: no key is lost or duplicated, and what is left passes
// checkInsertHeap and comes out in order.  Exit code 0 and "exchange ok".
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <set>
#include <vector>

#include "gpuheap.h"
#include "gpuheap_device.cuh"

using u64 = unsigned long long;

// ops[i] > 0: exchange ops[i] keys; 0: take a batch; < 0: insert -ops[i] keys.
// Block b runs operations b, b + gridDim.x ...; operation i's keys are at
// at[i] and its output at i * B.
template <typename H>
__global__ void __launch_bounds__(1024) mix(H heap, const uint64_t* keys, const int* ops, const int* at, int n, uint64_t* out, int* sizes,
                    uint64_t threshold, bool check) {
    const int B = heap.batchSize;
    for (int i = blockIdx.x; i < n; i += gridDim.x) {
        int size = 0;
        if (ops[i] > 0) heap.exchangeMin(keys + at[i], ops[i], out + static_cast<size_t>(i) * B, size, threshold, check, 0);
        else if (ops[i] == 0) heap.deleteMin(out + static_cast<size_t>(i) * B, size, 0);
        else heap.insertion(keys + at[i], -ops[i], 0, true);
        if (threadIdx.x == 0) sizes[i] = size;
        __syncthreads();
    }
}

template <int V>
static bool run(int B, int threads, int blocks, bool check, unsigned seed) {
    const int n = 120;
    u64 x = 0x9e3779b97f4a7c15ull * (seed + 1);
    auto rnd = [&] { x ^= x << 13; x ^= x >> 7; x ^= x << 17; return x; };
    std::vector<int> ops(n), at(n);
    std::vector<uint64_t> keys;
    for (int i = 0; i < n; ++i) {
        const int kind = static_cast<int>(rnd() % 8), some = 1 + static_cast<int>(rnd() % B);
        ops[i] = i < 3 ? -B : kind < 3 ? some : kind == 3 ? B : kind == 4 ? 0 : kind == 5 ? -B : kind == 6 ? -some : 1;
        at[i] = static_cast<int>(keys.size());
        for (int k = 0; k < std::abs(ops[i]); ++k) keys.push_back(rnd() % (seed % 3 ? 1ull << 40 : 50ull));
    }
    const uint64_t threshold = check ? (seed % 3 ? 1ull << 38 : 20ull) : ~0ull;
    gh_heap* h = nullptr;
    if (gh_heap_create(&h, GH_KEY_U64, V, 1, 256, B, nullptr) != GH_OK) return false;
    alignas(16) unsigned char view[64];
    gh_heap_device_view(h, view, sizeof(view));
    gh::Heap<uint64_t, V, true, 4> heap;
    std::memcpy(&heap, view, sizeof(heap));
    uint64_t *dk, *dout;
    int *dops, *dat, *dsizes;
    cudaMalloc(&dk, keys.size() * 8);
    cudaMalloc(&dout, static_cast<size_t>(n) * B * 8);
    cudaMalloc(&dops, n * 4);
    cudaMalloc(&dat, n * 4);
    cudaMalloc(&dsizes, n * 4);
    cudaMemcpy(dk, keys.data(), keys.size() * 8, cudaMemcpyHostToDevice);
    cudaMemcpy(dops, ops.data(), n * 4, cudaMemcpyHostToDevice);
    cudaMemcpy(dat, at.data(), n * 4, cudaMemcpyHostToDevice);
    const size_t smem = gh_heap_smem_bytes(GH_KEY_U64, B);
    cudaFuncSetAttribute(mix<gh::Heap<uint64_t, V, true, 4>>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    mix<<<blocks, threads, smem>>>(heap, dk, dops, dat, n, dout, dsizes, threshold, check);
    const gh_status st = gh_heap_sync(h, nullptr);
    bool ok = st == GH_OK;
    std::vector<uint64_t> out(static_cast<size_t>(n) * B), rest(keys.size() + B);
    std::vector<int> sizes(n);
    cudaMemcpy(out.data(), dout, out.size() * 8, cudaMemcpyDeviceToHost);
    cudaMemcpy(sizes.data(), dsizes, n * 4, cudaMemcpyDeviceToHost);
    int valid = 0;
    char msg[256] = "";
    gh_heap_check(h, &valid, msg, sizeof(msg), nullptr);
    ok = ok && valid;
    uint64_t* drest;
    long long left = 0;
    cudaMalloc(&drest, rest.size() * 8);
    ok = ok && gh_heap_delete(h, drest, static_cast<long long>(rest.size()), &left, nullptr) == GH_OK;
    cudaMemcpy(rest.data(), drest, left * 8, cudaMemcpyDeviceToHost);
    std::vector<uint64_t> all(rest.begin(), rest.begin() + left);
    ok = ok && std::is_sorted(all.begin(), all.end());
    std::multiset<uint64_t> held;
    for (int i = 0; i < n && ok; ++i) {
        const uint64_t* got = out.data() + static_cast<size_t>(i) * B;
        all.insert(all.end(), got, got + sizes[i]);
        if (blocks > 1) continue;
        for (int k = 0; k < std::abs(ops[i]); ++k) held.insert(keys[at[i] + k]);
        int want = ops[i] < 0 ? 0 : static_cast<int>(std::min<size_t>(B, held.size()));
        if (want && check && ops[i] > 0 && !(*held.begin() < threshold)) want = 0;
        ok = sizes[i] == want;
        for (int k = 0; k < want && ok; ++k) {
            ok = got[k] == *held.begin();
            held.erase(held.begin());
        }
        if (!ok) std::printf("operation %d (%d keys): got %d keys, want %d\n", i, ops[i], sizes[i], want);
    }
    std::sort(all.begin(), all.end());
    std::sort(keys.begin(), keys.end());
    ok = ok && all == keys;
    if (!ok)
        std::printf("variant %d B %d threads %d blocks %d check %d seed %u: %s, heap %s, %zu of %zu keys, %s\n", V, B, threads,
                    blocks, check, seed, gh_status_string(st), msg, all.size(), keys.size(), cudaGetErrorString(cudaGetLastError()));
    cudaFree(dk); cudaFree(dout); cudaFree(dops); cudaFree(dat); cudaFree(dsizes); cudaFree(drest);
    gh_heap_destroy(h);
    return ok;
}

int main() {
    const int shapes[][2] = {{64, 32}, {128, 64}, {256, 128}, {1024, 512}, {2048, 1024}};  // 4 keys a thread in the merges
    for (const auto& s : shapes)
        for (unsigned seed = 0; seed < 4; ++seed)
            for (int blocks : {1, 7})
                for (bool check : {false, true}) {
                    if (!run<gh::kTopDown>(s[0], s[1], blocks, check, seed)) return 1;
                    if (!run<gh::kBottomUp>(s[0], s[1], blocks, check, seed)) return 1;
                }
    std::printf("exchange ok\n");
    return 0;
}
