// Launchers for the heap kernels, instantiated once per key type in
// heap_inst_{u32,i32,u64}.cu so the three instantiation sets compile in
// parallel.  The merge width IPT = 2 * batchSize / threads is a template
// parameter of every kernel (1, 2, 4 or 8 keys per thread per merge).
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

#include "delete_plan.h"
#include "drain.cuh"
#include "heap_kernels.cuh"
#include "owner_delete.cuh"

namespace gh {
namespace impl {

struct LaunchArgs {
    const Desc* d;
    int threads;
    int grid;
    cudaStream_t stream;
    HostWords* words;  // null: nobody waits for the result
    bool autoThreads = false;  // `threads` / `grid` are the heap's automatic choice
    bool autoGrid = false;
    DeletePlan plan = DeletePlan::kAuto;
    void* tmp = nullptr;  // kPart: scratch for `expect` keys, of which the `take` smallest leave
    unsigned take = 0, expect = 0;
    int lim = -1;         // kWhole, kPart: room in the output
    bool prepared = false;  // bulk inserts: k_reset has reserved and marked the full batches' targets
    bool reserve = true;  // bulk inserts of full batches may reserve their targets (k_reserve)
};

// reset(), with the targets of `build` batches reserved and held if build > 0.
template <typename K>
cudaError_t launch_reset(const Desc& d, int numSMs, int build, cudaStream_t s) {
    const size_t bytes = (static_cast<size_t>(d.batchNum) + 1) * d.batchSize * sizeof(K);
    const size_t want = bytes / (16 * 256) + 1, most = static_cast<size_t>(numSMs) * 8;
    K fill;
    __builtin_memcpy(&fill, &d.initBits, sizeof(K));
    k_reset<K><<<static_cast<int>(want < most ? want : most), 256, 0, s>>>(
        static_cast<K*>(d.items), d.status, d.state, d.batchNum, d.batchSize, fill, static_cast<int*>(d.drain),
        d.drain ? kDrainWords : 0, build, d.variant == kTopDown ? TD::INUSE : BU::INUSE);
    count_launch();
    return cudaGetLastError();
}

template <typename K>
cudaError_t launch_insert(const LaunchArgs& a, const K* keys, long long n, int chunk);
template <typename K>
cudaError_t launch_erase(const LaunchArgs& a, K* out, const K* threshold = nullptr);
template <typename K>
cudaError_t launch_count_below(const LaunchArgs& a, K threshold);
template <typename K>
cudaError_t launch_erase_one(const LaunchArgs& a, K* out);
template <typename K>
cudaError_t launch_retrieve(const LaunchArgs& a, K* out, int want, K* scratch);
template <typename K>
cudaError_t launch_insert_counted(const LaunchArgs& a, const K* keys, const unsigned long long* n, int chunk);
template <typename K>
cudaError_t launch_concurrent(const LaunchArgs& a, const K* keys, long long n, int chunk, K* out, long long deletes);
// Bytes of gh::Heap<K, variant, pb> (IPT chosen at run time) for application kernels.
template <typename K>
void device_view(const Desc& d, void* out, size_t* bytes);

#ifdef GH_INSTANTIATE
template <typename H>
inline cudaError_t allow_smem(const void* fn, size_t smem) {
    if (smem <= 48 * 1024) return cudaSuccess;
    return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
}

// At most as many blocks as the GPU holds at once.  The reserved bulk insert
// hands batch j to block j mod grid, and an insert may wait for a parent
// target that an earlier batch fills; the owner-mode delete's owner waits
// for workers.  Both make progress only if every block runs, so a grid
// larger than the resident set would wait until the time limit.
inline int resident_grid(const void* fn, int threads, size_t smem, int want) {
    int per = 0, dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, threads, smem) != cudaSuccess || per < 1) {
        cudaGetLastError();
        return want;
    }
    const long long cap = static_cast<long long>(per) * sms;
    return want < cap ? want : static_cast<int>(cap);
}

// Calls f(Heap<K, V, PB, IPT>{}) for the run-time variant, pb flag and IPT.
template <typename K, typename F>
inline cudaError_t dispatch(const Desc& d, int threads, F&& f) {
    const int ipt = 2 * d.batchSize / threads;
    auto by_ipt = [&](auto v, auto pb) -> cudaError_t {
        constexpr int V = decltype(v)::value;
        constexpr bool PB = decltype(pb)::value;
        switch (ipt) {
            case 1: return f(Heap<K, V, PB, 1>{});
            case 2: return f(Heap<K, V, PB, 2>{});
            case 4: return f(Heap<K, V, PB, 4>{});
            case 8: return f(Heap<K, V, PB, 8>{});
            default: return cudaErrorInvalidValue;
        }
    };
    using TDv = std::integral_constant<int, kTopDown>;
    using BUv = std::integral_constant<int, kBottomUp>;
    using Yes = std::integral_constant<bool, true>;
    using No = std::integral_constant<bool, false>;
    if (d.variant == kTopDown) return d.pb ? by_ipt(TDv{}, Yes{}) : by_ipt(TDv{}, No{});
    return d.pb ? by_ipt(BUv{}, Yes{}) : by_ipt(BUv{}, No{});
}

template <typename H>
inline H view_of(const Desc& d, int sortOutput) {
    H h;
    h.heapItems = static_cast<typename H::key_type*>(d.items);
    h.status = d.status;
    h.state = d.state;
    __builtin_memcpy(&h.init_limits, &d.initBits, sizeof(typename H::key_type));
    h.batchNum = d.batchNum;
    h.batchSize = d.batchSize;
    h.sortOutput = sortOutput;
    h.timeoutNs = d.timeoutNs;
    return h;
}

// Threads of a heap build's blocks (k_build): 8 keys a thread in the merges,
// so that several blocks share an SM and hide each other's lock and load
// latency.  Measured on GB300: 2^28 u32, batch 2048: 5.7 ms at 512 threads,
// 10.2 at 1024; 2^24 u64, batch 1024: 0.72 ms at 256, 0.76 at 512.
// A build that is bound by the chain of sifts rather than by the SMs'
// instructions (few nodes, and 8-byte keys up to about 8192) runs faster at
// 4 keys a thread: 2^20 u64, batch 512: 107 us at 256 threads, 159 at 128;
// 2^14 u32, batch 256: 48 us at 128, 56 at 64.
inline int build_threads(int batchSize, int keyBytes, long long nodes) {
    const int t = batchSize >= 128 ? batchSize / 4 : 32;
    return 2 * t <= 512 && 2 * t <= 2 * batchSize && nodes <= (keyBytes == 8 ? 8192 : 512) ? 2 * t : t;
}

// The heap build of m reserved batches (and the `tail` keys after them).
template <typename K>
cudaError_t launch_build(const LaunchArgs& a, const K* keys, long long m, int tail) {
    const int threads = a.autoThreads ? build_threads(a.d->batchSize, a.d->keyBytes, m) : a.threads;
    return dispatch<K>(*a.d, threads, [&](auto proto) -> cudaError_t {
        using H = decltype(proto);
        const H h = view_of<H>(*a.d, 1);
        const size_t smem = H::smemBytes(a.d->batchSize);
        const void* fn = reinterpret_cast<const void*>(k_build<H, K>);
        cudaError_t e = allow_smem<H>(fn, smem);
        if (e != cudaSuccess) return e;
        long long g = a.autoGrid ? resident_grid(fn, threads, smem, INT_MAX) : a.grid;
        if (g == INT_MAX) g = a.grid;
        k_build<H, K><<<static_cast<int>(g < m ? g : m), threads, smem, a.stream>>>(h, keys, tail);
        count_launch();
        return cudaGetLastError();
    });
}

// Full batches (chunk == batchSize) go to targets reserved up front when the
// partial buffer is empty (k_reserve, k_mark_reserved, then k_build or
// k_insert_reserved);
// a ragged last chunk, or any other chunk size, goes through insertion().
template <typename K>
cudaError_t launch_insert(const LaunchArgs& a, const K* keys, long long n, int chunk) {
    return dispatch<K>(*a.d, a.threads, [&](auto proto) -> cudaError_t {
        using H = decltype(proto);
        const H h = view_of<H>(*a.d, 1);
        const int B = a.d->batchSize;
        const size_t smem = H::smemBytes(B);
        const long long m = (a.reserve && chunk == B) ? n / B : 0;
        if (m > 0) {
            if (!a.prepared) {
                const int nodeBytes = B * static_cast<int>(sizeof(K));
                if (a.d->batchNum <= kReserveOne || kBuildRatio * m <= kReserveOne) {
                    k_reserve_mark<H><<<1, 1024, 0, a.stream>>>(a.d->state, a.d->status, a.d->batchNum, nodeBytes, m);
                } else {
                    k_reserve<H><<<1, 1, 0, a.stream>>>(a.d->state, a.d->batchNum, nodeBytes, m);
                    count_launch();
                    const long long mb = (m + 255) / 256;
                    k_mark_reserved<H><<<static_cast<int>(mb < 1024 ? mb : 1024), 256, 0, a.stream>>>(a.d->state, a.d->status);
                }
                count_launch();
            }
            cudaError_t e = cudaSuccess;
            if (a.prepared || m >= kBuildLeast) e = launch_build<K>(a, keys, m, H::kHasPartialBuffer ? static_cast<int>(n - m * B) : 0);
            if (e != cudaSuccess) return e;
            if (a.prepared && (H::kHasPartialBuffer || n == m * B)) return cudaSuccess;
            if (!a.prepared) {
                e = allow_smem<H>(reinterpret_cast<const void*>(k_insert_reserved<H, K>), smem);
                if (e != cudaSuccess) return e;
                const int g = resident_grid(reinterpret_cast<const void*>(k_insert_reserved<H, K>), a.threads, smem,
                                            static_cast<int>(m < a.grid ? m : a.grid));
                k_insert_reserved<H, K><<<g, a.threads, smem, a.stream>>>(h, keys, m);
                count_launch();
                e = cudaGetLastError();
            }
            if (e != cudaSuccess) return e;
        }
        const long long rest = n - m * B;
        if (rest <= 0) return cudaSuccess;
        cudaError_t e = allow_smem<H>(reinterpret_cast<const void*>(k_insert<H, K>), smem);
        if (e != cudaSuccess) return e;
        const long long nchunks = (rest + chunk - 1) / chunk;
        const int g = static_cast<int>(nchunks < a.grid ? nchunks : a.grid);
        k_insert<H, K><<<g, a.threads, smem, a.stream>>>(h, keys + m * B, rest, chunk, m > 0);
        count_launch();
        return cudaGetLastError();
    });
}

template <typename K>
cudaError_t launch_insert_counted(const LaunchArgs& a, const K* keys, const unsigned long long* n, int chunk) {
    return dispatch<K>(*a.d, a.threads, [&](auto proto) -> cudaError_t {
        using H = decltype(proto);
        const H h = view_of<H>(*a.d, 1);
        const size_t smem = H::smemBytes(a.d->batchSize);
        cudaError_t e = allow_smem<H>(reinterpret_cast<const void*>(k_insert_counted<H, K>), smem);
        if (e != cudaSuccess) return e;
        k_insert_counted<H, K><<<a.grid, a.threads, smem, a.stream>>>(h, keys, n, chunk);
        count_launch();
        return cudaGetLastError();
    });
}

// The keys below `threshold` and the counters, for the host.
template <typename K>
cudaError_t launch_count_below(const LaunchArgs& a, K threshold) {
    DrainCtl* ctl = static_cast<DrainCtl*>(a.d->drain);
    const int blocks = (a.d->batchNum + 8) / 8 < 4 * a.grid ? (a.d->batchNum + 8) / 8 : 4 * a.grid;
    k_count_below<K><<<blocks, 256, 0, a.stream>>>(static_cast<const K*>(a.d->items), a.d->state, a.d->batchSize, threshold,
                                                   &ctl->below);
    count_launch();
    k_report_below<<<1, 1, 0, a.stream>>>(a.d->state, &ctl->below, a.words);
    count_launch();
    return cudaGetLastError();
}

// A bulk delete as one sort (k_drain).
template <typename K>
cudaError_t launch_drain(const LaunchArgs& a, K* out) {
    return dispatch<K>(*a.d, a.threads, [&](auto proto) -> cudaError_t {
        // the merge width plays no part: one instantiation per variant and partial buffer
        using P = decltype(proto);
        using H = Heap<K, P::kVariant, P::kHasPartialBuffer, 0>;
        H h = view_of<H>(*a.d, 1);
        const size_t smem = drain_smem(a.d->keyBytes);
        const void* fn = reinterpret_cast<const void*>(k_drain<H, K>);
        cudaError_t e = allow_smem<H>(fn, smem);
        if (e != cudaSuccess) return e;
        const int want = a.autoGrid || a.d->drainBlocks < a.grid ? a.d->drainBlocks : a.grid;
        const int g = resident_grid(fn, kDrainThreads, smem, want);
        DrainCtl* ctl = static_cast<DrainCtl*>(a.d->drain);
        unsigned* cnt = reinterpret_cast<unsigned*>(static_cast<char*>(a.d->drain) + sizeof(DrainCtl));
        int minNodes = drain_nodes(*a.d);
        K* tmp = a.plan == DeletePlan::kPart ? static_cast<K*>(a.tmp) : nullptr;
        unsigned take = a.take, expect = a.expect;
        int lim = a.lim;
        HostWords* words = a.lim < 0 ? nullptr : a.words;
        // no loops follow and nobody reads `words`: a sort that does not start is an error of the heap
        int must = a.lim >= 0 && !a.words;
        void* args[] = {&h, &out, &tmp, &take, &expect, &ctl, &cnt, &minNodes, &lim, &words, &must};
        e = cudaLaunchCooperativeKernel(fn, dim3(g), dim3(kDrainThreads), args, smem, a.stream);
        count_launch();
        return e;
    });
}

// Without a threshold, a heap with a mailbox first runs the owner-mode bulk
// delete (k_delete_owner, 1024-thread blocks) while it has nodes below its
// resident levels, then deleteKernel finishes; with a threshold,
// deleteKernel alone.
template <typename K>
cudaError_t launch_erase(const LaunchArgs& a, K* out, const K* threshold) {
    const bool sorts = a.plan == DeletePlan::kWhole || a.plan == DeletePlan::kPart;
    if (sorts || (a.plan == DeletePlan::kAuto && !threshold && a.d->drain && a.d->ownerDepth < 0)) {
        const cudaError_t e = launch_drain<K>(a, out);
        if (e != cudaSuccess || sorts) return e;
    }
    const int R = a.d->ownerDepth < 0 ? owner_depth(a.d->batchSize, a.d->keyBytes) : a.d->ownerDepth;
    if (!threshold && a.d->mbox && R > 0 && a.grid >= 2) {
        // all but the counters, which an owner that engages writes
        cudaError_t e = cudaMemsetAsync(a.d->mbox, 0, offsetof(Mailbox, stats), a.stream);
        if (e != cudaSuccess) return e;
        e = dispatch<K>(*a.d, 1024, [&](auto proto) -> cudaError_t {
            using H = decltype(proto);
            const H h = view_of<H>(*a.d, 1);
            const size_t smem = owner_smem(a.d->batchSize, a.d->keyBytes, R);
            cudaError_t e2 = allow_smem<H>(reinterpret_cast<const void*>(k_delete_owner<H, K>), smem);
            if (e2 != cudaSuccess) return e2;
            Mailbox* mb = static_cast<Mailbox*>(a.d->mbox);
            K* mdata = reinterpret_cast<K*>(static_cast<char*>(a.d->mbox) + sizeof(Mailbox));
            const int g = resident_grid(reinterpret_cast<const void*>(k_delete_owner<H, K>), 1024, smem, a.grid);
            k_delete_owner<H, K><<<g, 1024, smem, a.stream>>>(h, out, mb, mdata, R);
            count_launch();
            return cudaGetLastError();
        });
        if (e != cudaSuccess) return e;
    }
    return dispatch<K>(*a.d, a.threads, [&](auto proto) -> cudaError_t {
        using H = decltype(proto);
        const H h = view_of<H>(*a.d, 1);
        const size_t smem = H::smemBytes(a.d->batchSize);
        cudaError_t e = allow_smem<H>(reinterpret_cast<const void*>(k_delete<H, K>), smem);
        if (e != cudaSuccess) return e;
        k_delete<H, K><<<a.grid, a.threads, smem, a.stream>>>(h, out, threshold ? *threshold : h.init_limits,
                                                               threshold ? 1 : 0);
        count_launch();
        return cudaGetLastError();
    });
}

template <typename K>
cudaError_t launch_concurrent(const LaunchArgs& a, const K* keys, long long n, int chunk, K* out, long long deletes) {
    return dispatch<K>(*a.d, a.threads, [&](auto proto) -> cudaError_t {
        using H = decltype(proto);
        const H h = view_of<H>(*a.d, 1);
        const size_t smem = H::smemBytes(a.d->batchSize);
        cudaError_t e = allow_smem<H>(reinterpret_cast<const void*>(k_concurrent<H, K>), smem);
        if (e != cudaSuccess) return e;
        k_concurrent<H, K><<<a.grid, a.threads, smem, a.stream>>>(h, keys, n, chunk, out, deletes);
        count_launch();
        return cudaGetLastError();
    });
}

template <typename K>
cudaError_t launch_erase_one(const LaunchArgs& a, K* out) {
    return dispatch<K>(*a.d, a.threads, [&](auto proto) -> cudaError_t {
        using H = decltype(proto);
        const H h = view_of<H>(*a.d, 1);
        const size_t smem = H::smemBytes(a.d->batchSize);
        cudaError_t e = allow_smem<H>(reinterpret_cast<const void*>(k_delete_one<H, K>), smem);
        if (e != cudaSuccess) return e;
        k_delete_one<H, K><<<1, a.threads, smem, a.stream>>>(h, out, a.words);
        count_launch();
        return cudaGetLastError();
    });
}

template <typename K>
cudaError_t launch_retrieve(const LaunchArgs& a, K* out, int want, K* scratch) {
    return dispatch<K>(*a.d, a.threads, [&](auto proto) -> cudaError_t {
        using H = decltype(proto);
        const H h = view_of<H>(*a.d, 0);  // outputs at scratch[0]
        const size_t smem = H::smemBytes(a.d->batchSize);
        cudaError_t e = allow_smem<H>(reinterpret_cast<const void*>(k_retrieve<H, K>), smem);
        if (e != cudaSuccess) return e;
        k_retrieve<H, K><<<1, a.threads, smem, a.stream>>>(h, out, want, scratch, a.words);
        count_launch();
        return cudaGetLastError();
    });
}

template <typename K>
void device_view(const Desc& d, void* out, size_t* bytes) {
    auto put = [&](auto proto) {
        using H = decltype(proto);
        const H h = view_of<H>(d, 0);
        __builtin_memcpy(out, &h, sizeof(H));
        *bytes = sizeof(H);
    };
    if (d.variant == kTopDown) { if (d.pb) put(Heap<K, kTopDown, true>{}); else put(Heap<K, kTopDown, false>{}); }
    else { if (d.pb) put(Heap<K, kBottomUp, true>{}); else put(Heap<K, kBottomUp, false>{}); }
}

#define GH_INSTANTIATE_KEY(K)                                                                    \
    template cudaError_t launch_insert<K>(const LaunchArgs&, const K*, long long, int);          \
    template cudaError_t launch_erase<K>(const LaunchArgs&, K*, const K*);                       \
    template cudaError_t launch_count_below<K>(const LaunchArgs&, K);                            \
    template cudaError_t launch_insert_counted<K>(const LaunchArgs&, const K*, const unsigned long long*, int); \
    template cudaError_t launch_erase_one<K>(const LaunchArgs&, K*);                             \
    template cudaError_t launch_retrieve<K>(const LaunchArgs&, K*, int, K*);                     \
    template cudaError_t launch_concurrent<K>(const LaunchArgs&, const K*, long long, int, K*, long long); \
    template void device_view<K>(const Desc&, void*, size_t*);
#endif  // GH_INSTANTIATE

}  // namespace impl
}  // namespace gh
