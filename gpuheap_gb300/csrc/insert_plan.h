// How a bulk insert of full batches fills its reserved targets, decided on
// the device from the node count (no CUDA needed to compile this).
#pragma once

#ifdef __CUDACC__
#define GH_PLAN_HD __host__ __device__
#else
#define GH_PLAN_HD
#endif

namespace gh {
namespace impl {

// Fewest batches for which a heap build is looked at.
constexpr int kBuildLeast = 3;
// A build never makes the heap more than this many times the new batches.
constexpr int kBuildRatio = 48;

// Whether m new batches and their ancestors in a heap of n nodes are sifted
// from the bottom up (a heap build, k_build) rather than inserted one after
// another (k_insert_reserved).  A build looks at all n + m nodes with as many
// blocks as there are new batches, so few batches lose time on the nodes and
// many gain on the inserts that would meet at the top.  Measured on GB300, microseconds
// build / one by one:
//   bottom-up, u32, batch 512    m = 1, n = 20 47 / 28; m = 4, n = 4 34 / 32,
//     n = 44 51 / 39; m = 8, n = 32 44 / 49, n = 120 59 / 51; m = 16, n = 240
//     62 / 80, n = 736 84 / 75; m = 48, n = 2208 90 / 134
//   batch 16   m = 16, n = 64 44 / 61, n = 240 54 / 43; m = 64, n = 192
//     50 / 79, n = 704 59 / 52; m = 512, n = 11776 80 / 94
//   u64, batch 32   m = 16, n = 112 50 / 54, n = 176 55 / 45; m = 64, n = 704
//     62 / 76, n = 1472 73 / 66
//   top-down, u32, batch 512   m = 4, n = 8 37 / 36; m = 8, n = 56 45 / 51,
//     n = 248 60 / 56; m = 16, n = 736 68 / 86
// The lines cross near n = m^3 / 16 while there are few batches (m^3 / 32 for
// nodes below 512 bytes); small nodes, whose inserts cost little, stop at 6 to
// 24 times the batches (more once the inserts contend, from 128 on).  Top-down
// inserts go one at a time through the root and lose sooner, near m^3 / 4.
GH_PLAN_HD inline bool build_pays(bool topDown, long long nodeBytes, long long m, long long n) {
    if (m < kBuildLeast || n + m > kBuildRatio * m) return false;
    if (m < 64 && (topDown ? 4 : nodeBytes < 512 ? 32 : 16) * n > m * m * m) return false;
    if (topDown) return true;
    const long long most = nodeBytes < 128 ? 6 : nodeBytes < 512 ? 12 : nodeBytes < 1024 ? 24 : kBuildRatio;
    return n + m <= most * m * (m < 128 ? 128 : m < 1024 ? m : 1024) / 128;
}

}  // namespace impl
}  // namespace gh
