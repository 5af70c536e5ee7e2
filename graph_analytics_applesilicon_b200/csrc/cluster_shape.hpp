// cluster_shape.hpp -- how many blocks a source's cluster has (bfs_cluster.cu).
#pragma once

#include <cstddef>
#include <cstdint>

namespace gb {

constexpr uint32_t kClQueue = 2048;       // queue entries per block and level
constexpr size_t kClSmem = 220 * 1024;    // queues and bitmap of one block, at most
constexpr uint32_t kClMaxBlocks = 16;

// A block's shared memory: two queues of 16-byte entries and its share of the bitmap.
inline size_t clusterSmem(uint64_t n, uint32_t nc) { return 32 * kClQueue + ((n + 31) / 32 + nc - 1) / nc * 4; }

// Blocks per source.  More blocks make a level's passes fewer, until the
// sources together cover the SMs (64 sources, 1400 x 1400: 7.7 ms with 2
// blocks each, 12.2 with 4 and 13.2 with 8) or the frontier is too small to
// need them (150 x 150, about 100 vertices a level: 0.23 ms with 1 block, 0.31
// with 16; 700 x 700, about 600: 2.2 and 1.4 ms).  At least as many as hold
// the bitmap.  Of those only what `resident(blocks)` says the device can run at
// once: 16 blocks are more than every device must take and need as many free
// SMs side by side, so fewer are tried.  0: none, the grid forms run.
template <class Resident>
uint32_t clusterSize(uint64_t n, uint32_t k, uint32_t sms, Resident resident) {
    uint32_t nc = 1;
    while (nc < kClMaxBlocks && (uint64_t)k * nc * 2 <= sms && n >= (uint64_t)nc * 2 * 16384) nc *= 2;
    while (nc <= kClMaxBlocks && clusterSmem(n, nc) > kClSmem) nc *= 2;
    if (nc > kClMaxBlocks) return 0;
    while (nc && !resident(nc)) {
        nc /= 2;
        if (nc && clusterSmem(n, nc) > kClSmem) nc = 0;
    }
    return nc;
}

}  // namespace gb
