// split.cuh -- how a list of schedule records is cut for the GPU.
#pragma once
#include <algorithm>

#include "common.cuh"

namespace pti {

// Records per CTA of a list that may be cut anywhere (the CP model's values, and
// MTTKRP calls that allow it): as few turns of the GPU as tiles of `tile`
// records need, each as long as the next (1M records are 489 tiles of 2048 for
// 592 slots, or 592 of 1692), at least min_part, and a multiple of 4, so that
// bulk copies start on 16 bytes.  From the sixth turn on the CTAs are spread
// out anyway and whole tiles are the better size (20M records 0.87 ms, in 17
// even turns 0.89).
inline uint32_t tile_for(uint64_t n, uint32_t tile, uint64_t slots, uint32_t min_part)
{
    const uint64_t turns = std::max<uint64_t>(1, (n + slots * tile - 1) / (slots * tile));
    if (turns > 5) return tile;
    const uint64_t even = (n + slots * turns - 1) / (slots * turns);
    return std::min(tile, ((uint32_t)std::max<uint64_t>(even, min_part) + 3u) & ~3u);
}

// CTAs of kernel `k` the GPU holds at once.
template <class K>
uint64_t cta_slots(K k, int threads, size_t smem)
{
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, threads, smem) != cudaSuccess || n < 1) {
        cudaGetLastError();
        n = 1;
    }
    return (uint64_t)n * sm_count();
}

}  // namespace pti
