// split.cuh -- how many CTAs a tile of schedule records is given.
#pragma once
#include <algorithm>

#include "common.cuh"

namespace pti {

// Records per CTA when a tile is cut into `split` parts: a multiple of 4, so
// that every part's bulk copies start on 16 bytes.
inline uint32_t part_len(uint32_t tile, uint32_t split) { return ((tile + split - 1) / split + 3u) & ~3u; }

// Parts to cut each tile into.  The lane groups of a CTA walk their slices one
// batch of gathers after another, so a launch takes as long as its fullest SM
// slot: ceil(tiles * split / slots) turns of tile / split records, plus a
// fixed part per CTA (the bulk copy and the merge) worth about 200 records
// (60 and 600 time the same).  Few tiles therefore want many small parts, many
// tiles none.  A part gives each group at least one batch (min_part records).
// Measured on the HiCOO MTTKRP walks, all modes, whole tiles -> parts: 100,000
// Zipf R = 32 50 -> 25 us, 1.7M (1.1 waves of whole tiles) 120 -> 101; from
// about ten waves on whole tiles stay.
inline uint32_t split_for(uint64_t tiles, uint32_t tile, uint64_t slots, uint32_t min_part)
{
    constexpr uint64_t kFixed = 200;
    uint32_t best = 1;
    uint64_t cost = ~0ull;
    for (uint32_t split = 1; split <= tile / min_part; ++split) {
        const uint64_t c = (tiles * split + slots - 1) / slots * (part_len(tile, split) + kFixed);
        if (c < cost) {
            cost = c;
            best = split;
        }
        if (tiles * split >= 2 * slots) break;
    }
    return best;
}

// Records per CTA of a list that may be cut anywhere: as few turns as tiles of
// `tile` records need, each as long as the next (1M records are 489 tiles of
// 2048 for 592 slots, or 592 of 1692), and at least min_part.  From the sixth
// turn on the CTAs are spread out anyway and whole tiles are the better size
// (20M records of the CP model 0.87 ms, in 17 even turns 0.89).  COO MTTKRP,
// all modes, parts of a tile by split_for -> this: 1M R = 16 57.6 -> 51.3 us,
// 1.5M 92.6 -> 81, 3M Zipf R = 64 318 -> 281, 4-D 500,000 Zipf R = 24 90 -> 78;
// whole tiles -> this: 5,000 R = 10 22.6 -> 16.4, 30,000 Zipf R = 100 145 -> 23.
// Error against 64 bits over eight such tensors: whole tiles 1.72e-7, this 1.61e-7.
inline uint32_t tile_for(uint64_t n, uint32_t tile, uint64_t slots, uint32_t min_part)
{
    const uint64_t turns = std::max<uint64_t>(1, (n + slots * tile - 1) / (slots * tile));
    if (turns > 5) return tile;
    const uint64_t even = (n + slots * turns - 1) / (slots * turns);
    return std::min(tile, part_len((uint32_t)std::max<uint64_t>(even, min_part), 1));
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
