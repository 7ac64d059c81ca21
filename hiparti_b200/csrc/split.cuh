// split.cuh -- how many CTAs a tile of schedule records is given.
#pragma once
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
// Measured on the MTTKRP walks, all modes, whole tiles -> parts: COO 5,000
// nonzeros R = 10 22 -> 14 us, 30,000 Zipf R = 100 145 -> 25; HiCOO 100,000 Zipf
// R = 32 50 -> 25, 1.7M (1.1 waves of whole tiles) 120 -> 101; from about ten
// waves on whole tiles stay.
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
