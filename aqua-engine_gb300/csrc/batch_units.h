// batch_units.h — how a batch's pixels become the work items that the lanes of
// the batch kernel take (batch.cu). Host code without CUDA.
#pragma once

#include <stdint.h>

#include <algorithm>
#include <vector>

namespace aq {

// The items are dealt by a 32-bit counter, which the warps' last grabs push past
// their number by up to 32 each: a split batch keeps this far from its end.
constexpr uint64_t kMaxSplitItems = ((uint64_t)1 << 32) - ((uint64_t)1 << 22);

// Samples per run of a job (DevJob). The job alone sets it, so a pixel's sum has
// the same bits whether the batch around it, the GPU or the memory at hand split
// the job or not. The runs of a split job are stored, 16 bytes each: about
// kJobRuns of them (nine per lane of a GB300), and at least kPixelRuns per pixel
// with as many samples.
constexpr uint64_t kJobRuns = (uint64_t)1 << 20, kPixelRuns = 16;
inline uint32_t run_spp_of(uint32_t pixels, uint32_t spp) {
    const uint64_t runs = std::max(kPixelRuns, kJobRuns / pixels);
    return (uint32_t)((spp + runs - 1) / runs);
}

// Decides which jobs' pixels are split into runs, for about `lanes` lanes. A
// pixel's samples run one after another on one lane, so the last
// pixels of a small batch kept a few lanes busy long after the others had
// run dry (a 51 x 145 view of the interior at 43 spp took 19 ms alone). A job is
// split when its pixels hold more samples than a kShares-th of the paths that a
// lane runs in the whole batch (four views of up to 128^2 at 6 spp 2.41 -> 0.70 ms, ten of up to
// 300^2 at 16 spp 7.56 -> 2.42, twenty of up to 512^2 at 48 spp 41.4 -> 33.3). A
// large batch keeps whole pixels, and so do more and more jobs of one whose items
// would not fit 32 bits or whose stored runs would take more than 1 GB.
// Returns the items; pixels and stored runs of the split jobs by reference.
constexpr uint64_t kBatchLanes = 768;  // per SM
constexpr uint64_t kShares = 64;       // 16, 32, 128: 34.2, 33.4, 33.4 ms for the twenty views; 64 views at 64 spp
                                       // 190, 180, 175 ms against 177; others within 1%
constexpr uint64_t kMaxStoredRuns = (uint64_t)1 << 26;

template <class Job>
uint32_t split_jobs(std::vector<Job>& jobs, uint64_t lanes, bool split, uint32_t& split_pixels, uint32_t& parts) {
    uint64_t paths = 0;
    for (const Job& j : jobs) paths += (uint64_t)j.pixels * (uint64_t)j.spp;
    for (uint64_t share = std::max<uint64_t>(1, paths / (lanes * kShares));; share *= 2) {
        uint64_t items = 0, stored = 0, pixels = 0;
        for (Job& j : jobs) {
            const uint64_t spp = (uint64_t)j.spp, runs = (spp + j.run_spp - 1) / j.run_spp;
            j.units = (uint32_t)(split && spp > share ? runs : 1);
            j.item_begin = (uint32_t)items;
            j.part_begin = j.done_begin = 0;
            if (j.units > 1) {
                j.part_begin = (uint32_t)stored;
                j.done_begin = (uint32_t)pixels;
                stored += runs * j.pixels;
                pixels += j.pixels;
            }
            items += (uint64_t)j.units * j.pixels;
        }
        if (stored == 0 || (items <= kMaxSplitItems && stored <= kMaxStoredRuns)) {
            parts = (uint32_t)stored;
            split_pixels = (uint32_t)pixels;
            return (uint32_t)items;
        }
    }
}

}  // namespace aq
