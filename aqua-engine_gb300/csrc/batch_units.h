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

// Splits the pixels' samples into units (DevJob) for about `lanes` lanes (the
// GPU's at the default launch shape, so that an image's rounding does not
// depend on the shape). A pixel's samples run one after another on one lane, so the last
// pixels of a small batch kept a few lanes busy long after the others had
// run dry (a 51 x 145 view of the interior at 43 spp took 19 ms alone); units
// short enough that each lane takes kUnitsPerLane of them bound that tail
// (four views of up to 128^2 at 6 spp 2.41 -> 0.81 ms, ten of up to 300^2 at 16
// spp 7.56 -> 3.31, twenty of up to 512^2 at 48 spp 41.4 -> 35.7). A large
// batch keeps whole pixels, and so does one whose items would not fit 32 bits.
// Returns the items; pixels and partial sums of the split jobs by reference.
constexpr uint64_t kBatchLanes = 768;  // per SM
constexpr uint64_t kUnitsPerLane = 64;  // 16, 32 and 128: within 4%

template <class Job>
uint32_t split_jobs(std::vector<Job>& jobs, uint64_t lanes, bool split, uint32_t& split_pixels, uint32_t& parts) {
    uint64_t paths = 0;
    for (const Job& j : jobs) paths += (uint64_t)j.pixels * (uint64_t)j.spp;
    const uint64_t run = std::max<uint64_t>(1, paths / (lanes * kUnitsPerLane));
    auto unit_spp = [&](const Job& j) {
        return split && run < (uint64_t)j.spp ? (uint32_t)run : (uint32_t)j.spp;
    };
    uint64_t total = 0;
    for (const Job& j : jobs) total += ((uint64_t)j.spp + unit_spp(j) - 1) / unit_spp(j) * (uint64_t)j.pixels;
    if (total > kMaxSplitItems) split = false;
    uint32_t items = 0;
    split_pixels = parts = 0;
    for (Job& j : jobs) {
        j.unit_spp = unit_spp(j);
        j.units = ((uint32_t)j.spp + j.unit_spp - 1) / j.unit_spp;
        j.item_begin = items;
        j.part_begin = j.done_begin = 0;
        if (j.units > 1) {
            j.part_begin = parts;
            j.done_begin = split_pixels;
            parts += j.units * j.pixels;
            split_pixels += j.pixels;
        }
        items += j.units * j.pixels;
    }
    return items;
}

}  // namespace aq
