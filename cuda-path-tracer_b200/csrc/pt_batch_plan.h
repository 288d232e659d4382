// pt_batch_plan.h — the order in which batch_paths (pt_batch.cu) draws the samples of a batch.
//
// All pixels advance together, a sample at a time (pt_paths.h), but jobs may ask for very different numbers of
// samples.  A level is a range of passes in which the same jobs still have samples to draw: those with at least
// as many as the level's last pass.  With the jobs sorted by samples, most first, a level's pixels are the first
// `pixels` of the sorted order, so every item drawn is a sample of some pixel.  (Numbering items over all pixels
// and dropping those past a job's count made one 16x16 job of 256 samples beside 307,200 pixels of one draw 79
// million items for 370,000 samples.)  Once a level has fewer than `few` pixels (two per lane, the size below which a
// batch runs in the tail kernel alone), an item is a pixel with all its samples still to draw: from there on
// every pixel can have lanes of its own, and drawing pass after pass would only keep lanes from their paths.
#pragma once

#include <algorithm>
#include <vector>
#include "pt_internal.h"

namespace ptb {

struct BatchLevel {
    unsigned long long first_item;
    uint32_t pixels;            // of the sorted order
    int32_t drawn;              // samples of each pixel drawn by the levels before, when an item is all the others; -1: an item is one sample
};
static_assert(sizeof(BatchLevel) == 16, "level record is 16 bytes");

// The sample (or the rest of a pixel's samples) that `item` stands for: `place` in the sorted order of pixels.
struct BatchItem { uint32_t place; int32_t drawn; };
PT_HD inline BatchItem batch_item(const BatchLevel *levels, int32_t count, unsigned long long item) {
    int32_t lo = 0, hi = count - 1;
    while (lo < hi) {
        const int32_t mid = (lo + hi + 1) / 2;
        if (levels[mid].first_item <= item) lo = mid; else hi = mid - 1;
    }
    const BatchLevel l = levels[lo];
    item -= l.first_item;
    return {(item >> 32) ? uint32_t(item % l.pixels) : uint32_t(item) % l.pixels, l.drawn};
}
// Which sorted job holds the pixel at `place`: first[k] is the place of sorted job k's first pixel.
PT_HD inline int32_t batch_job_at(const uint32_t *first, int32_t jobs, uint32_t place) {
    int32_t lo = 0, hi = jobs - 1;
    while (lo < hi) {
        const int32_t mid = (lo + hi + 1) / 2;
        if (first[mid] <= place) lo = mid; else hi = mid - 1;
    }
    return lo;
}

struct BatchPlan {
    std::vector<int32_t> order;         // jobs, most samples first (equal ones as given)
    std::vector<uint32_t> first;        // per sorted job
    std::vector<BatchLevel> levels;
    unsigned long long items = 0;
};
// `pixels` and `samples` per job; all pixels together fewer than 2^32.
inline BatchPlan batch_plan(const std::vector<int32_t> &pixels, const std::vector<int32_t> &samples, int64_t few) {
    BatchPlan p;
    const size_t n = samples.size();
    for (size_t k = 0; k < n; k++) p.order.push_back(int32_t(k));
    std::stable_sort(p.order.begin(), p.order.end(), [&](int32_t a, int32_t b) { return samples[size_t(a)] > samples[size_t(b)]; });
    uint32_t place = 0;
    for (int32_t k : p.order) { p.first.push_back(place); place += uint32_t(pixels[size_t(k)]); }
    int32_t drawn = 0;
    for (size_t active = n; active > 0;) {      // jobs from the fewest samples up
        const int32_t upto = samples[size_t(p.order[active - 1])];
        const bool rest = int64_t(place) < few;
        p.levels.push_back({p.items, place, rest ? drawn : -1});
        p.items += (unsigned long long)place * (rest ? 1ull : (unsigned long long)(upto - drawn));
        if (rest) break;
        drawn = upto;
        while (active > 0 && samples[size_t(p.order[active - 1])] == upto) place -= uint32_t(pixels[size_t(p.order[--active])]);
    }
    return p;
}

} // namespace ptb
