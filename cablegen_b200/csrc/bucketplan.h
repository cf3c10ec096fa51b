// bucketplan.h -- sizes of one sort by buckets (bucketsort.cu), host arithmetic alone.
#pragma once
#include <algorithm>
#include <cmath>
#include <cstdint>

namespace cgb {

constexpr uint32_t BK_TARGET = 1800;   // keys per bucket aimed at
constexpr uint32_t BK_CAP = 4096;      // keys a bucket holds; 2.27 x the target: with 32 samples per bucket a
                                       // size is off by 18 % (one sigma), so this is seven sigma
constexpr uint32_t BK_FAN = 512;       // buckets of one partition step
constexpr uint32_t BK_ONE_STEP = 400 * BK_TARGET;  // keys up to which one step is taken: 8192 samples bound 400
                                       // buckets as well as 20 each do (2.27 x the size: one in a million)
constexpr uint32_t BK_COARSE = 512;    // coarse buckets of the two-step form
constexpr uint32_t BK_SAMPLES = 8192;
// The most keys one call takes: 512 coarse buckets of 901120 keys of room (seven
// sigma above 327680), which 512 fine buckets of the target size each take up.
constexpr uint64_t BUCKET_SORT_KEYS = 160ull << 20;

// arrays of one sort's control words (u32 indexes), which start with the counts of
// the coarse buckets
constexpr uint32_t A_COARSE = 0, A_BASE = A_COARSE + BK_COARSE, A_NUM = A_BASE + BK_COARSE, A_FINE = A_NUM + BK_COARSE;

struct BucketPlan {
    uint64_t n = 0;              // keys at most
    bool small = false;          // expected to fit one CTA: nothing but its sort is launched
    uint32_t coarse = 0, coarse_cap = 0;  // two steps: coarse buckets and their space
    uint32_t grid = 0;           // buckets at most
    uint64_t words = 0, arrays_at = 0;
};

// Sizes of one call.  Two steps above BK_ONE_STEP keys: coarse buckets of
// equal expected size, their space seven sigma above it (a coarse bucket is
// bounded by 64 samples, or by 8192 / coarse).  As many coarse buckets as fine ones
// in each, and more where one would hold more fine buckets than a step tells
// apart (above 99M keys; the space falls as their number grows).
inline bool plan_buckets(uint64_t n, BucketPlan *p)
{
    *p = BucketPlan{};
    p->n = n;
    if (n > BUCKET_SORT_KEYS) return false;
    if (n <= BK_CAP) {
        p->grid = 1;
    } else if (n <= BK_ONE_STEP) {
        p->grid = (uint32_t)((n + BK_TARGET - 1) / BK_TARGET);
    } else {
        auto space = [n](uint32_t c) {
            const double per = std::min(64.0, (double)BK_SAMPLES / c);
            return ((uint64_t)((double)n / c * (1.0 + 7.0 / std::sqrt(per))) + 63) / 64 * 64;
        };
        uint32_t c = (uint32_t)std::ceil(std::sqrt((double)n / BK_TARGET));
        while (c < BK_COARSE && space(c) > (uint64_t)BK_FAN * BK_TARGET) c++;
        if (c > BK_COARSE) c = BK_COARSE;
        const uint64_t cap = space(c);
        if (cap > (uint64_t)BK_FAN * BK_TARGET) return false;
        p->coarse = c;
        p->coarse_cap = (uint32_t)cap;
        p->grid = (uint32_t)(n / BK_TARGET) + c;
    }
    p->words = A_FINE + 2 * p->grid;
    return true;
}

}  // namespace cgb
