// Sizes of the sort by buckets for the key counts given: "n ok coarse coarse_cap grid words" each.
#include "../../cablegen_b200/csrc/bucketplan.h"
#include <cstdio>
#include <cstdlib>

int main(int argc, char **argv)
{
    std::printf("%llu\n", (unsigned long long)cgb::BUCKET_SORT_KEYS);
    for (int i = 1; i < argc; i++) {
        cgb::BucketPlan p;
        const unsigned long long n = std::strtoull(argv[i], nullptr, 10);
        const bool ok = cgb::plan_buckets(n, &p);
        std::printf("%llu %d %u %u %u %llu\n", n, ok ? 1 : 0, p.coarse, p.coarse_cap, p.grid, (unsigned long long)p.words);
    }
    return 0;
}
