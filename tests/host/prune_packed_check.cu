// Host-side check of prune_packed() (cablegen_b200/csrc/board.cuh): boards (u64
// file in argv[1]) under each parameter set "stsl,ltc,smallest_large" of argv[2..]
// against prune_board().  Prints "<on> <boards> <pruned> <mismatches>" per set.
#include "../../cablegen_b200/csrc/board.cuh"
#include <cstdio>
#include <vector>

int main(int argc, char **argv)
{
    std::vector<cgb::u64> b;
    FILE *f = argc > 2 ? std::fopen(argv[1], "rb") : nullptr;
    if (!f) return 2;
    for (cgb::u64 x; std::fread(&x, 8, 1, f) == 1;) b.push_back(x);
    std::fclose(f);
    for (int a = 2; a < argc; a++) {
        cgb::PruneParams p{0, 0, 0, 1};
        if (std::sscanf(argv[a], "%lld,%lld,%lld", &p.stsl, &p.ltc, &p.smallest_large) != 3) return 2;
        cgb::PackedPrune t;
        cgb::build_packed_prune(p, &t);
        size_t pruned = 0, bad = 0;
        for (cgb::u64 x : b) {
            const bool want = cgb::prune_board(x, p);
            pruned += want;
            if (t.on) bad += cgb::prune_packed(x, t.w, 1, t.add, t.test) != want;
        }
        std::printf("%u %zu %zu %zu\n", t.on, b.size(), pruned, bad);
    }
    return 0;
}
