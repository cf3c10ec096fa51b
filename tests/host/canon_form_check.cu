// Host-side check of canon_form() (cablegen_b200/csrc/board.cuh): for formation
// masks given as hex 16-bit cell sets in argv[1..] (bit c = cell c holds 0xf), in
// every orientation, random boards with those 0xf cells are taken in each view
// and the form the plan names is compared with the full canonical().  Prints
// "<mask> <form> <boards checked> <mismatches>" per mask and orientation.
#include "../../cablegen_b200/csrc/board.cuh"
#include <cstdio>
#include <cstdlib>
#include <random>

int main(int argc, char **argv)
{
    using namespace cgb;
    std::mt19937_64 rng(7);
    for (int a = 1; a < argc; a++) {
        const unsigned cells = (unsigned)std::strtoul(argv[a], nullptr, 16);
        u64 base = 0, shapes[8];
        for (int c = 0; c < 16; c++)
            if (cells >> c & 1) base |= 0xFull << (60 - 4 * c);
        images(base, shapes);
        for (u64 shape : shapes) {
            const CanonPlan plan = make_canon_plan(shape, false);
            u64 checked = 0, bad = 0;
            for (int it = 0; it < 5000 && plan.form != CANON_LIST; it++) {
                u64 x = shape, v[4];
                for (int c = 0; c < 16; c++)
                    if (!((shape >> (60 - 4 * c)) & 0xF) && rng() % 3) x |= (rng() % 15) << (60 - 4 * c);
                views(x, v);
                for (int k = 0; k < 4; k++) {
                    const u64 y = plan.form == CANON_ONE        ? canon_form<CANON_ONE>(v[k], plan, k)
                                  : plan.form == CANON_DIAGONAL ? canon_form<CANON_DIAGONAL>(v[k], plan, k)
                                                                : canon_form<CANON_MIRROR>(v[k], plan, k);
                    checked++;
                    bad += y != canonical(v[k]);
                }
            }
            std::printf("%04x %d %llu %llu\n", cells, plan.form, (unsigned long long)checked, (unsigned long long)bad);
        }
    }
    return 0;
}
