// Host build of the occupancy cache (cpabdiffeo_b200/csrc/cpab_occupancy.h) for tests/test_occupancy_cache.py.
#include "cpab_occupancy.h"

// How many queries `rounds` rounds of launches of `kernels` kernels at `sizes` sizes each make; -1: a wrong answer.
extern "C" long occupancy_queries(int kernels, int sizes, int rounds)
{
    static char kern[64];
    cpab::OccupancyCache cache;
    long asked = 0;
    for (int r = 0; r < rounds; ++r)
        for (int k = 0; k < kernels; ++k)
            for (int s = 0; s < sizes; ++s) {
                const int got = cache.get(kern + k, 128, 1024 + 16 * (size_t)s, [&] {
                    ++asked;
                    return 100 * k + s % 7;
                });
                if (got != 100 * k + s % 7) return -1;
            }
    return asked;
}
