// For every length up to 5,000 and a partner of as many 3-unit blocks: whether the
// profile of the first reaches as far as their strips. Prints the number of pairs and of
// those that do not. Touches no device.
#include <algorithm>
#include <cstdio>

#include "../../msa_b200/csrc/msa_internal.hpp"

int main()
{
    unsigned pairs = 0, short_of = 0;
    for(uint64_t a = 1; a <= 5000; ++a)
        for(uint64_t b = a; b <= a + 2; ++b) {
            if((a + 2) / 3 != (b + 2) / 3) continue;
            // Strips of one height, an even number of rows per lane, 32 at most.
            const uint64_t nst = (b + 1023) / 1024, R = ((b + 32 * nst - 1) / (32 * nst) + 1) & ~1ull;
            ++pairs;
            for(uint64_t rows : {32 * R * nst, (b + 511) / 512 * 512}) short_of += msa::prof_pitch(a) < rows;
        }
    std::printf("%u %u\n", pairs, short_of);
    return 0;
}
