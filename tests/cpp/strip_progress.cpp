// The plan of a job with one sequence of 70 million bases among 5,000 of 150 on bit
// planes, and the progress words of its strips: prints the strips of the longest
// chained set and how many neighbouring strips' words are out of order. Touches no
// device.
#include <cstdio>
#include <vector>

#include "../../msa_b200/csrc/nw_bits.hpp"

int main()
{
    std::vector<uint32_t> eff(5001, 150);
    eff[0] = 70000000;
    const msa::BitPlan plan = msa::plan_bits(eff, 148);
    uint32_t strips = 0, columns = 0;
    for(const msa::BitSet &s : plan.sets)
        if(s.first < plan.nchain && s.nst > strips) strips = s.nst;
    for(uint32_t q = plan.g0; q < plan.gcols.size(); ++q) columns = std::max(columns, plan.gcols[q]);
    uint64_t wrong = 0;
    for(uint32_t st = 0; st < strips; ++st) {
        // What a strip publishes grows with its columns, and lies below what any later
        // strip publishes or waits for; the words of a slot start from 0.
        const auto first = msa::strip_progress(st, 1), last = msa::strip_progress(st, columns),
                   end = msa::strip_progress(st, 0xffffffffu), next = msa::strip_progress(st + 1, 1);
        wrong += !(0 < first && (columns == 1 || first < last) && last < end && end < next);
    }
    std::printf("%u %u %llu\n", strips, columns, (unsigned long long) wrong);
    return 0;
}
