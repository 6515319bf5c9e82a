// Scoring on bit planes (nw_bits.cu): what the plan of a call takes from it.
#pragma once

#include "msa_internal.hpp"

namespace msa {

// A set of rows sequences: sorted a .. a + 32 / lanes - 1, R rows per lane, nst
// strips; its tasks (one per column group from its own, or from the first
// group of the launch) start at `first`.
struct BitSet {
    uint32_t a, first;
    uint16_t lanes, R;
    uint32_t nst;
};

struct BitParams {
    const uint8_t *units;
    const uint64_t *uoff;
    const uint32_t *eff;
    const uint32_t *sorted;
    uint32_t nclean, ngroups, g0;   // column groups; the first one scored here
    const BitSet *sets;
    uint32_t nsets, ntasks;
    uint32_t *match;                // match words of group q: kBitRows rows of bit_pitch(gcols[q]) at goff[q]
    const uint64_t *goff;
    const uint32_t *gcols;          // longest sequence of each group
    uint2 *bound;                   // bound_words per warp: a boundary row of bit_bound(columns) per sequence of a set
    uint64_t bound_words;
    int32_t *out;
    int32_t u, g;
    uint32_t letters;               // those that match themselves
    uint32_t nchain;                // tasks of the first sets, taken by whole CTAs
    int *err;                       // set when a wait between strips ran out
    unsigned long long *counter;    // of chained tasks, and of the others
    unsigned long long wait_ns;     // limit of the waits between strips
};

// Rows of match words: the letters, and which columns lie within a sequence.
constexpr int kBitLetters = 24, kBitRows = kBitLetters + 1;
// Rows of the ring: the letters, all ones (rows past a sequence's end), and the
// two planes of the row above a strip.
constexpr int kRingAll = kBitLetters, kRingTop = kRingAll + 1, kRingRows = kRingTop + 2;
constexpr int kBitWarps = 4;   // per CTA
// Longest columns: the sums of one lane's columns take 12 bits.
constexpr uint32_t kBitMaxCols = 40000;

// Progress of a chained set: `columns` columns of the last row of strip `strip` may be
// read. The word of any later strip is greater than every word of an earlier one: a
// sequence of 2^30 units has more than 2^20 strips.
__host__ __device__ constexpr unsigned long long strip_progress(uint32_t strip, uint32_t columns)
{
    return (unsigned long long) (strip + 1) << 32 | columns;
}

__host__ __device__ __forceinline__ uint32_t bit_pitch(uint32_t ncols) { return (ncols + 31) / 32 * 32 + 64; }
__host__ __device__ __forceinline__ uint32_t bit_bound(uint32_t ncols) { return (ncols + 31) / 32 * 32 + 96; }

// What of a job runs on bit planes: all pairs with a sequence of group g0 or
// later (the batched kernel takes the first 32 g0 sequences among themselves).
struct BitPlan {
    uint32_t g0 = 0;
    std::vector<BitSet> sets;
    std::vector<uint32_t> gcols;
    std::vector<uint64_t> goff;
    uint64_t ntasks = 0, nchain = 0, match_words = 0, bound_words = 0;
};

// u of a table of this kind (0 for others), and the letters that score M against themselves.
struct BitTable {
    int32_t u;
    uint32_t letters;
};
BitTable bit_table(const ExtTable &t);
// Sets and split for the sorted lengths `eff`; no tasks where the batched kernel is the faster one.
BitPlan plan_bits(const std::vector<uint32_t> &eff, uint32_t num_sms);
// CTAs of a plan's launch.
int bits_grid(msa_ctx *ctx, const BitPlan &plan, uint64_t *grid);
cudaError_t launch_match(const BitParams &p, cudaStream_t s);
cudaError_t launch_bits(const BitParams &p, uint64_t grid, cudaStream_t s);

}  // namespace msa
