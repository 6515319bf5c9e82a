// All-pairs Needleman-Wunsch kernels for sm_100a.
//
// Recurrence (linear gap, global alignment), exactly the one of
// sequential::align_pair (src/pairwise/needleman/impl/sequential.cpp:29-68):
//   H[0][j] = -j*g, H[i][0] = -i*g,
//   H[i][j] = max(H[i-1][j-1] + T[a_i][b_j], H[i][j-1] - g, H[i-1][j] - g).
// Scores are small integers, so int32 (or, where a host-side bound proves it
// cannot overflow, 16-bit lanes) reproduces the reference's float scores
// exactly.
//
// Work layout: one warp runs one task. A task is one (rows, cols) pair, or on
// the 16-bit path two pairs sharing the column sequence (the two rows
// sequences of a rows pair, one per 16-bit half). Lane k owns R consecutive
// rows of a 32*R-row strip and sweeps the columns one step behind lane k-1:
// the cell above its first row arrives from lane k-1 by __shfl_up_sync, so a
// strip advances one anti-diagonal per step with no block-wide barrier. Strips
// of a long rows sequence are chained through a per-warp boundary row in
// global memory. Substitution scores come from a per-sequence score profile
// (one int8 row per residue code) staged per strip in shared memory, in planes
// whose 16-byte (or 8-byte) loads are bank-conflict free whatever codes the
// lanes hold; the batched kernel keeps part of each strip as packed bytes
// (Layout) to halve those rows' shared-memory traffic.
#include <cstdio>
#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>

#include "nw_bits.hpp"

namespace msa {
namespace dev {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kEnd = MSA_UNIT_END;

// Sign-extended byte K of w.
template <int K>
__device__ __forceinline__ int32_t sbyte(uint32_t w)
{
    int32_t r;
    asm("prmt.b32 %0, %1, 0, %2;" : "=r"(r) : "r"(w), "n"((K) | ((K | 8) << 4) | ((K | 8) << 8) | ((K | 8) << 12)));
    return r;
}

// Two sign-extended bytes K of lo and hi packed as int16x2 (lo in bits 0-15).
template <int K>
__device__ __forceinline__ uint32_t sbyte2(uint32_t lo, uint32_t hi)
{
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(lo), "r"(hi),
        "n"((K) | ((K | 8) << 4) | ((4 + K) << 8) | (((4 + K) | 8) << 12)));
    return r;
}

__device__ __forceinline__ uint32_t dup16(int32_t v) { return ((uint32_t) v & 0xffffu) | ((uint32_t) v << 16); }

// One cell: max(up - g, max(left - g, diag + s)). The inner max depends only on
// the previous column, so the serial chain down a lane's rows is one DPX op.
struct Wide {
    using W = int32_t;
    __device__ static __forceinline__ W cell(W d, W s, W left, W up, W ng)
    {
        const W ds = d + s;
        const W t = __viaddmax_s32(left, ng, ds);
        return __viaddmax_s32(up, ng, t);
    }
    __device__ static __forceinline__ W splat(int32_t v) { return v; }
    // max(left - g, diag + s): the part of a cell that needs only the previous column.
    __device__ static __forceinline__ W cell_part(W d, W s, W left, W ng) { return __viaddmax_s32(left, ng, d + s); }
    // max(up - g, part): the serial part down a lane's rows.
    __device__ static __forceinline__ W cell_chain(W up, W ng, W part) { return __viaddmax_s32(up, ng, part); }
};

// Two cells per 32-bit lane (16-bit halves: the two rows sequences of a rows
// pair). The lane state is not H but T(i,j) = H(i,j) + g*(i + j), unsigned per
// half. The gap terms cancel out of the recurrence:
//   T = max(T_left, T_up, T_diag + (s + 2g)),
// one vadd2 (FMA pipe, off the row chain) and one vimax3_u16x2 (ALU pipe, the
// only operation on the chain down a lane's rows); the staged profile words
// hold s + 2g. Row 0 and column 0 of T are 0. Over every path T = the sum of
// (s + 2g) over its matched cells, so 0 <= T(i,j) <= min(i,j)*(smax + 2g) when
// smin + 2g >= 0 (narrow_ok checks both), and the diagonal candidate never
// exceeds the cell it competes for: no half leaves [0, 0xffff]. Every operation
// stays inside its 16-bit half, so rows past a sequence's end (padding, or the
// shorter sequence of the pair) hold values that never reach a scored cell.
struct Narrow {
    using W = uint32_t;
    // H(rows, cols) from the low or high half of T(rows, cols).
    __device__ static __forceinline__ int32_t lo(W w, int32_t g, int rows, int cols) { return (int32_t) (w & 0xffffu) - g * (rows + cols); }
    __device__ static __forceinline__ int32_t hi(W w, int32_t g, int rows, int cols) { return (int32_t) (w >> 16) - g * (rows + cols); }
    __device__ static __forceinline__ W splat(int32_t v) { return dup16(v); }
};

// R profile bytes of one lane for residue code b, from the staged strip.
// Layout [code][plane][lane][16] with R/16 planes (R >= 16) or [code][lane][R].
template <int R>
struct ProfWords {
    static constexpr int NW = R / 4;
    uint32_t w[NW];
    __device__ __forceinline__ void load(const int8_t *sprof, int b, int lane)
    {
        constexpr int SH = 32 * R;
        if constexpr(R >= 16) {
#pragma unroll
            for(int p = 0; p < R / 16; ++p) {
                const uint4 v = *reinterpret_cast<const uint4 *>(sprof + b * SH + p * 512 + lane * 16);
                w[4 * p + 0] = v.x; w[4 * p + 1] = v.y; w[4 * p + 2] = v.z; w[4 * p + 3] = v.w;
            }
        } else if constexpr(R == 8) {
            const uint2 v = *reinterpret_cast<const uint2 *>(sprof + b * SH + lane * 8);
            w[0] = v.x; w[1] = v.y;
        } else {
            static_assert(R == 4, "R must be 4, 8, 16 or 32");
            w[0] = *reinterpret_cast<const uint32_t *>(sprof + b * SH + lane * 4);
        }
    }
};

// Copies strip rows [i0, i0 + 32R) of a sequence profile ([code][Lp] int8,
// global) into the warp's shared staging area.
template <int R>
__device__ __forceinline__ void stage_profile(int8_t *sprof, const int8_t *__restrict__ gprof,
                                              uint32_t lp, int i0, int lane)
{
    constexpr int SH = 32 * R;
    constexpr int CH = SH / 16;   // 16-byte chunks per code row
    for(int c = lane; c < kAlpha * CH; c += 32) {
        const int b = c / CH, w = c - b * CH;
        const uint4 v = __ldg(reinterpret_cast<const uint4 *>(gprof + (size_t) b * lp + i0) + w);
        int dst;
        if constexpr(R >= 16) {
            const int ln = w / (R / 16), pl = w - ln * (R / 16);
            dst = b * SH + pl * 512 + ln * 16;
        } else {
            dst = b * SH + w * 16;   // [code][lane][R] is the natural order for R <= 16
        }
        *reinterpret_cast<uint4 *>(sprof + dst) = v;
    }
}

// Runs one task in 32-bit lanes on the calling warp (the plain and the
// reference-orientation kernels): ncolsA columns of colsA against nrows rows.
// kSkip: END units in the columns copy the left neighbour
// (sequential.cpp:53-60) instead of scoring. Returns H[nrows][ncolsA] (resA);
// colsB, ncolsB and resB are unused (resB = 0).
template <int R, class K, bool kSkip>
__device__ __forceinline__ void run_task(const int8_t *__restrict__ gprof, uint32_t lp, int nrows,
                                         const uint8_t *__restrict__ colsA, int ncolsA,
                                         const uint8_t *__restrict__ colsB, int ncolsB,
                                         int8_t *sprof, uint32_t *__restrict__ bound,
                                         int32_t g, int lane, int32_t &resA, int32_t &resB)
{
    static_assert(std::is_same<K, Wide>::value, "run_task sweeps 32-bit lanes");
    using W = typename K::W;
    constexpr int SH = 32 * R;
    const int nstrips = (nrows + SH - 1) / SH;
    const W ng = K::splat(-g);
    int32_t outA = 0, outB = 0;

    for(int s = 0; s < nstrips; ++s) {
        const int i0 = s * SH;
        const bool first = (s == 0);
        const bool last = (s == nstrips - 1);
        const int rl = nrows - 1 - i0;              // last row's offset (meaningful in the last strip)
        const int klast = last ? rl / R : 31;
        const int rlast = rl - (rl / R) * R;

        __syncwarp();
        stage_profile<R>(sprof, gprof, lp, i0, lane);
        __syncwarp();

        W H[R];
#pragma unroll
        for(int r = 0; r < R; ++r) H[r] = K::splat(-(i0 + lane * R + r + 1) * g);
        W diag = K::splat(-(i0 + lane * R) * g);    // H[row_top - 1][0]
        W hlast = H[R - 1];

        // Boundary row of the previous strip, prefetched 32 columns at a time
        // (lane q holds column c0 + q); lane 0 picks its column by shuffle.
        uint32_t bq_cur = 0, bq_nxt = 0;
        if(!first) {
            bq_cur = bound[lane];
            bq_nxt = bound[32 + lane];
        }
        int clampA = ncolsA - 1;
        uint32_t curA = colsA[min(max(-lane, 0), clampA)];

        const int tend = ncolsA + klast;
        for(int t = 0; t < tend; ++t) {
            W up = __shfl_up_sync(kFull, hlast, 1);
            if(!first) {
                if((t & 31) == 0 && t > 0) {
                    bq_cur = bq_nxt;
                    bq_nxt = bound[t + 32 + lane];
                }
                const uint32_t bv = __shfl_sync(kFull, bq_cur, t & 31);
                if(lane == 0) up = (W) bv;
            } else if(lane == 0) {
                up = K::splat(-(t + 1) * g);
            }
            const int j = t - lane;
            const int jn = min(max(j + 1, 0), clampA);
            const uint32_t nxtA = colsA[jn];

            if(j >= 0 && j < ncolsA) {
                const bool skip = kSkip && curA == (uint32_t) kEnd;
                if(!skip) {
                    ProfWords<R> pa;
                    pa.load(sprof, (int) curA, lane);
                    W d = diag, u = up;
#pragma unroll
                    for(int q = 0; q < R / 4; ++q) {
#pragma unroll
                        for(int k = 0; k < 4; ++k) {
                            const int r = 4 * q + k;
                            W sc;
                            if(k == 0) sc = sbyte<0>(pa.w[q]);
                            else if(k == 1) sc = sbyte<1>(pa.w[q]);
                            else if(k == 2) sc = sbyte<2>(pa.w[q]);
                            else sc = sbyte<3>(pa.w[q]);
                            const W h = K::cell(d, sc, H[r], u, ng);
                            d = H[r];
                            H[r] = h;
                            u = h;
                        }
                    }
                }
                hlast = H[R - 1];
                if(!last && lane == 31) bound[j] = (uint32_t) hlast;
                if(last && lane == klast && j == ncolsA - 1) {
                    W v = H[0];
#pragma unroll
                    for(int r = 1; r < R; ++r) if(r == rlast) v = H[r];
                    outA = (int32_t) v;
                }
                diag = up;
            }
            curA = nxtA;
        }
        if(last) {
            resA = __shfl_sync(kFull, outA, klast);
            resB = __shfl_sync(kFull, outB, klast);
        }
    }
    __syncwarp();
}

__device__ __forceinline__ uint64_t tri_index(uint32_t i, uint32_t j)
{
    const uint64_t hi = i > j ? i : j, lo = i > j ? j : i;
    return hi * (hi - 1) / 2 + lo;
}

}  // namespace dev

// ---------------------------------------------------------------- params

struct NwParams {
    const uint8_t *units;
    const uint64_t *uoff;
    const uint32_t *eff;
    const uint32_t *plen;
    const int8_t *prof;
    const uint64_t *poff;
    const uint32_t *plp;
    const uint32_t *sorted;     // clean sequences, eff descending
    uint32_t nclean;
    const uint64_t *row_task;   // persistent: first task of each sorted row (nclean + 1)
    const uint8_t *row_narrow;  // persistent: 16-bit tasks for this row
    uint64_t ntasks;
    const uint32_t *gpairs;     // generic path: (rows orig, cols orig) pairs
    uint64_t ngeneric;
    uint32_t *bound;            // per resident warp: bound_stride words
    uint64_t bound_stride;
    int32_t *out;
    int32_t g;
    unsigned long long *counter;
};

// Sorted-space pair (a, b), a < b, from its a-major linear index k.
__device__ __forceinline__ void decode_pair(uint64_t k, uint32_t n, uint32_t &a, uint32_t &b)
{
    // Row a starts at a*(2n - a - 1)/2.
    const double nn = (double) n - 0.5;
    double x = nn - sqrt(nn * nn - 2.0 * (double) k);
    int64_t aa = (int64_t) floor(x);
    if(aa < 0) aa = 0;
    auto start = [n](int64_t r) -> uint64_t { return (uint64_t) r * (2 * (uint64_t) n - (uint64_t) r - 1) / 2; };
    while(aa > 0 && start(aa) > k) --aa;
    while(start(aa + 1) <= k) ++aa;
    a = (uint32_t) aa;
    b = (uint32_t) (aa + 1 + (k - start(aa)));
}

template <int R>
__device__ __forceinline__ void clean_pair_task(const NwParams &p, uint32_t a, uint32_t b,
                                                int8_t *sprof, uint32_t *bound, int lane)
{
    const uint32_t ri = p.sorted[a], ci = p.sorted[b];
    int32_t ra = 0, rb = 0;
    dev::run_task<R, dev::Wide, false>(p.prof + p.poff[ri], p.plp[ri], (int) p.eff[ri],
                                       p.units + p.uoff[ci], (int) p.eff[ci], nullptr, 0,
                                       sprof, bound, p.g, lane, ra, rb);
    if(lane == 0) p.out[dev::tri_index(ri, ci)] = ra;
}

// Plain: one launch per length bucket (a range of the a-major pair order),
// each warp takes pairs k_lo + w, k_lo + w + W, ... in a fixed stride.
template <int R, int WPB>
__global__ void __launch_bounds__(WPB * 32) nw_plain_kernel(NwParams p, uint64_t k_lo, uint64_t k_hi)
{
    extern __shared__ __align__(16) int8_t smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int8_t *sprof = smem + warp * (kAlpha * 32 * R);
    const uint64_t gw = (uint64_t) blockIdx.x * WPB + warp;
    const uint64_t nw = (uint64_t) gridDim.x * WPB;
    uint32_t *bound = p.bound + gw * p.bound_stride;
    for(uint64_t k = k_lo + gw; k < k_hi; k += nw) {
        uint32_t a, b;
        decode_pair(k, p.nclean, a, b);
        clean_pair_task<R>(p, a, b, sprof, bound, lane);
    }
}

// ---------------------------------------------------------------- batched kernel
//
// One persistent launch over every clean pair. The length-sorted sequences
// are taken two at a time as a rows pair (X1, X2) = (sorted 2k, sorted 2k+1);
// a task is one rows pair against a group of W consecutive column sequences,
// one per warp of the CTA. On the 16-bit path the two rows sequences share
// every 32-bit lane: X1 in the low half, X2 in the high half, against the same
// column residue, so one staged profile word is already the packed score pair
// and each lane does two cells per instruction. The profile strip is staged
// once per CTA and shared by its W warps. Where the 16-bit bound fails the
// task runs both rows sequences one after the other in 32-bit lanes.
// CTAs take tasks from a global counter in cost order (longest rows pairs
// first), so the tail of the launch is the cheapest work.

// One all-pairs job as the batched kernels see it: its store, score profiles,
// length order, per-rows-pair 16-bit flags and output triangle.
struct JobView {
    const uint8_t *units;
    const uint64_t *uoff;
    const uint32_t *eff;
    const int8_t *prof;
    const uint64_t *poff;
    const uint32_t *plp;
    const uint32_t *sorted;     // clean sequences, eff descending
    const uint8_t *row_narrow;  // per rows pair k: kRowNarrow and the flags beside it; for stacked ones on the first
    int32_t *out;
    uint32_t nclean;
    int32_t g;
};

// row_narrow flags: 16-bit lanes; rows pairs k and k + 1 (kRowQuad), or k to
// k + 3 (kRowOct), stacked in one warp (stack_task), their tasks all under k.
// Rows pairs of several strips: kRowLong runs its 16-bit lanes on a moving base
// (sweep_long), kRowChain makes every strip a task of its own, of up to 32 x 32
// rows or 32 x 16 (chain_form).
constexpr uint8_t kRowNarrow = 1, kRowQuad = 2, kRowLong = 4, kRowChain = 8, kRowR16 = 16, kRowOct = 64;

// Steps between moves of a long strip's base; see sweep_long.
constexpr int kRebase = 512;
// Columns between two publications of a chained strip's progress.
constexpr int kPublish = 64;
// A chained strip waits at most this long for the one above it, unless the context
// says otherwise (msa_nw_set_wait).
constexpr uint32_t kStripWaitUs = 5000000;
// Entries of a boundary row's base table for ncols columns, and the tables it
// has: strip s writes table s mod 8 and reads the one before. A chained strip is
// at least 128 steps behind the one it follows when it moves its base, so the
// strip that writes a table again, 8 on, is 896 steps behind the last reader of
// an entry that serves 512 columns.
__host__ __device__ __forceinline__ uint32_t base_entries(uint32_t ncols) { return (ncols + 31) / kRebase + 2; }
constexpr uint32_t kBaseTables = 8;
// Words of a boundary row and its base tables.
__host__ __device__ __forceinline__ uint64_t bound_words(uint32_t ncols)
{
    return ((uint64_t) ncols + 160 + 2 * kBaseTables * base_entries(ncols) + 31) / 32 * 32;
}
// The same for the columns of a rows pair, its second sequence and those after
// it in the sorted order, which may be longer by the rest of a 3-unit block.
__host__ __device__ __forceinline__ uint64_t chain_words_of(uint32_t second) { return bound_words((second + 2) / 3 * 3); }

struct BatchParams {
    JobView job;
    uint32_t npairs_rows;       // number of rows pairs, ceil(nclean / 2)
    const uint64_t *row_task;   // first task of each rows pair (npairs_rows + 1)
    uint64_t ntasks;            // tasks of this launch: task_base .. task_base + ntasks - 1
    uint64_t task_base;
    uint32_t gchunk;            // column groups per task of a single-strip rows pair
    uint32_t *bound;
    uint64_t bound_stride;
    unsigned long long *counter;
    // Chained rows pairs (the first ones of the launch): boundary rows of rows
    // pair k, group g, warp w at chain_bound + chain_off[k] + (g W + w) words;
    // progress of task q, warp w at chain_flag[(q - task_base) W + w].
    uint32_t *chain_bound;
    const uint64_t *chain_off;
    uint32_t *chain_flag;
    int *err;                   // set when a wait between strips ran out
    unsigned long long wait_ns; // limit of those waits
    uint32_t step;              // largest s + 2g, for the moving base
};

// Merged launches of the serving loop: explicit (job slot, rows pair, column
// group) tasks over several jobs.
struct ServeParams {
    const JobView *jobs;
    const uint4 *tasks;
    uint64_t ntasks;
    uint32_t *bound;
    uint64_t bound_stride;
    unsigned long long *counter;
};

namespace dev {

// Shared-memory layout of one strip's profile for R rows per lane, per code:
// R16 rows as 32-bit words in planes [lane][4 words] of 4 rows (one 16-byte
// load per lane and plane, bank-conflict free whatever codes the lanes hold),
// then a half plane [lane][2 words] when R16 is 2 mod 4; then, on 16-bit lanes,
// R8 rows as packed bytes, one word holding rows r and r + 1 of both sequences,
// in planes [lane][4 words] of 8 rows and a half plane [lane][2 words] of 4
// rows when R8 is 4 mod 8. A packed row costs one PRMT (ALU pipe) and half the
// shared-memory bytes of a 16-bit row. R8 = 8 floor(R/16) (a third to a half of
// a long strip's rows) balances the shared-memory data pipe, the bound of
// 16-bit rows alone, against the ALU pipe and issue: on c3 it measured 16.07
// TCUPS against 14.81 with no packed rows and 15.96 with R8 = 4 floor(R/8).
template <int R, bool kNarrow, bool kPack = true> struct Layout {
    static constexpr int R8 = kNarrow && kPack ? 8 * (R / 16) : 0;
    static constexpr int R16 = R - R8;
    static constexpr int P16 = R16 / 4;                      // full 16-bit planes
    static constexpr bool kHalf = R16 % 4 != 0;
    static constexpr int HALF = P16 * 128;                   // word offset of the 16-bit half plane
    static constexpr int PACK = HALF + (kHalf ? 64 : 0);     // word offset of the packed planes
    static constexpr int P8 = R8 / 8;                        // full packed planes
    static constexpr int PHALF = PACK + P8 * 128;            // word offset of the packed half plane
    static constexpr int SH = PHALF + (R8 % 8 ? 64 : 0);     // words per code
};

// PRMT of w with a zero second operand.
template <int SEL>
__device__ __forceinline__ uint32_t prmt0(uint32_t w)
{
    uint32_t r;
    asm("prmt.b32 %0, %1, 0, %2;" : "=r"(r) : "r"(w), "n"(SEL));
    return r;
}

// Stages strip rows [i0, i0 + 32R) of the profile in shared memory (Layout).
// Narrow: word = (s(X1_i, b) + 2g, s(X2_i, b) + 2g) as 16x2 (see Narrow), or
// bytes (s1_i, s1_i+1, s2_i, s2_i+1) + 2g in the packed planes; rows of X2 past
// its profile (lp2) score 0, X1's reaches as far as the strips (prof_pitch). Wide: word = s(X1_i, b) as int32.
// The profile is read in 16-byte chunks (16 rows of one code), each thread
// issuing the loads of up to kStageBatch chunks before it converts and stores
// any, so one staging costs about one L2 round trip instead of one per chunk.
// Profile rows are 16-byte aligned: the per-sequence pitch is a multiple of
// 1024 and i0 a multiple of 64; lp2 is a multiple of 1024, so a chunk lies
// wholly inside or wholly past X2's profile. Stacked rows pairs have at most 512 rows.
constexpr int kStageBatch = 4;

// A rows pair's score profiles as staging reads them.
struct RowsProf {
    const int8_t *g1, *g2;
    uint32_t lp1, lp2;
};

// With kPairs > 1 (16-bit lanes only) the strip stacks that many rows pairs,
// each on 32 / kPairs lanes from its row 0: `stack` holds their profiles.
template <int R, bool kNarrow, bool kPack = true, int kPairs = 1>
__device__ __forceinline__ void stage_words(uint32_t *sprof, const int8_t *__restrict__ g1, uint32_t lp1,
                                            const int8_t *__restrict__ g2, uint32_t lp2, int i0, int32_t gap = 0,
                                            const RowsProf *stack = nullptr)
{
    using L = Layout<R, kNarrow, kPack>;
    constexpr int SH = L::SH;
    constexpr int CH = 2 * R;                 // 16-byte chunks per code row (32R rows)
    constexpr int TOTAL = kAlpha * CH;
    const int nt = blockDim.x;
    if constexpr(kNarrow) {
        static_assert(R % 2 == 0, "16-bit lanes take an even number of rows");
        const uint32_t gg = ((uint32_t) (2 * gap) & 0xffffu) * 0x10001u;
        for(int c0 = threadIdx.x; c0 < TOTAL; c0 += kStageBatch * nt) {
            uint4 va[kStageBatch], vb[kStageBatch];
#pragma unroll
            for(int u = 0; u < kStageBatch; ++u) {
                const int c = c0 + u * nt;
                va[u] = vb[u] = make_uint4(0, 0, 0, 0);
                if(c < TOTAL) {
                    const int b = c / CH, m = c - b * CH;
                    if constexpr(kPairs == 1) {
                        va[u] = __ldg(reinterpret_cast<const uint4 *>(g1 + (size_t) b * lp1 + i0) + m);
                        if((uint32_t) (i0 + 16 * m) < lp2)
                            vb[u] = __ldg(reinterpret_cast<const uint4 *>(g2 + (size_t) b * lp2 + i0) + m);
                    } else {
                        constexpr int CPP = CH / kPairs;   // chunks per rows pair
                        const RowsProf &rp = stack[m / CPP];
                        const int mb = m % CPP;
                        va[u] = __ldg(reinterpret_cast<const uint4 *>(rp.g1 + (size_t) b * rp.lp1) + mb);
                        vb[u] = __ldg(reinterpret_cast<const uint4 *>(rp.g2 + (size_t) b * rp.lp2) + mb);
                    }
                }
            }
#pragma unroll
            for(int u = 0; u < kStageBatch; ++u) {
                const int c = c0 + u * nt;
                if(c >= TOTAL) break;
                const int b = c / CH, m = c - b * CH;
                uint32_t *code = sprof + b * SH;
                const uint32_t wa[4] = {va[u].x, va[u].y, va[u].z, va[u].w};
                const uint32_t wb[4] = {vb[u].x, vb[u].y, vb[u].z, vb[u].w};
#pragma unroll
                for(int k = 0; k < 8; ++k) {   // two-row group k: rows 16m + 2k, 16m + 2k + 1
                    uint2 o;
                    if(k & 1) {
                        o.x = __vadd2(sbyte2<2>(wa[k >> 1], wb[k >> 1]), gg);
                        o.y = __vadd2(sbyte2<3>(wa[k >> 1], wb[k >> 1]), gg);
                    } else {
                        o.x = __vadd2(sbyte2<0>(wa[k >> 1], wb[k >> 1]), gg);
                        o.y = __vadd2(sbyte2<1>(wa[k >> 1], wb[k >> 1]), gg);
                    }
                    const int row = 16 * m + 2 * k, ln = row / R, r = row - ln * R;
                    if(r < 4 * L::P16) {
                        *reinterpret_cast<uint2 *>(code + (r >> 2) * 128 + ln * 4 + (r & 3)) = o;
                    } else if(r < L::R16) {
                        *reinterpret_cast<uint2 *>(code + L::HALF + ln * 2) = o;
                    } else {
                        const int wi = (r - L::R16) >> 1;   // packed word of rows r, r + 1
                        uint32_t pk;
                        asm("prmt.b32 %0, %1, %2, 0x6240;" : "=r"(pk) : "r"(o.x), "r"(o.y));
                        if(wi < 4 * L::P8) code[L::PACK + (wi >> 2) * 128 + ln * 4 + (wi & 3)] = pk;
                        else code[L::PHALF + ln * 2 + (wi - 4 * L::P8)] = pk;
                    }
                }
            }
        }
    } else {
        static_assert(R % 4 == 0, "32-bit lanes use full planes");
        constexpr int PL = R / 4;        // planes per lane
        for(int c0 = threadIdx.x; c0 < TOTAL; c0 += kStageBatch * nt) {
            uint4 va[kStageBatch];
#pragma unroll
            for(int u = 0; u < kStageBatch; ++u) {
                const int c = c0 + u * nt;
                va[u] = make_uint4(0, 0, 0, 0);
                if(c < TOTAL) {
                    const int b = c / CH, m = c - b * CH;
                    va[u] = __ldg(reinterpret_cast<const uint4 *>(g1 + (size_t) b * lp1 + i0) + m);
                }
            }
#pragma unroll
            for(int u = 0; u < kStageBatch; ++u) {
                const int c = c0 + u * nt;
                if(c >= TOTAL) break;
                const int b = c / CH, m = c - b * CH;
                const uint32_t wa[4] = {va[u].x, va[u].y, va[u].z, va[u].w};
#pragma unroll
                for(int k = 0; k < 4; ++k) {   // 4-row group 4m + k
                    const int rg = 4 * m + k, ln = rg / PL, pl = rg - ln * PL;
                    uint4 o;
                    o.x = (uint32_t) sbyte<0>(wa[k]);
                    o.y = (uint32_t) sbyte<1>(wa[k]);
                    o.z = (uint32_t) sbyte<2>(wa[k]);
                    o.w = (uint32_t) sbyte<3>(wa[k]);
                    *reinterpret_cast<uint4 *>(sprof + b * SH + pl * 128 + ln * 4) = o;
                }
            }
        }
    }
}

template <bool V> struct Guard { static constexpr bool value = V; };

// Where the row above a strip comes from (sweep_strip's kTop):
//   kTopBound  the boundary row in `bound` (any strip; the last row is stored
//              back when store_bound);
//   kTopZero   row zero of the gap-free state, 0, above lane 0 (a strip that
//              is the first and the last one, 16-bit lanes only);
//   kTopStack  as kTopZero, with a rows pair of its own on every LP lanes, row
//              zero above the first of them (see stack_task).
constexpr int kTopBound = 0, kTopZero = 1, kTopStack = 2;

// Sweeps one strip (rows [i0, i0 + 32R)) of one column sequence on the calling
// warp. `bound` holds the row above the strip on entry (column j at index j)
// and, when store_bound, the strip's last row on exit. After the call, lane k's
// H registers hold the strip's rows at the last column it reached
// (tend - 1 - lane). Steps run in groups of 8 (the loop bookkeeping of a group
// is shared by 8 columns); only the fill and drain groups, where some lanes
// sit outside [0, ncols), test the lane's column. Lane k is one step behind lane
// k - 1 of its rows pair.
template <int R, class K, bool kPack = true, int kTop = kTopBound, int LP = 32>
__device__ __forceinline__ void sweep_strip(const uint32_t *__restrict__ sprof, const uint8_t *__restrict__ cols,
                                            int ncols, uint32_t *__restrict__ bound, int i0, int tend,
                                            bool store_bound, int32_t g, int lane, typename K::W (&H)[R])
{
    using W = typename K::W;
    constexpr bool kB = std::is_same<K, Narrow>::value;
    using L = Layout<R, kB, kPack>;
    constexpr int SH = L::SH;
    const W ng = K::splat(-g);
    W diag;
    if constexpr(kB) {
#pragma unroll
        for(int r = 0; r < R; ++r) H[r] = 0u;   // column 0 of T
        diag = 0u;
    } else {
#pragma unroll
        for(int r = 0; r < R; ++r) H[r] = K::splat(-(i0 + lane * R + r + 1) * g);
        diag = K::splat(-(i0 + lane * R) * g);
    }
    W hlast = H[R - 1];
    static_assert(kTop == kTopBound || kB, "row zero is 0 only in the gap-free 16-bit state");
    uint32_t bq_cur = 0, bq_nxt = 0;
    if constexpr(kTop == kTopBound) {
        bq_cur = bound[lane];
        bq_nxt = bound[32 + lane];
    }
    const uint32_t *prow = sprof + lane * 4;
    const int half_off = L::HALF - lane * 2;      // the 16-bit half plane, from prow
    const int phalf_off = L::PHALF - lane * 2;    // the packed half plane, from prow
    const bool st31 = store_bound && lane == 31;
    int j = -(lane & (LP - 1));
    uint32_t cur = cols[j], nxt = cols[j + 1];   // columns -32..ncols+35 lie in the padded store

    auto group = [&](int t0, auto guard) {
        constexpr bool kG = decltype(guard)::value;
        if(kTop == kTopBound && (t0 & 31) == 0 && t0 > 0) {
            bq_cur = bq_nxt;
            bq_nxt = bound[t0 + 32 + lane];
        }
#pragma unroll
        for(int u = 0; u < 8; ++u) {
            W up = __shfl_up_sync(kFull, hlast, 1);
            if constexpr(kTop == kTopBound) {
                const uint32_t bv = __shfl_sync(kFull, bq_cur, (t0 & 31) + u);
                if(lane == 0) up = (W) bv;
            } else if constexpr(kTop == kTopZero) {
                if(lane == 0) up = 0u;
            } else {
                if((lane & (LP - 1)) == 0) up = 0u;
            }
            if(!kG || (unsigned) j < (unsigned) ncols) {
                const uint32_t *pb = prow + cur * SH;
                W sc[4];
                auto load_plane = [&](int q) {   // 16-bit plane q (q == P16: the half plane)
                    if(q < L::P16) {
                        const uint4 v = *reinterpret_cast<const uint4 *>(pb + q * 128);
                        sc[0] = (W) v.x; sc[1] = (W) v.y; sc[2] = (W) v.z; sc[3] = (W) v.w;
                    } else {
                        const uint2 v = *reinterpret_cast<const uint2 *>(pb + half_off);
                        sc[0] = (W) v.x; sc[1] = (W) v.y;
                    }
                };
                load_plane(0);
                if constexpr(kB) {
                    // T = max(T_left, T_up, T_diag + s + 2g); see Narrow.
                    W above = up, dprev = diag;
                    uint4 pk;
#pragma unroll
                    for(int r = 0; r < R; ++r) {
                        W sr;
                        if(r < L::R16) {
                            if(r > 0 && (r & 3) == 0) load_plane(r >> 2);
                            sr = sc[r & 3];
                        } else {
                            const int rr = r - L::R16;
                            if((rr & 7) == 0) {
                                if((rr >> 3) < L::P8) {
                                    pk = *reinterpret_cast<const uint4 *>(pb + L::PACK + (rr >> 3) * 128);
                                } else {
                                    const uint2 v = *reinterpret_cast<const uint2 *>(pb + phalf_off);
                                    pk.x = v.x;
                                    pk.y = v.y;
                                }
                            }
                            const int wi = (rr >> 1) & 3;
                            const uint32_t w = wi == 0 ? pk.x : wi == 1 ? pk.y : wi == 2 ? pk.z : pk.w;
                            sr = (rr & 1) ? prmt0<0x4341>(w) : prmt0<0x4240>(w);
                        }
                        const W D = __vadd2(dprev, sr);
                        dprev = H[r];
                        H[r] = __vimax3_u16x2(H[r], above, D);
                        above = H[r];
                    }
                } else {
                static_assert(R % 4 == 0, "32-bit lanes use full planes");
                // Row r needs the old H[r-1] (diagonal) and old H[r] (left): the
                // off-chain part for row r+1 is computed before row r is
                // overwritten, so no register copies are needed.
                W pn = K::cell_part(diag, sc[0], H[0], ng);
                W u_ = up;
#pragma unroll
                for(int r = 0; r < R; ++r) {
                    const W pr = pn;
                    if(r + 1 < R) {
                        if(((r + 1) & 3) == 0) load_plane((r + 1) >> 2);
                        pn = K::cell_part(H[r], sc[(r + 1) & 3], H[r + 1], ng);
                    }
                    H[r] = K::cell_chain(u_, ng, pr);
                    u_ = H[r];
                }
                }
                hlast = H[R - 1];
                if constexpr(kTop == kTopBound)
                    if(st31) bound[j] = (uint32_t) hlast;
                diag = up;
            }
            cur = nxt;
            nxt = cols[j + 2];
            ++j;
        }
    };

    const int tend4 = (tend + 7) & ~7;
    int t0 = 0;
#pragma unroll 1
    for(; t0 < tend4 && t0 < LP; t0 += 8) group(t0, Guard<true>{});
#pragma unroll 1
    for(; t0 + 7 < ncols; t0 += 8) group(t0, Guard<false>{});   // every lane inside [0, ncols)
#pragma unroll 1
    for(; t0 < tend4; t0 += 8) group(t0, Guard<true>{});
}

template <int R, class K>
__device__ __forceinline__ typename K::W pick_row(const typename K::W (&H)[R], int r)
{
    typename K::W v = H[0];
#pragma unroll
    for(int q = 1; q < R; ++q) if(q == r) v = H[q];
    return v;
}

__device__ __forceinline__ uint32_t ld_acquire(const uint32_t *p)
{
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release(uint32_t *p, uint32_t v)
{
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// The strip above a chained one: its progress (columns of its last row that
// may be read) and where this strip publishes its own; null where there is none.
struct Chain {
    const uint32_t *above;
    uint32_t *mine;
    int *err;
    unsigned long long wait_ns;
};

// Waits until *flag >= want and returns its value, or gives up: then, and in
// every later wait of the launch, the strip runs on with what is there and the
// call fails.
__device__ __noinline__ uint32_t chain_wait(const uint32_t *flag, uint32_t want, int *err, unsigned long long wait_ns)
{
    unsigned long long t0, t1;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    for(;;) {
        const uint32_t v = ld_acquire(flag);
        if(v >= want) return v;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
        if(*(volatile int *) err != 0) return want;
        if(t1 - t0 > wait_ns) {
            atomicExch(err, 1);
            return want;
        }
        __nanosleep(100);
    }
}

// sweep_strip for strips whose T outgrows 16 bits, and for chained strips: the
// lanes hold T minus a base of the warp (one per 16-bit half), moved up every
// kRebase steps by the smallest first-row value of the 32 lanes less one step.
// T grows along rows and columns by at most `step` = smax + 2g per cell, so the
// cells in flight (32R rows, 32 columns) and all that a lane can still read lie
// within (32R + 33) step above that, and grow by kRebase step until the next
// move: long_ok keeps the sum within 16 bits, whatever the sequences' lengths.
// A boundary word is relative to its writer's base at the step that wrote it
// (column j: step j + 31), which the writer leaves in tab_out and its reader
// finds in tab_in.
// 24 genomes of 30,000 bases: 334 ms in 32-bit lanes with all 30 strips of a
// column in one warp (42 tasks on 296 resident CTAs), 27.9 ms with moving bases
// and a task per strip; 50 genomes of 2,000 to 10,000 bases 15.8 -> 4.7 ms.
template <int R, bool kPack>
__device__ __forceinline__ void sweep_long(const uint32_t *__restrict__ sprof, const uint8_t *__restrict__ cols,
                                           int ncols, uint32_t *bound, const int2 *tab_in, int2 *tab_out,
                                           bool first, int tend,
                                           bool store_bound, const Chain &chain, uint32_t step, int lane,
                                           Narrow::W (&H)[R], int2 &base)
{
    using W = Narrow::W;
    using L = Layout<R, true, kPack>;
    constexpr int SH = L::SH;
#pragma unroll
    for(int r = 0; r < R; ++r) H[r] = 0u;   // column 0 of T
    W diag = 0u, hlast = 0u;
    base = make_int2(0, 0);
    // Columns c0 + lane of the row above, relative to this warp's base. The
    // progress above is read again only when the last value read falls short.
    uint32_t known = 0;
    auto load_above = [&](int c0) -> uint32_t {
        if(first) return 0u;
        if(chain.above) {
            const uint32_t want = (uint32_t) min(c0 + 32, ncols);
            if(known < want) known = chain_wait(chain.above, want, chain.err, chain.wait_ns);
        }
        const int c = c0 + lane;
        if(c >= ncols) return 0u;
        const uint32_t w = __ldcg(bound + c);
        const int2 b = __ldcg(tab_in + (c + 31) / kRebase);
        return __vadd2(w, ((uint32_t) (b.x - base.x) & 0xffffu) | ((uint32_t) (b.y - base.y) << 16));
    };
    uint32_t bq_cur = load_above(0), bq_nxt = load_above(32);
    const uint32_t *prow = sprof + lane * 4;
    const int half_off = L::HALF - lane * 2, phalf_off = L::PHALF - lane * 2;
    const bool st31 = store_bound && lane == 31;
    __syncwarp();
    if(st31) tab_out[0] = base;
    int j = -lane;
    uint32_t cur = cols[j], nxt = cols[j + 1];

    auto group = [&](int t0, auto guard) {
        constexpr bool kG = decltype(guard)::value;
        if((t0 & 31) == 0 && t0 > 0) {
            bq_cur = bq_nxt;
            if(t0 % kRebase == 0) {
                // Unsigned halves: the smallest H[0] of the lanes, less one step.
                const uint32_t lo = __reduce_min_sync(kFull, H[0] & 0xffffu), hi = __reduce_min_sync(kFull, H[0] >> 16);
                const uint32_t dlo = lo > step ? lo - step : 0u, dhi = hi > step ? hi - step : 0u;
                const uint32_t d = dlo | dhi << 16;
#pragma unroll
                for(int r = 0; r < R; ++r) H[r] = __vsub2(H[r], d);
                diag = __vsub2(diag, d);
                hlast = __vsub2(hlast, d);
                bq_cur = __vsub2(bq_cur, d);
                base.x += (int) dlo;
                base.y += (int) dhi;
                if(st31) tab_out[t0 / kRebase] = base;
            }
            bq_nxt = load_above(t0 + 32);
        }
#pragma unroll
        for(int u = 0; u < 8; ++u) {
            W up = __shfl_up_sync(kFull, hlast, 1);
            const uint32_t bv = __shfl_sync(kFull, bq_cur, (t0 & 31) + u);
            if(lane == 0) up = bv;
            if(!kG || (unsigned) j < (unsigned) ncols) {
                const uint32_t *pb = prow + cur * SH;
                W sc[4];
                auto load_plane = [&](int q) {
                    if(q < L::P16) {
                        const uint4 v = *reinterpret_cast<const uint4 *>(pb + q * 128);
                        sc[0] = v.x; sc[1] = v.y; sc[2] = v.z; sc[3] = v.w;
                    } else {
                        const uint2 v = *reinterpret_cast<const uint2 *>(pb + half_off);
                        sc[0] = v.x; sc[1] = v.y;
                    }
                };
                load_plane(0);
                W above = up, dprev = diag;
                uint4 pk;
#pragma unroll
                for(int r = 0; r < R; ++r) {
                    W sr;
                    if(r < L::R16) {
                        if(r > 0 && (r & 3) == 0) load_plane(r >> 2);
                        sr = sc[r & 3];
                    } else {
                        const int rr = r - L::R16;
                        if((rr & 7) == 0) {
                            if((rr >> 3) < L::P8) {
                                pk = *reinterpret_cast<const uint4 *>(pb + L::PACK + (rr >> 3) * 128);
                            } else {
                                const uint2 v = *reinterpret_cast<const uint2 *>(pb + phalf_off);
                                pk.x = v.x;
                                pk.y = v.y;
                            }
                        }
                        const int wi = (rr >> 1) & 3;
                        const uint32_t w = wi == 0 ? pk.x : wi == 1 ? pk.y : wi == 2 ? pk.z : pk.w;
                        sr = (rr & 1) ? prmt0<0x4341>(w) : prmt0<0x4240>(w);
                    }
                    const W Dg = __vadd2(dprev, sr);
                    dprev = H[r];
                    H[r] = __vimax3_u16x2(H[r], above, Dg);
                    above = H[r];
                }
                hlast = H[R - 1];
                if(st31) bound[j] = hlast;
                diag = up;
            }
            cur = nxt;
            nxt = cols[j + 2];
            ++j;
        }
        // Columns 0 .. t0 + 7 - 31 of the last row are stored.
        if(st31 && chain.mine && ((t0 + 8) & (kPublish - 1)) == 0 && t0 + 8 > 31)
            st_release(chain.mine, (uint32_t) min(t0 + 8 - 31, ncols));
    };

    const int tend8 = (tend + 7) & ~7;
    int t0 = 0;
#pragma unroll 1
    for(; t0 < tend8 && t0 < 32; t0 += 8) group(t0, Guard<true>{});
#pragma unroll 1
    for(; t0 + 7 < ncols; t0 += 8) group(t0, Guard<false>{});
#pragma unroll 1
    for(; t0 < tend8; t0 += 8) group(t0, Guard<true>{});
    if(st31 && chain.mine) st_release(chain.mine, (uint32_t) ncols);
}

// The column sequences of one task: sorted b0, b0 + bstep, ... (ngrp of them
// for this warp), each against the rows pair (x1, x2) of a job.
struct TaskCols {
    const JobView *jv;
    uint32_t x1, x2, a2;   // rows sequences (original index) and x2's sorted index
    uint32_t b0, bstep, ngrp;
};

// One task's work for a 16-bit rows pair with strips of 32R rows. With a
// single strip (nst == 1) the strip is staged once and swept against every
// column sequence of the task; otherwise the task has one column sequence per
// warp and every strip is staged in turn. Only the first staging of a
// single-strip task and the stagings of a multi-strip task synchronise the
// CTA, so the loop counts and nst are CTA-uniform.
template <int R, bool kPack>
__device__ __noinline__ void narrow_task(uint32_t *sprof, const int8_t *g1, uint32_t lp1, const int8_t *g2,
                                         uint32_t lp2, int e1, int e2, int nst, const TaskCols &tc, uint32_t *bound,
                                         int32_t g, int lane)
{
    constexpr int SH = 32 * R;
    const JobView &jv = *tc.jv;
    const int em = max(e1, e2), s1 = (e1 - 1) / SH, s2 = (e2 - 1) / SH;
    for(uint32_t t = 0; t < tc.ngrp; ++t) {
        const uint32_t b = tc.b0 + t * tc.bstep;
        const bool has = b < jv.nclean;
        const uint32_t y = has ? jv.sorted[b] : tc.x1;
        const int ncols = has ? (int) jv.eff[y] : 0;
        const uint8_t *cols = jv.units + jv.uoff[y];
        // Row zero of the DP (0 in the T state) as the boundary above the
        // first of several strips (a single strip takes it as a constant).
        if(has && nst > 1) for(int jj = lane; jj < ncols + 96; jj += 32) bound[jj] = 0u;
        int32_t r1 = 0, r2 = 0;
        for(int s = 0; s < nst; ++s) {
            const int i0 = s * SH;
            if(t == 0 || nst > 1) {
                __syncthreads();
                stage_words<R, true, kPack>(sprof, g1, lp1, g2, lp2, i0, g);
                __syncthreads();
            }
            if(has) {
                const bool last = s == nst - 1;
                const int k1 = last ? (em - 1 - i0) / R : 31;
                Narrow::W H[R];
                __syncwarp();
                if(nst == 1)
                    sweep_strip<R, Narrow, kPack, kTopZero>(sprof, cols, ncols, bound, i0, ncols + k1, false, g, lane, H);
                else
                    sweep_strip<R, Narrow, kPack>(sprof, cols, ncols, bound, i0, ncols + k1, !last, g, lane, H);
                __syncwarp();
                if(s == s2) {
                    const int rr = e2 - 1 - i0;
                    r2 = __shfl_sync(kFull, Narrow::hi(pick_row<R, Narrow>(H, rr % R), g, e2, ncols), rr / R);
                }
                if(s == s1) {
                    const int rr = e1 - 1 - i0;
                    r1 = __shfl_sync(kFull, Narrow::lo(pick_row<R, Narrow>(H, rr % R), g, e1, ncols), rr / R);
                }
            }
        }
        if(has && lane == 0) {
            jv.out[tri_index(tc.x1, y)] = r1;
            if(b != tc.a2) jv.out[tri_index(tc.x2, y)] = r2;
        }
    }
}

// Strips [s0, s1) of a 16-bit rows pair with strips of 32R rows on a moving
// base, against one column sequence per warp: all of them, or one chained strip.
template <int R, bool kPack>
__device__ __noinline__ void long_task(uint32_t *sprof, const int8_t *g1, uint32_t lp1, const int8_t *g2, uint32_t lp2,
                                       int e1, int e2, int s0, int s1, const TaskCols &tc, uint32_t *bound,
                                       uint64_t words, const Chain &chain, uint32_t step, int32_t g, int lane)
{
    constexpr int SH = 32 * R;
    const JobView &jv = *tc.jv;
    const int em = max(e1, e2), slast = (em - 1) / SH, sr1 = (e1 - 1) / SH, sr2 = (e2 - 1) / SH;
    const bool has = tc.b0 < jv.nclean;
    const uint32_t y = has ? jv.sorted[tc.b0] : tc.x1;
    const int ncols = has ? (int) jv.eff[y] : 0;
    const uint8_t *cols = jv.units + jv.uoff[y];
    const uint32_t entries = base_entries((uint32_t) ncols);
    int2 *tabs = reinterpret_cast<int2 *>(bound + words) - kBaseTables * entries;
    for(int s = s0; s < s1; ++s) {
        const int i0 = s * SH;
        __syncthreads();
        stage_words<R, true, kPack>(sprof, g1, lp1, g2, lp2, i0, g);
        __syncthreads();
        if(!has) continue;
        const bool last = s == slast;
        const int k1 = last ? (em - 1 - i0) / R : 31;
        Narrow::W H[R];
        int2 base;
        __syncwarp();
        sweep_long<R, kPack>(sprof, cols, ncols, bound, tabs + (uint32_t) (s - 1) % kBaseTables * entries,
                             tabs + (uint32_t) s % kBaseTables * entries, s == 0, ncols + k1, !last, chain, step, lane,
                             H, base);
        __syncwarp();
        if(s == sr2) {
            const int rr = e2 - 1 - i0;
            const int32_t v = __shfl_sync(kFull, base.y + Narrow::hi(pick_row<R, Narrow>(H, rr % R), g, e2, ncols), rr / R);
            if(lane == 0 && tc.b0 != tc.a2) jv.out[tri_index(tc.x2, y)] = v;
        }
        if(s == sr1) {
            const int rr = e1 - 1 - i0;
            const int32_t v = __shfl_sync(kFull, base.x + Narrow::lo(pick_row<R, Narrow>(H, rr % R), g, e1, ncols), rr / R);
            if(lane == 0) jv.out[tri_index(tc.x1, y)] = v;
        }
    }
}

// One rows sequence (x1 when h == 0, x2 when h == 1) in 32-bit lanes with
// strips of 32R rows, against the task's column sequences; staging as in
// narrow_task.
template <int R>
__device__ __noinline__ void wide_task(uint32_t *sprof, const int8_t *g1, uint32_t lp1, int e1, int nst, int h,
                                       const TaskCols &tc, uint32_t *bound, int32_t g, int lane)
{
    constexpr int SH = 32 * R;
    const JobView &jv = *tc.jv;
    const uint32_t xr = h ? tc.x2 : tc.x1;
    for(uint32_t t = 0; t < tc.ngrp; ++t) {
        const uint32_t b = tc.b0 + t * tc.bstep;
        const bool mine = b < jv.nclean && !(h == 1 && b == tc.a2);
        const uint32_t y = mine ? jv.sorted[b] : xr;
        const int ncols = mine ? (int) jv.eff[y] : 0;
        const uint8_t *cols = jv.units + jv.uoff[y];
        if(mine) for(int jj = lane; jj < ncols + 96; jj += 32) bound[jj] = (uint32_t) (-(jj + 1) * g);
        int32_t res = 0;
        for(int s = 0; s < nst; ++s) {
            const int i0 = s * SH;
            if(t == 0 || nst > 1) {
                __syncthreads();
                stage_words<R, false>(sprof, g1, lp1, nullptr, 0, i0);
                __syncthreads();
            }
            if(mine) {
                const bool last = s == nst - 1;
                const int k1 = last ? (e1 - 1 - i0) / R : 31;
                Wide::W H[R];
                __syncwarp();
                sweep_strip<R, Wide>(sprof, cols, ncols, bound, i0, ncols + k1, !last, g, lane, H);
                __syncwarp();
                if(last) {
                    const int rr = e1 - 1 - i0;
                    res = __shfl_sync(kFull, pick_row<R, Wide>(H, rr % R), rr / R);
                }
            }
        }
        if(mine && lane == 0) jv.out[tri_index(xr, y)] = res;
    }
}

// kPairs short rows pairs (2 or 4) in one warp: pair k + p (sorted 2(k + p),
// 2(k + p) + 1) on LP = 32 / kPairs lanes from p LP on, R rows per lane, so each
// pair has LP R >= its rows in one strip; all sweep the same column sequences
// (those of pair k: sorted 2k + 1 + q W + warp). In the gap-free state row zero
// is 0, so the first lane of a pair takes 0 from above instead of the last row
// of the pair before, and they never mix. A column is scored for a rows sequence
// only when it comes after it in the sorted order; the lane that holds a
// sequence's last row writes its score. A step's fixed cost (about 28
// instructions) is shared by kPairs times the cells of a strip on 32 lanes, and
// filling and draining the lanes takes LP - 1 steps per column sequence instead
// of 31: 3,000 reads of 100 to 250 bases 13.9 -> 9.06 ms (two by two before).
template <int R, int kPairs, bool kPack>
__device__ __noinline__ void stack_task(uint32_t *sprof, RowsProf *stack, const JobView &jv, uint32_t k, uint32_t b0,
                                        uint32_t bstep, uint32_t ngrp, int32_t g, int lane)
{
    constexpr int LP = 32 / kPairs;
    if(threadIdx.x < kPairs) {   // read after the barrier below; the last task's stagings are over
        const uint32_t s1 = jv.sorted[2 * (k + threadIdx.x)], s2 = jv.sorted[2 * (k + threadIdx.x) + 1];
        stack[threadIdx.x] = RowsProf{jv.prof + jv.poff[s1], jv.prof + jv.poff[s2], jv.plp[s1], jv.plp[s2]};
    }
    __syncthreads();
    stage_words<R, true, kPack, kPairs>(sprof, nullptr, 0, nullptr, 0, 0, g, stack);
    __syncthreads();
    // The lane's rows pair, and whether it holds the last row of either sequence.
    const uint32_t a1 = 2 * (k + lane / LP), x1 = jv.sorted[a1], x2 = jv.sorted[a1 + 1];
    const int l1 = (int) jv.eff[x1] - 1, l2 = (int) jv.eff[x2] - 1, at = lane % LP;
    for(uint32_t t = 0; t < ngrp; ++t) {
        const uint32_t b = b0 + t * bstep;
        if(b >= jv.nclean) break;
        const uint32_t y = jv.sorted[b];
        const int ncols = (int) jv.eff[y];
        Narrow::W H[R];
        __syncwarp();
        sweep_strip<R, Narrow, kPack, kTopStack, LP>(sprof, jv.units + jv.uoff[y], ncols, nullptr, 0, ncols + LP - 1,
                                                     false, g, lane, H);
        __syncwarp();
        const Narrow::W w1 = pick_row<R, Narrow>(H, l1 % R), w2 = pick_row<R, Narrow>(H, l2 % R);
        if(at == l1 / R && b > a1) jv.out[tri_index(x1, y)] = Narrow::lo(w1, g, l1 + 1, ncols);
        if(at == l2 / R && b > a1 + 1) jv.out[tri_index(x2, y)] = Narrow::hi(w2, g, l2 + 1, ncols);
    }
}

// Strip plan for `rows` rows with at most 32*RMAX rows per strip: the fewest
// strips, each of 32R rows with R the smallest even number that covers them.
template <int RMAX>
__device__ __forceinline__ void strip_plan(int rows, int &nst, int &R)
{
    nst = (rows + 32 * RMAX - 1) / (32 * RMAX);
    R = (rows + 32 * nst - 1) / (32 * nst);
    R = (R + 1) & ~1;
}

}  // namespace dev

// Rows per lane of a rows pair's strips, from its flags: the plan's, or for a
// chained one with lower strips, 16.
template <int RMAX>
__host__ __device__ __forceinline__ int strip_rows(int rows, uint8_t flags)
{
    if(flags & kRowR16) return 16;
    const int nst = (rows + 32 * RMAX - 1) / (32 * RMAX);
    const int R = (rows + 32 * nst - 1) / (32 * nst);
    return (R + 1) & ~1;
}

// Resident CTAs per SM the batched kernel is compiled for (register budget).
template <int RMAX, int W> struct BatchOcc { static constexpr int value = (RMAX == 32 ? 16 : 24) / W; };

// Column groups of W per task for rows pair k of a job with nclean clean
// sequences: `chunk` groups when its rows fit one strip of 32 RMAX rows (the
// strip is then staged once for all of them), else one. The host's task
// tables use the same rule.
__host__ __device__ __forceinline__ uint32_t groups_per_task(uint32_t e1, int rmax, uint32_t chunk)
{
    return e1 <= (uint32_t) (32 * rmax) ? chunk : 1u;
}

// One task: rows pair k (sorted 2k, 2k+1) of job `jv` against `ngrp` column
// groups starting at `grp` (group q: sorted 2k+1 + q*W + warp for each warp).
// All threads of the CTA call it.
template <int RMAX, int W, bool kPack>
__device__ __forceinline__ void rows_pair_task(const JobView &jv, uint32_t k, uint32_t grp, uint32_t ngrp,
                                               uint32_t *sprof_b, uint32_t *bound, int warp, int lane,
                                               uint64_t words = 0, uint32_t step = 0, int strip = -1,
                                               const dev::Chain &chain = dev::Chain{nullptr, nullptr, nullptr, 0})
{
    const uint32_t a1 = 2 * k, a2 = min(2 * k + 1, jv.nclean - 1);
    const uint32_t x1 = jv.sorted[a1], x2 = jv.sorted[a2];
    // In the reference's orientation the second may be up to two rows longer.
    const int e1 = (int) jv.eff[x1], e2 = (int) jv.eff[x2], em = max(e1, e2);
    dev::TaskCols tc{&jv, x1, x2, a2, 2 * k + 1 + grp * W + warp, (uint32_t) W, ngrp};

    if constexpr(RMAX == 32) {
        __shared__ dev::RowsProf stack[4];
        // Stacked rows pairs: R rows per lane, enough for the longest sequence.
        auto longest = [&](uint32_t pairs) {
            int e = em;
            for(uint32_t a = 2 * k + 2; a < 2 * (k + pairs); ++a) e = max(e, (int) jv.eff[jv.sorted[a]]);
            return e;
        };
#define MSA_STACK(RR, NP) case RR: dev::stack_task<RR, NP, kPack>(sprof_b, stack, jv, k, tc.b0, tc.bstep, ngrp, jv.g, lane); break;
#define MSA_STACKS(NP)                                                                                              \
    switch(R) {                                                                                                     \
        MSA_STACK(2, NP) MSA_STACK(4, NP) MSA_STACK(6, NP) MSA_STACK(8, NP) MSA_STACK(10, NP) MSA_STACK(12, NP)     \
        MSA_STACK(14, NP) MSA_STACK(16, NP) MSA_STACK(18, NP) MSA_STACK(20, NP) MSA_STACK(22, NP) MSA_STACK(24, NP) \
        MSA_STACK(26, NP) MSA_STACK(28, NP) MSA_STACK(30, NP) MSA_STACK(32, NP) default: break;                     \
    }
        if(jv.row_narrow[k] & kRowQuad) {
            const int R = ((longest(2) + 15) / 16 + 1) & ~1;
            MSA_STACKS(2)
            return;
        }
        if constexpr(kPack) {
            if(jv.row_narrow[k] & kRowOct) {
                const int R = ((longest(4) + 7) / 8 + 1) & ~1;
                MSA_STACKS(4)
                return;
            }
        }
#undef MSA_STACKS
#undef MSA_STACK
        if(jv.row_narrow[k] & kRowLong) {
            const int R = strip_rows<RMAX>(em, jv.row_narrow[k]), nst = (em + 32 * R - 1) / (32 * R);
            const int s0 = strip < 0 ? 0 : strip, s1 = strip < 0 ? nst : strip + 1;
            const int8_t *g1 = jv.prof + jv.poff[x1], *g2 = jv.prof + jv.poff[x2];
            const uint32_t lp1 = jv.plp[x1], lp2 = jv.plp[x2];
#define MSA_LONG(RR) case RR: dev::long_task<RR, kPack>(sprof_b, g1, lp1, g2, lp2, e1, e2, s0, s1, tc, bound, words, chain, step, jv.g, lane); break;
            switch(R) {   // strips of several per rows pair: 18 rows per lane and more, or 16
                MSA_LONG(16) MSA_LONG(18) MSA_LONG(20) MSA_LONG(22) MSA_LONG(24) MSA_LONG(26) MSA_LONG(28)
                MSA_LONG(30) MSA_LONG(32) default: break;
            }
#undef MSA_LONG
            return;
        }
    }
    if(jv.row_narrow[k]) {
        int nst, R;
        dev::strip_plan<RMAX>(em, nst, R);
        const int8_t *g1 = jv.prof + jv.poff[x1], *g2 = jv.prof + jv.poff[x2];
        const uint32_t lp1 = jv.plp[x1], lp2 = jv.plp[x2];
#define MSA_NARROW(RR) case RR: dev::narrow_task<RR, kPack>(sprof_b, g1, lp1, g2, lp2, e1, e2, nst, tc, bound, jv.g, lane); break;
        switch(R) {
            MSA_NARROW(2) MSA_NARROW(4) MSA_NARROW(6) MSA_NARROW(8) MSA_NARROW(10) MSA_NARROW(12) MSA_NARROW(14)
            MSA_NARROW(16)
            default:
                if constexpr(RMAX > 16) {
                    switch(R) {
                        MSA_NARROW(18) MSA_NARROW(20) MSA_NARROW(22) MSA_NARROW(24) MSA_NARROW(26) MSA_NARROW(28)
                        MSA_NARROW(30) MSA_NARROW(32) default: break;
                    }
                }
                break;
        }
#undef MSA_NARROW
    } else {
        for(int h = 0; h < 2; ++h) {
            if(h == 1 && a2 == a1) break;   // CTA-uniform
            const uint32_t xr = h ? x2 : x1;
            const int er = h ? e2 : e1;
            const int nst = (er + 32 * RMAX - 1) / (32 * RMAX);
            dev::wide_task<RMAX>(sprof_b, jv.prof + jv.poff[xr], jv.plp[xr], er, nst, h, tc, bound, jv.g, lane);
        }
    }
}

// kPack = false stages every profile row as 16-bit words (no packed-byte
// rows); it exists to measure what the packed rows contribute.
template <int RMAX, int W, bool kPack = true>
__global__ void __launch_bounds__(W * 32, BatchOcc<RMAX, W>::value) nw_batched_kernel(BatchParams p)
{
    extern __shared__ __align__(16) uint32_t sprof_b[];
    __shared__ unsigned long long task_q;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t *bound = p.bound + ((uint64_t) blockIdx.x * W + warp) * p.bound_stride;

    for(;;) {
        __syncthreads();
        if(threadIdx.x == 0) task_q = atomicAdd(p.counter, 1ull);
        __syncthreads();
        if(task_q >= p.ntasks) break;
        const unsigned long long q = task_q + p.task_base;
        uint32_t lo = 0, hi = p.npairs_rows - 1;
        while(lo < hi) {
            const uint32_t mid = (lo + hi + 1) >> 1;
            if(p.row_task[mid] <= q) lo = mid; else hi = mid - 1;
        }
        if constexpr(RMAX == 32) {
            const uint8_t fl = p.job.row_narrow[lo];
            if(fl & kRowChain) {
                // Task (group, strip); the strip above is the task before it.
                const uint32_t second = p.job.eff[p.job.sorted[min(2 * lo + 1, p.job.nclean - 1)]];
                const int em = (int) max(p.job.eff[p.job.sorted[2 * lo]], second), SH = 32 * strip_rows<RMAX>(em, fl);
                const uint32_t nst = (uint32_t) ((em + SH - 1) / SH), qq = (uint32_t) (q - p.row_task[lo]);
                const uint32_t grp = qq / nst, strip = qq - grp * nst;
                const uint64_t words = chain_words_of(second);
                uint32_t *flag = p.chain_flag + task_q * W + warp;
                const dev::Chain chain{strip ? flag - W : nullptr, flag, p.err, p.wait_ns};
                rows_pair_task<RMAX, W, kPack>(p.job, lo, grp, 1, sprof_b,
                                               p.chain_bound + p.chain_off[lo] + (grp * W + warp) * words, warp, lane,
                                               words, p.step, (int) strip, chain);
                continue;
            }
        }
        const uint32_t groups = (p.job.nclean - 2 * lo - 1 + W - 1) / W;
        const uint32_t chunk = groups_per_task(max(p.job.eff[p.job.sorted[2 * lo]],
                                                   p.job.eff[p.job.sorted[min(2 * lo + 1, p.job.nclean - 1)]]),
                                               RMAX, p.gchunk);
        const uint32_t grp = (uint32_t) (q - p.row_task[lo]) * chunk;
        rows_pair_task<RMAX, W, kPack>(p.job, lo, grp, min(chunk, groups - grp), sprof_b, bound, warp, lane,
                                       p.bound_stride, p.step);
    }
}

template <int RMAX, int W>
__global__ void __launch_bounds__(W * 32, BatchOcc<RMAX, W>::value) nw_serve_kernel(ServeParams p)
{
    extern __shared__ __align__(16) uint32_t sprof_b[];
    __shared__ unsigned long long task_q;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t *bound = p.bound + ((uint64_t) blockIdx.x * W + warp) * p.bound_stride;

    for(;;) {
        __syncthreads();
        if(threadIdx.x == 0) task_q = atomicAdd(p.counter, 1ull);
        __syncthreads();
        const unsigned long long q = task_q;
        if(q >= p.ntasks) break;
        const uint4 t = p.tasks[q];
        const JobView jv = p.jobs[t.x];
        rows_pair_task<RMAX, W, true>(jv, t.y, t.z, 1, sprof_b, bound, warp, lane);
    }
}

// Pairs that involve a sequence with END units before its last letter, or an
// empty one: the reference's orientation (rows = more 3-unit blocks, ties to
// the pair's second element) and its END handling (rows stop at the first END,
// END columns copy the left neighbour over the full padded width).
template <int R, int WPB>
__global__ void __launch_bounds__(WPB * 32) nw_generic_kernel(NwParams p)
{
    extern __shared__ __align__(16) int8_t smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int8_t *sprof = smem + warp * (kAlpha * 32 * R);
    const uint64_t gw = (uint64_t) blockIdx.x * WPB + warp;
    const uint64_t nw = (uint64_t) gridDim.x * WPB;
    uint32_t *bound = p.bound + gw * p.bound_stride;
    for(uint64_t k = gw; k < p.ngeneric; k += nw) {
        const uint32_t ri = p.gpairs[2 * k], ci = p.gpairs[2 * k + 1];
        const int nrows = (int) p.eff[ri], ncols = (int) p.plen[ci];
        int32_t ra = -ncols * p.g, rb = 0;
        if(nrows > 0 && ncols > 0) {
            dev::run_task<R, dev::Wide, true>(p.prof + p.poff[ri], p.plp[ri], nrows,
                                              p.units + p.uoff[ci], ncols, nullptr, 0,
                                              sprof, bound, p.g, lane, ra, rb);
        } else if(nrows > 0) {
            ra = -nrows * p.g;   // no columns: every row copies column 0
        }
        if(lane == 0) p.out[dev::tri_index(ri, ci)] = ra;
    }
}

// Score profile of every sequence: prof[off + b*Lp + i] = T[unit_i][b] for
// i < eff, 0 beyond. One block per sequence, 16 bytes per thread step.
__global__ void build_profiles_kernel(const uint8_t *__restrict__ units, const uint64_t *__restrict__ uoff,
                                      const uint32_t *__restrict__ eff, const uint64_t *__restrict__ poff,
                                      const uint32_t *__restrict__ plp, const int8_t *__restrict__ ext,
                                      int8_t *__restrict__ prof)
{
    __shared__ int8_t tbl[kAlpha * kAlpha];
    for(int i = threadIdx.x; i < kAlpha * kAlpha; i += blockDim.x) tbl[i] = ext[i];
    __syncthreads();
    const uint32_t s = blockIdx.x;
    const uint8_t *u = units + uoff[s];
    const uint32_t e = eff[s], lp = plp[s];
    int8_t *dst = prof + poff[s];
    const uint32_t chunks = lp / 16;
    for(uint32_t c = threadIdx.x; c < chunks * kAlpha; c += blockDim.x) {
        const uint32_t b = c / chunks, w = c - b * chunks;
        const uint32_t i = w * 16;
        uint32_t out[4] = {0, 0, 0, 0};
        if(i < e) {
            const uint4 v = *reinterpret_cast<const uint4 *>(u + i);
            const uint32_t in[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for(int q = 0; q < 4; ++q) {
#pragma unroll
                for(int k = 0; k < 4; ++k) {
                    const uint32_t x = (in[q] >> (8 * k)) & 0xffu;
                    const int8_t sc = (i + 4 * q + k < e && x < (uint32_t) kAlpha) ? tbl[x * kAlpha + b] : 0;
                    out[q] |= ((uint32_t) (uint8_t) sc) << (8 * k);
                }
            }
        }
        *reinterpret_cast<uint4 *>(dst + (size_t) b * lp + i) = make_uint4(out[0], out[1], out[2], out[3]);
    }
}

// ---------------------------------------------------------------- host side

static constexpr int kPlainR = 16;
static constexpr int kWPB = 4;

template <int R>
static size_t smem_bytes() { return (size_t) kWPB * kAlpha * 32 * R; }

struct Launch {
    int blocks_per_sm = 0;
};

template <class KernelT>
static int occupancy(KernelT kernel, size_t smem, int *blocks)
{
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem);
    if(e != cudaSuccess) return -1;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, kernel, kWPB * 32, smem);
    if(e != cudaSuccess || *blocks < 1) return -1;
    return 0;
}

// 16-bit lanes are exact when every scored cell of a task fits them. In the
// lane state T(i,j) = H(i,j) + g(i+j) every path scores the sum of s + 2g over
// its matched cells, so with smin + 2g >= 0 the state and its diagonal
// candidate lie in [0, min(i,j)*(smax + 2g)], with min(i,j) <= min(rows, cols).
// Cells outside the sequences (padding rows, the shorter sequence's tail) may
// wrap within their half but never feed a scored cell. smin and smax are taken
// over the letter block, or, where sequences hold GAP units, over every entry
// but END's.
struct ScoreRange { int64_t pos, neg; };   // largest score, largest magnitude of a negative one
static inline ScoreRange range_of(const ExtTable &t, bool gap)
{
    return gap ? ScoreRange{t.max_pos, t.max_neg} : ScoreRange{t.letter_pos, t.letter_neg};
}
static inline bool narrow_ok(int64_t rows_p, int64_t cols, const ExtTable &t, bool gap = false)
{
    const ScoreRange sr = range_of(t, gap);
    const int64_t g2 = 2 * (int64_t) t.penalty;
    if(sr.neg > g2) return false;
    const int64_t step = std::max<int64_t>(sr.pos + g2, 0);
    if(step > 0xff) return false;   // s + 2g is staged as a byte in packed rows
    return step * std::min(rows_p, cols) <= 0xffff;
}

// The largest s + 2g of the letters (and of padding rows, which score 0).
static inline int64_t largest_step(const ExtTable &t, bool gap)
{
    return std::max<int64_t>(range_of(t, gap).pos, 0) + 2 * (int64_t) t.penalty;
}

// 16-bit lanes on a moving base are exact for any lengths when what lies
// between the base and the largest cell in flight fits (sweep_long).
static inline bool long_ok(const ExtTable &t, bool gap)
{
    return range_of(t, gap).neg <= 2 * (int64_t) t.penalty && largest_step(t, gap) <= 0xff &&
           largest_step(t, gap) * (32 * 32 + 34 + kRebase) <= 0xffff;
}

// Batched-kernel tile shapes (pick_tiles: rows per lane R and warps per CTA
// W) and column groups per single-strip task (pick_chunk), autotuned; the
// context may override either (msa_nw_set_tiles, msa_nw_set_variant).
#include "autotune.inc"

Tiles pick_tiles_for(const SeqStore *st) { return pick_tiles(st, (uint32_t) st->clean_sorted.size()); }

cudaError_t launch_profiles(const SeqStore *st, const int8_t *d_ext, int8_t *d_prof, cudaStream_t s)
{
    if(st->n == 0) return cudaSuccess;
    build_profiles_kernel<<<st->n, 256, 0, s>>>(st->d_units, st->d_off, st->d_eff, st->d_prof_off, st->d_prof_lp,
                                                d_ext, d_prof);
    return cudaGetLastError();
}

void plan_rows_pairs(const SeqStore *st, const ExtTable &tbl, Tiles tiles, std::vector<uint8_t> &narrow,
                     std::vector<uint32_t> &groups)
{
    const uint32_t nclean = (uint32_t) st->clean_sorted.size();
    const uint32_t K = (nclean + 1) / 2;
    const int SH = 32 * tiles.R;
    narrow.assign(K, 0);
    groups.assign(K, 0);
    for(uint32_t k = 0; k < K; ++k) {
        const int64_t ncol = (int64_t) nclean - (2 * (int64_t) k + 1);
        if(ncol <= 0) continue;
        const int64_t rows_p = (int64_t) round_up(st->eff[st->clean_sorted[2 * k]], SH);
        const int64_t cols = st->eff[st->clean_sorted[2 * k + 1]];
        narrow[k] = narrow_ok(rows_p, cols, tbl) ? 1 : 0;
        groups[k] = (uint32_t) ((ncol + tiles.W - 1) / tiles.W);
    }
}

size_t job_view_bytes() { return sizeof(JobView); }

void fill_job_view(void *dst, const SeqStore *st, const int8_t *d_prof, const uint8_t *d_narrow, int32_t *d_out,
                   int32_t g)
{
    JobView v{};
    v.units = st->d_units;
    v.uoff = st->d_off;
    v.eff = st->d_eff;
    v.prof = d_prof;
    v.poff = st->d_prof_off;
    v.plp = st->d_prof_lp;
    v.sorted = st->d_clean_sorted;
    v.row_narrow = d_narrow;
    v.out = d_out;
    v.nclean = (uint32_t) st->clean_sorted.size();
    v.g = g;
    std::memcpy(dst, &v, sizeof(v));
}

cudaError_t load_profiles_kernel()
{
    cudaFuncAttributes a{};
    return cudaFuncGetAttributes(&a, build_profiles_kernel);
}

int serve_grid(msa_ctx *ctx, uint64_t *grid)
{
    auto kern = nw_serve_kernel<32, 8>;
    const size_t smem = (size_t) kAlpha * 32 * 32 * 4;
    MSA_CUDA_TRY(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem));
    int bps = 0;
    MSA_CUDA_TRY(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, kern, 8 * 32, smem));
    if(bps < 1) return set_error(ctx, MSA_ERR_CUDA, "serving kernel cannot be resident");
    *grid = (uint64_t) ctx->num_sms * bps;
    return MSA_OK;
}

cudaError_t launch_serve(const ServeLaunch &l, uint64_t grid, cudaStream_t s)
{
    ServeParams p{};
    p.jobs = (const JobView *) l.jobs;
    p.tasks = (const uint4 *) l.tasks;
    p.ntasks = l.ntasks;
    p.bound = l.bound;
    p.bound_stride = l.bound_stride;
    p.counter = l.counter;
    const size_t smem = (size_t) kAlpha * 32 * 32 * 4;
    nw_serve_kernel<32, 8><<<(unsigned) std::min<uint64_t>(grid, std::max<uint64_t>(l.ntasks, 1)), 8 * 32, smem, s>>>(p);
    return cudaGetLastError();
}


// ---------------------------------------------------------------- plans and graphs
//
// A plan is everything a call needs besides the store: the host-side task
// tables, and device buffers it owns (score profiles, the table, boundary
// rows, task tables, the work counter). Plans are cached per context, keyed by
// store, table, mode, tile shape and output pointer; for the persistent mode
// the launch sequence is captured once into a CUDA graph and replayed.

struct PlainLaunch { uint64_t k_lo, k_hi, blocks; };

struct NwPlan {
    uint64_t store_serial = 0;
    int mode = 0;
    int32_t *d_out = nullptr;
    Tiles tiles{0, 0};
    ExtTable tbl{};
    msa_ctx *home = nullptr;    // whose block cache `mem` goes back to
    void *mem = nullptr;
    size_t mem_bytes = 0;
    std::vector<uint8_t> staged;   // host copy of the tables at the start of `mem`
    const int8_t *d_ext = nullptr;
    NwParams p{};
    BatchParams bp{};
    BitParams bits{};           // of the pairs on bit planes, if any (ntasks > 0)
    uint64_t bits_grid = 0;
    uint32_t n = 0;
    uint64_t ngeneric = 0, gen_blocks = 0;
    std::vector<PlainLaunch> plain;
    uint64_t batch_grid = 0;
    uint32_t launches = 0, narrow_tasks = 0;
    uint64_t cells = 0, pairs = 0;
    uint32_t part = 0, nparts = 1;
    int variant = 0;            // msa_nw_set_variant flags the plan was built with
    uint32_t chunk = 0;         // and its groups-per-task override
    uint32_t wait_us = 0;       // and its waits (msa_nw_set_wait)
    bool fixed_tiles = false;   // and whether it says the tiles (msa_nw_set_tiles)
    size_t clear_bytes = 64;    // of the work counter and what follows it
    bool chained = false;
    bool profiles = true;       // whether any kernel of the plan reads score profiles
    cudaGraphExec_t exec = nullptr;
    cudaStream_t captured_on = nullptr;
    ~NwPlan()
    {
        if(exec) cudaGraphExecDestroy(exec);
        if(mem) home->blocks.give(mem, mem_bytes);
    }
};

struct GraphCache {
    std::vector<NwPlan *> plans;   // most recent last
    // Executable graphs of dropped plans: a new plan's sequence mostly has the
    // same nodes, and updating one costs a fraction of instantiating it.
    std::vector<cudaGraphExec_t> spare;
    void drop(NwPlan *pl)
    {
        if(pl->exec && spare.size() < 4) {
            spare.push_back(pl->exec);
            pl->exec = nullptr;
        }
        delete pl;
    }
    // `g` as an executable graph.
    cudaError_t instantiate(cudaGraph_t g, cudaGraphExec_t *exec)
    {
        while(!spare.empty()) {
            cudaGraphExec_t x = spare.back();
            spare.pop_back();
            cudaGraphExecUpdateResultInfo info{};
            if(cudaGraphExecUpdate(x, g, &info) == cudaSuccess) {
                *exec = x;
                return cudaSuccess;
            }
            cudaGetLastError();
            cudaGraphExecDestroy(x);
        }
        return cudaGraphInstantiate(exec, g, 0);
    }
};

// Plans kept per context: as many as a program rotates its stores through, and
// at most kMaxPlanBytes beyond the newest.
static constexpr size_t kMaxPlans = 8;
static constexpr size_t kMaxPlanBytes = size_t(2) << 30;
// Device memory that the boundary rows of chained rows pairs may take.
static constexpr uint64_t kChainBytes = 2ull << 30;

void release_graphs(msa_ctx *ctx)
{
    if(!ctx->graphs) return;
    for(NwPlan *pl : ctx->graphs->plans) delete pl;
    for(cudaGraphExec_t x : ctx->graphs->spare) cudaGraphExecDestroy(x);
    delete ctx->graphs;
    ctx->graphs = nullptr;
}

void drop_plans(msa_ctx *ctx)
{
    if(!ctx->graphs) return;
    for(NwPlan *pl : ctx->graphs->plans) ctx->graphs->drop(pl);
    ctx->graphs->plans.clear();
}

void drop_plans_for_store(msa_ctx *ctx, uint64_t serial)
{
    if(!ctx->graphs) return;
    auto &v = ctx->graphs->plans;
    for(size_t i = 0; i < v.size();) {
        if(v[i]->store_serial == serial) { ctx->graphs->drop(v[i]); v.erase(v.begin() + i); }
        else ++i;
    }
}

// Grid of an instance of the batched kernel (`slot`: its place in the context's
// occupancy cache).
template <int R, int W, bool kPack = true>
static int batched_grid(msa_ctx *ctx, int slot, uint64_t ntasks, uint64_t *grid)
{
    int &bps = ctx->batch_blocks_per_sm[slot];
    if(bps == 0) {
        auto kern = nw_batched_kernel<R, W, kPack>;
        const size_t smem = (size_t) kAlpha * 32 * R * 4;
        MSA_CUDA_TRY(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem));
        int k = 0;
        MSA_CUDA_TRY(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&k, kern, W * 32, smem));
        if(k < 1) return set_error(ctx, MSA_ERR_CUDA, "batched NW kernel cannot be resident");
        bps = k;
    }
    *grid = std::min<uint64_t>((uint64_t) ctx->num_sms * bps, std::max<uint64_t>(ntasks, 1));
    return MSA_OK;
}

template <int R, int W, bool kPack = true>
static void launch_batched(const NwPlan &pl, cudaStream_t s)
{
    const size_t smem = (size_t) kAlpha * 32 * R * 4;
    nw_batched_kernel<R, W, kPack><<<(unsigned) pl.batch_grid, W * 32, smem, s>>>(pl.bp);
}

// Instructions of a warp's step besides its cells, and what a moving base adds.
constexpr uint64_t kStepCost = 28, kMovingCost = 22;

// Whether the longest rows pairs are chained, and with strips of how many rows: the
// form with the least estimated time, from the longest of them (`rows`, `columns`;
// `moving`: on a moving base also when not chained) and the work of all rows pairs as
// one task each (`tasks`), of the chained ones' strips of up to 1,024 rows (`high`) and
// of 512 (`low`), counted in the longest's own tasks or strips. A strip is columns + 31
// steps; it follows the one above by about 100 steps more than its own lanes need. Up to
// one CTA per SM runs undisturbed, two share the SM's shared-memory pipe, and beyond
// that tasks wait for a CTA; strips that wait for each other hold theirs. The factors
// are fitted to 178 jobs of 2 to 700 sequences of up to 60,000 residues, alike, log-normal
// and one long among short ones, each measured unchained, with strips of 1,024 and of
// 512 rows: the form taken is within 2.1% of the best in the mean and 24% at worst, and
// nowhere more than 9% slower than unchained. Chaining wherever the launch's share
// allows, with strips as low as 256 rows where they do not fill the CTAs, was 12% slower
// in the mean: 64 sequences of 1,030 residues 528 us (299 not chained), one of 20,000
// among 49 of 200 2.37 ms (0.94 not chained, 0.71 with strips of 1,024 rows), 24 of 6,000
// 2.57 ms (6.95, 1.46).
static uint8_t chain_form(uint64_t rows, uint64_t columns, bool moving, double tasks, double high, double low,
                          double resident)
{
    const double steps = (double) columns + 31;
    auto share = [&](double n, double two, double base, double slope) {
        return 2 * n <= resident ? 1.0 : n <= resident ? two : std::max(two, base + slope * n / resident);
    };
    auto chained = [&](uint64_t nst, int R, double n) {
        const double line = std::max(1.0, n / resident) * (1.0 + (double) (nst - 1) * 100.0 / steps);
        return std::max(share(n, 1.25, 0.3, 1.5), line) * steps * (double) (R + kStepCost + kMovingCost);
    };
    const int R = strip_rows<32>((int) rows, 0);
    const uint64_t nst = (rows + 32 * R - 1) / (32 * (uint64_t) R);
    const double apart = (double) nst * steps * (double) (R + kStepCost + (moving ? kMovingCost : 0)) *
                         share(tasks, 1.65, 0.5, 1.8);
    const double tall = chained(nst, R, high), halved = chained((rows + 511) / 512, 16, low);
    if(apart <= std::min(tall, halved)) return 0;
    return tall <= halved ? kRowLong | kRowChain : kRowLong | kRowChain | kRowR16;
}

static int build_plan(msa_ctx *ctx, SeqStore *st, const ExtTable &tbl, int mode, int32_t *d_out, Tiles tiles,
                      uint32_t part, uint32_t nparts, NwPlan *pl)
{
    const uint32_t n = st->n;
    pl->store_serial = st->serial;
    pl->mode = mode;
    pl->d_out = d_out;
    pl->tiles = tiles;
    pl->tbl = tbl;
    pl->n = n;
    pl->part = part;
    pl->nparts = nparts;
    pl->variant = ctx->nw_variant;
    pl->chunk = ctx->nw_chunk;
    pl->wait_us = ctx->nw_wait_us;
    pl->fixed_tiles = ctx->tile_r != 0;

    const uint32_t nclean = (uint32_t) st->clean_sorted.size();
    const uint64_t nclean_pairs = (uint64_t) nclean * (nclean > 0 ? nclean - 1 : 0) / 2;

    // What runs on bit planes (nw_bits.cu): where the table allows it, pairs
    // beyond the first 32 g0 sequences; `nrows` sequences are left to the
    // batched kernel. Parts of a job and overridden tiles stay on that kernel.
    BitPlan bits;
    const BitTable planes = bit_table(tbl);
    uint32_t nrows = nclean;
    if(mode == MSA_NW_PERSISTENT && planes.u && nparts == 1 && nclean > 32 && !st->any_gap && !ctx->nw_variant &&
       !ctx->tile_r && !ctx->nw_chunk) {
        std::vector<uint32_t> eff(nclean);
        for(uint32_t a = 0; a < nclean; ++a) eff[a] = st->eff[st->clean_sorted[a]];
        bits = plan_bits(eff, (uint32_t) ctx->num_sms);
        if(bits.ntasks) nrows = 32 * bits.g0;
    }

    // Pairs with at least one dirty sequence, in the reference's orientation,
    // and this part's runs of rows pairs and generic pairs.
    std::vector<uint32_t> gpairs_all;
    list_generic_pairs(st->dirty, st->len, gpairs_all);
    const JobSplit split = split_job(st->eff, st->plen, st->clean_sorted, gpairs_all, nparts);
    const uint32_t k_lo = split.k[part], k_hi = split.k[part + 1];
    const uint64_t g_lo = split.g[part], g_hi = split.g[part + 1];
    const std::vector<uint32_t> gpairs(gpairs_all.begin() + 2 * g_lo, gpairs_all.begin() + 2 * g_hi);
    pl->ngeneric = gpairs.size() / 2;

    // Pairs and cells (given lengths) of this part.
    {
        using u128 = unsigned __int128;
        const auto &cs = st->clean_sorted;
        std::vector<u128> suffix(nclean + 1, 0);
        for(uint32_t b = nclean; b-- > 0;) suffix[b] = suffix[b + 1] + st->len[cs[b]];
        u128 cells = 0;
        uint64_t pairs = 0;
        for(uint32_t a = 2 * k_lo; a < std::min<uint32_t>(2 * k_hi, nclean); ++a) {
            cells += (u128) st->len[cs[a]] * suffix[a + 1];
            pairs += nclean - 1 - a;
        }
        for(uint64_t q = 0; q < pl->ngeneric; ++q) cells += (u128) st->len[gpairs[2 * q]] * st->len[gpairs[2 * q + 1]];
        pl->cells = (uint64_t) cells;
        pl->pairs = pairs + pl->ngeneric;
    }

    uint32_t max_cols = 1;
    for(uint32_t i = 0; i < n; ++i) max_cols = std::max(max_cols, st->plen[i]);
    const uint64_t stride = bound_words(max_cols);

    // Occupancy of the per-warp kernels, where they run.
    uint64_t resident_blocks = 0;
    if(mode == MSA_NW_PLAIN || pl->ngeneric) {
        if(ctx->plain_blocks_per_sm == 0) {
            const size_t smem = smem_bytes<kPlainR>();
            int bps = 0, bps3 = 0;
            if(occupancy(nw_plain_kernel<kPlainR, kWPB>, smem, &bps) || occupancy(nw_generic_kernel<kPlainR, kWPB>, smem, &bps3))
                return set_error(ctx, MSA_ERR_CUDA, "occupancy query failed (no sm_100a image?)");
            ctx->plain_blocks_per_sm = std::min(bps, bps3);
        }
        resident_blocks = (uint64_t) ctx->num_sms * (uint64_t) ctx->plain_blocks_per_sm;
    }
    uint64_t warps_needed = resident_blocks * kWPB;

    // Persistent task tables: rows pairs (sorted 2k, 2k+1) x column groups of W.
    std::vector<uint64_t> row_task;
    std::vector<uint8_t> row_narrow;
    std::vector<uint64_t> chain_off;
    uint64_t chain_words = 0, chain_tasks = 0;
    uint64_t ntasks = 0;
    uint32_t K = 0;
    uint64_t task_base = 0;
    uint32_t gchunk = 1;
    if(mode == MSA_NW_PERSISTENT && nclean_pairs > 0 && nrows > 1) {
        K = (nrows + 1) / 2;
        const uint32_t k_hi = std::min(split.k[part + 1], K);
        const int SH = 32 * tiles.R;
        const bool gap = st->any_gap;
        auto eff_at = [&](uint32_t a) { return (uint64_t) st->eff[st->clean_sorted[std::min(a, nrows - 1)]]; };
        // Rows of rows pair k, and its longest column sequence.
        auto rows_at = [&](uint32_t k) { return std::max(eff_at(2 * k), eff_at(2 * k + 1)); };
        const bool oriented = gap || !table_is_symmetric(tbl);
        auto cols_at = [&](uint32_t k) { return oriented ? (eff_at(2 * k + 1) + 2) / 3 * 3 : eff_at(2 * k + 1); };
        row_narrow.assign(K, 0);
        std::vector<uint64_t> groups_k(K, 0);
        for(uint32_t k = 0; k < K; ++k) {
            const int64_t ncol = (int64_t) nrows - (2 * (int64_t) k + 1);
            if(ncol <= 0) continue;
            const bool nar = narrow_ok((int64_t) round_up(rows_at(k), SH), (int64_t) cols_at(k), tbl, gap) && !(ctx->nw_variant & MSA_NW_VARIANT_INT32);
            row_narrow[k] = nar ? kRowNarrow : 0;
            if(!nar && tiles.R == 32 && long_ok(tbl, gap) && !(ctx->nw_variant & MSA_NW_VARIANT_INT32))
                row_narrow[k] = kRowNarrow | kRowLong;
            groups_k[k] = (uint64_t) (ncol + tiles.W - 1) / tiles.W;
            if(nar && k >= k_lo && k < k_hi) pl->narrow_tasks += (uint32_t) groups_k[k];
        }
        const uint64_t resident = 2 * (uint64_t) ctx->num_sms;
        // A task's time in instructions of one warp: steps times (rows per lane + kStepCost).
        auto task_cost = [&](uint32_t k) {
            const uint64_t R = strip_rows<32>((int) rows_at(k), 0), nst = (rows_at(k) + 32 * R - 1) / (32 * R);
            return nst * (cols_at(k) + 31) * (R + kStepCost);
        };
        // Short rows pairs stacked in one warp (stack_task), four by four up to
        // 256 rows and two by two up to 512: all on 16-bit lanes with the state
        // bound holding for 512 rows, the first's longer sequence within the
        // lanes, the last with two sequences and columns, and all in this
        // part. The others' tasks are the first's. Stacking leaves fewer and
        // longer tasks, so it is used where at least two per resident CTA are
        // left (257 proteins of 150 to 400 residues: 274 us stacked two by two,
        // 350 us not), and two by two also where the tasks are more than the
        // resident CTAs, none stands out and all can be stacked, since then a
        // second round of them costs more: stacked against not, 100 proteins of 20 residues 45 and 50
        // us, of 100 to 150 56 and 67, of 300 to 400 122 and 136, 170 of 200 to
        // 256 122 and 157. 120 of 80 to 600, whose mean task is 0.63 of the
        // longest: 153 and 141; 100 of 480 to 600: 261 and 206; 64 of 100 to 150,
        // one round: 56 and 55.
        if(tiles.R == 32 && narrow_ok(512, 512, tbl, gap)) {
            uint64_t groups_all = 0, total = 0, longest = 0;
            for(uint32_t k = k_lo; k < k_hi; ++k) {
                groups_all += groups_k[k];
                total += groups_k[k] * task_cost(k);
                longest = std::max(longest, task_cost(k));
            }
            const uint64_t fill = 2 * resident;
            const bool even = groups_all > resident && 10 * total >= 7 * longest * groups_all && rows_at(k_lo) <= 16 * 32;
            auto stack = [&](uint32_t pairs, uint32_t rows, uint8_t flag) {
                if(groups_all < pairs * fill && !(pairs == 2 && even)) return;
                for(uint32_t k = k_lo; k + pairs <= k_hi;) {
                    bool ok = 2 * ((uint64_t) k + pairs) <= nrows;
                    for(uint32_t p = 0; p < pairs; ++p)
                        ok = ok && row_narrow[k + p] == kRowNarrow && groups_k[k + p] != 0 && rows_at(k + p) <= rows;
                    if(!ok) {
                        ++k;
                        continue;
                    }
                    row_narrow[k] |= flag;
                    for(uint32_t p = 1; p < pairs; ++p) groups_k[k + p] = 0;
                    k += pairs;
                }
            };
            if(tiles.W == 8 && !(ctx->nw_variant & MSA_NW_VARIANT_NO_PACKED)) stack(4, 8 * 32, kRowOct);
            stack(2, 16 * 32, kRowQuad);
        }
        // Where the strips of the longest rows pair, one after the other, take
        // more than the launch's share per resident CTA, it and those down to
        // half of that share may be chained: every strip a task, each waiting for
        // the boundary row of the one above as it comes. (50 genomes: 4.7 ms,
        // 5.4 when only those above the whole share are; where the longest is
        // below it, the order of the tasks balances them, and chaining would
        // cost 1,200 uneven sequences 0.3%.)
        chain_off.assign(K + 1, 0);
        if(tiles.R == 32 && tiles.W == 8 && !ctx->nw_variant && !ctx->tile_r && long_ok(tbl, gap)) {
            uint64_t total = 0;
            for(uint32_t k = k_lo; k < k_hi; ++k) total += groups_k[k] * task_cost(k);
            uint32_t kc = k_lo;
            double high = 0, low = 0;
            for(; kc < k_hi; ++kc) {
                const uint64_t rows = rows_at(kc), words = groups_k[kc] * 8 * chain_words_of((uint32_t) eff_at(2 * kc + 1));
                if(rows <= 32 * 32 || !row_narrow[kc] || (kc == k_lo ? 1 : 2) * resident * task_cost(kc) < total) break;
                if(chain_words + words > (kChainBytes >> 2)) break;
                chain_off[kc] = chain_words;
                chain_words += words;
                const double steps = (double) (groups_k[kc] * (cols_at(kc) + 31));
                const uint64_t R = strip_rows<32>((int) rows, 0);
                high += steps * (double) ((rows + 1023) / 1024 * (R + kStepCost + kMovingCost));
                low += steps * (double) ((rows + 511) / 512 * (16 + kStepCost + kMovingCost));
            }
            uint8_t form = 0;
            if(kc > k_lo) {
                const double steps = (double) (cols_at(k_lo) + 31);
                const uint64_t R = strip_rows<32>((int) rows_at(k_lo), 0);
                form = chain_form(rows_at(k_lo), cols_at(k_lo), row_narrow[k_lo] & kRowLong,
                                  (double) total / (double) task_cost(k_lo),
                                  high / (steps * (double) (R + kStepCost + kMovingCost)),
                                  low / (steps * (double) (16 + kStepCost + kMovingCost)), (double) resident);
            }
            if(!(form & kRowChain)) {
                kc = k_lo;
                chain_words = 0;
                chain_off.assign(K + 1, 0);
            }
            for(uint32_t k = k_lo; k < kc; ++k) {
                row_narrow[k] |= form;
                const uint64_t SH = 32 * (uint64_t) strip_rows<32>((int) rows_at(k), row_narrow[k]);
                groups_k[k] *= (rows_at(k) + SH - 1) / SH;   // tasks
                chain_tasks += groups_k[k];
            }
        }
        // Tasks of a single-strip rows pair take up to gchunk column groups
        // (one staging of the strip for all of them) while this part keeps at
        // least 16 tasks per resident CTA for the work-stealing tail.
        auto tables = [&](uint32_t chunk) {
            row_task.assign(K + 1, 0);
            uint64_t nt = 0;
            for(uint32_t k = 0; k < K; ++k) {
                row_task[k] = nt;
                const uint32_t c = groups_per_task((uint32_t) rows_at(k), tiles.R, chunk);
                nt += (groups_k[k] + c - 1) / c;
            }
            row_task[K] = nt;
            return row_task[k_hi] - row_task[k_lo];
        };
        int rc;
        const uint64_t all_groups = tables(1);
        if(ctx->nw_variant & MSA_NW_VARIANT_NO_PACKED) rc = batched_grid<32, 8, false>(ctx, 0, all_groups, &pl->batch_grid);
        else if(tiles.R == 16 && tiles.W == 4) rc = batched_grid<16, 4>(ctx, 1, all_groups, &pl->batch_grid);
        else if(tiles.R == 16 && tiles.W == 8) rc = batched_grid<16, 8>(ctx, 2, all_groups, &pl->batch_grid);
        else if(tiles.R == 32 && tiles.W == 4) rc = batched_grid<32, 4>(ctx, 3, all_groups, &pl->batch_grid);
        else rc = batched_grid<32, 8>(ctx, 4, all_groups, &pl->batch_grid);
        if(rc) return rc;
        const uint32_t want = ctx->nw_chunk ? ctx->nw_chunk : pick_chunk(st, nclean);
        for(gchunk = want; gchunk > 1 && tables(gchunk) < 16 * pl->batch_grid; gchunk /= 2) {}
        ntasks = tables(gchunk);
        // This part's tasks: those of rows pairs [k_lo, k_hi).
        task_base = row_task[k_lo];
        warps_needed = std::max<uint64_t>(warps_needed, pl->batch_grid * tiles.W);
    }

    if(bits.ntasks) {
        const int rc = bits_grid(ctx, bits, &pl->bits_grid);
        if(rc) return rc;
        pl->narrow_tasks += (uint32_t) bits.ntasks;
    }

    // One device block owned by the plan; the tables that come from the host
    // lie at its start and are copied at once.
    size_t off = 0;
    auto take = [&off](size_t b) { size_t o = off; off = round_up(off + b, 256); return o; };
    const size_t o_ext = take(kAlpha * kAlpha), o_rt = take((K + 1) * sizeof(uint64_t)), o_rn = take(K + 16),
                 o_co = take((K + 1) * sizeof(uint64_t)), o_gp = take(gpairs.size() * sizeof(uint32_t) + 16),
                 o_ord = take(nclean * sizeof(uint32_t) + 16), o_bs = take(bits.sets.size() * sizeof(BitSet) + 16),
                 o_go = take(bits.goff.size() * sizeof(uint64_t) + 16),
                 o_gc = take(bits.gcols.size() * sizeof(uint32_t) + 16), staged = off;
    pl->profiles = mode != MSA_NW_PERSISTENT || ntasks || pl->ngeneric;
    const size_t o_prof = take((pl->profiles ? st->prof_bytes : 0) + 64), o_bound = take(warps_needed * stride * sizeof(uint32_t)),
                 o_cb = take(chain_words * sizeof(uint32_t)), o_match = take(bits.match_words * sizeof(uint32_t)),
                 o_bb = take(pl->bits_grid * kBitWarps * bits.bound_words * sizeof(uint2)),
                 // the work counter, the error word and the chained strips' progress, cleared by every launch
                 o_cnt = take(64 + chain_tasks * 8 * sizeof(uint32_t));
    MSA_CUDA_TRY(ctx, take_block(ctx, off, &pl->mem, &pl->mem_bytes));
    pl->home = ctx;
    char *base = (char *) pl->mem;
    cudaStream_t s = ctx->stream;
    pl->staged.assign(staged, 0);
    auto put = [&](size_t o, const void *src, size_t b) { if(b) std::memcpy(pl->staged.data() + o, src, b); };
    put(o_ext, tbl.score, kAlpha * kAlpha);
    put(o_rt, row_task.data(), row_task.size() * sizeof(uint64_t));
    put(o_rn, row_narrow.data(), row_narrow.size());
    put(o_co, chain_off.data(), chain_off.size() * sizeof(uint64_t));
    put(o_gp, gpairs.data(), gpairs.size() * sizeof(uint32_t));
    put(o_ord, st->clean_sorted.data(), nclean * sizeof(uint32_t));
    if(bits.ntasks) {
        put(o_bs, bits.sets.data(), bits.sets.size() * sizeof(BitSet));
        put(o_go, bits.goff.data(), bits.goff.size() * sizeof(uint64_t));
        put(o_gc, bits.gcols.data(), bits.gcols.size() * sizeof(uint32_t));
    }
    MSA_CUDA_TRY(ctx, cudaMemcpyAsync(base, pl->staged.data(), staged, cudaMemcpyHostToDevice, s));

    pl->d_ext = (const int8_t *) (base + o_ext);
    NwParams &p = pl->p;
    p.units = st->d_units;
    p.uoff = st->d_off;
    p.eff = st->d_eff;
    p.plen = st->d_plen;
    p.prof = (const int8_t *) (base + o_prof);
    p.poff = st->d_prof_off;
    p.plp = st->d_prof_lp;
    p.sorted = (const uint32_t *) (base + o_ord);   // the call's order, not always the store's
    p.nclean = nclean;
    p.out = d_out;
    p.g = tbl.penalty;
    p.bound_stride = stride;
    p.bound = (uint32_t *) (base + o_bound);
    p.gpairs = (const uint32_t *) (base + o_gp);
    p.ngeneric = pl->ngeneric;
    pl->gen_blocks = std::min<uint64_t>(resident_blocks, (pl->ngeneric + kWPB - 1) / kWPB);

    BatchParams &bp = pl->bp;
    bp.job.units = st->d_units;
    bp.job.uoff = st->d_off;
    bp.job.eff = st->d_eff;
    bp.job.prof = p.prof;
    bp.job.poff = st->d_prof_off;
    bp.job.plp = st->d_prof_lp;
    bp.job.sorted = p.sorted;
    bp.job.nclean = nrows;
    bp.job.row_narrow = (const uint8_t *) (base + o_rn);
    bp.job.out = d_out;
    bp.job.g = tbl.penalty;
    bp.npairs_rows = K;
    bp.row_task = (const uint64_t *) (base + o_rt);
    bp.ntasks = ntasks;
    bp.task_base = task_base;
    bp.gchunk = gchunk;
    bp.bound = p.bound;
    bp.bound_stride = stride;
    bp.counter = (unsigned long long *) (base + o_cnt);
    bp.err = (int *) (base + o_cnt + 8);
    bp.wait_ns = (unsigned long long) (ctx->nw_wait_us ? ctx->nw_wait_us : kStripWaitUs) * 1000ull;
    bp.chain_flag = (uint32_t *) (base + o_cnt + 64);
    bp.chain_bound = (uint32_t *) (base + o_cb);
    bp.chain_off = (const uint64_t *) (base + o_co);
    bp.step = (uint32_t) std::min<int64_t>(largest_step(tbl, st->any_gap), 0xffff);
    pl->clear_bytes = 64 + chain_tasks * 8 * sizeof(uint32_t);
    pl->chained = chain_tasks != 0 || bits.nchain != 0;

    if(bits.ntasks) {
        BitParams &q = pl->bits;
        q.units = st->d_units;
        q.uoff = st->d_off;
        q.eff = st->d_eff;
        q.sorted = p.sorted;
        q.nclean = nclean;
        q.ngroups = (uint32_t) bits.gcols.size();
        q.g0 = bits.g0;
        q.sets = (const BitSet *) (base + o_bs);
        q.nsets = (uint32_t) bits.sets.size();
        q.ntasks = (uint32_t) bits.ntasks;
        q.match = (uint32_t *) (base + o_match);
        q.goff = (const uint64_t *) (base + o_go);
        q.gcols = (const uint32_t *) (base + o_gc);
        q.bound = (uint2 *) (base + o_bb);
        q.bound_words = bits.bound_words;
        q.out = d_out;
        q.u = planes.u;
        q.letters = planes.letters;
        q.g = tbl.penalty;
        q.nchain = (uint32_t) bits.nchain;
        q.err = bp.err;
        q.wait_ns = bp.wait_ns;
        q.counter = (unsigned long long *) (base + o_cnt + 16);   // cleared with the batched kernel's
    }

    pl->launches = (pl->profiles ? 1 : 0) + (pl->ngeneric ? 1 : 0) + (bits.ntasks ? 2 : 0);
    if(mode == MSA_NW_PLAIN && nclean_pairs > 0) {
        // Buckets: runs of sorted rows with the same strip count.
        constexpr int SH = 32 * kPlainR;
        // This part's rows: sorted [2 k_lo, 2 k_hi).
        const uint32_t a_end = std::min<uint32_t>(2 * k_hi, nclean);
        uint32_t a = std::min<uint32_t>(2 * k_lo, nclean);
        while(a < a_end && a + 1 < nclean) {
            const uint32_t strips = (st->eff[st->clean_sorted[a]] + SH - 1) / SH;
            uint32_t a2 = a + 1;
            while(a2 < a_end && a2 + 1 < nclean && (st->eff[st->clean_sorted[a2]] + SH - 1) / SH == strips) ++a2;
            const uint64_t k_lo = (uint64_t) a * (2 * (uint64_t) nclean - a - 1) / 2;
            const uint64_t k_hi = (uint64_t) a2 * (2 * (uint64_t) nclean - a2 - 1) / 2;
            pl->plain.push_back({k_lo, k_hi, std::min<uint64_t>(resident_blocks, (k_hi - k_lo + kWPB - 1) / kWPB)});
            a = a2;
        }
        pl->launches += (uint32_t) pl->plain.size();
    } else if(ntasks > 0) {
        pl->launches += 1;
    }
    return MSA_OK;
}

// Enqueues one scoring pass. Events are recorded with cudaEventRecordExternal
// while capturing so they stay real timing records inside the graph.
static cudaError_t enqueue(msa_ctx *ctx, const NwPlan &pl, const SeqStore *st, cudaStream_t s, bool capturing)
{
    const unsigned flags = capturing ? cudaEventRecordExternal : cudaEventRecordDefault;
    cudaError_t e = cudaEventRecordWithFlags(ctx->ev[0], s, flags);
    if(e) return e;
    if(pl.profiles) {
        build_profiles_kernel<<<pl.n, 256, 0, s>>>(st->d_units, st->d_off, st->d_eff, st->d_prof_off, st->d_prof_lp,
                                                   pl.d_ext, const_cast<int8_t *>(pl.p.prof));
        if((e = cudaGetLastError())) return e;
    }
    if(pl.bits.ntasks) {
        if((e = launch_match(pl.bits, s))) return e;
    }
    if((e = cudaEventRecordWithFlags(ctx->ev[1], s, flags))) return e;
    const size_t smem = smem_bytes<kPlainR>();
    if(pl.ngeneric) {
        nw_generic_kernel<kPlainR, kWPB><<<(unsigned) pl.gen_blocks, kWPB * 32, smem, s>>>(pl.p);
        if((e = cudaGetLastError())) return e;
    }
    if(pl.mode == MSA_NW_PLAIN) {
        for(const PlainLaunch &L : pl.plain) {
            nw_plain_kernel<kPlainR, kWPB><<<(unsigned) L.blocks, kWPB * 32, smem, s>>>(pl.p, L.k_lo, L.k_hi);
            if((e = cudaGetLastError())) return e;
        }
        return cudaEventRecordWithFlags(ctx->ev[2], s, flags);
    }
    if(pl.bp.ntasks || pl.bits.ntasks)
        if((e = cudaMemsetAsync(pl.bp.counter, 0, pl.clear_bytes, s))) return e;
    if(pl.bp.ntasks) {
        const Tiles t = pl.tiles;
        if(pl.variant & MSA_NW_VARIANT_NO_PACKED) launch_batched<32, 8, false>(pl, s);
        else if(t.R == 16 && t.W == 4) launch_batched<16, 4>(pl, s);
        else if(t.R == 16 && t.W == 8) launch_batched<16, 8>(pl, s);
        else if(t.R == 32 && t.W == 4) launch_batched<32, 4>(pl, s);
        else launch_batched<32, 8>(pl, s);
        if((e = cudaGetLastError())) return e;
    }
    if(pl.bits.ntasks) {
        if((e = launch_bits(pl.bits, pl.bits_grid, s))) return e;
    }
    return cudaEventRecordWithFlags(ctx->ev[2], s, flags);
}

static bool same_table(const ExtTable &a, const ExtTable &b)
{
    return std::memcmp(a.score, b.score, sizeof(a.score)) == 0 && std::memcmp(a.valid, b.valid, sizeof(a.valid)) == 0 &&
           a.penalty == b.penalty;
}

int nw_run(msa_ctx *ctx, SeqStore *st, const ExtTable &tbl, int mode, int32_t *d_out, uint32_t part,
           uint32_t nparts)
{
    cudaStream_t s = ctx->stream;
    const uint32_t n = st->n;
    msa_nw_stats stats{};
    stats.pairs = (uint64_t) n * (n > 0 ? n - 1 : 0) / 2;
    ctx->last_plane_tasks = 0;
    if(n < 2) { ctx->last = stats; return MSA_OK; }

    const uint32_t nclean = (uint32_t) st->clean_sorted.size();
    const Tiles tiles = mode != MSA_NW_PERSISTENT ? Tiles{0, 0}
                      : (ctx->nw_variant & MSA_NW_VARIANT_NO_PACKED) ? Tiles{32, 8}
                      : ctx->tile_r ? Tiles{ctx->tile_r, ctx->tile_w} : pick_tiles(st, nclean);

    if(!ctx->graphs) ctx->graphs = new GraphCache;
    auto &plans = ctx->graphs->plans;
    NwPlan *pl = nullptr;
    for(size_t i = 0; i < plans.size(); ++i) {
        NwPlan *c = plans[i];
        if(c->store_serial == st->serial && c->mode == mode && c->d_out == d_out && c->tiles.R == tiles.R &&
           c->tiles.W == tiles.W && c->part == part && c->nparts == nparts && same_table(c->tbl, tbl) &&
           c->variant == ctx->nw_variant && c->chunk == ctx->nw_chunk && c->wait_us == ctx->nw_wait_us &&
           c->fixed_tiles == (ctx->tile_r != 0)) {
            pl = c;
            plans.erase(plans.begin() + i);
            plans.push_back(pl);
            break;
        }
    }
    if(!pl) {
        auto held = [&plans] {
            size_t b = 0;
            for(const NwPlan *c : plans) b += c->mem_bytes;
            return b;
        };
        while(!plans.empty() && (plans.size() >= kMaxPlans || held() > kMaxPlanBytes)) {
            ctx->graphs->drop(plans.front());
            plans.erase(plans.begin());
        }
        pl = new NwPlan;
        const int rc = build_plan(ctx, st, tbl, mode, d_out, tiles, part, nparts, pl);
        if(rc) { delete pl; return rc; }
        plans.push_back(pl);
    }

    // The persistent mode replays a captured graph; the legacy default stream
    // cannot be captured, so there the same sequence is launched directly.
    bool use_graph = mode == MSA_NW_PERSISTENT && s != nullptr;
    if(use_graph && (!pl->exec || pl->captured_on != s)) {
        if(pl->exec) { cudaGraphExecDestroy(pl->exec); pl->exec = nullptr; }
        cudaGraph_t g = nullptr;
        cudaError_t e = cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal);
        if(!e) {
            const cudaError_t e2 = enqueue(ctx, *pl, st, s, true);
            e = cudaStreamEndCapture(s, &g);
            if(!e) e = e2;
        }
        if(!e) e = ctx->graphs->instantiate(g, &pl->exec);
        if(g) cudaGraphDestroy(g);
        if(e) {
            cudaGetLastError();
            pl->exec = nullptr;
            use_graph = false;   // launch the same kernels directly
        } else {
            pl->captured_on = s;
        }
    }
    if(use_graph) {
        MSA_CUDA_TRY(ctx, cudaGraphLaunch(pl->exec, s));
    } else {
        MSA_CUDA_TRY(ctx, enqueue(ctx, *pl, st, s, false));
    }
    ctx->launches += pl->launches;

    MSA_CUDA_TRY(ctx, cudaEventSynchronize(ctx->ev[2]));
    if(pl->chained) {
        int err = 0;
        MSA_CUDA_TRY(ctx, cudaMemcpyAsync(&err, pl->bp.err, sizeof(err), cudaMemcpyDeviceToHost, s));
        MSA_CUDA_TRY(ctx, cudaStreamSynchronize(s));
        if(err) return set_error(ctx, MSA_ERR_DEVICE_TIMEOUT, "a wait between the strips of a sequence ran out");
    }
    float ms_k = 0, ms_t = 0;
    cudaEventElapsedTime(&ms_k, ctx->ev[1], ctx->ev[2]);
    cudaEventElapsedTime(&ms_t, ctx->ev[0], ctx->ev[2]);
    stats.kernel_ms = ms_k;
    stats.total_ms = ms_t;
    stats.cells = pl->cells;
    stats.launches = pl->launches;
    stats.narrow_tasks = pl->narrow_tasks;
    ctx->last_plane_tasks = pl->bits.ntasks;
    stats.graph = use_graph ? 1 : 0;
    ctx->last = stats;
    return MSA_OK;
}

}  // namespace msa
