// All-pairs scores on bit planes, 32 column sequences to a word, for tables in
// which letters score M against themselves and I against any other with
// M + 2g = 3u and I + 2g = u, u > 0 (the DNA table: M = 1, I = -1, g = 1; a letter
// may score I against itself, as X does there).
//
// In the gap-free state T(i,j) = (H(i,j) + g (i + j)) / u a cell is
//   T = max(T_left, T_up, T_diag + w), w = 3 on a match, 1 otherwise,
// and T grows by 0 to 3 from a cell to its right or lower neighbour. With
// a = T(i,j-1) - T(i-1,j-1) and b = T(i-1,j) - T(i-1,j-1) the cell turns (a, b)
// into a' = T(i,j) - T(i-1,j) and b' = T(i,j) - T(i,j-1):
//   a' = t - b, b' = t - a, t = max(a, b, w),
// with a = 0 in column 0 and b = 0 in row 0. Both are two bits, so 32 pairs take
// a cell in four words (a and b as a high and a low bit) and a match word: eight
// three-input logic operations (bit_cell; found by a search over such circuits),
// with no carries between the bits. The 16-bit lanes of the batched kernel take
// two instructions and half a shared-memory load for two cells. What bounds the
// kernel is the ALU pipe (64 lanes per SM and clock, so 74 TCUPS at 1,965 MHz; ncu:
// 84% busy on 3,000 reads, three in four of its instructions in cells).
// 3,000 DNA reads of 100 to 250 bases 9.0 -> 2.96 ms, 1,200 uneven DNA sequences of
// 200 to 16,000 bases 177 -> 65 ms.
//
// A task is a set of 1, 2 or 4 rows sequences against one group of 32 sequences
// that are neighbours in the length order; one warp runs it. Lanes own R
// consecutive rows and advance one column per step behind the lane above, as in
// the batched kernel; the lanes of a warp are split between the sequences of a
// set. What a row needs of a column is the match word of its letter, from a ring
// of the group's last 32 to 64 columns that the warp keeps in shared memory (one row
// of words per letter). The last row's b words go to the warp's boundary row:
// they are the row above the next strip, and their sum over a sequence's columns
// is its T.
#include <algorithm>

#include "nw_bits.hpp"

namespace msa {
namespace dev {

constexpr unsigned kFull = 0xffffffffu;
__device__ __forceinline__ uint64_t tri_index(uint32_t i, uint32_t j)
{
    const uint64_t hi = i > j ? i : j, lo = i > j ? j : i;
    return hi * (hi - 1) / 2 + lo;
}


template <int LUT>
__device__ __forceinline__ uint32_t lop3(uint32_t a, uint32_t b, uint32_t c)
{
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, %4;" : "=r"(r) : "r"(a), "r"(b), "r"(c), "n"(LUT));
    return r;
}

// (a, b) -> (a', b') of 32 cells; a1, b1 are the high bits, m the match word.
__device__ __forceinline__ void bit_cell(uint32_t &a1, uint32_t &a0, uint32_t &b1, uint32_t &b0, uint32_t m)
{
    const uint32_t p = lop3<0x06>(b1, a0, a1);
    const uint32_t q = lop3<0xc4>(b0, b1, a0);
    const uint32_t nb1 = lop3<0x54>(q, m, a1);
    const uint32_t r = lop3<0x54>(m, b0, a0);
    const uint32_t s = lop3<0x06>(r, nb1, a1);
    const uint32_t nb0 = lop3<0x0b>(s, p, m);
    a1 = lop3<0x54>(s, m, b1);
    a0 = lop3<0x16>(nb0, b0, a0);
    b1 = nb1;
    b0 = nb0;
}

// Lane s: the number of set bits s of x over the lanes (a 32 x 32 transposition).
__device__ __forceinline__ int count_bits(uint32_t x, int lane)
{
    uint32_t low = 0xffffu;
#pragma unroll
    for(int d = 16; d; d >>= 1, low ^= low << d) {
        const uint32_t y = __shfl_xor_sync(kFull, x, d);
        x = lane & d ? (x & ~low) | ((y & ~low) >> d) : (x & low) | ((y & low) << d);
    }
    return __popc(x);
}

// Waits until *done >= want, or gives up: then, and in every later wait of the
// launch, the strip runs on with what is there and the call fails.
__device__ __noinline__ void strip_wait(const BitParams &p, volatile unsigned long long *done, unsigned long long want)
{
    unsigned long long t0, t1;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    while(*done < want) {
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
        if(*(volatile int *) p.err != 0) break;
        if(t1 - t0 > p.wait_ns) {
            atomicExch(p.err, 1);
            break;
        }
        __nanosleep(100);
    }
}

// One task. `ring`: the warp's kRingRows rows of S words. S is 0 mod 32 where the
// lanes are on 32 different columns, and 8 or 16 where 4 or 2 lanes are on one: equal
// columns of the first letters then lie in different banks. `done`: the progress of the
// warps of a CTA that share a task's strips, as strip_progress gives it (null: one warp
// has all of them).
template <int R, int LP>
__device__ __noinline__ void bit_task(const BitParams &p, const BitSet &set, uint32_t grp, uint32_t *ring,
                                      uint2 *bound, int lane, int s0 = 0, int ds = 1,
                                      volatile unsigned long long *done = nullptr)
{
    constexpr int S = 96 + (LP == 8 ? 8 : LP == 16 ? 16 : 0), U = R <= 8 ? 4 : R <= 16 ? 2 : 1;
    const int at = lane % LP, ncols = (int) p.gcols[grp];
    const uint32_t pitch = bit_pitch((uint32_t) ncols);
    const uint32_t *match = p.match + p.goff[grp];
    const uint32_t x = p.sorted[set.a + lane / LP];
    const int ex = (int) p.eff[x], nst = LP == 32 ? (int) set.nst : 1;
    const uint8_t *ux = p.units + p.uoff[x];
    const uint32_t bstride = bit_bound((uint32_t) ncols);
    uint2 *mine = bound + (lane / LP) * bstride;

    // Rows past the sequence's end, in the lane that holds its last row, match
    // every column: pad such rows move the last row's cells pad columns on.
    const int last_lane = (ex - 1 - (nst - 1) * 32 * R) / R;
    const int pad = R - 1 - (ex - 1 - (nst - 1) * 32 * R) % R;
    __syncwarp();
    for(int k = lane; k < S; k += 32) ring[kRingAll * S + k] = kFull;

    for(int st = s0; st < nst; st += ds) {
        const bool last = st == nst - 1;
        const int i0 = st * 32 * R + at * R;
        uint32_t off[R], a1[R], a0[R], letters = 0;
        const uint32_t base = (uint32_t) __cvta_generic_to_shared(ring) + (32 - at) * 4;
#pragma unroll
        for(int r = 0; r < R; ++r) {
            const uint32_t c = i0 + r < ex ? ux[i0 + r] : (uint32_t) kRingAll;
            letters |= 1u << c;
            off[r] = base + c * (S * 4);
            a1[r] = a0[r] = 0u;
        }
        letters = __reduce_or_sync(kFull, letters) & ~(1u << kRingAll);
        const int width = ncols + (last ? pad : 0);
        const bool keeps = at == (last ? last_lane : LP - 1);
        const int tend = (int) __reduce_max_sync(kFull, (uint32_t) (width + (last ? last_lane : LP - 1)));
        const uint32_t top = base + kRingTop * (S * 4);
        uint32_t b1 = 0, b0 = 0;

        // Columns c0 + lane behind the 32 before them.
        auto load = [&](int c0) {
            const bool in = c0 + lane < (int) pitch;
            __syncwarp();
            for(uint32_t m = letters; m;) {
                uint32_t w[4], c[4];
#pragma unroll
                for(int q = 0; q < 4; ++q) {
                    c[q] = m ? (uint32_t) __ffs((int) m) - 1 : kRingAll;
                    m &= m - 1;
                    w[q] = c[q] == kRingAll ? kFull : in ? __ldg(match + c[q] * pitch + c0 + lane) : 0u;
                }
#pragma unroll
                for(int q = 0; q < 4; ++q) {
                    uint32_t *dst = ring + c[q] * S + lane;
                    dst[0] = dst[32];
                    dst[32] = w[q];
                }
            }
            if(LP == 32 && done) {
                // Lane 31 has stored the columns up to c0 - 32.
                if(lane == 31 && c0 > 31) {
                    __threadfence_block();
                    done[st % ds] = strip_progress((uint32_t) st, (uint32_t) (c0 - 31));
                }
                if(st > 0) {
                    const unsigned long long want = strip_progress((uint32_t) st - 1, (uint32_t) min(c0 + 32, ncols));
                    if(done[(st - 1) % ds] < want)
                        strip_wait(p, done + (st - 1) % ds, want);
                    __threadfence_block();
                }
                __syncwarp();
            }
            if(st > 0) {   // lane 0 reads these, at its own column only
                const uint2 v = c0 + lane < (int) bstride ? mine[c0 + lane] : make_uint2(0, 0);
                uint32_t *dst = ring + kRingTop * S + 32 + lane;
                dst[0] = v.x;
                dst[S] = v.y;
            }
            __syncwarp();
        };
#pragma unroll 1
        for(int c0 = 0; c0 < tend; c0 += 32) {
            load(c0);
            const int steps = min(32, tend - c0);
            int j = c0 - at;
#pragma unroll 1
            for(int t = 0; t < steps; t += U) {
#pragma unroll
                for(int u = 0; u < U; ++u, ++j) {
                    uint32_t u1 = __shfl_up_sync(kFull, b1, 1), u0 = __shfl_up_sync(kFull, b0, 1);
                    if(at == 0) {
                        u1 = u0 = 0u;
                        if(LP == 32 && st > 0) {
                            asm volatile("ld.shared.u32 %0, [%1];" : "=r"(u1) : "r"(top + 4 * (t + u)) : "memory");
                            asm volatile("ld.shared.u32 %0, [%1];" : "=r"(u0) : "r"(top + 4 * (t + u) + S * 4) : "memory");
                        }
                    }
                    if(j >= 0) {
#pragma unroll
                        for(int r = 0; r < R; ++r) {
                            uint32_t m;
                            asm volatile("ld.shared.u32 %0, [%1];" : "=r"(m) : "r"(off[r] + 4 * (t + u)) : "memory");
                            bit_cell(a1[r], a0[r], u1, u0, m);
                        }
                        b1 = u1;
                        b0 = u0;
                        if(keeps && j < width) mine[j] = make_uint2(b1, b0);
                    }
                }
            }
        }
        __syncwarp();
        if(LP == 32 && done && lane == 31) {
            __threadfence_block();
            done[st % ds] = strip_progress((uint32_t) st, 0xffffffffu);
        }
    }
    if((nst - 1) % ds != s0) return;   // another warp has the last row

    // T of every pair: the sum of the last row's b over the sequence's columns.
    // Lanes take every 32nd column and add into 12 bit planes; then the planes'
    // bits are counted over the lanes.
    const int planes = 32 - __clz(3 * ((ncols + 31) / 32));
    const uint32_t b = 32 * grp + lane;
    const bool has = b < p.nclean;
    const uint32_t y = has ? p.sorted[b] : 0;
    for(int k = 0; k < 32 / LP; ++k) {
        const int shift = __shfl_sync(kFull, pad, k * LP);
        const uint32_t xk = __shfl_sync(kFull, x, k * LP);
        const uint2 *row = bound + k * bstride + shift;
        uint32_t sum[12];
#pragma unroll
        for(int q = 0; q < 12; ++q) sum[q] = 0u;
        for(int j = lane; j < ncols; j += 32) {
            const uint32_t in = __ldg(match + kBitLetters * pitch + j);
            const uint2 v = row[j];
            uint32_t carry = v.y & in, hi = v.x & in;
#pragma unroll
            for(int q = 0; q < 12; ++q) {
                if(q >= planes) break;
                uint32_t next = sum[q] & carry;
                sum[q] ^= carry;
                if(q == 1) {   // the high bit comes in here
                    next |= sum[q] & hi;
                    sum[q] ^= hi;
                }
                carry = next;
            }
        }
        int t = 0;
#pragma unroll
        for(int q = 0; q < 12; ++q) if(q < planes) t += count_bits(sum[q], lane) << q;
        if(has && b > set.a + k) p.out[tri_index(xk, y)] = p.u * t - p.g * ((int32_t) p.eff[xk] + (int32_t) p.eff[y]);
    }
}

}  // namespace dev

// Match words of 32 columns of a group per warp.
__global__ void __launch_bounds__(128) nw_match_kernel(BitParams p)
{
    const uint32_t q = p.g0 + blockIdx.x, n = p.gcols[q], pitch = bit_pitch(n);
    const int lane = threadIdx.x & 31;
    const uint32_t b = 32 * q + lane, y = p.sorted[min(b, p.nclean - 1)], e = b < p.nclean ? p.eff[y] : 0;
    const uint8_t *units = p.units + p.uoff[y];
    uint32_t *dst = p.match + p.goff[q];
    for(uint32_t c0 = 32 * (blockIdx.y * 4 + threadIdx.x / 32); c0 < pitch; c0 += 32 * 4 * gridDim.y) {
        uint32_t w[8];
#pragma unroll
        for(int h = 0; h < 2; ++h) {
            uint4 v = make_uint4(~0u, ~0u, ~0u, ~0u);
            if(c0 + 16 * h < e) v = __ldg(reinterpret_cast<const uint4 *>(units + c0 + 16 * h));
            w[4 * h] = v.x; w[4 * h + 1] = v.y; w[4 * h + 2] = v.z; w[4 * h + 3] = v.w;
        }
        for(uint32_t c = 0; c < (uint32_t) kBitRows; ++c) {
            uint32_t mine = 0;
#pragma unroll
            for(int j = 0; j < 32; ++j) {
                const bool in = c0 + j < e;
                const uint32_t word = __ballot_sync(dev::kFull, in && (c == (uint32_t) kBitLetters || (((w[j / 4] >> (8 * (j % 4))) & 0xffu) == c && p.letters >> c & 1)));
                if(lane == j) mine = word;
            }
            dst[c * pitch + c0 + lane] = mine;
        }
    }
}

// Words of a warp's ring, enough for every stride.
constexpr int kRingWords = kRingRows * 112;
constexpr size_t kRingBytes = kBitWarps * kRingWords * sizeof(uint32_t);

// Four warps per CTA, four CTAs per SM. 1,200 uneven sequences, before the split of a
// job counted a warp's pace beside three others (65 ms since): with three CTAs, and
// registers to spare, 76.5 ms instead of 71.8. A step of R rows is one pass of the loop
// where R is above 16: two steps to a pass save an addition per row, but the warps'
// places in the code then outgrow the instruction caches (78.1 ms; four steps 98.6).
// Every warp takes its own tasks, longest rows first. ptxas spills 4 to 52 bytes in the
// tasks of 22 rows and more.
__global__ void __launch_bounds__(kBitWarps * 32, 4) nw_bits_kernel(BitParams p)
{
    extern __shared__ __align__(16) uint32_t rings[];
    __shared__ unsigned long long done[kBitWarps];
    __shared__ unsigned long long task;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t *ring = rings + warp * kRingWords;
    auto find = [&](uint32_t q) {
        uint32_t lo = 0, hi = p.nsets - 1;
        while(lo < hi) {
            const uint32_t mid = (lo + hi + 1) >> 1;
            if(p.sets[mid].first <= q) lo = mid; else hi = mid - 1;
        }
        return p.sets[lo];
    };
    // Chained tasks: strip s on warp s mod kBitWarps (1,200 uneven sequences, with four
    // steps to a pass: 117 ms with every task on one warp, 98.6 chained).
    while(p.nchain) {
        __syncthreads();
        if(threadIdx.x == 0) task = atomicAdd(p.counter, 1ull);
        if(lane == 0) done[warp] = 0;
        __syncthreads();
        const unsigned long long q = task;
        if(q >= p.nchain) break;
        const BitSet set = find((uint32_t) q);
        const uint32_t grp = max(p.g0, set.a / 32) + (uint32_t) q - set.first;
        uint2 *bound = p.bound + blockIdx.x * kBitWarps * p.bound_words;
#define MSA_BITS(RR) case RR: dev::bit_task<RR, 32>(p, set, grp, ring, bound, lane, warp, kBitWarps, done); break;
        if(warp < (int) set.nst)
            switch(set.R) {
                MSA_BITS(18) MSA_BITS(20) MSA_BITS(22) MSA_BITS(24) MSA_BITS(26) MSA_BITS(28) MSA_BITS(30) MSA_BITS(32)
                default: break;
            }
#undef MSA_BITS
    }
    uint2 *bound = p.bound + (blockIdx.x * kBitWarps + warp) * p.bound_words;
    for(;;) {
        unsigned long long q = 0;
        if(lane == 0) q = p.nchain + atomicAdd(p.counter + 1, 1ull);
        q = __shfl_sync(dev::kFull, q, 0);
        if(q >= p.ntasks) break;
        const BitSet set = find((uint32_t) q);
        const uint32_t grp = max(p.g0, set.a / 32) + (uint32_t) q - set.first;
#define MSA_BITS(RR, LL) case RR: dev::bit_task<RR, LL>(p, set, grp, ring, bound, lane); break;
        if(set.lanes == 8) {
            switch(set.R) {
                MSA_BITS(4, 8) MSA_BITS(6, 8) MSA_BITS(8, 8) MSA_BITS(10, 8) MSA_BITS(12, 8) MSA_BITS(14, 8)
                MSA_BITS(16, 8) MSA_BITS(18, 8) MSA_BITS(20, 8) MSA_BITS(22, 8) MSA_BITS(24, 8) MSA_BITS(26, 8)
                MSA_BITS(28, 8) MSA_BITS(30, 8) MSA_BITS(32, 8) default: break;
            }
        } else if(set.lanes == 16) {
            switch(set.R) {
                MSA_BITS(18, 16) MSA_BITS(20, 16) MSA_BITS(22, 16) MSA_BITS(24, 16) MSA_BITS(26, 16)
                MSA_BITS(28, 16) MSA_BITS(30, 16) MSA_BITS(32, 16) default: break;
            }
        } else {
            switch(set.R) {
                MSA_BITS(18, 32) MSA_BITS(20, 32) MSA_BITS(22, 32) MSA_BITS(24, 32) MSA_BITS(26, 32)
                MSA_BITS(28, 32) MSA_BITS(30, 32) MSA_BITS(32, 32) default: break;
            }
        }
#undef MSA_BITS
    }
}

// ---------------------------------------------------------------- host side

BitTable bit_table(const ExtTable &t)
{
    const int32_t g2 = 2 * t.penalty;
    BitTable b{t.score[1] + g2, 0};
    if(b.u <= 0) return BitTable{0, 0};
    for(int x = 0; x < kBitLetters; ++x)
        for(int y = 0; y < kBitLetters; ++y) {
            const int32_t s = t.score[x * kAlpha + y] + g2;
            if(x == y && s == 3 * b.u) b.letters |= 1u << x;
            else if(s != b.u) return BitTable{0, 0};
        }
    return b;
}

// Sets and split for the sorted lengths `eff`. The first groups hold the
// longest and most unequal sequences, so their words are the emptiest and their
// tasks the longest serial ones; g0 is where the sum of both kernels' times is
// least. A warp's step takes about 16 R + 40 cycles of its scheduler; the
// batched kernel runs a few long sequences at about 10 TCUPS and whole jobs at
// 11 to 16 by their median length.
BitPlan plan_bits(const std::vector<uint32_t> &eff, uint32_t num_sms)
{
    BitPlan bp;
    const uint32_t n = (uint32_t) eff.size(), ng = (n + 31) / 32;
    bp.gcols.assign(ng, 0);
    for(uint32_t a = 0; a < n; ++a) bp.gcols[a / 32] = std::max(bp.gcols[a / 32], eff[a]);
    auto longest = [&](uint32_t a, uint32_t k) {
        uint32_t e = 0;
        for(uint32_t i = a; i < a + k; ++i) e = std::max(e, eff[i]);
        return e;
    };
    auto even = [](uint32_t rows, uint32_t lanes) { return ((rows + lanes - 1) / lanes + 1) & ~1u; };
    for(uint32_t a = 0; a + 1 < n;) {
        BitSet s{a, 0, 32, 0, 1};
        if(a % 4 == 0 && a + 4 <= n && longest(a, 4) <= 8 * 32) {
            s.lanes = 8;
            s.R = (uint16_t) std::max(even(longest(a, 4), 8), 4u);
        } else if(a % 2 == 0 && a + 2 <= n && longest(a, 2) <= 16 * 32) {
            s.lanes = 16;
            s.R = (uint16_t) std::max(even(longest(a, 2), 16), 18u);
        } else {
            const uint32_t strips = (eff[a] + 1023) / 1024;
            s.R = (uint16_t) std::max(even(eff[a], 32 * strips), 18u);
            s.nst = (eff[a] + 32 * s.R - 1) / (32 * s.R);
        }
        bp.sets.push_back(s);
        a += 32 / s.lanes;
    }
    // Cycles of a set per column, and of its task against group q.
    auto rate = [](const BitSet &s) { return (double) s.nst * (16 * s.R + 40); };
    auto steps = [&](const BitSet &s, uint32_t q) { return (double) bp.gcols[q] + s.lanes + s.R / 2 + 20; };
    std::vector<double> work(ng + 1, 0), cells(ng + 1, 0);   // of groups q and later; of the first q groups' sequences
    {
        std::vector<double> sum(ng, 0), fixed(ng, 0);   // over the sets with a / 32 <= q
        for(const BitSet &s : bp.sets) {
            sum[s.a / 32] += rate(s);
            fixed[s.a / 32] += rate(s) * (steps(s, s.a / 32) - bp.gcols[s.a / 32]);
        }
        for(uint32_t q = 1; q < ng; ++q) sum[q] += sum[q - 1], fixed[q] += fixed[q - 1];
        for(uint32_t q = ng; q-- > 0;) work[q] = work[q + 1] + sum[q] * bp.gcols[q] + fixed[q];
        double len = 0, got = 0;
        for(uint32_t a = 0; a < n; ++a) {
            got += len * eff[a];
            len += eff[a];
            cells[a / 32 + 1] = got;
        }
    }
    // A warp's pace beside three others on its scheduler. Taken as 2, 1,200 uneven
    // sequences put the longest 32 against themselves here: 71 ms, most of it that task.
    constexpr double kShare = 4;
    auto rounds = [](const BitSet &s) { return (s.nst + kBitWarps - 1) / kBitWarps; };
    const double hz = 1.9e9, med = eff[n / 2], whole = med < 384 ? 11e12 : med < 1024 ? 13e12 : med < 2048 ? 15e12 : 16e12;
    double best = cells[ng] / whole;
    bp.g0 = ng;
    for(uint32_t q = 0; q < ng; ++q) {
        if(bp.gcols[q] > kBitMaxCols) continue;
        double serial = 0;   // the longest task: of the first set, or of a later group's own
        if(!bp.sets.empty()) serial = kShare * rate(bp.sets[0]) / bp.sets[0].nst * rounds(bp.sets[0]) * steps(bp.sets[0], q);
        const double both = q ? cells[q] / 10e12 + 20e-6 : 0;   // profiles, and another kernel's start and tail
        const double t = both + std::max(work[q] / (4.0 * num_sms), serial) / hz + 10e-6;
        if(t < best) best = t, bp.g0 = q;
    }
    if(bp.g0 == ng) return bp;
    std::vector<uint32_t> widest(bp.gcols);   // of groups q and later
    for(uint32_t q = ng - 1; q-- > 0;) widest[q] = std::max(widest[q], widest[q + 1]);
    for(BitSet &s : bp.sets) {
        const uint32_t q = std::max(bp.g0, s.a / 32);
        s.first = (uint32_t) bp.ntasks;
        bp.ntasks += ng - q;
        bp.bound_words = std::max(bp.bound_words, 32 / s.lanes * (uint64_t) bit_bound(widest[q]));
    }
    // The tasks that would take more than half of the launch on one warp are chained
    // (a quarter and the whole of it measured within 2%). Sets are in falling order of length.
    for(const BitSet &s : bp.sets) {
        if(s.nst < 2 || kShare * rate(s) * steps(s, std::max(bp.g0, s.a / 32)) < work[bp.g0] / (8.0 * num_sms)) break;
        bp.nchain = s.first + (ng - std::max(bp.g0, s.a / 32));
    }
    bp.goff.assign(ng, 0);
    for(uint32_t q = bp.g0; q < ng; ++q) {
        bp.goff[q] = bp.match_words;
        bp.match_words += (uint64_t) kBitRows * bit_pitch(bp.gcols[q]);
    }
    return bp;
}

int bits_grid(msa_ctx *ctx, const BitPlan &plan, uint64_t *grid)
{
    int &bps = ctx->bits_blocks_per_sm;
    if(bps == 0) {
        int k = 0;
        MSA_CUDA_TRY(ctx, cudaFuncSetAttribute(nw_bits_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
        MSA_CUDA_TRY(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&k, nw_bits_kernel, kBitWarps * 32, kRingBytes));
        if(k < 1) return set_error(ctx, MSA_ERR_CUDA, "the bit-plane NW kernel cannot be resident");
        bps = k;
    }
    *grid = std::min<uint64_t>((uint64_t) ctx->num_sms * bps, plan.nchain + (plan.ntasks - plan.nchain + kBitWarps - 1) / kBitWarps);
    return MSA_OK;
}

cudaError_t launch_match(const BitParams &p, cudaStream_t s)
{
    nw_match_kernel<<<dim3(p.ngroups - p.g0, 8), 128, 0, s>>>(p);
    return cudaGetLastError();
}

cudaError_t launch_bits(const BitParams &p, uint64_t grid, cudaStream_t s)
{
    nw_bits_kernel<<<(unsigned) grid, kBitWarps * 32, kRingBytes, s>>>(p);
    return cudaGetLastError();
}

}  // namespace msa
