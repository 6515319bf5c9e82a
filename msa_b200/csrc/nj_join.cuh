// The joining kernels of neighbor-joining.
//
// State. D is a full symmetric float matrix over *slots*; a node keeps its slot
// while it lives. The reference numbers the live nodes logically and moves one
// of them at every join (sequential.cpp:189-224); here only the number moves:
// pos[slot] is the node's logical index (plus t in the symmetric order, whose
// indices all shift down by one per join).
//
// nj_join_kernel: one cluster of K CTAs, the matrix in global memory. A join
// of (x, y) puts the new node into a slot freed at an earlier join (`spare`;
// one slot more than nodes is allocated), so nothing that this join reads is
// overwritten by it.
//
// Search. Every live node has a row state: its best partner jb among the
// nodes of its last scan with their distance db, and an upper bound on Q over
// all its other partners. With S the row sums as stored, k joins after the
// bound B was taken and for every partner j,
//   Q_ij(now) = Q_ij(then) - k D_ij - (S_i(now) - S_i(then)) - (S_j(now) - S_j(then))
//            <= B(then) - k min_j D_ij - (S_i(now) - S_i(then)) + (C(now) - C(then)),
// where C adds up, join by join, the largest fall of any row sum; every
// operation on bounds rounds up. `slack` covers the rounding of the float
// evaluation of Q (three roundings of values at most (c-2) max|D| + 2 max|S|,
// here with a factor of more than two to spare). A row whose bound stays
// strictly below a Q already known to be attained cannot hold the maximum, nor
// tie with it, and is not read; a row that can is scanned in full with the
// reference's operations and order, which renews its state. A new node's
// pairs enter the state of the *other* node (one Q per row and join), so
// every live pair is covered by the row of its older node. Rows start without
// a bound, so the first search of a launch reads the whole matrix. Any
// non-finite or huge value switches the bounds off and every row is scanned
// every time. On matrices of related, of independent and of very uneven
// sequences 14 to 28 rows of 2,000 to 5,000 are read per join, 158 where only four
// distinct scores make many pairs tie, and all of them among copies of one sequence;
// there the launch gives up (kManyRows).
//
// Phases of a join:
//   search  every CTA owns the rows of slots = rank mod K: it scans those whose
//           bound reaches the best value known, while two warps fold the last
//           new node's row sum (sequential.cpp:259, a serial float sum); then
//           each row takes in its pair with that node and evaluates its best
//           pair exactly;
//   A       each CTA's best candidate goes to every CTA (distributed shared
//           memory), one cluster barrier;
//   join    every CTA computes all new distances and row sums for its own
//           copy of S (sequential.cpp:247-267): two row reads from L2 and no
//           second exchange; the new row and column are written by slices.
// The new column is not read before the next barrier A (its slot's S is +inf
// until then, which keeps it out of every scan), so the writes need no barrier
// of their own.
//
// nj_small_kernel: one CTA, the matrix in its shared memory and the live slots
// kept dense, so a plain search of every pair is cheaper than any bookkeeping.
//
// Measured beside a search of the whole lower triangle at every join (one
// cluster of 16 CTAs, slices of the join exchanged over a second barrier):
// 5,000 proteins 90.6 -> 38.3 ms, 2,000 proteins 15.2 -> 10.0 ms, 257 proteins
// 1.34 -> 0.76 ms with its upload, 120 proteins 0.55 -> 0.23 ms. What bounds a join
// now is the latency of its phases, not the matrix: at 2,000 nodes about 3,600 cycles
// for the rows scanned (the fold beside them 3,300), 1,500 to take in the new node,
// 1,900 to the barrier and across it, 2,900 for the join.
#pragma once

#include "nj_device.cuh"

namespace msa {
namespace njdev {

constexpr int kJoinThreads = 512;
constexpr int kJoinWarps = kJoinThreads / 32;
static_assert(kJoinWarps == 16, "half a warp reads one candidate per warp");
constexpr int kFoldWarps = 2;                   // fold a row sum while the others scan
constexpr int kScanWarps = kJoinWarps - kFoldWarps;
constexpr int kFoldParts = kFoldWarps * 8;      // four lanes each
constexpr uint32_t kDead = 0xffffu;             // pos of a slot without a live node; no partner
// Where copies of a sequence or few distinct scores make many pairs tie, every row
// that ties is read at every join, and a search of every pair (nj_cluster_kernel,
// on a matrix that holds the live nodes alone) is quicker. A CTA's rows beyond
// `rows_allowed` are added up over the joins; where they come to kExcessJoins joins'
// worth, the launch ends with kManyRows and the host goes on with that kernel.
constexpr int kManyRows = 5, kExcessJoins = 16;
constexpr uint32_t kGiveUp = 0x80000000u;   // in a candidate's slots, which take 14 bits each
// Float4 loads each lane keeps in flight while it scans a row.
constexpr int kRowBatch = 4;
constexpr size_t kMaxSmem = 227 * 1024 - 4096;   // dynamic, beside up to 4 KB of static shared memory

// One launch: joins from N nodes (slot k = logical k) down to c_end.
struct Stage {
    float *D;                  // (N + 1) rows of P floats
    const float *S0;           // row sums by slot
    float *S_out;              // row sums by logical index at the end
    uint32_t *order_out;       // slot of each logical index at the end
    uint32_t *mabs;            // bits of the largest |D| so far (above 0x7f7fffff: not finite)
    uint32_t *rec_x, *rec_y;   // logical indices joined at each step
    float *rec_dx, *rec_dy;
    int *err;                  // 2: no joinable pair; 4: an invalid pair; kManyRows
    uint32_t *left;            // kManyRows: nodes of the launch that gave up, and those it left
    uint32_t rows_allowed;     // rows per join and CTA beyond which the launch gives up (0: any number)
    unsigned long long *cycles;
    uint32_t N, P, c_end, step0;
    // nj_small_kernel only: the packed triangle (float, or int32 converted
    // exactly) when the launch is the first one, else null.
    const void *tri;
    int tri_int;
};

// Dynamic shared memory of nj_join_kernel with `own` row states per CTA.
__host__ __device__ __forceinline__ size_t join_smem(uint32_t P, uint32_t own)
{
    return (size_t) P * 16 + ((size_t) own + 1) / 2 * 2 * 22 + 16;
}

__device__ __forceinline__ float warp_fmax(float v)   // NaN loses
{
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float warp_fmin(float v)
{
    float r;
    asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

// A join as the next search records it: its division is off the way from one
// search to the next.
struct Joined {
    float sx, sy, dxy;   // row sums before the join's update (those of x and y are not updated)
    uint32_t x, y, c;
};

// raise_candidate (sequential.cpp:142-152).
__device__ __noinline__ void record_join(uint32_t *rec_x, uint32_t *rec_y, float *rec_dx, float *rec_dy, const Joined &j)
{
    const float pairsum = __fsub_rn(j.sx, j.sy);
    const float den = (float) (2u * (j.c - 2));
    const float q = __fdiv_rn(pairsum, den);
    float dx = __double2float_rn(__dadd_rn(__dmul_rn(0.5, (double) j.dxy), (double) q));
    float dy = __fsub_rn(j.dxy, dx);
    // The last join divides by 2(c-2) = 0; for 0/0 the reference's x86 SSE
    // arithmetic yields the default NaN 0xFFC00000 and propagates it into dx
    // and dy, where the GPU would give its canonical 0x7FFFFFFF.
    if(dx != dx) dx = __uint_as_float(0xFFC00000u);
    if(dy != dy) dy = __uint_as_float(0xFFC00000u);
    *rec_x = j.x;
    *rec_y = j.y;
    *rec_dx = dx;
    *rec_dy = dy;
}

// The serial fold of a new row sum over values V[i], i ascending, as a float
// chain: where every value is a float, a double add rounded to float is the
// float add (double has >= 2*24+2 significand bits). V is padded to a multiple
// of 4 with -0 (x + -0 = x).
__device__ __forceinline__ float fold_serial(const float *V, uint32_t lo, uint32_t hi, float s)
{
#pragma unroll 4
    for(uint32_t i = lo; i < hi; i += 4) {
        const float4 v = *reinterpret_cast<const float4 *>(V + i);
        s = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(s, v.x), v.y), v.z), v.w);
    }
    return s;
}

// The same out of line, where it is rare.
__device__ __noinline__ float fold_again(const float *V, uint32_t lo, uint32_t hi, float s) { return fold_serial(V, lo, hi, s); }

// The literal double chain over 0.5 W[i] (some value is not a float).
__device__ __noinline__ float fold_wide(const float *W, uint32_t n)
{
    float s = 0.0f;
#pragma unroll 1
    for(uint32_t i = 0; i < n; ++i) s = __double2float_rn(__dadd_rn((double) s, 0.5 * (double) W[i]));
    return s;
}

// fold_serial in kFoldParts parts at once. A part is run from four starting
// values, an estimate of the sum before it with its last two significand bits
// set to 0..3. From a start s that equals one of them but for a multiple of 4
// ulps, d, the chain takes the same path shifted by d, because every rounding
// on the way is the same: rounding to a multiple of an ulp u, ties to even,
// commutes with adding an even multiple of u, as long as shifted and unshifted
// values share a binade (no lower than the start's and at most one above, so
// that d is an even multiple of their ulp). Each run keeps how close to an
// edge of its binade it came; where d is not smaller, or another binade was
// met, the part is run again from s itself (one join in a hundred on matrices
// of protein scores). The parts are then chained by one shift each. Called by
// the folding warps, `ft` their thread number; thread 0 gets the sum.
__device__ __forceinline__ float fold_parts(const float *V, uint32_t n, float4 *fp, float *psum, int ft)
{
    const uint32_t g = (uint32_t) ft >> 2, r = (uint32_t) ft & 3u;
    const uint32_t len = ((n + kFoldParts - 1) / kFoldParts + 3) & ~3u, n4 = (n + 3) & ~3u;
    const uint32_t lo = min(g * len, n4), hi = min(lo + len, n4);
    float e = 0.0f;
#pragma unroll 4
    for(uint32_t i = lo + 4 * r; i < hi; i += 16) {
        const float4 v = *reinterpret_cast<const float4 *>(V + i);
        e += (v.x + v.y) + (v.z + v.w);
    }
    e += __shfl_xor_sync(kFull, e, 1);
    e += __shfl_xor_sync(kFull, e, 2);
    if(r == 0) psum[g] = e;
    asm volatile("barrier.sync 2, %0;" ::"n"(kFoldWarps * 32) : "memory");
    float before[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
    for(int k = 0; k < kFoldParts; k += 4) {
        const float4 v = *reinterpret_cast<const float4 *>(psum + k);
        before[0] += (uint32_t) k < g ? v.x : 0.0f;
        before[1] += (uint32_t) k + 1 < g ? v.y : 0.0f;
        before[2] += (uint32_t) k + 2 < g ? v.z : 0.0f;
        before[3] += (uint32_t) k + 3 < g ? v.w : 0.0f;
    }
    const uint32_t b0 = g == 0 ? 0u : (__float_as_uint((before[0] + before[1]) + (before[2] + before[3])) & ~3u) | r;
    float s = __uint_as_float(b0);
    // Over the run: smallest and largest bits (sign, exponent, significand),
    // and of the significand as a signed number centred in its binade.
    uint32_t bmin = b0, bmax = b0;
    int32_t cmin = (int32_t) ((b0 << 9) ^ 0x80000000u), cmax = cmin;
    auto add2 = [&](float v0, float v1) {
        s = __fadd_rn(s, v0);
        const uint32_t x0 = __float_as_uint(s);
        s = __fadd_rn(s, v1);
        const uint32_t x1 = __float_as_uint(s);
        const int32_t c0 = (int32_t) (x0 * 512u + 0x80000000u), c1 = (int32_t) (x1 * 512u + 0x80000000u);
        bmin = __vimin3_u32(bmin, x0, x1);
        bmax = __vimax3_u32(bmax, x0, x1);
        cmin = __vimin3_s32(cmin, c0, c1);
        cmax = __vimax3_s32(cmax, c0, c1);
    };
#pragma unroll 4
    for(uint32_t i = lo; i < hi; i += 4) {
        const float4 v = *reinterpret_cast<const float4 *>(V + i);
        add2(v.x, v.y);
        add2(v.z, v.w);
    }
    const uint32_t ex = b0 >> 23;   // sign and exponent
    // Ulps between the run and the nearest edge of a binade.
    const uint32_t edge = min((uint32_t) cmin + 0x80000000u, 0x7fffffffu - (uint32_t) cmax) >> 9;
    float margin = -1.0f;
    if((bmin >> 23) >= ex && (bmax >> 23) <= ex + 1 && (ex & 255u) > 24u && (ex & 255u) < 253u && edge > 1u)
        margin = (float) (edge - 1u) * __uint_as_float(((ex & 255u) - 23u) << 23);
    fp[ft] = make_float4(__uint_as_float(b0), s, margin, 0.0f);
    asm volatile("barrier.sync 2, %0;" ::"n"(kFoldWarps * 32) : "memory");
    float t = 0.0f;
    if(ft < 32) {
        bool ok = true;
#pragma unroll
        for(int k = 0; k < kFoldParts; ++k) {
            const float4 p = fp[4 * k + (k ? (__float_as_uint(t) & 3u) : 0u)];
            const float d = __fsub_rn(t, p.x);
            ok = ok && (d == 0.0f || fabsf(d) <= p.z);
            t = __fadd_rn(p.y, d);
        }
        if(!ok) {
            t = 0.0f;
#pragma unroll 1
            for(uint32_t k = 0; k < kFoldParts; ++k) {
                const float4 p = fp[4 * k + (k ? (__float_as_uint(t) & 3u) : 0u)];
                const float d = __fsub_rn(t, p.x);
                const uint32_t a = min(k * len, n4);
                t = d == 0.0f || fabsf(d) <= p.z ? __fadd_rn(p.y, d) : fold_again(V, a, min(a + len, n4), t);
            }
        }
    }
    return t;
}

// A candidate pair: its Q and D, the slots (logically larger << 16 | smaller)
// and the logical indices likewise, which order equal Q as the reference's
// row-major scan of the lower triangle does. q = -inf: none (the reference's
// strict `q > best`, best starting at -inf, takes neither -inf nor NaN).
struct alignas(16) Cand {
    float q, d;
    uint32_t slots, order;
};
__device__ __forceinline__ Cand no_cand() { return Cand{-INFINITY, 0.0f, 0u, 0xffffffffu}; }
__device__ __forceinline__ bool better(float q, uint32_t order, const Cand &c)
{
    return q > c.q || (q == c.q && q > -INFINITY && order < c.order);
}

// The lane holding the warp's best candidate (lane 0 when there is none).
__device__ __forceinline__ int best_lane(const Cand &c, int lane)
{
    const float m = warp_fmax(c.q);
    uint32_t who = __ballot_sync(kFull, c.q == m);
    if(__popc(who) > 1) {
        const bool in = (who >> lane) & 1u;
        const uint32_t first = __reduce_min_sync(kFull, in ? c.order : 0xffffffffu);
        who = __ballot_sync(kFull, in && c.order == first);
    }
    return who ? __ffs(who) - 1 : 0;
}
__device__ __forceinline__ Cand shfl_cand(const Cand &c, int src)
{
    return Cand{__shfl_sync(kFull, c.q, src), __shfl_sync(kFull, c.d, src), __shfl_sync(kFull, c.slots, src),
                __shfl_sync(kFull, c.order, src)};
}

// Of two pairs of one node, the reference's row-major scan meets the one with the
// smaller logical partner first: partners below the node are columns of its row,
// those above it are rows further down.
struct RowScan {
    float m1, m2, d1, dmin;   // best Q, best of the others, D of the best, smallest D
    uint32_t j1;
};

// Q of the pair (i, j): the row sum of the logically later node is subtracted
// first, as the reference does.
__device__ __forceinline__ float pair_q(float cm2, float d, float si, uint32_t pi, float sj, uint32_t pj)
{
    const bool later = pj > pi;
    return __fsub_rn(__fsub_rn(__fmul_rn(cm2, d), later ? sj : si), later ? si : sj);
}

// A row scanned by `wpr` warps of which this is number `sub`: the lane's two
// largest Q, the pair of the first and the smallest distance. The loop holds
// no branch; equal Q show as m2 == m1 (see merge_row).
__device__ __forceinline__ RowScan scan_row(const float *__restrict__ row, const float *S, const uint16_t *pos,
                                            uint32_t i, uint32_t P, float cm2, uint32_t sub, uint32_t wpr, int lane)
{
    RowScan r{-INFINITY, -INFINITY, 0.0f, 3.0e38f, kDead};
    const float si = S[i];
    const uint32_t pi = pos[i], nch = P >> 2, stride = 32 * wpr;
#pragma unroll 1
    for(uint32_t g0 = sub * 32 + lane; g0 < nch; g0 += kRowBatch * stride) {
        float4 d[kRowBatch];
#pragma unroll
        for(int u = 0; u < kRowBatch; ++u) {
            const uint32_t g = g0 + u * stride;
            if(g < nch) d[u] = __ldcg(reinterpret_cast<const float4 *>(row) + g);
        }
#pragma unroll
        for(int u = 0; u < kRowBatch; ++u) {
            const uint32_t g = g0 + u * stride;
            if(g >= nch) break;
            const float4 s4 = *reinterpret_cast<const float4 *>(S + 4 * g);
            const uint2 p4 = *reinterpret_cast<const uint2 *>(pos + 4 * g);
            const float dd[4] = {d[u].x, d[u].y, d[u].z, d[u].w}, ss[4] = {s4.x, s4.y, s4.z, s4.w};
            const uint32_t pp[4] = {p4.x & 0xffffu, p4.x >> 16, p4.y & 0xffffu, p4.y >> 16};
#pragma unroll
            for(int k = 0; k < 4; ++k) {
                // Slots without a live node, the new node's, padding, itself.
                const bool live = ss[k] != INFINITY && pp[k] != pi;
                const float q = live ? pair_q(cm2, dd[k], si, pi, ss[k], pp[k]) : -INFINITY;
                r.dmin = fminf(r.dmin, live ? dd[k] : 3.0e38f);
                const bool more = q > r.m1;
                r.m2 = fmaxf(r.m2, fminf(r.m1, q));
                r.m1 = fmaxf(r.m1, q);
                r.d1 = more ? dd[k] : r.d1;
                r.j1 = more ? 4 * g + k : r.j1;
            }
        }
    }
    return r;
}

// The lanes' scans of one row as one; every lane gets it.
__device__ __forceinline__ RowScan merge_scans(const RowScan &r, const uint16_t *pos, int lane)
{
    RowScan o;
    o.m1 = warp_fmax(r.m1);
    o.dmin = warp_fmin(r.dmin);
    uint32_t who = __ballot_sync(kFull, r.m1 == o.m1 && r.j1 != kDead);
    if(__popc(who) > 1) {   // equal Q: the first pair in the reference's order
        const bool in = (who >> lane) & 1u;
        const uint32_t pj = in ? pos[r.j1] : kDead;
        const uint32_t first = __reduce_min_sync(kFull, pj);
        who = __ballot_sync(kFull, pj == first);
    }
    const int src = who ? __ffs(who) - 1 : 0;
    o.m2 = warp_fmax(who && lane == src ? r.m2 : r.m1);
    o.d1 = __shfl_sync(kFull, r.d1, src);
    o.j1 = __shfl_sync(kFull, r.j1, src);
    if(who == 0u) o.j1 = kDead;
    return o;
}

// The same after a scan of the row: lanes with several cells of the row's largest Q
// go through their cells again, with the scan's loads, for the first of them (2,000
// nodes, a quarter of them copies of one: 17.6 ms with one load at a time, 10.6 so).
__device__ __noinline__ RowScan merge_row(RowScan r, const float *__restrict__ row, const float *S,
                                          const uint16_t *pos, uint32_t i, uint32_t P, float cm2, uint32_t sub,
                                          uint32_t wpr, int lane)
{
    const float top = warp_fmax(r.m1);
    if(r.m1 == r.m2 && r.m1 == top && r.j1 != kDead) {
        const float si = S[i];
        const uint32_t pi = pos[i], nch = P >> 2, stride = 32 * wpr;
        uint32_t first = pos[r.j1];
#pragma unroll 1
        for(uint32_t g0 = sub * 32 + lane; g0 < nch; g0 += kRowBatch * stride) {
            float4 d[kRowBatch];
#pragma unroll
            for(int u = 0; u < kRowBatch; ++u)
                if(g0 + u * stride < nch) d[u] = __ldcg(reinterpret_cast<const float4 *>(row) + g0 + u * stride);
#pragma unroll
            for(int u = 0; u < kRowBatch; ++u) {
                const uint32_t g = g0 + u * stride;
                if(g >= nch) break;
                const float4 s4 = *reinterpret_cast<const float4 *>(S + 4 * g);
                const uint2 p4 = *reinterpret_cast<const uint2 *>(pos + 4 * g);
                const float dd[4] = {d[u].x, d[u].y, d[u].z, d[u].w}, ss[4] = {s4.x, s4.y, s4.z, s4.w};
                const uint32_t pp[4] = {p4.x & 0xffffu, p4.x >> 16, p4.y & 0xffffu, p4.y >> 16};
#pragma unroll
                for(int k = 0; k < 4; ++k)
                    if(pp[k] < first && pp[k] != pi && ss[k] != INFINITY &&
                       pair_q(cm2, dd[k], si, pi, ss[k], pp[k]) == r.m1) {
                        first = pp[k];
                        r.j1 = 4 * g + k;
                        r.d1 = dd[k];
                    }
            }
        }
    }
    __syncwarp();
    return merge_scans(r, pos, lane);
}

template <bool Linear>
__global__ void __launch_bounds__(kJoinThreads, 1) nj_join_kernel(Stage st)
{
    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t K = cluster.num_blocks(), rank = cluster.block_rank();   // K is a power of two
    const uint32_t kbits = __ffs(K) - 1;
    const uint32_t N = st.N, P = st.P, own = (N + K) >> kbits;   // slots rank, rank + K, ... <= N
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float *S = reinterpret_cast<float *>(smem_raw);         // row sums by slot (+inf: not to be scanned)
    float *NDl = S + P;                                     // new distances by logical index
    float *Wl = NDl + P;                                    // twice their value before rounding
    uint16_t *pos = reinterpret_cast<uint16_t *>(Wl + P), *l2s = pos + P;
    float *ND = reinterpret_cast<float *>(l2s + P);         // new distances of the own rows
    float *Zb = ND + own;                                   // bound of the row's other pairs (see `bound`)
    float *Dm = Zb + own;                                   // smallest D among them
    float *db = Dm + own;                                   // D of the best pair
    uint16_t *jb = reinterpret_cast<uint16_t *>(db + own);  // its partner's slot
    uint16_t *tau = jb + own;                               // join at which the bound was taken
    uint16_t *list = tau + own;                             // rows to scan

    __shared__ Cand parts[2][kMaxCluster];                  // every CTA's candidate
    __shared__ Cand wcand[kJoinWarps];                      // every warp's
    __shared__ RowScan wscan[kScanWarps];
    __shared__ float4 fparts[kFoldParts * 4];
    __shared__ __align__(16) float fsum[kFoldParts];
    __shared__ float wA[kJoinWarps];
    __shared__ uint32_t wV[kJoinWarps];
    __shared__ float sz_sh;
    __shared__ Joined joined;
    __shared__ uint32_t nlist;
    __shared__ int excess;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if(*st.err != 0) return;   // an earlier launch failed (the same for every CTA)
    float *D = st.D;

    auto record = [&](uint32_t k) {
        const uint32_t at = st.step0 + k;
        record_join(st.rec_x + at, st.rec_y + at, st.rec_dx + at, st.rec_dy + at, joined);
    };
    auto scan_sync = [] { asm volatile("barrier.sync 1, %0;" ::"n"(kScanWarps * 32) : "memory"); };
    // Size of values that Q is made of, as float bits (a NaN is the largest):
    // N |D| and 2 |S|; bit 0 marks a new distance that is not a float.
    const float fN = (float) N;
    auto size_of = [&](float d, float s) {
        return max(__float_as_uint(fN * fabsf(d)), __float_as_uint(2.0f * fabsf(s))) & ~1u;
    };

    if(tid < kJoinWarps) wcand[tid] = no_cand();
    if(tid < 2 * (int) kMaxCluster) parts[tid / kMaxCluster][tid % kMaxCluster] = no_cand();
    if(tid == 0) {
        nlist = 0;
        excess = 0;
        sz_sh = 0.0f;
    }
    uint32_t sv = size_of(__uint_as_float(*st.mabs), 0.0f);
    for(uint32_t k = tid; k < P; k += kJoinThreads) {
        const float s = k < N ? st.S0[k] : INFINITY;
        S[k] = s;
        pos[k] = (uint16_t) (k < N ? k : kDead);
        l2s[k] = (uint16_t) k;
        if(k < N) sv = max(sv, size_of(0.0f, s));
    }
    for(uint32_t l = tid; l < own; l += kJoinThreads) {
        Zb[l] = INFINITY;
        Dm[l] = 0.0f;
        db[l] = 0.0f;
        jb[l] = (uint16_t) kDead;
        tau[l] = 0;
    }
    sv = __reduce_max_sync(kFull, sv);
    if(lane == 0) wV[warp] = sv;
    __syncthreads();
    sv = __reduce_max_sync(kFull, lane < kJoinWarps ? wV[lane] : 0u);
    cluster.sync();   // every CTA runs before any exchange

    uint32_t c = N, t = 0, step = 0, spare = N, z = kDead;
    float C = 0.0f;                // falls of row sums, added up
    bool exact = true, failed = false, bad = false;
    // Phase counters of one thread of CTA 0 (and of thread 0 for the fold).
    const bool timer = rank == 0 && tid == 32 * kFoldWarps;
    uint32_t t_last = (uint32_t) clock64();
    unsigned long long cyc_scan = 0, cyc_wait = 0, cyc_join = 0, cyc_fold_wait = 0, cyc_new = 0, cyc_fold = 0;
    auto mark = [&](unsigned long long &to) {
        if(timer) {
            const uint32_t now = (uint32_t) clock64();
            to += now - t_last;
            t_last = now;
        }
    };
    while(c > st.c_end) {
        const float cm2 = (float) (c - 2), size = __uint_as_float(sv);
        const bool prune = size < 1e30f;
        const float slack = __fadd_ru(__fmul_ru(size, 1.0f / (1 << 19)), 1e-37f);
        // Q of the live nodes at distance d with logical indices pi and pj, and its key.
        auto q_of = [&](uint32_t pi, float si, uint32_t pj, float sj, float d) { return pair_q(cm2, d, si, pi, sj, pj); };
        auto order_of = [&](uint32_t pi, uint32_t pj) { return (max(pi, pj) - t) << 16 | (min(pi, pj) - t); };
        // The bound of own row l (row sum si), and what to store for a bound b taken now.
        auto bound = [&](uint32_t l, float si) {
            return __fadd_ru(__fsub_ru(Zb[l], si), __fsub_ru(C, __fmul_rd((float) (step - tau[l]), Dm[l])));
        };
        auto stored = [&](float b, float si) { return __fsub_ru(__fadd_ru(b, si), C); };

        // ---- search
        if(warp < kFoldWarps) {
            if(z != kDead) {
                const uint32_t f0 = (uint32_t) clock64();
                // Its row sum over the c + 1 values of its join.
                const float ns = exact ? fold_parts(NDl, c + 1, fparts, fsum, tid) : fold_wide(Wl, c + 1);
                if(tid == 0) {
                    sz_sh = ns;
                    cyc_fold += (uint32_t) clock64() - f0;
                }
            }
        } else {
            const uint32_t w = (uint32_t) warp - kFoldWarps, sid = (uint32_t) tid - 32 * kFoldWarps;
            if(rank == 0 && step > 0 && tid == kJoinThreads - 1) record(step - 1);
            // A Q that some live pair attains, from what is left of the last
            // search: this CTA's candidates by warp and every CTA's.
            float L = -INFINITY;
            {
                const Cand v = lane < 16 ? wcand[lane] : parts[(step - 1) & 1u][lane - 16];
                const uint32_t i = v.slots >> 16 & 0x7fffu, j = v.slots & 0xffffu;
                if(v.q > -INFINITY && i != z && j != z) {
                    const uint32_t pi = pos[i], pj = pos[j];
                    if(pi != kDead && pj != kDead) L = q_of(pi, S[i], pj, S[j], v.d);
                }
                L = warp_fmax(L);
            }
#pragma unroll 1
            for(uint32_t l = sid; l < own; l += kScanWarps * 32) {
                const uint32_t i = l * K + rank;
                if(i > N || pos[i] == kDead || i == z) continue;
                const uint32_t j = jb[l];
                if(j != kDead && pos[j] == kDead) jb[l] = (uint16_t) kDead;   // joined away
                if(!prune || !(__fadd_ru(bound(l, S[i]), slack) < L)) list[atomicAdd(&nlist, 1u)] = (uint16_t) l;
            }
            scan_sync();
            const uint32_t m = nlist;
            // A row's new state, by lane 0 of the warp that holds its scan.
            auto renew = [&](uint32_t l, const RowScan &r) {
                if(lane != 0) return;
                jb[l] = (uint16_t) r.j1;
                db[l] = r.d1;
                Dm[l] = r.dmin;
                tau[l] = (uint16_t) step;
                Zb[l] = stored(__fadd_ru(r.m2, slack), S[l * K + rank]);
            };
            // Warps per row, a power of two: as many as there are for m rows,
            // down to one load a lane each.
            const uint32_t lg = min(m <= 1 ? 3u : m <= 3 ? 2u : m <= 7 ? 1u : 0u, P > 512 ? 3u : P > 256 ? 2u : 1u);
            const uint32_t wpr = 1u << lg, rows = kScanWarps >> lg;   // rows scanned at once
#pragma unroll 1
            for(uint32_t k = w >> lg; k < m; k += rows) {   // once where warps share a row: m <= rows
                const uint32_t l = list[k], i = l * K + rank;
                const float *row = D + (size_t) i * P;
                const RowScan o = merge_row(scan_row(row, S, pos, i, P, cm2, w & (wpr - 1), wpr, lane), row, S, pos, i,
                                            P, cm2, w & (wpr - 1), wpr, lane);
                if(wpr > 1) {
                    if(lane == 0) wscan[w] = o;
                } else {
                    renew(l, o);
                }
            }
            if(wpr > 1) {
                scan_sync();
                if(w < m) {
                    const uint32_t l = list[w];
                    RowScan r{-INFINITY, -INFINITY, 0.0f, 3.0e38f, kDead};
                    if((uint32_t) lane < wpr) r = wscan[(w << lg) + lane];
                    renew(l, merge_scans(r, pos, lane));
                }
            }
            mark(cyc_scan);
        }
        __syncthreads();
        mark(cyc_fold_wait);
        // Each row takes in its pair with the new node z; the CTA's best pair.
        {
            const float sz = sz_sh;
            const uint32_t pz = z != kDead ? pos[z] : kDead;
            if(tid == 0) {
                if(z != kDead) S[z] = sz;   // read again only after the next barrier
                // Rows read beyond the allowance of each join (the first one reads all).
                if(step > 0) excess = max(excess + (int) nlist - (int) st.rows_allowed, 0);
                nlist = 0;
            }
            Cand best = no_cand();
#pragma unroll 1
            for(uint32_t l = tid; l < own; l += kJoinThreads) {
                const uint32_t i = l * K + rank, pi = i <= N ? pos[i] : kDead;
                if(pi == kDead || i == z) continue;
                const float si = S[i];
                uint32_t j = jb[l], pj = kDead;
                float d = db[l], q = -INFINITY;
                if(j != kDead) {
                    pj = pos[j];
                    q = q_of(pi, si, pj, S[j], d);
                }
                if(z != kDead) {
                    const float dz = ND[l], qz = q_of(pi, si, pz, sz, dz);
                    const bool take = qz > q || (qz == q && pz < pj);
                    const float B = bound(l, si), other = __fadd_ru(take ? q : qz, slack);
                    if(other > B || dz < Dm[l]) {
                        Dm[l] = fminf(Dm[l], dz);
                        tau[l] = (uint16_t) step;
                        Zb[l] = stored(fmaxf(B, other), si);
                    }
                    if(take) {
                        q = qz;
                        d = dz;
                        j = z;
                        pj = pz;
                        jb[l] = (uint16_t) z;
                        db[l] = dz;
                    }
                }
                const uint32_t order = order_of(pi, pj);
                if(better(q, order, best)) best = Cand{q, d, pi > pj ? i << 16 | j : j << 16 | i, order};
            }
            if(lane == best_lane(best, lane)) wcand[warp] = best;
        }
        __syncthreads();
        const uint32_t buf = step & 1u;
        if(warp == 0) {
            const Cand v = lane < kJoinWarps ? wcand[lane] : no_cand();
            Cand o = shfl_cand(v, best_lane(v, lane));
            if(st.rows_allowed != 0 && excess > kExcessJoins * (int) st.rows_allowed) o.slots |= kGiveUp;
            if((uint32_t) lane < K) *cluster.map_shared_rank(&parts[buf][rank], (unsigned) lane) = o;
        }
        mark(cyc_new);
        cluster_arrive();   // A
        cluster_wait();
        mark(cyc_wait);

        // ---- join
        Cand win = (uint32_t) lane < K ? parts[buf][lane] : no_cand();
        const bool give_up = __any_sync(kFull, (win.slots & kGiveUp) != 0u);
        win = shfl_cand(win, best_lane(win, lane));
        win.slots &= ~kGiveUp;
        if(win.q == -INFINITY) {   // no selectable Q (all NaN): the reference would index an undefined pair
            failed = true;
            break;
        }
        const uint32_t x = win.order >> 16, y = win.order & 0xffffu, X = win.slots >> 16, Y = win.slots & 0xffffu;
        if(x >= c || y >= x || X > N || Y > N) {   // never a pair of this join: report it, touch nothing
            bad = true;
            break;
        }
        const float dxy = win.d;
        const uint32_t znew = spare;
        // The new node takes x's number; then logical 0 (symmetric: all numbers
        // shift down by one) or the last one (linear), ps, takes y's.
        const uint32_t px = x + t, py = y + t, ps = Linear ? c - 1 : t;
        const float *rx = D + (size_t) X * P, *ry = D + (size_t) Y * P;
        float fall = -INFINITY;
        bool ex = true;
        uint32_t moved = kDead;
        if((uint32_t) tid < ((4u - (c & 3u)) & 3u)) NDl[c + tid] = -0.0f;
        // join_pair (sequential.cpp:247-267) for every live slot; X and Y read
        // the diagonal and D[x][y], as the reference does.
        constexpr int U = 4;
#pragma unroll 1
        for(uint32_t s0 = tid; s0 <= N; s0 += U * kJoinThreads) {
            float a[U], b[U];
            uint32_t p[U];
#pragma unroll
            for(int u = 0; u < U; ++u) {
                const uint32_t s = s0 + u * kJoinThreads;
                p[u] = s <= N && s != znew ? pos[s] : kDead;
                if(p[u] != kDead) {
                    a[u] = __ldcg(rx + s);
                    b[u] = __ldcg(ry + s);
                }
            }
#pragma unroll
            for(int u = 0; u < U; ++u) {
                const uint32_t s = s0 + u * kJoinThreads;
                if(p[u] == kDead) continue;
                const float prev = __fadd_rn(a[u], b[u]);
                const float w = __fsub_rn(prev, dxy);
                const float nd = __fmul_rn(w, 0.5f);   // the double 0.5 w, rounded
                ex = ex && __fadd_rn(nd, nd) == w;
                Wl[p[u] - t] = w;
                NDl[p[u] - t] = nd;
                if((s & (K - 1)) == rank) ND[s >> kbits] = nd;
                if(p[u] == ps) moved = s;
                if(s == X || s == Y) continue;   // their numbers and sums below
                const float s_old = S[s];
                const double uu = __dmul_rn((double) w, 0.5);
                const float sn = __double2float_rn(__dadd_rn((double) s_old, __dsub_rn(uu, (double) prev)));
                S[s] = sn;
                fall = fmaxf(fall, __fsub_ru(s_old, sn));
                sv = max(sv, size_of(nd, sn));
                if(((s >> 5) & (K - 1)) == rank) {
                    D[(size_t) znew * P + s] = nd;
                    D[(size_t) s * P + znew] = nd;
                }
            }
        }
        // The node that changes its number: its thread alone reads pos here.
        if(moved != kDead && moved != X && moved != Y) {
            pos[moved] = (uint16_t) py;
            l2s[py] = (uint16_t) moved;
        }
        if((uint32_t) tid == (Y & (kJoinThreads - 1))) {
            if(rank == 0) joined = Joined{S[X], S[Y], dxy, x, y, c};
            S[X] = INFINITY;
            S[Y] = INFINITY;
            pos[Y] = (uint16_t) kDead;
        }
        if((uint32_t) tid == (X & (kJoinThreads - 1))) {
            const uint32_t pz = px == ps ? py : px;
            pos[X] = (uint16_t) kDead;
            pos[znew] = (uint16_t) pz;
            l2s[pz] = (uint16_t) znew;
            S[znew] = INFINITY;   // until its row sum is folded and its column is written
            // Its diagonal, as the join gives it for x.
            if(rank == 0) D[(size_t) znew * P + znew] = NDl[px - t];
            if((znew & (K - 1)) == rank) {
                // Nothing is covered by the new node's own row yet.
                const uint32_t l = znew >> kbits;
                Zb[l] = -INFINITY;
                Dm[l] = 3.0e38f;
                jb[l] = (uint16_t) kDead;
                tau[l] = (uint16_t) (step + 1);
            }
        }
        fall = warp_fmax(fall);
        const uint32_t wv = __reduce_max_sync(kFull, sv) | (__any_sync(kFull, !ex) ? 1u : 0u);
        if(lane == 0) {
            wA[warp] = fall;
            wV[warp] = wv;
        }
        __syncthreads();
        fall = warp_fmax(lane < kJoinWarps ? wA[lane] : -INFINITY);
        if(fall > -INFINITY) C = __fadd_ru(C, fall);
        sv = __reduce_max_sync(kFull, lane < kJoinWarps ? wV[lane] : 0u);
        exact = __all_sync(kFull, lane >= kJoinWarps || !(wV[lane] & 1u));
        sv &= ~1u;
        spare = X;
        z = znew;
        if(!Linear) ++t;
        ++step;
        --c;
        mark(cyc_join);
        if(give_up) break;
    }
    if(rank == 0 && tid == 0) {
        if(failed) atomicExch(st.err, 2);
        if(bad) atomicExch(st.err, 4);
        if(!failed && !bad && c > st.c_end) {
            st.left[0] = N;
            st.left[1] = c;
            atomicExch(st.err, kManyRows);
        }
    }
    if(rank == 0) {
        if(!failed && !bad) {
            if(tid == kJoinThreads - 1) record(step - 1);
            // What the next launch starts from.
            if(warp == 0) {
                const float ns = exact ? fold_again(NDl, 0, (c + 4) & ~3u, 0.0f) : fold_wide(Wl, c + 1);
                if(lane == 0) S[z] = ns;
            }
            __syncthreads();
            for(uint32_t k = tid; k < c; k += kJoinThreads) {
                const uint32_t s = l2s[t + k];
                st.order_out[k] = s;
                st.S_out[k] = S[s];
            }
            // An upper bound on |D| is enough for the next launch's slack.
            if(tid == 0) *st.mabs = __float_as_uint(__uint_as_float(sv) / fN * 1.0001f);
        }
        __syncthreads();
        if(timer) {
            atomicAdd(st.cycles + 0, cyc_scan);
            atomicAdd(st.cycles + 1, cyc_wait);
            atomicAdd(st.cycles + 2, cyc_join);
            atomicAdd(st.cycles + 6, cyc_new);
            atomicAdd(st.cycles + 7, cyc_fold_wait);
        }
        if(tid == 0) atomicAdd(st.cycles + 5, cyc_fold);
    }
    cluster.sync();   // no CTA leaves while another may still write its shared memory
}

// ---------------------------------------------------------------- one CTA

// Matrices of up to this many nodes live in one CTA's shared memory.
constexpr uint32_t kSmallNodes = 230;
// Columns of a row that a lane goes through: 32 k + lane, k < kSmallCols.
constexpr int kSmallCols = (kSmallNodes + 31) / 32;

__host__ __device__ __forceinline__ size_t small_smem(uint32_t N, uint32_t P)
{
    // Rows past the last one are read (and ignored) up to 32 kSmallCols cells.
    return ((size_t) N * P + 32 * kSmallCols) * 4 + (size_t) P * 16 + 32 * kSmallCols * 4;
}

// All joins from N <= kSmallNodes nodes on. The live nodes' slots are their
// logical indices plus t (0 in the linear order; the joins so far in the
// symmetric one, which drops logical 0), so the data of the node that the
// reference moves is moved here too. Per join: warps 1.. search every pair but
// the new node's (its row sum is +inf until then) in row-major order, which
// needs no rule for equal Q within a lane, while warp 0 folds that row sum;
// then every thread adds its pair with the new node, and the block's best pair
// is joined, one slot per thread.
template <bool Linear, int kThreads>
__global__ void __launch_bounds__(kThreads, 1) nj_small_kernel(Stage st)
{
    constexpr int kWarps = kThreads / 32;
    const uint32_t N = st.N, P = st.P;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float *D = reinterpret_cast<float *>(smem_raw);
    float *NDl = D + (size_t) N * P + 32 * kSmallCols;   // new distances by logical index
    float *Wl = NDl + P;                                 // twice their value before rounding
    float *dg = Wl + P;                                  // the diagonal (0 unless a distance is not finite)
    float *S = dg + P;                                   // row sums (+inf: not to be searched)
    __shared__ Cand wcand[kWarps];
    __shared__ float sz_sh;
    __shared__ Joined joined;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if(*st.err != 0) return;

    if(st.tri) {
        // A warp per row of the triangle.
#pragma unroll 1
        for(uint32_t i = 1 + warp; i < N; i += kWarps) {
            const uint32_t at = i * (i - 1) / 2;
#pragma unroll 2
            for(uint32_t j = lane; j < i; j += 32) {
                const float v = st.tri_int ? (float) static_cast<const int32_t *>(st.tri)[at + j]
                                           : static_cast<const float *>(st.tri)[at + j];
                D[i * P + j] = v;
                D[j * P + i] = v;
            }
        }
        for(uint32_t k = tid; k < N; k += kThreads) D[k * P + k] = dg[k] = 0.0f;
        __syncthreads();
        // cache_init (sequential.cpp:80-94): ascending over j != k, from 0.
        for(uint32_t k = tid; k < N; k += kThreads) {
            float s = 0.0f;
#pragma unroll 8
            for(uint32_t j = 0; j < N; ++j)
                if(j != k) s = __fadd_rn(s, D[j * P + k]);
            S[k] = s;
        }
    } else {
        const float4 *src = reinterpret_cast<const float4 *>(st.D);
        for(uint32_t k = tid; k < N * P / 4; k += kThreads) reinterpret_cast<float4 *>(D)[k] = src[k];
        __syncthreads();
        for(uint32_t k = tid; k < N; k += kThreads) {
            dg[k] = D[k * P + k];
            S[k] = st.S0[k];
        }
    }
    for(uint32_t k = N + tid; k < P + 32 * kSmallCols; k += kThreads) S[k] = INFINITY;
    __syncthreads();

    auto record = [&](uint32_t k) {
        const uint32_t at = st.step0 + k;
        record_join(st.rec_x + at, st.rec_y + at, st.rec_dx + at, st.rec_dy + at, joined);
    };
    uint32_t c = N, t = 0, step = 0, z = kDead;
    bool exact = true;
    unsigned long long scan_cyc = 0, fold_cyc = 0, rest_cyc = 0, t_last = clock64();
    while(c > 1) {
        const float cm2 = (float) (c - 2);
        Cand best = no_cand();
        if(warp == 0) {
            if(z != kDead) {
                const float ns = exact ? fold_serial(NDl, 0, (c + 4) & ~3u, 0.0f) : fold_wide(Wl, c + 1);
                if(lane == 0) sz_sh = ns;
                fold_cyc += clock64() - t_last;
            }
        } else {
            if(tid == kThreads - 1 && step > 0) record(step - 1);
            float sb[kSmallCols];
#pragma unroll
            for(int k = 0; k < kSmallCols; ++k) sb[k] = S[t + 32 * k + lane];
            float bq = -INFINITY;
            uint32_t bij = 0;
#pragma unroll 1
            for(uint32_t a = warp; a < c; a += kWarps - 1) {
                const float sa = S[t + a];
                const float *row = D + (t + a) * P + t + lane;
#pragma unroll
                for(int k = 0; k < kSmallCols; ++k) {
                    if(32 * k >= a) break;
                    float q = __fsub_rn(__fsub_rn(__fmul_rn(cm2, row[32 * k]), sa), sb[k]);
                    if(32 * k + 32 > a) q = 32 * k + lane < a ? q : -INFINITY;
                    const bool more = q > bq;
                    bij = more ? (a << 16) + 32 * k : bij;
                    bq = fmaxf(bq, q);
                }
            }
            if(bq > -INFINITY) {
                bij += lane;
                best = Cand{bq, D[(t + (bij >> 16)) * P + t + (bij & 0xffffu)], bij, bij};
            }
        }
        if(tid == 32) {
            const unsigned long long now = clock64();
            scan_cyc += now - t_last;
            t_last = now;
        }
        __syncthreads();
        const uint32_t s = tid, o = t + s;   // logical index and slot of this thread
        float ss = INFINITY;
        if(32u * warp < c) {
            if(s < c) ss = S[o];
            if(z != kDead) {
                const float sz = sz_sh;
                if(s == z) ss = sz;
                else if(s < c) {
                    const float d = D[(t + z) * P + o];
                    const float q = pair_q(cm2, d, ss, s, sz, z);
                    const uint32_t order = s > z ? s << 16 | z : z << 16 | s;
                    if(better(q, order, best)) best = Cand{q, d, order, order};
                }
            }
        }
        if(lane == best_lane(best, lane)) wcand[warp] = best;
        __syncthreads();
        Cand win = lane < kWarps ? wcand[lane] : no_cand();
        win = shfl_cand(win, best_lane(win, lane));
        const uint32_t x = win.order >> 16, y = win.order & 0xffffu;
        const bool none = win.q == -INFINITY;
        if(none || x >= c || y >= x) {
            if(tid == 0) atomicExch(st.err, none ? 2 : 4);
            break;
        }
        const float dxy = win.d;
        // src is moved into y (nothing to move when it is y itself); in the
        // linear order, when x is the last, the new node goes to y instead.
        const uint32_t src = Linear ? c - 1 : 0u, A = Linear && x == src ? y : x;
        const bool move = src != x && src != y;
        // join_pair (sequential.cpp:247-267), one node per thread; x and y read
        // the diagonal and D[x][y], as the reference does.
        float prev = 0.0f, w = 0.0f, nd = 0.0f, ve = 0.0f;
        bool ex = true;
        if(s < c) {
            const float a = s == y ? dxy : s == x ? dg[o] : D[(t + x) * P + o];
            const float b = s == x ? dxy : s == y ? dg[o] : D[(t + y) * P + o];
            ve = s == src ? dg[o] : D[(t + src) * P + o];
            prev = __fadd_rn(a, b);
            w = __fsub_rn(prev, dxy);
            nd = __fmul_rn(w, 0.5f);   // the double 0.5 w, rounded
            ex = __fadd_rn(nd, nd) == w;
            Wl[s] = w;
            NDl[s] = nd;
            // The last new node's row sum may not be in S yet.
            if(s == x) joined = Joined{ss, y == z ? sz_sh : S[t + y], dxy, x, y, c};
        } else if(s < ((c + 3) & ~3u)) {
            NDl[s] = -0.0f;
        }
        exact = __syncthreads_and(ex) != 0;
        if(s < c) {
            if(s == x) {
                S[t + A] = INFINITY;   // until its row sum is folded
                dg[t + A] = nd;
            } else if(s != y) {
                const uint32_t to = t + (move && s == src ? y : s);
                const double uu = __dmul_rn((double) w, 0.5);
                S[to] = __double2float_rn(__dadd_rn((double) ss, __dsub_rn(uu, (double) prev)));
                D[(t + A) * P + to] = nd;
                D[to * P + t + A] = nd;
                if(move) {
                    if(s == src) {
                        dg[to] = ve;
                    } else {
                        D[(t + y) * P + o] = ve;
                        D[o * P + t + y] = ve;
                    }
                }
            }
        }
        // Numbers shift down by one in the symmetric order; the linear order's
        // dropped slot leaves the search (as do cells past a row's end).
        if(Linear && tid == 0) S[c - 1] = INFINITY;
        z = Linear ? A : x - 1;
        if(!Linear) ++t;
        ++step;
        --c;
        __syncthreads();
        if(tid == 32) {
            const unsigned long long now = clock64();
            rest_cyc += now - t_last;
            t_last = now;
        }
        if(warp == 0) t_last = clock64();
    }
    if(c == 1 && tid == kThreads - 1) record(step - 1);
    if(tid == 32) {
        atomicAdd(st.cycles + 0, scan_cyc);
        atomicAdd(st.cycles + 2, rest_cyc);
    }
    if(tid == 0) atomicAdd(st.cycles + 5, fold_cyc);
}

// Packed triangle (float or int32) -> full symmetric matrix of n + 1 rows of
// pitch P, diagonal, row n and padding 0. One block per 32 x 32 tile at or
// below the diagonal: the tile is written as read and, through shared memory,
// transposed, both coalesced. mabs receives the bits of the largest |value|.
template <class T>
__global__ void __launch_bounds__(256) inflate_kernel(const T *__restrict__ tri, float *__restrict__ D, uint32_t n,
                                                      uint32_t P, uint32_t *mabs)
{
    __shared__ float tile[32][33];
    const uint32_t bi = blockIdx.y, bj = blockIdx.x;
    if(bj > bi) return;
    const uint32_t tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    uint32_t mx = 0;
    for(uint32_t r = ty; r < 32; r += 8) {
        const uint32_t i = bi * 32 + r, j = bj * 32 + tx;
        const float v = (i < n && j < i) ? (float) tri[(uint64_t) i * (i - 1) / 2 + j] : 0.0f;
        tile[r][tx] = v;
        mx = max(mx, __float_as_uint(v) & 0x7fffffffu);
    }
    __syncthreads();
    for(uint32_t r = ty; r < 32; r += 8) {
        const uint32_t i = bi * 32 + r, j = bj * 32 + tx;
        if(i <= n && j < P) D[(size_t) i * P + j] = bi == bj && tx > r ? tile[tx][r] : tile[r][tx];
        const uint32_t it = bj * 32 + r, jt = bi * 32 + tx;   // the transposed tile
        if(bi != bj && it <= n && jt < P) D[(size_t) it * P + jt] = tile[tx][r];
    }
    mx = __reduce_max_sync(kFull, mx);
    if(tx == 0 && mx != 0u) atomicMax(mabs, mx);
}

// cache_init (sequential.cpp:80-94): S[k] folds D[k][j] over j != k ascending,
// from 0. Thread k reads column k (= row k by symmetry), so a warp's reads
// coalesce; each sum is a serial chain, so the loads of a batch are issued
// before its additions, and one-warp blocks spread the rows over the SMs.
__global__ void __launch_bounds__(32) row_sums_kernel(const float *__restrict__ D, float *__restrict__ S, uint32_t n,
                                                      uint32_t P)
{
    const uint32_t k = blockIdx.x * 32 + threadIdx.x;
    if(k >= n) return;
    constexpr int B = 32;
    float s = 0.0f, v[B];
    for(uint32_t j0 = 0; j0 < n; j0 += B) {
#pragma unroll
        for(int u = 0; u < B; ++u) v[u] = j0 + u < n ? __ldcg(D + (size_t) (j0 + u) * P + k) : 0.0f;
#pragma unroll
        for(int u = 0; u < B; ++u)
            if(j0 + u < n && j0 + u != k) s = __fadd_rn(s, v[u]);
    }
    S[k] = s;
}

// The live nodes of a finished launch in logical order: the next launch's matrix.
__global__ void compact_kernel(const float *__restrict__ D, uint32_t P, const uint32_t *__restrict__ order,
                               float *__restrict__ D2, uint32_t n2, uint32_t P2, const int *err)
{
    if(*err != 0) return;
    for(uint32_t r = blockIdx.x; r <= n2; r += gridDim.x) {
        const float *src = r < n2 ? D + (size_t) order[r] * P : nullptr;
        for(uint32_t k = threadIdx.x; k < P2; k += blockDim.x)
            D2[(size_t) r * P2 + k] = (r < n2 && k < n2) ? __ldg(src + order[k]) : 0.0f;
    }
}

}  // namespace njdev
}  // namespace msa
