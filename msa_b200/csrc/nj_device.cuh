// Device pieces shared by the neighbor-joining kernels: candidate keys, warp
// maxima and cluster barriers.
#pragma once

#include <cmath>
#include <cstdint>

#include <cooperative_groups.h>

namespace msa {
namespace njdev {

namespace cg = cooperative_groups;

constexpr unsigned kFull = 0xffffffffu;
constexpr unsigned kMaxCluster = 16;
constexpr uint32_t kNone = 0xffffffffu;
// Phase counters of a run (msa_nj_stats).
constexpr int kCycleSlots = 8;

// Orderable key of a finite or +inf Q value; 0 for NaN and -inf, which the
// reference's strict `q > best` (best starting at -inf) never selects.
// -0 and +0 compare equal there, so both map to the +0 key.
__device__ __forceinline__ uint32_t order_key(float q)
{
    if(q != q || q == -INFINITY) return 0u;
    uint32_t b = __float_as_uint(q);
    if(b == 0x80000000u) b = 0u;
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

// A candidate pair (i, j), j < i, as one 64-bit key: larger Q wins; on equal
// Q the pair earlier in the reference's row-major scan of the lower triangle
// (smaller i, then smaller j) wins, which is the order of i << 16 | j (i, j <
// 2^16). 0 means "no candidate"; the low word names the pair.
__device__ __forceinline__ unsigned long long pack(uint32_t key, uint32_t i, uint32_t j)
{
    return key ? (((unsigned long long) key << 32) | (0xffffffffu - ((i << 16) | j))) : 0ull;
}
__device__ __forceinline__ uint32_t pair_of(unsigned long long v) { return 0xffffffffu - (uint32_t) v; }

__device__ __forceinline__ unsigned long long umax64(unsigned long long a, unsigned long long b) { return a > b ? a : b; }

// The warp's maximum of a 64-bit key in two 32-bit warp reductions: the
// largest high word, then the largest low word among the lanes holding it.
__device__ __forceinline__ unsigned long long warp_max(unsigned long long v)
{
    const uint32_t hi = (uint32_t) (v >> 32), lo = (uint32_t) v;
    const uint32_t mhi = __reduce_max_sync(kFull, hi);
    const uint32_t mlo = __reduce_max_sync(kFull, hi == mhi ? lo : 0u);
    return ((unsigned long long) mhi << 32) | mlo;
}

// Two floats in one 64-bit register and the packed operations of sm_100 on them:
// each half is rounded to nearest as the scalar operation (no flush to zero), so
// `sub2(sub2(fma2(a, b, nz), c), d)` gives per half the bits of
// __fsub_rn(__fsub_rn(__fmul_rn(a, b), c), d) with half the issues. The product is
// a fused operation with the addend -0, which changes no product, handed to the
// kernel as an argument: mul.rn.f32x2 followed by sub.rn.f32x2 is compiled into one
// fused operation (nine in ten of random operands gave its bits on the device), and
// a constant -0 would let the compiler see the product.
__device__ __forceinline__ unsigned long long f2(float a, float b)
{
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void f2_split(unsigned long long v, float &a, float &b)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c)
{
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ unsigned long long sub2(unsigned long long a, unsigned long long b)
{
    unsigned long long r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

}  // namespace njdev
}  // namespace msa
