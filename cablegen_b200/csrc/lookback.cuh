// lookback.cuh -- decoupled look-back over one count per tile, shared by the
// compacting kernels (unique, merge, bucket sort).
#pragma once
#include "common.cuh"

namespace cgb {

__device__ __forceinline__ u64 ld_relaxed64(const u64 *p)
{
    u64 v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed64(u64 *p, u64 v)
{
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Polls of a look-back wait, and the test switch that keeps the first tile from
// publishing its count (options "lookback_spin_limit", "lookback_hold_first_tile")
struct LookbackLimit {
    u32 polls = SPIN_LIMIT;
    u32 hold = 0;
};
extern LookbackLimit g_lookback;

// Warp-wide form of the walk back over one count per tile, called by all 32
// lanes of one warp: lane i reads the word of tile j - i, so one round trip
// covers 32 predecessors.  The words from tile j down to the nearest inclusive
// prefix (or down to the first one not yet published, which is polled again)
// are summed with a warp reduction.  Every lane returns the same prefix.  A
// wait gives up after `limit` polls (ERR_LOOKBACK_TIMEOUT in *err).
template <typename W>
__device__ __forceinline__ W warp_lookback_sum(const W *words, int j, u32 *err, u32 limit)
{
    constexpr W PRE = (W)2 << (8 * sizeof(W) - 2);
    constexpr W MASK = ((W)1 << (8 * sizeof(W) - 2)) - 1;
    const int lane = threadIdx.x & 31;
    W excl = 0;
    u32 spins = 0;
    while (j >= 0) {
        const int k = j - lane;
        W v;
        if (k >= 0) {
            if constexpr (sizeof(W) == 8) v = ld_relaxed64((const u64 *)words + k);
            else v = ld_relaxed((const u32 *)words + k);
        } else {
            v = PRE;  // before tile 0: an empty inclusive prefix ends the walk
        }
        const W flag = v & ~MASK;
        const u32 pre = __ballot_sync(0xffffffffu, flag == PRE);
        const u32 unready = __ballot_sync(0xffffffffu, flag == 0);
        // lanes that count: up to the nearest inclusive prefix, and short of
        // the first word not yet published
        const u32 upto = pre ? ((pre & (0u - pre)) << 1) - 1 : 0xffffffffu;
        const u32 stop = unready & upto;
        const u32 take = stop ? (stop & (0u - stop)) - 1 : upto;
        W c = ((take >> lane) & 1) ? (v & MASK) : (W)0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
        excl += c;
        if (!stop && pre) break;
        j -= __popc(take);
        // a round trip to L2 per poll is the wait; the poll count bounds it
        if (stop && ++spins > limit) {
            if (lane == 0) atomicOr(err, ERR_LOOKBACK_TIMEOUT);
            break;
        }
    }
    return excl;
}

// empty cells (0 nibbles) of a board
__device__ __forceinline__ u32 zero_nibbles(u64 k)
{
    const u64 x = k | (k >> 1) | (k >> 2) | (k >> 3);
    return (u32)__popcll(~x & 0x1111111111111111ull);
}

}  // namespace cgb
