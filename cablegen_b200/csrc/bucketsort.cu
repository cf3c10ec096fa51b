// bucketsort.cu -- sort of u64 keys, with or without their repeats, by sampled
// splitters and a merge sort of each bucket by one CTA.
//
// The layer streams (move results, spawns) are sorted in every layer step.  An LSD
// radix sort moves every key once per varying byte (six times for an LL board) and
// pays a fixed latency per pass, so both large and small streams are slow.  Here a
// key moves two or three times whatever its width:
//   1. split:     one CTA sorts a sample of the input (20 to 64 keys per bucket) and
//                 keeps the bucket boundaries;
//   2. partition: each tile of 4096 keys finds its keys' buckets by binary
//                 search over the boundaries in shared memory, ranks them with
//                 shared-memory counters, reserves its space in every bucket
//                 with one global add and writes the buckets' parts coalesced;
//                 above 400 buckets this runs twice: coarse buckets first, then
//                 every coarse bucket by boundaries of its own;
//   3. bucket:    one CTA per bucket (at most 4096 keys, 1800 on average) sorts
//                 it -- 16 keys per thread through a register network, the 512
//                 of a warp by bitonic merges across its lanes, runs of 512 by
//                 merge-path steps in shared memory -- drops repeats when asked
//                 (equal keys always share a bucket) and writes at the offset
//                 that a look-back over the buckets' counts gives.
// Inputs of up to 16384 keys are one bucket, sorted by one CTA of 1024 threads
// (of 256 up to 4096 keys).
//
// Bounds: the partition is bound by its shared-memory accesses (50 wavefronts
// per 32 keys: search, counters, staging; 62 % of the peak), the bucket sort by
// instruction issue (280 warp instructions per 32 keys at 2.3 per cycle), neither
// by HBM.  Measured on B200, against byte-digit passes over 4096-key tiles:
// 11.5M LL moves 0.73 -> 0.40 ms, 1.27M DPDF moves 141 -> 92 us, 34M moves of
// LL with free formation 2.18 -> 1.33 ms, 4100 2x4 moves (one CTA) 53 -> 15 us; against
// those over 8192-key tiles, 120M keys of 48 bits 4.94 -> 4.36 ms, 168M 6.81 -> 5.82.
//
// The space of a bucket is fixed, so an input whose keys repeat so often that
// one bucket cannot hold them (or whose sample misleads) sets a flag and
// nothing is written; the caller then sorts by digit passes, which take any
// input.  The input itself is only read.
#include "engine.h"
#include "lookback.cuh"
#include <cstring>

namespace cgb {

constexpr u32 BK_TILE = 4096;     // keys per partition CTA
constexpr int BK_KPT = 16;        // keys per thread, every kernel
constexpr int SPLIT_THREADS = 512;
constexpr int PART_THREADS = 256;
constexpr int BUCKET_THREADS = 256;
constexpr int SMALL_THREADS = 1024;
constexpr u32 BK_SMALL = SMALL_THREADS * BK_KPT;  // keys that one CTA sorts in a single launch

constexpr u64 KEY_MAX = ~0ull;
constexpr u32 BK_OVERFLOW = 1u << 16;   // a bucket ran full (beside the ERR_* bits)

// control words of a sort's head (u32 indexes); its arrays: A_* of bucketplan.h
constexpr u32 H_TICKET = 0, H_FLAGS = 1, H_BUCKETS = 2, H_COUNT = BUCKET_COUNT_AT, H_EMPTIES = 6, H_ZEROS = 8,
              H_ONES = 10,  // bits that are 0 (1) in some key, each low word first
              H_STAMP = BUCKET_STAMP_AT,
              H_HEAVY = 14;  // a step's sample holds a key that no bucket has room for: one word a step

// The number of keys of a call: known on the host, or counted by a kernel before
// it (at most n, which sizes grids and buckets).
struct KeyCount {
    u32 n;
    const u64 *counted;
    __device__ __forceinline__ u32 get() const { return counted ? (u32)min((u64)n, *counted) : n; }
};

__device__ __forceinline__ u32 pad16(u32 i) { return i + (i >> 4); }
constexpr u32 SAMPLE_WORDS = BK_SAMPLES + BK_SAMPLES / 16;

// ---- sorting inside a CTA ---------------------------------------------------
// Keys are u64, or u32 where a bucket's keys differ in at most 32 bits.
template <typename K>
__device__ __forceinline__ K key_max() { return (K)~(K)0; }

__device__ __forceinline__ void order(u64 &a, u64 &b)
{
    const bool s = b < a;
    const u64 x = s ? b : a;
    b = s ? a : b;
    a = x;
}
__device__ __forceinline__ void order(u32 &a, u32 &b)
{
    const u32 x = min(a, b);
    b = max(a, b);
    a = x;
}

// Batcher's odd-even merge sort (Batcher 1968) of v[LO .. LO + N) in registers,
// unrolled by the templates
template <int LO, int N, int R, typename K>
__device__ __forceinline__ void odd_even_merge(K (&v)[BK_KPT])
{
    if constexpr (2 * R < N) {
        odd_even_merge<LO, N, 2 * R>(v);
        odd_even_merge<LO + R, N, 2 * R>(v);
#pragma unroll
        for (int i = LO + R; i + R < LO + N; i += 2 * R) order(v[i], v[i + R]);
    } else {
        order(v[LO], v[LO + R]);
    }
}
template <int LO, int N, typename K>
__device__ __forceinline__ void odd_even_sort(K (&v)[BK_KPT])
{
    if constexpr (N > 1) {
        odd_even_sort<LO, N / 2>(v);
        odd_even_sort<LO + N / 2, N / 2>(v);
        odd_even_merge<LO, N, 1>(v);
    }
}

// Sorts the 512 keys of a warp, 16 per lane: lane l ends with the keys of
// positions 16 l .. 16 l + 15.  Each lane sorts its own keys, then bitonic
// merges double the runs: the first stage of a merge compares a key with its
// mirror image in the other run, the others halve the distance, across lanes
// by shuffles and inside a lane in registers.  No shared memory, no barrier.
// A level costs 19 to 47 instructions per 64-bit key against about 50 of a
// merge-path step through shared memory, and a fraction of its latency.
template <typename K>
__device__ __forceinline__ void warp_sort(K (&v)[BK_KPT])
{
    const u32 lane = threadIdx.x & 31;
    odd_even_sort<0, BK_KPT>(v);
#pragma unroll 1
    for (u32 run = 1; run < 32; run *= 2) {
        {
            const bool up = lane & run;
#pragma unroll
            for (int i = 0; i < BK_KPT / 2; i++) {
                const K a = __shfl_xor_sync(0xffffffffu, v[BK_KPT - 1 - i], 2 * run - 1);
                const K b = __shfl_xor_sync(0xffffffffu, v[i], 2 * run - 1);
                v[i] = (v[i] < a) != up ? v[i] : a;
                v[BK_KPT - 1 - i] = (v[BK_KPT - 1 - i] < b) != up ? v[BK_KPT - 1 - i] : b;
            }
        }
#pragma unroll 1
        for (u32 d = run / 2; d; d /= 2) {
            const bool up = lane & d;
#pragma unroll
            for (int i = 0; i < BK_KPT; i++) {
                const K a = __shfl_xor_sync(0xffffffffu, v[i], d);
                v[i] = (v[i] < a) != up ? v[i] : a;  // the smaller of the two, or the larger
            }
        }
#pragma unroll
        for (int d = BK_KPT / 2; d; d /= 2)
#pragma unroll
            for (int i = 0; i < BK_KPT; i++)
                if (!(i & d)) order(v[i], v[i + d]);
    }
}

// Sorts n keys of a CTA, 16 per thread (the keys beyond n are the largest
// value), into position order: thread t ends with positions 16t .. 16t + 15.
// Warps that hold no key below n leave their registers alone.  Runs of 512
// come from the warps; merge-path steps through buf (at least n + n / 16
// words, padded so that a thread's 16 consecutive keys, and merge starts about
// 8 keys apart, lie on different banks) join them.  A side of a merge that has
// run out stands at the largest value: a tie with a real one takes an equal
// value, so no bounds test decides the order.
template <typename K>
__device__ __forceinline__ void block_sort(K *buf, u32 n, K (&v)[BK_KPT])
{
    const u32 t = threadIdx.x, n16 = (n + 15) & ~15u;
    const bool on = 16 * t < n;
    if ((t & ~31u) * 16 < n) warp_sort(v);
    for (u32 w = 512; w < n16; w *= 2) {
        __syncthreads();
        if (on) {
#pragma unroll
            for (int i = 0; i < BK_KPT; i++) buf[17 * t + i] = v[i];
        }
        __syncthreads();
        if (!on) continue;
        const u32 a0 = (16 * t) & ~(2 * w - 1), ae = min(a0 + w, n16), be = min(a0 + 2 * w, n16);
        const u32 diag = 16 * t - a0, la = ae - a0, lb = be - ae;
        u32 lo = diag > lb ? diag - lb : 0, hi = min(diag, la);
        while (lo < hi) {
            const u32 mid = (lo + hi) >> 1;
            if (buf[pad16(a0 + mid)] <= buf[pad16(ae + diag - 1 - mid)]) lo = mid + 1;
            else hi = mid;
        }
        u32 ia = a0 + lo, ib = ae + diag - lo;
        K xa = ia < ae ? buf[pad16(ia)] : key_max<K>(), xb = ib < be ? buf[pad16(ib)] : key_max<K>();
#pragma unroll
        for (int i = 0; i < BK_KPT; i++) {
            const bool ta = xa <= xb;
            v[i] = ta ? xa : xb;
            if (i + 1 < BK_KPT) {
                ia += ta ? 1 : 0;
                ib += ta ? 0 : 1;
                const u32 ni = ta ? ia : ib, ne = ta ? ae : be;
                const K x = ni < ne ? buf[pad16(ni)] : key_max<K>();
                xa = ta ? x : xa;
                xb = ta ? xb : x;
            }
        }
    }
}

// index of a CTA's i-th key of this thread: warp w takes keys 512 w .. 512 w + 511
__device__ __forceinline__ u32 warp_key(int i) { return (threadIdx.x & ~31u) * BK_KPT + i * 32 + (threadIdx.x & 31); }

// ---- keys that differ in at most 32 bits -------------------------------------
// The bits of x under mask m moved together, in order, by five steps of moves
// by 1, 2, 4, 8 and 16 places (Warren, Hacker's Delight, the compress and
// expand functions); mv[i] marks the bits that step i moves.
struct BitMoves {
    u32 m, mv[5];
};
__device__ inline void plan_moves(u32 m, BitMoves *b)
{
    b->m = m;
    u32 mk = ~m << 1;  // bits with an unselected bit just below
#pragma unroll
    for (int i = 0; i < 5; i++) {
        u32 p = mk;    // parity of the unselected bits below each position
#pragma unroll
        for (int s = 1; s < 32; s *= 2) p ^= p << s;
        const u32 mv = p & m;
        b->mv[i] = mv;
        m = (m ^ mv) | (mv >> (1 << i));
        mk &= ~p;
    }
}
__device__ __forceinline__ u32 compress_bits(u32 x, const BitMoves &b)
{
    x &= b.m;
#pragma unroll
    for (int i = 0; i < 5; i++) {
        const u32 t = x & b.mv[i];
        x = (x ^ t) | (t >> (1 << i));
    }
    return x;
}
__device__ __forceinline__ u32 expand_bits(u32 x, const BitMoves &b)
{
#pragma unroll
    for (int i = 4; i >= 0; i--) x = (x & ~b.mv[i]) | ((x << (1 << i)) & b.mv[i]);
    return x & b.m;
}

// key as u32 and back: the low word's selected bits below the high word's
__device__ __forceinline__ u32 narrow_key(u64 k, const BitMoves &lo, const BitMoves &hi, u32 low)
{
    const u32 y = hi.m ? compress_bits((u32)(k >> 32), hi) << (low & 31) : 0u;  // low < 32 where hi.m
    return y | compress_bits((u32)k, lo);
}
__device__ __forceinline__ u64 wide_key(u32 x, const BitMoves &lo, const BitMoves &hi, u32 low)
{
    return make64(hi.m ? expand_bits(x >> (low & 31), hi) : 0u, expand_bits(x, lo));
}

// AND and OR over a warp's values into and_or[0..1] (low, high word), [2..3]
__device__ __forceinline__ void reduce_and_or(u64 a, u64 o, u32 *and_or)
{
    constexpr u32 ALL = 0xffffffffu;
    const u32 lane = threadIdx.x & 31;
    const u32 r[4] = {__reduce_and_sync(ALL, (u32)a), __reduce_and_sync(ALL, (u32)(a >> 32)),
                      __reduce_or_sync(ALL, (u32)o), __reduce_or_sync(ALL, (u32)(o >> 32))};
    if (lane < 2) atomicAnd(and_or + lane, lane ? r[1] : r[0]);
    else if (lane < 4) atomicOr(and_or + lane, lane == 3 ? r[3] : r[2]);
}

// lowbias32 (Wellons, Hash Prospector, 2018)
__device__ __forceinline__ u32 mix32(u32 x)
{
    x = (x ^ (x >> 16)) * 0x7feb352du;
    x = (x ^ (x >> 15)) * 0x846ca68bu;
    return x ^ (x >> 16);
}

// The sorted sample (16 keys per thread, in v) turned into boundaries, in the
// order of a search tree: the children of node j are 2j and 2j + 1, so the
// nodes of one level are consecutive and a warp's lanes spread over the banks
// (in sorted order the candidates of a level are a power of two apart, on one
// bank).  Unused boundaries stay at KEY_MAX: no key is above them.
//
// `heavy`, if given, is set where the sample of cnt keys holds one that repeats about
// twice as often as a bucket has room: whole threads of equal keys, as many of them
// in a row as stand for 2 BK_CAP copies.  What follows is then skipped: an input half
// of which is one key takes 0.49 ms instead of 0.55 for 3M keys (0.44 with nothing tried
// before the digit passes), 1.81 instead of 2.21 for 30M (1.69).
template <typename K, class Emit>
__device__ __forceinline__ void write_bounds(K (&v)[BK_KPT], K *buf, u32 m, u32 cnt, u32 nb, u64 *bounds, u32 *heavy,
                                             Emit emit)
{
    block_sort(buf, m, v);
    __syncthreads();
    if (16 * threadIdx.x < m) {
#pragma unroll
        for (int i = 0; i < BK_KPT; i++) buf[17 * threadIdx.x + i] = v[i];
    }
    __syncthreads();
    if (heavy && v[0] == v[BK_KPT - 1]) {
        const u32 last = 16 * (threadIdx.x + (2 * BK_CAP / 16 * m + cnt - 1) / cnt) - 1;  // of that many threads
        if (last < m && buf[pad16(last)] == v[0]) *heavy = 1;
    }
    const u32 leaves = nb > 1 ? 2u << (31 - __clz(nb - 1)) : 1;
    for (u32 j = threadIdx.x; j < leaves; j += SPLIT_THREADS) {
        const u32 level = j ? 31 - __clz(j) : 0, half = (leaves >> level) >> 1;
        const u32 i = (2 * (j - (1u << level)) + 1) * half;  // this node's place in sorted order, from 1
        bounds[j] = j && i < nb ? emit(buf[pad16(i * m / nb)]) : KEY_MAX;
    }
}

// Boundaries from a sorted sample.  FINE false: of the whole input, into buckets
// of the target size where one step does (BK_ONE_STEP), else into `buckets`
// coarse buckets; true: CTA c, the boundaries inside coarse bucket c, whose number
// follows its size.  A sample is one random key out of
// each of equally long stretches, so that neither a regular pattern nor a
// sorted input biases it.  (Nothing to do for the keys of one bucket: the bucket
// sort takes them from the input.)
template <bool FINE>
__global__ void __launch_bounds__(SPLIT_THREADS, 1) bucket_split_kernel(const u64 *src, KeyCount n,
                                                                        u32 buckets, u32 coarse_cap, u32 *head,
                                                                        u32 *arrays, u64 *bounds)
{
    extern __shared__ __align__(16) u64 split_buf[];
    __shared__ u32 scratch[33];
    __shared__ BitMoves moves[2];
    after_previous();
    if (!FINE) stamp((u64 *)(head + H_STAMP));
    u32 cnt = n.get(), nb = buckets;
    const bool one_step = cnt <= BK_ONE_STEP;
    if (cnt <= BK_CAP || (FINE && (one_step || head[H_HEAVY]))) return;
    if (FINE) {
        const u32 c = blockIdx.x;
        // this coarse bucket's first fine bucket: the numbers of those before it, summed
        u32 mine = 0, all = 0;
        for (u32 i = threadIdx.x; i < buckets; i += SPLIT_THREADS) {
            const u32 f = (min(arrays[A_COARSE + i], coarse_cap) + BK_TARGET - 1) / BK_TARGET;
            all += f;
            mine += i < c ? f : 0;
        }
        u32 base, total;
        block_exclusive_scan<u32>(mine, scratch, &base);
        block_exclusive_scan<u32>(all, scratch, &total);
        cnt = min(arrays[A_COARSE + c], coarse_cap);
        nb = (cnt + BK_TARGET - 1) / BK_TARGET;
        if (threadIdx.x == 0) {
            arrays[A_BASE + c] = base;
            arrays[A_NUM + c] = nb;
            if (c == 0) head[H_BUCKETS] = total;
        }
        if (nb <= 1) return;
        src += (u64)c * coarse_cap;
        bounds += (u64)c * BK_FAN;
    } else if (one_step) {
        nb = (cnt + BK_TARGET - 1) / BK_TARGET;
        if (threadIdx.x == 0) head[H_BUCKETS] = nb;
    }
    const u32 m = min(min(nb * (FINE ? 32u : one_step ? 24u : 64u), BK_SAMPLES), cnt);
    if (threadIdx.x < 4) scratch[threadIdx.x] = threadIdx.x < 2 ? 0xffffffffu : 0u;
    __syncthreads();
    u64 k[BK_KPT];
    u64 a = KEY_MAX, o = 0;
    const bool on = (threadIdx.x & ~31u) * BK_KPT < m;
    if (on) {
        const u32 q = cnt / m, r = cnt % m;  // stretch i: q keys, one more for the first r
#pragma unroll
        for (int s = 0; s < BK_KPT; s++) {
            const u32 i = min(warp_key(s), m - 1);
            k[s] = src[i * q + min(i, r) + __umulhi(mix32(i), q + (i < r ? 1 : 0))];
        }
#pragma unroll
        for (int s = 0; s < BK_KPT; s++) {
            a &= k[s];
            o |= k[s];
        }
        reduce_and_or(a, o, scratch);
    }
    __syncthreads();
    u64 used = make64(scratch[1] ^ scratch[3], scratch[0] ^ scratch[2]);
    const u64 fixed = make64(scratch[1], scratch[0]) & ~used;
    u32 *heavy = head + H_HEAVY + (FINE ? 1 : 0);
    if (__popcll(used) <= 40) {
        if (__popcll(used) > 32) heavy = nullptr;  // equal words need not be equal keys
        // a boundary need not be a key: up to eight of the lowest bits are left
        // out, which moves it past 255 distinct keys at most
        while (__popcll(used) > 32) used &= used - 1;
        const u32 low = __popc((u32)used);
        if (threadIdx.x == 0) plan_moves((u32)used, &moves[0]);
        if (threadIdx.x == 32) plan_moves((u32)(used >> 32), &moves[1]);
        __syncthreads();
        u32 v[BK_KPT];
        if (on) {
#pragma unroll
            for (int s = 0; s < BK_KPT; s++)
                v[s] = warp_key(s) < m ? narrow_key(k[s], moves[0], moves[1], low) : 0xffffffffu;
        }
        write_bounds(v, (u32 *)split_buf, m, cnt, nb, bounds, heavy,
                     [&](u32 x) { return wide_key(x, moves[0], moves[1], low) | fixed; });
    } else {
#pragma unroll
        for (int s = 0; s < BK_KPT; s++)
            if (!on || warp_key(s) >= m) k[s] = KEY_MAX;
        write_bounds(k, split_buf, m, cnt, nb, bounds, heavy, [](u64 x) { return x; });
    }
}

struct PartSmem {
    u64 keys[BK_TILE];
    u64 bounds[BK_FAN];
    unsigned short id[BK_TILE];
    u32 count[BK_FAN], first[BK_FAN], delta[BK_FAN];
    u32 scan[33];
};

// One tile of a partition step.  FINE: the tile belongs to coarse bucket
// blockIdx.x / tiles and goes to that bucket's fine buckets; else the input is
// the source and goes to the coarse buckets, or to the fine ones where one step
// does.
template <bool FINE>
__global__ void __launch_bounds__(PART_THREADS, 4)
    bucket_partition_kernel(const u64 *src, KeyCount n, u32 src_cap, u32 tiles, u32 buckets, const u64 *bounds, u32 *head, u32 *arrays, u64 *coarse, u32 coarse_cap,
                            u64 *fine)
{
    extern __shared__ __align__(16) unsigned char part_smem[];
    PartSmem &S = *reinterpret_cast<PartSmem *>(part_smem);
    after_previous();
    const u32 t = threadIdx.x;
    const u32 c = FINE ? blockIdx.x / tiles : 0, tile = FINE ? blockIdx.x % tiles : blockIdx.x;
    const u32 all = n.get();
    // nothing to do where a key is too frequent for a bucket: the caller's digit passes
    // take the input (the words are read beside the counts, so they cost no time)
    const u32 heavy = FINE ? head[H_HEAVY] | head[H_HEAVY + 1] : head[H_HEAVY];
    const u32 cnt = heavy ? 0 : FINE ? min(arrays[A_COARSE + c], src_cap) : all;
    const u32 start = tile * BK_TILE;
    const bool one_step = all <= BK_ONE_STEP;
    if (start >= cnt || all <= BK_CAP || (FINE && one_step)) return;
    const bool to_fine = FINE || one_step;
    u64 *dst = to_fine ? fine : coarse;
    const u32 dst_cap = to_fine ? BK_CAP : coarse_cap, counters = to_fine ? A_FINE : A_COARSE;
    const u32 nb = FINE ? arrays[A_NUM + c] : one_step ? head[H_BUCKETS] : buckets;
    const u32 base = FINE ? arrays[A_BASE + c] : 0;
    if (FINE) {
        src += (u64)c * src_cap;
        bounds += (u64)c * BK_FAN;
    }
    const u32 tile_n = min(BK_TILE, cnt - start);
    u64 k[BK_KPT];
#pragma unroll
    for (int i = 0; i < BK_KPT; i++) {
        const u32 j = i * PART_THREADS + t;
        k[i] = j < tile_n ? src[start + j] : KEY_MAX;
    }
    const u32 leaves = nb > 1 ? 2u << (31 - __clz(nb - 1)) : 1;
    for (u32 i = t; i < BK_FAN; i += PART_THREADS) S.count[i] = 0;
    for (u32 i = t; i < leaves; i += PART_THREADS) S.bounds[i] = bounds[i];
    __syncthreads();
    // bucket = boundaries below the key; 16 independent searches per thread
    u32 at[BK_KPT];
#pragma unroll
    for (int i = 0; i < BK_KPT; i++) at[i] = 1;
    for (u32 w = leaves; w > 1; w >>= 1) {
#pragma unroll
        for (int i = 0; i < BK_KPT; i++) at[i] = 2 * at[i] + (S.bounds[at[i]] < k[i] ? 1 : 0);
    }
#pragma unroll
    for (int i = 0; i < BK_KPT; i++) {
        at[i] -= leaves;
        if (i * PART_THREADS + t < tile_n) at[i] |= atomicAdd(&S.count[at[i]], 1u) << 16;
    }
    __syncthreads();
    {
        // two neighbouring buckets per thread; their space is reserved before the
        // scan, whose barriers hide the round trip
        u32 num[2], g[2];
#pragma unroll
        for (int q = 0; q < 2; q++) {
            num[q] = S.count[2 * t + q];
            g[q] = num[q] ? atomicAdd(arrays + counters + base + 2 * t + q, num[q]) : 0;
        }
        u32 total;
        u32 first = block_exclusive_scan<u32>(num[0] + num[1], S.scan, &total);
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const u32 b = 2 * t + q;
            S.first[b] = first;
            u32 delta = 0xFFFFFFFFu;
            if (num[q]) {
                if (g[q] + num[q] <= dst_cap) delta = (base + b) * dst_cap + g[q] - first;
                else atomicOr(head + H_FLAGS, BK_OVERFLOW);
            }
            S.delta[b] = delta;
            first += num[q];
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < BK_KPT; i++) {
        if (i * PART_THREADS + t < tile_n) {
            const u32 b = at[i] & 0xFFFFu, p = S.first[b] + (at[i] >> 16);
            S.keys[p] = k[i];
            S.id[p] = (unsigned short)b;
        }
    }
    __syncthreads();
#pragma unroll 4
    for (u32 j = t; j < tile_n; j += PART_THREADS) {
        const u32 delta = S.delta[S.id[j]];
        if (delta != 0xFFFFFFFFu) dst[(u32)(delta + j)] = S.keys[j];
    }
}

template <int THREADS>
struct BucketSmem {
    static constexpr u32 WORDS = THREADS * BK_KPT + THREADS;  // padded
    union {
        u64 wide[WORDS];
        u32 narrow[WORDS];
    };
    u64 last64[THREADS];
    u32 warp[THREADS / 32];
    u32 and_or[4];
    BitMoves lo, hi;
    u32 tile, prefix, kept;
};

// Everything after the sort key type is known: sort, flag the keys to keep,
// their offset by look-back, write.  EMIT turns a sorted key into the u64.
template <bool UNIQUE, bool DIRECT, int THREADS, typename K, class Emit>
__device__ __forceinline__ void finish_bucket(K (&v)[BK_KPT], K *buf, K *last_sh, u32 cnt, u32 tile, u32 tiles, u32 *look,
                                              u32 *head, u64 *__restrict__ out, u32 count_empties, LookbackLimit lb,
                                              BucketSmem<THREADS> &S, Emit emit)
{
    constexpr u32 ALL = 0xffffffffu;
    constexpr u32 AGG = 1u << 30, PRE = 2u << 30;
    const u32 t = threadIdx.x, lane = t & 31, warp = t >> 5;
    block_sort(buf, cnt, v);
    const u32 mine = 16 * t < cnt ? min(16u, cnt - 16 * t) : 0;
    u32 flags = mine == 16 ? 0xFFFFu : (1u << mine) - 1;
    if (UNIQUE) {
        // a thread before one that holds keys holds 16
        last_sh[t] = v[BK_KPT - 1];
        __syncthreads();
        K prev = t ? last_sh[t - 1] : 0;
        u32 same = 0;
#pragma unroll
        for (int i = 0; i < BK_KPT; i++) {
            if (v[i] == prev) same |= 1u << i;
            prev = v[i];
        }
        if (t == 0) same &= ~1u;
        flags &= ~same;
    }
    const u32 kept = __popc(flags);
    const u32 inc = warp_inclusive_scan(kept);
    if (lane == 31) S.warp[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        const u32 c = lane < THREADS / 32 ? S.warp[lane] : 0u;
        const u32 wi = warp_inclusive_scan(c);
        const u32 total = __shfl_sync(ALL, wi, 31);
        u32 prefix = 0;
        if (!DIRECT) {
            if (tile > 0) {
                if (UNIQUE && lane == 0) st_relaxed(look + tile, AGG | total);
                prefix = warp_lookback_sum<u32>(look, (int)tile - 1, head + H_FLAGS, lb.polls);
            }
            if (lane == 0 && !(lb.hold && tile == 0)) st_relaxed(look + tile, PRE | (prefix + total));
        }
        if (lane < THREADS / 32) S.warp[lane] = wi - c;
        if (lane == 0) {
            S.prefix = prefix;
            S.kept = total;
            if (tile + 1 == tiles) *(u64 *)(head + H_COUNT) = prefix + total;
        }
    }
    __syncthreads();
    u32 w = S.warp[warp] + inc - kept;
#pragma unroll
    for (int i = 0; i < BK_KPT; i++)
        if (flags & (1u << i)) {
            buf[pad16(w)] = v[i];
            w++;
        }
    __syncthreads();
    const u32 prefix = S.prefix, num = S.kept;
    u32 empty = 0;
    for (u32 j = t; j < num; j += THREADS) {
        const u64 key = emit(buf[pad16(j)]);
        out[prefix + j] = key;
        if (UNIQUE && count_empties) empty += zero_nibbles(key);
    }
    if (UNIQUE && count_empties) {
        empty = __reduce_add_sync(ALL, empty);
        if (lane == 0 && empty) atomicAdd((unsigned long long *)(head + H_EMPTIES), (unsigned long long)empty);
    }
}

// One bucket: sorted, repeats dropped with UNIQUE, written at the sum of the
// counts of the buckets before it.  Buckets are taken in ticket order, so every
// predecessor that a look-back waits for is already running.  An input that
// fits one bucket is taken as it is (DIRECT: known on the host).
//
// The keys of a bucket share their high cells, and the constant bits of the
// others (fixed cells, the top bits of small tiles) hold no order: in buckets
// of LL, DPDF and 2x4 layers 22 to 30 bits differ, at most 32 in 94 to 100 % of
// them.  Such a bucket is sorted as u32 keys of those bits alone, where a
// compare-exchange is two instructions instead of six (the low words as they
// are where the high words agree); the others are sorted as they are.
template <bool UNIQUE, bool DIRECT, int THREADS>
__device__ __forceinline__ void sort_bucket(const u64 *src, u32 cnt, u32 tile, u32 tiles, u32 *look, u32 *head,
                                            u64 *__restrict__ out, u32 count_empties, LookbackLimit lb,
                                            BucketSmem<THREADS> &S)
{
    constexpr u32 ALL = 0xffffffffu;
    const u32 t = threadIdx.x;
    u64 k[BK_KPT];
    u64 a = KEY_MAX, o = 0;
    const bool on = (t & ~31u) * BK_KPT < cnt;
    if (on) {
#pragma unroll
        for (int i = 0; i < BK_KPT; i++) {
            const u32 j = warp_key(i);
            k[i] = j < cnt ? src[j] : KEY_MAX;
        }
#pragma unroll
        for (int i = 0; i < BK_KPT; i++) {
            a &= k[i];  // the padding does not change it
            if (warp_key(i) < cnt) o |= k[i];
        }
        reduce_and_or(a, o, S.and_or);
    } else {
#pragma unroll
        for (int i = 0; i < BK_KPT; i++) k[i] = KEY_MAX;
    }
    __syncthreads();
    if (UNIQUE && t < 4) {
        const u32 bits = t < 2 ? ~S.and_or[t] : S.and_or[t];
        if (bits & ~ld_relaxed(head + H_ZEROS + t)) atomicOr(head + H_ZEROS + t, bits);
    }
    const u32 vary_lo = S.and_or[0] ^ S.and_or[2], vary_hi = S.and_or[1] ^ S.and_or[3];
    const u32 low = __popc(vary_lo);
    if (vary_hi == 0) {
        const u32 high = S.and_or[1];
        u32 v[BK_KPT];
#pragma unroll
        for (int i = 0; i < BK_KPT; i++) v[i] = (u32)k[i];  // KEY_MAX beyond cnt
        finish_bucket<UNIQUE, DIRECT, THREADS>(v, S.narrow, (u32 *)S.last64, cnt, tile, tiles, look, head, out,
                                               count_empties, lb, S, [=](u32 x) { return make64(high, x); });
    } else if (low + __popc(vary_hi) <= 32) {
        if (t == 0) plan_moves(vary_lo, &S.lo);
        if (t == 32) plan_moves(vary_hi, &S.hi);
        const u64 fixed = make64(S.and_or[1] & ~vary_hi, S.and_or[0] & ~vary_lo);
        __syncthreads();
        u32 v[BK_KPT];
        {
            const BitMoves lo = S.lo, hi = S.hi;
#pragma unroll
            for (int i = 0; i < BK_KPT; i++) v[i] = warp_key(i) < cnt ? narrow_key(k[i], lo, hi, low) : ALL;
        }
        finish_bucket<UNIQUE, DIRECT, THREADS>(v, S.narrow, (u32 *)S.last64, cnt, tile, tiles, look, head, out,
                                               count_empties, lb, S,
                                               [&](u32 x) { return wide_key(x, S.lo, S.hi, low) | fixed; });
    } else {
        finish_bucket<UNIQUE, DIRECT, THREADS>(k, S.wide, S.last64, cnt, tile, tiles, look, head, out, count_empties, lb,
                                               S, [](u64 x) { return x; });
    }
}

template <bool UNIQUE, bool DIRECT>
__global__ void __launch_bounds__(BUCKET_THREADS, 4)
    bucket_sort_kernel(const u64 *input, KeyCount n, const u64 *slots, u32 counters, u32 words, u32 *head, u32 *arrays,
                       u64 *__restrict__ out, u32 count_empties, LookbackLimit lb)
{
    __shared__ BucketSmem<BUCKET_THREADS> S;
    after_previous();
    const u32 t = threadIdx.x;
    if (!slots || gridDim.x == 1) stamp((u64 *)(head + H_STAMP));  // no split before it
    const u32 all = n.get();
    // one thread reads the flags for all: another CTA's wait may run out and set one
    // while this CTA starts
    if (t == 0 && !DIRECT) {
        const u32 ticket = atomicAdd(head + H_TICKET, 1u);  // (with the flags on their way too)
        S.tile = ld_relaxed(head + H_FLAGS) | ld_relaxed(head + H_HEAVY) | ld_relaxed(head + H_HEAVY + 1) ? 0xFFFFFFFFu : ticket;
    }
    if (t < 4) S.and_or[t] = t < 2 ? 0xffffffffu : 0u;
    const bool whole = DIRECT || all <= BK_CAP;
    __syncthreads();
    const u32 tile = DIRECT ? 0 : S.tile, tiles = whole ? 1 : head[H_BUCKETS];
    if (!DIRECT && tile >= tiles) return;
    const u32 cnt = whole ? all : arrays[counters + tile];
    u32 *look = arrays + words;
    if (!UNIQUE && t == 0 && tile > 0) st_relaxed(look + tile, (1u << 30) | cnt);
    const u64 *src = whole ? input : slots + (u64)tile * BK_CAP;
    sort_bucket<UNIQUE, DIRECT, BUCKET_THREADS>(src, cnt, tile, tiles, look, head, out, count_empties, lb, S);
}

// Up to 16384 keys in one CTA of 1024 threads: a launch in place of three, whose
// kernels would each leave the chip idle.  The two sorts of the 149 layers of the
// 2x4 table (3400 moves and 14000 spawns each): 7.8 -> 6.0 ms.
template <bool UNIQUE>
__global__ void __launch_bounds__(SMALL_THREADS, 1)
    small_sort_kernel(const u64 *input, KeyCount n, u32 *head, u64 *__restrict__ out, u32 count_empties)
{
    extern __shared__ __align__(16) unsigned char small_smem[];
    BucketSmem<SMALL_THREADS> &S = *reinterpret_cast<BucketSmem<SMALL_THREADS> *>(small_smem);
    after_previous();
    stamp((u64 *)(head + H_STAMP));
    const u32 cnt = n.get();
    if (cnt > BK_SMALL && threadIdx.x == 0) head[H_FLAGS] = BK_OVERFLOW;
    if (cnt == 0 || cnt > BK_SMALL) return;
    if (threadIdx.x < 4) S.and_or[threadIdx.x] = threadIdx.x < 2 ? 0xffffffffu : 0u;
    __syncthreads();
    sort_bucket<UNIQUE, true, SMALL_THREADS>(input, cnt, 0, 1, nullptr, head, out, count_empties, LookbackLimit{}, S);
}

// ---------------------------------------------------------------------------
void BucketWorkspace::release(cudaStream_t s)
{
    dev_free(ctl.p, s);
    dev_free(coarse.p, s);
    dev_free(fine.p, s);
    dev_free(bounds.p, s);
    ctl = DevBuf<u32>{};
    coarse = fine = bounds = DevBuf<u64>{};
}

static bool attributes()
{
    static bool done = false;
    if (done) return true;
    const int part = (int)sizeof(PartSmem), split = (int)(SAMPLE_WORDS * sizeof(u64));
    const auto smem = cudaFuncAttributeMaxDynamicSharedMemorySize;
    done = CGB_CUDA(cudaFuncSetAttribute(bucket_split_kernel<false>, smem, split)) &&
           CGB_CUDA(cudaFuncSetAttribute(bucket_split_kernel<true>, smem, split)) &&
           CGB_CUDA(cudaFuncSetAttribute(small_sort_kernel<false>, smem, (int)sizeof(BucketSmem<SMALL_THREADS>))) &&
           CGB_CUDA(cudaFuncSetAttribute(small_sort_kernel<true>, smem, (int)sizeof(BucketSmem<SMALL_THREADS>))) &&
           CGB_CUDA(cudaFuncSetAttribute(bucket_partition_kernel<false>, smem, part)) &&
           CGB_CUDA(cudaFuncSetAttribute(bucket_partition_kernel<true>, smem, part));
    return done;
}

bool bucket_prepare(const u64 *n, int calls, BucketPlan *plans, BucketWorkspace &w, cudaStream_t s, const u64 *likely)
{
    u64 words = BUCKET_HEADS * BUCKET_HEAD_WORDS, fine = 0, coarse = 0, bounds = 0;
    for (int i = 0; i < calls; i++) {
        BucketPlan &p = plans[i];
        if (!plan_buckets(n[i], &p)) return false;
        p.small = (likely && likely[i] <= BK_SMALL) || (n[i] > BK_CAP && n[i] <= BK_SMALL);
        p.arrays_at = words;
        words += (p.words + 1) / 2 * 2;
        if (p.n <= BK_CAP || p.small) continue;
        fine = std::max(fine, (u64)p.grid * BK_CAP);
        coarse = std::max(coarse, (u64)p.coarse * p.coarse_cap);
        bounds = std::max(bounds, (u64)BK_FAN * (p.coarse + 1));
    }
    w.used_words = words;
    auto room = [&](auto &b, u64 want) { return (b.p && b.cap >= want) || !want || grow(b, want * 5 / 4, s); };
    w.growing = true;
    const bool have = room(w.ctl, words) && room(w.bounds, bounds) && room(w.fine, fine) && room(w.coarse, coarse);
    w.growing = false;
    if (!have) {  // the digit passes take over, and their caller may need the room
        w.release(s);
        return false;
    }
    if (!w.host && !CGB_CUDA(cudaHostAlloc((void **)&w.host, BUCKET_HEADS * BUCKET_HEAD_WORDS * 4, cudaHostAllocDefault)))
        return false;
    return attributes();
}

bool bucket_clear(BucketWorkspace &w, cudaStream_t s)
{
    return CGB_CUDA(cudaMemsetAsync(w.ctl.p, 0, w.used_words * sizeof(u32), s));
}

template <bool UNIQUE>
static void launch_sort(const BucketPlan &p, const u64 *keys, KeyCount kc, u64 *out, bool empties, u32 *head, u32 *arrays,
                        BucketWorkspace &w, cudaStream_t s)
{
    if (p.n <= BK_CAP && !kc.counted)
        launch_after(bucket_sort_kernel<UNIQUE, true>, 1, BUCKET_THREADS, 0, s, keys, kc, nullptr, A_FINE,
                     A_FINE + p.grid, head, arrays, out, empties, g_lookback);
    else
        launch_after(bucket_sort_kernel<UNIQUE, false>, p.grid, BUCKET_THREADS, 0, s, keys, kc, w.fine.p, A_FINE,
                     A_FINE + p.grid, head, arrays, out, empties, g_lookback);
}

int bucket_enqueue(const BucketPlan &p, int slot, const u64 *keys, const u64 *counted, u64 *out, bool unique, bool empties,
                   BucketWorkspace &w, cudaStream_t s)
{
    const u32 split_smem = SAMPLE_WORDS * sizeof(u64);
    u32 *head = w.ctl.p + slot * BUCKET_HEAD_WORDS, *arrays = w.ctl.p + p.arrays_at;
    const KeyCount kc{(u32)p.n, counted};
    const u32 tiles = (u32)((p.n + BK_TILE - 1) / BK_TILE);
    int np = 1;
    if (p.small) {
        constexpr u32 smem = sizeof(BucketSmem<SMALL_THREADS>);
        launch_after(unique ? small_sort_kernel<true> : small_sort_kernel<false>, 1, SMALL_THREADS, smem, s, keys, kc,
                     head, out, unique && empties);
        return np;
    }
    if (p.n > BK_CAP) {
        launch_after(bucket_split_kernel<false>, 1, SPLIT_THREADS, split_smem, s, keys, kc, p.coarse, 0, head, arrays,
                     w.bounds.p);
        launch_after(bucket_partition_kernel<false>, tiles, PART_THREADS, sizeof(PartSmem), s, keys, kc, 0, 1, p.coarse,
                     w.bounds.p, head, arrays, w.coarse.p, p.coarse_cap, w.fine.p);
        np = 2;
    }
    if (p.coarse) {
        const u32 fine_tiles = (p.coarse_cap + BK_TILE - 1) / BK_TILE;
        u64 *fine_bounds = w.bounds.p + BK_FAN;
        launch_after(bucket_split_kernel<true>, p.coarse, SPLIT_THREADS, split_smem, s, w.coarse.p, kc, p.coarse,
                     p.coarse_cap, head, arrays, fine_bounds);
        launch_after(bucket_partition_kernel<true>, p.coarse * fine_tiles, PART_THREADS, sizeof(PartSmem), s, w.coarse.p,
                     kc, p.coarse_cap, fine_tiles, 0, fine_bounds, head, arrays, nullptr, 0, w.fine.p);
        np = 3;
    }
    if (unique) launch_sort<true>(p, keys, kc, out, empties, head, arrays, w, s);
    else launch_sort<false>(p, keys, kc, out, false, head, arrays, w, s);
    kstats().launches += np == 1 ? 0 : np == 2 ? 2 : 4;
    return np;
}

BucketResult bucket_result(const u32 *heads, int slot)
{
    const u32 *h = heads + slot * BUCKET_HEAD_WORDS;
    BucketResult r;
    r.error = h[H_FLAGS] & ~BK_OVERFLOW;
    r.overflow = (h[H_FLAGS] & BK_OVERFLOW) || h[H_HEAVY] || h[H_HEAVY + 1];
    memcpy(&r.count, h + H_COUNT, 8);
    memcpy(&r.started, h + H_STAMP, 8);
    memcpy(&r.empties, h + H_EMPTIES, 8);
    memcpy(&r.bits.all, h + H_ZEROS, 8);
    memcpy(&r.bits.any, h + H_ONES, 8);
    r.bits.all = ~r.bits.all;
    r.bits.known = r.count > 0;
    return r;
}

bool bucket_sort(const u64 *keys, u64 n, u64 *out, bool unique, u64 *n_out, u64 *empties, int *passes,
                 BucketWorkspace &w, cudaStream_t s, bool *done, KeyBits *bits)
{
    *done = false;
    BucketPlan p;
    // without room for the buckets the caller's digit passes take over
    if (n < 2 || !bucket_prepare(&n, 1, &p, w, s)) return true;
    if (!bucket_clear(w, s)) return false;
    kclock().begin(s, &kstats().onesweep_ms);
    const int np = bucket_enqueue(p, 0, keys, nullptr, out, unique, empties != nullptr, w, s);
    kclock().end(s);
    if (!CGB_CUDA(cudaGetLastError()) ||
        !words_to_host(w.host, w.ctl.p, BUCKET_HEAD_WORDS, s) ||
        !CGB_CUDA(cudaStreamSynchronize(s)))
        return false;
    kclock().flush();
    const BucketResult r = bucket_result(w.host, 0);
    if (r.error) {
        set_error("bucket_sort: device error " + err_string(r.error));
        return false;
    }
    if (r.overflow) return true;
    *n_out = r.count;
    if (empties) *empties = r.empties;
    if (bits) *bits = r.bits;
    kstats().onesweep_bytes += 16 * n * np;
    kstats().onesweep_launches += np;
    if (passes) *passes = np;
    *done = true;
    return true;
}

}  // namespace cgb
