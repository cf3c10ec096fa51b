// solve.cu -- backward expectimax over one layer (src/solve.c:226-302).
//
// One thread per board of layer s:
//   * satisfied (src/solve.c:233-244): with nox the board wins (1.0) when it
//     holds tile nox; otherwise when it matches any winstate image.
//   * otherwise expectimax (src/solve.c:257-281): for every empty cell in
//     cell order 0..15, a 2 (weight 0.9) and a 4 (weight 0.1) are placed; the
//     value of each spawn is the best of the four moves (src/solve.c:246-256),
//     each successor looked up, canonicalised, in the s+2 / s+4 table; a miss
//     is 0.0 (src/solve.c:108-164).  res = 0.9*S2/k + 0.1*S4/k.
//
// Two kernels: solve_items_kernel (the default) spreads the (board, empty
// cell) pairs of 32 boards over a warp's lanes; solve_direct_kernel runs one
// thread per board.  Canonical forms take the maximum over the images a
// CanonPlan allows for the board's 0xf mask (all eight without a plan).
//
// FP64 evaluates exactly the reference's operation sequence with
// round-to-nearest intrinsics (no FMA contraction): bit-identical values.
// FP32 keeps table values in FP32, accumulates the two spawn sums with Kahan
// compensation and forms the weighted mean in FP64 before rounding once (a
// 0.9f weight alone would bias every layer by 2.6e-8 relative).
//
// Lookup structures (all exact; a miss returns 0 like the reference):
//   INDEX_BISECT  branch-free bisection over the sorted layer
//   INDEX_BUCKET  top bits after the layer's common prefix select a bucket of
//                 the sorted layer, then bisection inside it
//   INDEX_HASH    open addressing with linear probing; a 16-byte slot holds
//                 the key and the value, so a hit costs one sector
#include "engine.h"
#include "hashidx.cuh"

namespace cgb {

constexpr int TABLE_BYTES_S = 65536 * 2;  // left-move rows, ROW_LOCKED for locked ones

// ---- lookup ---------------------------------------------------------------
template <typename V>
struct DevTable {
    int kind;
    const u64 *keys;
    const V *vals;
    u64 n;
    const u32 *bucket;
    int prefix, bits;
    u64 prefix_value;
    const ulonglong2 *slots;
    u64 cap;
    CompactHash ch;  // INDEX_HASH with 8-byte slots (ch.on)
};

template <typename V>
__device__ __forceinline__ V from_bits(u64 b);
template <>
__device__ __forceinline__ double from_bits<double>(u64 b) { return __longlong_as_double((long long)b); }
template <>
__device__ __forceinline__ float from_bits<float>(u64 b) { return __uint_as_float((u32)b); }

template <typename V>
__device__ __forceinline__ u64 to_bits(V v);
template <>
__device__ __forceinline__ u64 to_bits<double>(double v) { return (u64)__double_as_longlong(v); }
template <>
__device__ __forceinline__ u64 to_bits<float>(float v) { return (u64)__float_as_uint(v); }

template <typename V>
__device__ __forceinline__ V sorted_lookup(const DevTable<V> &t, u64 key)
{
    if (t.n == 0) return V(0);
    u64 lo = 0, len = t.n;
    if (t.kind == INDEX_BUCKET) {
        if (t.prefix > 0 && (key >> (64 - t.prefix)) != t.prefix_value) return V(0);
        const u32 bk = (u32)((key << t.prefix) >> (64 - t.bits));
        const u32 b0 = __ldg(t.bucket + bk), b1 = __ldg(t.bucket + bk + 1);
        lo = b0;
        len = b1 - b0;
        if (len == 0) return V(0);
    }
    while (len > 1) {
        const u64 half = len >> 1;
        lo = (__ldg(t.keys + lo + half) <= key) ? lo + half : lo;
        len -= half;
    }
    return __ldg(t.keys + lo) == key ? __ldg(t.vals + lo) : V(0);
}

// continue a linear probe after the first slot missed (plain arguments: a
// reference to the kernel's table would force a copy of it to local memory)
template <typename V>
__device__ __noinline__ V hash_probe_rest(const ulonglong2 *slots, u64 cap, u64 key, u64 s)
{
    for (u64 i = 1; i < cap; i++) {
        s = (s + 1 == cap) ? 0 : s + 1;
        const ulonglong2 e = __ldg(slots + s);
        if (e.x == key) return from_bits<V>(e.y);
        if (e.x == 0) return V(0);
    }
    return V(0);
}

// continue a compact probe after the home slot held another key
template <typename V>
__device__ __noinline__ V compact_probe_rest(const u64 *slots, u64 cap, int dbits, u64 home, u32 tag0)
{
    const u32 last = (1u << dbits) - 1u;  // probe distances stay below it (the build checks)
    for (u32 d = 1; d + 1 < last; d++) {
        const u64 e = __ldg(slots + ((home + d) & (cap - 1)));
        if ((u32)e == tag0 + d) return from_bits<V>(e >> 32);
        if ((u32)e == 0u) return V(0);
    }
    return V(0);
}

template <typename V>
__device__ __forceinline__ V vmax(V a, V b) { return a > b ? a : b; }

template <typename V>
__device__ __forceinline__ V table_value(const DevTable<V> &t, u64 key)
{
    if (t.kind == INDEX_HASH && t.ch.on) {
        if ((key & t.ch.cmask) != t.ch.cval) return V(0);
        u32 tag0;
        const u64 h = compact_home(t.ch, key, &tag0);
        const u64 e = __ldg((const u64 *)t.slots + h);
        if ((u32)e == tag0) return from_bits<V>(e >> 32);
        if ((u32)e == 0u) return V(0);
        return compact_probe_rest<V>((const u64 *)t.slots, t.cap, t.ch.dbits, h, tag0);
    }
    if (t.kind == INDEX_HASH) {
        if (t.cap == 0) return V(0);
        const u64 s = home_slot(key, t.cap);
        const ulonglong2 e = __ldg(t.slots + s);
        if (e.x == key) return from_bits<V>(e.y);
        if (e.x == 0) return V(0);
        return hash_probe_rest<V>(t.slots, t.cap, key, s);
    }
    return sorted_lookup(t, key);
}

__device__ __forceinline__ void add_probes(u32 probes, u64 *counter)
{
    const u32 w = __reduce_add_sync(0xffffffffu, probes);
    if ((threadIdx.x & 31) == 0 && w) atomicAdd((unsigned long long *)counter, (unsigned long long)w);
}

__device__ __forceinline__ bool satisfied(u64 b, const SolveRules &r)
{
    if (r.nox && !r.score) return has_tile(b, r.nox);
    if (r.score) return false;
    int lo = 0, hi = r.n_winstates;
    if (r.fid) {
        const u32 f = __ldg(r.fid + fixed_pattern(b));
        if (f == 0xFF) return false;
        lo = (int)__ldg(r.ws_begin + f);
        hi = (int)__ldg(r.ws_begin + f + 1);
    }
    for (int i = lo; i < hi; i++)
        if (matches(b, __ldg(r.winstates + i))) return true;
    return false;
}

__device__ __forceinline__ void stage_table_s(unsigned char *smem, const unsigned short *g_move)
{
    const uint4 *src = (const uint4 *)g_move;
    uint4 *dst = (uint4 *)smem;
    for (int i = threadIdx.x; i < TABLE_BYTES_S / 16; i += blockDim.x) dst[i] = __ldg(src + i);
    __syncthreads();
}

// Spawn-weighted mean of one board from its per-cell best values, in cell
// order (src/solve.c:257-281): FP64 adds in order, FP32 Kahan-compensated sums;
// the weighted mean is formed in FP64 and rounded once.
template <typename V>
struct SpawnSums {
    V s2 = 0, s4 = 0, c2 = 0, c4 = 0;
    __device__ __forceinline__ void add(V best2, V best4)
    {
        if constexpr (sizeof(V) == 8) {  // cell order, plain IEEE adds
            s2 = __dadd_rn(s2, best2);
            s4 = __dadd_rn(s4, best4);
        } else {  // Kahan-compensated
            const float y2 = __fsub_rn(best2, c2), u2 = __fadd_rn(s2, y2);
            c2 = __fsub_rn(__fsub_rn(u2, s2), y2);
            s2 = u2;
            const float y4 = __fsub_rn(best4, c4), u4 = __fadd_rn(s4, y4);
            c4 = __fsub_rn(__fsub_rn(u4, s4), y4);
            s4 = u4;
        }
    }
    __device__ __forceinline__ V result(int spaces, u64 b, const SolveRules &r) const
    {
        double d = 0.0;
        if (spaces) {
            const double k = (double)spaces;
            const double S2 = (double)s2 - (double)c2, S4 = (double)s4 - (double)c4;
            d = __dadd_rn(__ddiv_rn(__dmul_rn(0.9, S2), k), __ddiv_rn(__dmul_rn(0.1, S4), k));
        }
        if (r.score && d == 0.0) d = (double)tile_sum(b);
        return (V)d;
    }
};

// Direct variant: one thread per board, no queue.  The eight successors of
// one cell (2 spawns x 4 moves) are formed from the board's four views (the
// spawned nibble is OR-ed into each view), canonicalised and probed together,
// so a thread keeps up to eight independent loads in flight.
constexpr int DIRECT_THREADS = 1024;

template <typename V>
__device__ __forceinline__ void probe4(const DevTable<V> &t, const u64 *key, u32 legal, V *out)
{
    if (t.kind == INDEX_HASH && t.ch.on) {
        u64 h[4], e[4];
        u32 tag[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const bool on = (legal >> j) & 1 && (key[j] & t.ch.cmask) == t.ch.cval;
            h[j] = compact_home(t.ch, key[j], &tag[j]);
            e[j] = on ? __ldg((const u64 *)t.slots + h[j]) : 0ull;
        }
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if ((u32)e[j] == tag[j]) out[j] = from_bits<V>(e[j] >> 32);
            else if ((u32)e[j] == 0u) out[j] = V(0);
            else out[j] = compact_probe_rest<V>((const u64 *)t.slots, t.cap, t.ch.dbits, h[j], tag[j]);
        }
        return;
    }
    if (t.kind == INDEX_HASH) {
        u64 s[4];
        ulonglong2 e[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const bool on = (legal >> j) & 1 && t.cap;
            s[j] = on ? home_slot(key[j], t.cap) : 0;
            e[j] = on ? __ldg(t.slots + s[j]) : make_ulonglong2(0, 0);
        }
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if (!((legal >> j) & 1) || e[j].x == 0) out[j] = V(0);
            else if (e[j].x == key[j]) out[j] = from_bits<V>(e[j].y);
            else out[j] = hash_probe_rest<V>(t.slots, t.cap, key[j], s[j]);
        }
    } else {
#pragma unroll
        for (int j = 0; j < 4; j++) out[j] = ((legal >> j) & 1) ? sorted_lookup(t, key[j]) : V(0);
    }
}

// The best values of one empty cell: its eight successors (2 and 4 spawned
// into each of the board's four views, then the left move), canonicalised --
// over the plan's images when PLANNED, which the caller picks once per warp so
// that the image choice is a uniform branch -- and looked up in the s+2 and s+4
// tables, eight loads in flight.
template <bool PLANNED, typename V>
__device__ __forceinline__ void cell_bests(const RowTable &rt, const u64 v[4], int cell, const CanonPlan &plan,
                                           const DevTable<V> &t2, const DevTable<V> &t4, V &best2, V &best4,
                                           u32 &probes)
{
    u64 k2[4], k4[4];
    u32 l2 = 0, l4 = 0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const int sh = 60 - 4 * view_cell(k, cell);
        u64 m;
        if (move_left(rt, v[k] | (1ull << sh), &m) == 2) l2 |= 1u << k;
        k2[k] = PLANNED ? canon_cand(m, plan.cand(k)) : canonical(m);
        if (move_left(rt, v[k] | (2ull << sh), &m) == 2) l4 |= 1u << k;
        k4[k] = PLANNED ? canon_cand(m, plan.cand(k)) : canonical(m);
    }
    probes += __popc(l2) + __popc(l4);
    V p2[4], p4[4];
    probe4(t2, k2, l2, p2);
    probe4(t4, k4, l4, p4);
    best2 = vmax(vmax(p2[0], p2[1]), vmax(p2[2], p2[3]));
    best4 = vmax(vmax(p4[0], p4[1]), vmax(p4[2], p4[3]));
}

// One probe of a table (the successor is looked up only when its move was legal).
template <typename V>
__device__ __forceinline__ V probe1(const DevTable<V> &t, u64 key, bool legal)
{
    if (!legal) return V(0);
    if (t.kind == INDEX_HASH && t.ch.on) {
        if ((key & t.ch.cmask) != t.ch.cval) return V(0);
        u32 tag0;
        const u64 h = compact_home(t.ch, key, &tag0);
        const u64 e = __ldg((const u64 *)t.slots + h);
        if ((u32)e == tag0) return from_bits<V>(e >> 32);
        if ((u32)e == 0u) return V(0);
        return compact_probe_rest<V>((const u64 *)t.slots, t.cap, t.ch.dbits, h, tag0);
    }
    if (t.kind == INDEX_HASH) {
        if (t.cap == 0) return V(0);
        const u64 s = home_slot(key, t.cap);
        const ulonglong2 e = __ldg(t.slots + s);
        if (e.x == key) return from_bits<V>(e.y);
        if (e.x == 0) return V(0);
        return hash_probe_rest<V>(t.slots, t.cap, key, s);
    }
    return sorted_lookup(t, key);
}

// cell_bests with the four views in a loop that is not unrolled: one view's two
// successors per iteration, a quarter of the code (the unrolled body of all
// eight successors is large enough that warps wait on instruction fetch).  Both
// successors' first slots are loaded before either is looked at: 1.06 -> 0.96 ms
// for 5M LL boards, the kernel being bound by the latency of these loads.
//
// The views k0, k0 + step, ... only (all: 0 and 1); with step 4 the one view's values.
template <int FORM, typename V>
__device__ __forceinline__ void cell_bests_rolled(const RowTable &rt, u64 b, int cell, const CanonPlan &plan,
                                                  const DevTable<V> &t2, const DevTable<V> &t4, V &best2, V &best4,
                                                  u32 &probes, int k0, int step)
{
    const Half h = halves(b), t = transpose(h);
    const int r0 = cell >> 2, q0 = cell & 3;
    best2 = V(0);
    best4 = V(0);
    const bool wide = t2.kind == INDEX_HASH && t4.kind == INDEX_HASH && !t2.ch.on && !t4.ch.on;
    const bool compact = sizeof(V) == 4 && t2.kind == INDEX_HASH && t4.kind == INDEX_HASH && t2.ch.on && t4.ch.on;
#pragma unroll 1
    for (int k = k0; k < 4; k += step) {
        // view k: id, H, T, H.T; the cell of the spawn in it
        const Half x = (k & 2) ? t : h;
        const u64 y = (k & 1) ? whole(flip_h(x)) : whole(x);
        const int row = (k & 2) ? q0 : r0;
        const int col = ((k & 2) ? r0 : q0) ^ ((k & 1) ? 3 : 0);
        const int sh = 60 - 4 * (4 * row + col);
        u64 m2, m4;
        const bool ok2 = move_left(rt, y | (1ull << sh), &m2) == 2;
        const bool ok4 = move_left(rt, y | (2ull << sh), &m4) == 2;
        const u64 c2 = canon_planned<FORM>(m2, plan, k);
        const u64 c4 = canon_planned<FORM>(m4, plan, k);
        probes += (u32)ok2 + (u32)ok4;
        V v2 = V(0), v4 = V(0);
        if (wide) {
            const u64 s2 = home_slot(c2, t2.cap), s4 = home_slot(c4, t4.cap);
            ulonglong2 e2 = make_ulonglong2(0, 0), e4 = e2;
            if (ok2) e2 = __ldg(t2.slots + s2);
            if (ok4) e4 = __ldg(t4.slots + s4);
            v2 = from_bits<V>(e2.y);
            v4 = from_bits<V>(e4.y);
            // an empty slot (and a move that was not looked up) holds key 0 and value 0
            if (e2.x != c2) v2 = e2.x == 0 ? V(0) : hash_probe_rest<V>(t2.slots, t2.cap, c2, s2);
            if (e4.x != c4) v4 = e4.x == 0 ? V(0) : hash_probe_rest<V>(t4.slots, t4.cap, c4, s4);
        } else if (compact) {
            u32 g2, g4;
            const u64 s2 = compact_home(t2.ch, c2, &g2), s4 = compact_home(t4.ch, c4, &g4);
            u64 e2 = 0, e4 = 0;
            if (ok2 && (c2 & t2.ch.cmask) == t2.ch.cval) e2 = __ldg((const u64 *)t2.slots + s2);
            if (ok4 && (c4 & t4.ch.cmask) == t4.ch.cval) e4 = __ldg((const u64 *)t4.slots + s4);
            v2 = from_bits<V>(e2 >> 32);
            v4 = from_bits<V>(e4 >> 32);
            if ((u32)e2 != g2)
                v2 = (u32)e2 == 0u ? V(0)
                                   : compact_probe_rest<V>((const u64 *)t2.slots, t2.cap, t2.ch.dbits, s2, g2);
            if ((u32)e4 != g4)
                v4 = (u32)e4 == 0u ? V(0)
                                   : compact_probe_rest<V>((const u64 *)t4.slots, t4.cap, t4.ch.dbits, s4, g4);
        } else {
            v2 = probe1(t2, c2, ok2);
            v4 = probe1(t4, c4, ok4);
        }
        best2 = step == 4 ? v2 : vmax(best2, v2);
        best4 = step == 4 ? v4 : vmax(best4, v4);
    }
}

template <typename V>
__global__ void __launch_bounds__(DIRECT_THREADS, 1) solve_direct_kernel(const u64 *__restrict__ keys, u64 n,
                                                                         V *__restrict__ out, DevTable<V> t2,
                                                                         DevTable<V> t4, SolveRules r,
                                                                         const unsigned short *g_move,
                                                                         u64 *probes_out, CanonPlan plan)
{
    extern __shared__ __align__(16) unsigned char smem[];
    stage_table_s(smem, g_move);
    const RowTable rt{(const unsigned short *)smem};
    u32 probes = 0;
    for (u64 i = (u64)blockIdx.x * DIRECT_THREADS + threadIdx.x; i < n; i += (u64)gridDim.x * DIRECT_THREADS) {
        const u64 b = keys[i];
        // the images that can be canonical: the plan's when every board of the warp has its mask
        const bool planned = __all_sync(__activemask(), fixed_pattern(b) == plan.mask);
        V res;
        if (satisfied(b, r)) {
            res = V(1);
        } else {
            u64 e = empty_mask(b);
            const int spaces = popc64(e);
            u64 v[4];
            views(b, v);
            SpawnSums<V> sums;
            while (e) {  // cells in order 0..15 = highest nibble first
                const int bit = 63 - __clzll(e);
                e &= ~(1ull << bit);
                const int cell = (60 - bit) >> 2;
                V best2, best4;
                if (planned) cell_bests<true>(rt, v, cell, plan, t2, t4, best2, best4, probes);
                else cell_bests<false>(rt, v, cell, plan, t2, t4, best2, best4, probes);
                sums.add(best2, best4);
            }
            res = sums.result(spaces, b, r);
        }
        out[i] = res;
    }
    add_probes(probes, probes_out);
}

// ---- insertion into a hash index ---------------------------------------------
template <typename V>
__device__ __forceinline__ bool insert_wide(ulonglong2 *slots, u64 cap, u64 key, V val)
{
    u64 s = home_slot(key, cap);
    for (u64 p = 0; p < cap; p++) {
        if (atomicCAS((unsigned long long *)&slots[s].x, 0ull, (unsigned long long)key) == 0ull) {
            slots[s].y = to_bits<V>(val);
            return true;
        }
        s = (s + 1 == cap) ? 0 : s + 1;
    }
    return false;
}

// false when the probe distance runs past what the tag holds
__device__ __forceinline__ bool insert_compact(unsigned long long *slots, u64 cap, const CompactHash &c, u64 key, float val)
{
    const u32 last = (1u << c.dbits) - 1u;
    u32 tag0;
    const u64 h = compact_home(c, key, &tag0), vbits = (u64)__float_as_uint(val) << 32;
    for (u32 d = 0; d + 1 < last; d++)
        if (atomicCAS(slots + ((h + d) & (cap - 1)), 0ull, (unsigned long long)(vbits | (tag0 + d))) == 0ull) return true;
    return false;
}

// The index that a solve fills with the boards it solves: none, 16-byte or 8-byte
// slots, cleared before.
enum : int { FILL_NONE = 0, FILL_WIDE = 1, FILL_COMPACT = 2 };
struct IndexFill {
    int kind = FILL_NONE;
    void *slots = nullptr;
    u64 cap = 0;
    CompactHash ch;
    u32 *err = nullptr;
    template <typename V>
    __device__ __forceinline__ void add(u64 key, V val) const
    {
        bool placed = true;
        if (kind == FILL_WIDE) placed = insert_wide((ulonglong2 *)slots, cap, key, val);
        else if (sizeof(V) == 4 && kind == FILL_COMPACT)
            placed = insert_compact((unsigned long long *)slots, cap, ch, key, (float)val);
        if (!placed) atomicOr(err, ERR_CAPACITY);
    }
};

// Item form: the work of a warp is its boards' (board, empty cell) pairs, not
// its boards.  Boards have 0..16 empty cells, so one thread per board leaves a
// warp waiting on its fullest board; here the 32 lanes take the pairs of 32
// boards 32 at a time, every lane busy except in the last round.  A pair forms
// the eight successors of its cell (2 spawns x 4 moves, from the owner's four
// views), canonicalises them over the images its CanonPlan allows, probes the
// s+2 and s+4 tables, and leaves the two best values in shared memory; the
// owning lane then adds its pairs' values in cell order.
constexpr int ITEM_THREADS = 1024;
constexpr int ITEM_WARPS = ITEM_THREADS / 32;
constexpr int ITEM_MAX = 32 * 16;  // pairs of 32 boards at most
template <typename V>
constexpr int item_smem() { return TABLE_BYTES_S + ITEM_WARPS * (ITEM_MAX * 2 + 2 * 32 * (int)sizeof(V)); }

//
// With VIEWS, for layers that leave the chip idle, four lanes share a pair, one view
// each: the chain of four views, a move, a canonical form and a probe each, is what
// such a layer's solve takes.  Every lane then takes the maximum of the four values in
// the views' order, as one lane does, so that a NaN of a given table counts the same.
template <typename V, int FORM, bool VIEWS>
__global__ void __launch_bounds__(ITEM_THREADS, 1)
    solve_items_kernel(const u64 *__restrict__ keys, u64 n, V *__restrict__ out, DevTable<V> t2, DevTable<V> t4,
                       SolveRules r, const unsigned short *g_move, u64 *probes_out, CanonPlan plan, u32 per,
                       IndexFill fill)
{
    extern __shared__ __align__(16) unsigned char smem[];
    stage_table_s(smem, g_move);
    const RowTable rt{(const unsigned short *)smem};
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned short *items = (unsigned short *)(smem + TABLE_BYTES_S) + warp * ITEM_MAX;  // (lane << 4) | cell
    V *best_sh = (V *)(smem + TABLE_BYTES_S + ITEM_WARPS * ITEM_MAX * 2) + warp * 64;   // [2][32]
    u32 probes = 0;
    const u64 stride = (u64)gridDim.x * ITEM_WARPS * per;
    for (u64 base = ((u64)blockIdx.x * ITEM_WARPS + warp) * per; base < n; base += stride) {
        const u64 i = base + lane;
        const bool active = lane < (int)per && i < n;
        const u64 b = active ? keys[i] : 0;
        const bool sat = active && satisfied(b, r);
        u64 e = (active && !sat) ? empty_mask(b) : 0;
        const int spaces = popc64(e);
        const u32 inc = warp_inclusive_scan((u32)spaces);
        const u32 off = inc - (u32)spaces;
        const u32 total = __shfl_sync(0xffffffffu, inc, 31);
        // this board's pairs, cells in order 0..15 (highest nibble first)
        for (u32 j = off; e; j++) {
            const int bit = 63 - __clzll(e);
            e &= ~(1ull << bit);
            items[j] = (unsigned short)((lane << 4) | ((60 - bit) >> 2));
        }
        // the images that can be canonical: the plan's when every board of the batch has its mask
        const bool planned = __all_sync(0xffffffffu, !active || fixed_pattern(b) == plan.mask);
        __syncwarp();
        SpawnSums<V> sums;
        constexpr u32 PAIRS = VIEWS ? 8 : 32;  // of a round
        for (u32 r0 = 0; r0 < total; r0 += PAIRS) {
            const u32 j = r0 + (u32)lane / (32 / PAIRS);
            const bool has = j < total;
            const u32 it = has ? items[j] : 0u;
            const int owner = (int)(it >> 4), cell = (int)(it & 15u);
            const u64 ob = __shfl_sync(0xffffffffu, b, owner);
            V best2 = 0, best4 = 0;
            if (has) {
                const int k0 = VIEWS ? lane & 3 : 0, step = VIEWS ? 4 : 1;
                if (planned) cell_bests_rolled<FORM>(rt, ob, cell, plan, t2, t4, best2, best4, probes, k0, step);
                else cell_bests_rolled<-1>(rt, ob, cell, plan, t2, t4, best2, best4, probes, k0, step);
            }
            if (VIEWS) {
                const V v2 = best2, v4 = best4;
                best2 = best4 = V(0);
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    best2 = vmax(best2, __shfl_sync(0xffffffffu, v2, (lane & ~3) | k));
                    best4 = vmax(best4, __shfl_sync(0xffffffffu, v4, (lane & ~3) | k));
                }
            }
            best_sh[j - r0] = best2;
            best_sh[32 + j - r0] = best4;
            __syncwarp();
            // the owner adds the pairs of this round that are its own, in cell order
            const u32 lo = off > r0 ? off : r0;
            const u32 hi = (off + (u32)spaces) < r0 + PAIRS ? off + (u32)spaces : r0 + PAIRS;
            for (u32 q = lo; q < hi; q++) sums.add(best_sh[q - r0], best_sh[32 + q - r0]);
            __syncwarp();
        }
        if (active) {
            const V val = sat ? V(1) : sums.result(spaces, b, r);
            out[i] = val;
            fill.add(b, val);
        }
        __syncwarp();
    }
    add_probes(probes, probes_out);
}

// ---- index construction ----------------------------------------------------
__global__ void bucket_offsets_kernel(const u64 *__restrict__ keys, u64 n, u32 *__restrict__ off, int prefix,
                                      int bits)
{
    const u64 nb = 1ull << bits;
    for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i <= n; i += (u64)gridDim.x * blockDim.x) {
        const u64 bk = i < n ? (keys[i] << prefix) >> (64 - bits) : nb;
        const u64 bp = i ? (keys[i - 1] << prefix) >> (64 - bits) : 0;
        const u64 from = i ? bp + 1 : 0;
        for (u64 j = from; j <= bk && j <= nb; j++) off[j] = (u32)i;
    }
}

template <typename V>
__global__ void hash_build_kernel(const u64 *__restrict__ keys, const V *__restrict__ vals, u64 n,
                                  ulonglong2 *slots, u64 cap, u32 *err)
{
    for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x) {
        if (!insert_wide(slots, cap, keys[i], vals[i])) atomicOr(err, ERR_CAPACITY);
    }
}

// AND and OR over the keys, as the bits that are 0 in some key (bits[0]) and 1 in
// some key (bits[1]), which start at zero
__global__ void key_bits_kernel(const u64 *__restrict__ keys, u64 n, unsigned long long *bits)
{
    u64 z = 0, o = 0;
    for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x) {
        const u64 k = keys[i];
        z |= ~k;
        o |= k;
    }
    for (int d = 16; d; d >>= 1) {
        z |= __shfl_xor_sync(0xffffffffu, z, d);
        o |= __shfl_xor_sync(0xffffffffu, o, d);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicOr(bits, (unsigned long long)z);
        atomicOr(bits + 1, (unsigned long long)o);
    }
}

__global__ void compact_build_kernel(const u64 *__restrict__ keys, const float *__restrict__ vals, u64 n,
                                     unsigned long long *slots, CompactHash c, u64 cap, u32 *err)
{
    for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x)
        // where this fails the host falls back to 16-byte slots
        if (!insert_compact(slots, cap, c, keys[i], vals[i])) atomicOr(err, ERR_CAPACITY);
}

// ---- region-partitioned build of the 16-byte-slot index ----------------------
// The atomic build inserts every key with a compare-and-swap on a random slot of
// a table that was zeroed first: a random read-modify-write per key.  This form
// partitions the keys by region of their home slot (1024 slots = 16 KiB), builds
// each region in shared memory and writes it out whole: the table is written
// once, sequentially, and never zeroed.  A key whose linear probe runs past its
// region's end (or whose region's bucket is full) goes to an overflow list,
// inserted afterwards into the finished table with the atomic probe from its
// home slot; the slots a placed key skipped were taken when it was placed and
// stay taken, so every key stays reachable by the linear probe from its home.
constexpr u32 BUILD_REGION = 1024;
// u32 words from one region's cursor to the next: a sector each, which spreads
// the atomic adds over the L2 slices
constexpr u32 CURSOR_PAD = 8;

// Each region owns a bucket of `bcap` pairs in the scratch (the mean count of
// a region plus eight standard deviations and a margin, so that a bucket runs
// full almost never); a pair that finds its bucket full joins the overflow
// list.  Four keys per thread per step keep four cursor atomics in flight.
// Measured over 12.2M keys (two LL layers, FP64, scatter and build): cursors side
// by side and 2048-slot regions in CTAs of 512 threads 506 us, a sector per cursor
// 477 us, and 1024-slot regions in CTAs of 256, whose clearing, filling and
// writing overlap more, 465 us; eight keys per step gave nothing.
template <typename V>
__global__ void __launch_bounds__(256) region_scatter_kernel(const u64 *__restrict__ keys, const V *__restrict__ vals,
                                                             u64 n, u64 cap, u32 bcap, u32 *cursor,
                                                             ulonglong2 *tmp, ulonglong2 *overflow, u32 max_over,
                                                             u32 *n_over, u32 *err)
{
    constexpr int U = 4;
    const u64 stride = (u64)gridDim.x * blockDim.x;
    for (u64 i0 = (u64)blockIdx.x * blockDim.x + threadIdx.x; i0 < n; i0 += U * stride) {
        u64 key[U];
        V val[U];
        u32 r[U], p[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const u64 i = i0 + u * stride;
            key[u] = i < n ? keys[i] : 0ull;
            val[u] = i < n ? vals[i] : V(0);
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            r[u] = (u32)(home_slot(key[u], cap) / BUILD_REGION);
            p[u] = i0 + u * stride < n ? atomicAdd(cursor + r[u] * CURSOR_PAD, 1u) : 0u;
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            if (i0 + u * stride >= n) continue;
            const ulonglong2 e = make_ulonglong2(key[u], to_bits<V>(val[u]));
            if (p[u] < bcap) {
                tmp[(u64)r[u] * bcap + p[u]] = e;
            } else {
                const u32 k = atomicAdd(n_over, 1u);
                if (k < max_over) overflow[k] = e;
                else atomicOr(err, ERR_CAPACITY);
            }
        }
    }
}

__global__ void __launch_bounds__(256) region_build_kernel(const ulonglong2 *__restrict__ tmp,
                                                           const u32 *__restrict__ cursor, u32 bcap, u32 nreg,
                                                           u64 cap, ulonglong2 *slots, ulonglong2 *overflow,
                                                           u32 max_over, u32 *n_over, u32 *err)
{
    __shared__ ulonglong2 tab[BUILD_REGION];
    for (u32 r = blockIdx.x; r < nreg; r += gridDim.x) {
        for (u32 j = threadIdx.x; j < BUILD_REGION; j += blockDim.x) tab[j] = make_ulonglong2(0, 0);
        __syncthreads();
        const u64 base = (u64)r * BUILD_REGION;
        const u32 len = (u32)min((u64)BUILD_REGION, cap - base);
        const u32 cnt = min(cursor[r * CURSOR_PAD], bcap);
        const ulonglong2 *bucket = tmp + (u64)r * bcap;
        for (u32 j = threadIdx.x; j < cnt; j += blockDim.x) {
            const ulonglong2 e = bucket[j];
            bool placed = false;
            for (u32 sl = (u32)(home_slot(e.x, cap) - base); sl < len; sl++) {
                if (atomicCAS((unsigned long long *)&tab[sl].x, 0ull, (unsigned long long)e.x) == 0ull) {
                    tab[sl].y = e.y;
                    placed = true;
                    break;
                }
            }
            if (!placed) {
                const u32 k = atomicAdd(n_over, 1u);
                if (k < max_over) overflow[k] = e;
                else atomicOr(err, ERR_CAPACITY);
            }
        }
        __syncthreads();
        for (u32 j = threadIdx.x; j < len; j += blockDim.x) slots[base + j] = tab[j];
        __syncthreads();
    }
}

// the overflow keys, inserted into the finished table by the atomic linear probe
__global__ void overflow_insert_kernel(const ulonglong2 *__restrict__ over, const u32 *n_over, u32 max_over,
                                       ulonglong2 *slots, u64 cap, u32 *err)
{
    const u32 n = min(*n_over, max_over);
    for (u32 i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const ulonglong2 e = over[i];
        if (!insert_wide(slots, cap, e.x, __longlong_as_double((long long)e.y))) atomicOr(err, ERR_CAPACITY);
    }
}

static int grid_for(u64 n, int threads, int per_sm)
{
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms <= 0) sms = NUM_SMS_B200;
    const u64 need = (n + threads - 1) / threads;
    return (int)std::max<u64>(1, std::min<u64>(need, (u64)sms * per_sm));
}

bool ensure_storage(IndexStorage &st, u64 bytes, cudaStream_t s)
{
    if (st.bytes >= bytes && st.p) return true;
    if (st.p) dev_free(st.p, s);
    st.p = nullptr;
    st.bytes = 0;
    if (!dev_alloc(&st.p, bytes, s)) return false;
    st.bytes = bytes;
    return true;
}

bool key_bits(const KeySet &a, const KeySet &b, KeyBits *bits, const u64 *first, Counters &c, cudaStream_t s)
{
    // device words 16..19: the two sets' bits, 20: the first key of *first
    static u64 *host = nullptr;
    if (!host && !CGB_CUDA(cudaHostAlloc((void **)&host, 5 * sizeof(u64), cudaHostAllocDefault))) return false;
    u64 *d = c.d + 16;
    if (!CGB_CUDA(cudaMemsetAsync(d, 0, 4 * sizeof(u64), s))) return false;
    if (first && !CGB_CUDA(cudaMemcpyAsync(d + 4, first, sizeof(u64), cudaMemcpyDeviceToDevice, s))) return false;
    if (a.n) key_bits_kernel<<<grid_for(a.n, 256, 8), 256, 0, s>>>(a.keys, a.n, (unsigned long long *)d);
    if (b.n) key_bits_kernel<<<grid_for(b.n, 256, 8), 256, 0, s>>>(b.keys, b.n, (unsigned long long *)(d + 2));
    if (!CGB_CUDA(cudaGetLastError()) || !words_to_host((u32 *)host, (const u32 *)d, 10, s) ||
        !CGB_CUDA(cudaStreamSynchronize(s)))
        return false;
    for (int i = 0; i < 2; i++)
        if (i ? b.n : a.n) bits[i] = KeyBits{~host[2 * i], host[2 * i + 1], true};
    if (first) bits[2].any = host[4];
    return true;
}

int g_hash_compact = 1;  // FP32 hash tables in 8-byte slots where the keys allow it

// a begun build's error word, on the device and its pinned copy, by ix.slot
static u32 *h_index_err = nullptr;
static u32 *index_err(const LayerIndex &ix, Counters &c) { return (u32 *)(c.d + 40 + ix.slot); }

// a cleared table of 8-byte slots for ix, where its keys allow one (ix.kind says so)
static bool start_compact(LayerIndex &ix, IndexStorage &st, Counters &c, cudaStream_t s, const KeyBits &bits)
{
    int cbits = 0;
    const CompactHash ch = plan_compact(bits.all, bits.any, ix.n, &cbits);
    if (!ch.on) return true;
    const u64 cap = 1ull << cbits;
    if (!ensure_storage(st, cap * 8, s)) return false;
    if (!CGB_CUDA(cudaMemsetAsync(st.p, 0, cap * 8, s))) return false;
    if (!CGB_CUDA(cudaMemsetAsync(index_err(ix, c), 0, sizeof(u32), s))) return false;
    ix.kind = INDEX_HASH;
    ix.slots = st.p;
    ix.cap = cap;
    ix.ch = ch;
    return true;
}

// launches the build of the 8-byte-slot index of an FP32 layer: AND/OR of the keys
// give the constant bytes; the table is the power of two at or above twice the
// layer; the tag holds the remainder bits (at most 26) and the probe distance.
// Leaves ix.kind == INDEX_BISECT (nothing launched) when the keys vary in too
// many bytes.
static bool begin_compact(LayerIndex &ix, IndexStorage &st, Counters &c, cudaStream_t s, KeyBits bits)
{
    if (!bits.known && !key_bits(KeySet{ix.keys, ix.n}, KeySet{}, &bits, nullptr, c, s)) return false;
    if (!start_compact(ix, st, c, s, bits)) return false;
    if (ix.kind != INDEX_HASH) return true;
    kclock().begin(s, &kstats().index_ms);
    compact_build_kernel<<<grid_for(ix.n, 256, 16), 256, 0, s>>>(
        ix.keys, (const float *)ix.vals, ix.n, (unsigned long long *)st.p, ix.ch, ix.cap, index_err(ix, c));
    kclock().end(s);
    if (!CGB_CUDA(cudaGetLastError()) || !words_to_host(h_index_err + ix.slot, index_err(ix, c), 1, s))
        return false;
    ix.unchecked = true;
    return true;
}

// the region-partitioned build's cursors, buckets and overflow list, kept from one
// build to the next until index_release_scratch
static IndexStorage region_scratch;

int g_region_build = 1;  // 16-byte-slot indexes of 2^16..2^28 keys built region by region

// launches the region-partitioned build (above); the overflow keys are inserted
// by a kernel that reads their number, so nothing is waited for in between
static bool begin_regions(LayerIndex &ix, int vbytes, IndexStorage &st, Counters &c, cudaStream_t s)
{
    const u64 n = ix.n;
    const u64 cap = hash_capacity(n);
    const u32 nreg = (u32)((cap + BUILD_REGION - 1) / BUILD_REGION);
    const u32 max_over = (u32)(n / 32 + 4096);
    // bucket size: the mean pairs of a region plus eight standard deviations and a margin
    const double mean = (double)n * BUILD_REGION / (double)cap;
    const u32 bcap = (u32)((mean + 8.0 * sqrt(mean) + 64.0 + 15.0) / 16.0) * 16u;
    if (!ensure_storage(st, cap * 16, s)) return false;
    // scratch: the cursors and the overflow count (u32), the region buckets, the overflow list
    const u64 bytes = 4ull * nreg * CURSOR_PAD + 64 + 16ull * nreg * bcap + 16ull * max_over;
    if (!ensure_storage(region_scratch, bytes, s)) return false;
    u32 *cursor = (u32 *)region_scratch.p, *n_over = cursor + (u64)nreg * CURSOR_PAD;
    ulonglong2 *tmp = (ulonglong2 *)(((uintptr_t)(n_over + 1) + 15) & ~(uintptr_t)15);
    ulonglong2 *over = tmp + (u64)nreg * bcap;
    bool ok = CGB_CUDA(cudaMemsetAsync(cursor, 0, 4ull * nreg * CURSOR_PAD + 4, s)) && CGB_CUDA(cudaMemsetAsync(index_err(ix, c), 0, 4, s));
    if (ok) {
        kclock().begin(s, &kstats().index_ms);
        const int grid = grid_for((n + 3) / 4, 256, 8);
        if (vbytes == 8)
            region_scatter_kernel<double><<<grid, 256, 0, s>>>(ix.keys, (const double *)ix.vals, n, cap, bcap,
                                                                cursor, tmp, over, max_over, n_over, index_err(ix, c));
        else
            region_scatter_kernel<float><<<grid, 256, 0, s>>>(ix.keys, (const float *)ix.vals, n, cap, bcap,
                                                               cursor, tmp, over, max_over, n_over, index_err(ix, c));
        region_build_kernel<<<std::min<u32>(nreg, (u32)NUM_SMS_B200 * 8), 256, 0, s>>>(
            tmp, cursor, bcap, nreg, cap, (ulonglong2 *)st.p, over, max_over, n_over, index_err(ix, c));
        overflow_insert_kernel<<<NUM_SMS_B200, 256, 0, s>>>(over, n_over, max_over, (ulonglong2 *)st.p, cap, index_err(ix, c));
        kclock().end(s);
        kstats().launches += 2;
        ok = CGB_CUDA(cudaGetLastError()) &&
             words_to_host(h_index_err + ix.slot, index_err(ix, c), 1, s);
    }
    if (!ok) return false;
    ix.kind = INDEX_HASH;
    ix.slots = st.p;
    ix.cap = cap;
    ix.unchecked = true;
    return true;
}

void index_release_scratch(cudaStream_t s)
{
    dev_free(region_scratch.p, s);
    region_scratch = IndexStorage{};
}

// a cleared table of 16-byte slots for ix
static bool start_atomic(LayerIndex &ix, IndexStorage &st, cudaStream_t s)
{
    // load factor <= g_hash_load_pct: capacity rounded up to a multiple of 64 slots
    const u64 cap = hash_capacity(ix.n);
    if (!ensure_storage(st, cap * 16, s)) return false;
    if (!CGB_CUDA(cudaMemsetAsync(st.p, 0, cap * 16, s))) return false;
    ix.kind = INDEX_HASH;
    ix.slots = st.p;
    ix.cap = cap;
    return true;
}

// launches the atomic build into a zeroed table, which cannot fail: the table
// has more slots than keys
static bool begin_atomic(LayerIndex &ix, int vbytes, IndexStorage &st, Counters &c, cudaStream_t s)
{
    if (!start_atomic(ix, st, s)) return false;
    const u64 cap = ix.cap;
    kclock().begin(s, &kstats().index_ms);
    if (vbytes == 8)
        hash_build_kernel<double><<<grid_for(ix.n, 256, 16), 256, 0, s>>>(ix.keys, (const double *)ix.vals, ix.n,
                                                                         (ulonglong2 *)st.p, cap, index_err(ix, c));
    else
        hash_build_kernel<float><<<grid_for(ix.n, 256, 16), 256, 0, s>>>(ix.keys, (const float *)ix.vals, ix.n,
                                                                        (ulonglong2 *)st.p, cap, index_err(ix, c));
    kclock().end(s);
    if (!CGB_CUDA(cudaGetLastError())) return false;
    kstats().index_builds++;
    return true;
}

// ix without an index yet, which its `slot`-th error word belongs to
static bool reset_index(LayerIndex &ix, int slot)
{
    ix.slot = slot;
    ix.kind = INDEX_BISECT;
    ix.bucket = nullptr;
    ix.slots = nullptr;
    ix.cap = 0;
    ix.unchecked = false;
    ix.ch = CompactHash{};
    if (h_index_err) return true;
    void *h = nullptr;
    if (!CGB_CUDA(cudaHostAlloc(&h, INDEX_SLOTS * sizeof(u32), cudaHostAllocDefault))) return false;
    h_index_err = (u32 *)h;
    return true;
}

bool index_begin(LayerIndex &ix, int kind, int vbytes, IndexStorage &st, int bucket_bits, Counters &c, cudaStream_t s,
                 const KeyBits &bits, int slot)
{
    if (!reset_index(ix, slot)) return false;
    if (ix.n == 0 || kind == INDEX_BISECT) return true;
    if (kind == INDEX_HASH && vbytes == 4 && g_hash_compact && ix.n >= 64) {
        if (!begin_compact(ix, st, c, s, bits)) return false;
        if (ix.kind == INDEX_HASH) return true;
    }
    if (kind == INDEX_HASH && g_region_build && ix.n >= (1u << 16) && ix.n <= (1u << 28))
        return begin_regions(ix, vbytes, st, c, s);
    if (kind == INDEX_HASH) return begin_atomic(ix, vbytes, st, c, s);
    // INDEX_BUCKET
    if (ix.n < 64 || bucket_bits <= 0) return true;
    u64 first, last;
    if (!CGB_CUDA(cudaMemcpyAsync(&first, ix.keys, 8, cudaMemcpyDeviceToHost, s))) return false;
    if (!CGB_CUDA(cudaMemcpyAsync(&last, ix.keys + ix.n - 1, 8, cudaMemcpyDeviceToHost, s))) return false;
    if (!CGB_CUDA(cudaStreamSynchronize(s))) return false;
    const u64 x = first ^ last;
    const int prefix = x ? __builtin_clzll(x) : 64;
    int nb = bucket_bits;
    if (nb > 64 - prefix) nb = 64 - prefix;
    if (nb <= 0) return true;
    const u64 need = ((1ull << nb) + 1) * sizeof(u32);
    if (!ensure_storage(st, need, s)) return false;
    kclock().begin(s, &kstats().index_ms);
    bucket_offsets_kernel<<<grid_for(ix.n + 1, 256, 16), 256, 0, s>>>(ix.keys, ix.n, (u32 *)st.p, prefix, nb);
    kclock().end(s);
    if (!CGB_CUDA(cudaGetLastError())) return false;
    ix.kind = INDEX_BUCKET;
    ix.bucket = (const u32 *)st.p;
    ix.prefix = prefix;
    ix.bits = nb;
    ix.prefix_value = prefix ? first >> (64 - prefix) : 0;
    return true;
}

bool index_finish(LayerIndex &ix, int vbytes, IndexStorage &st, Counters &c, cudaStream_t s, bool *again)
{
    if (!ix.unchecked) return true;
    if (!CGB_CUDA(cudaStreamSynchronize(s))) return false;
    kclock().flush();
    ix.unchecked = false;
    if (h_index_err[ix.slot] == 0) {
        kstats().index_builds++;
        if (ix.ch.on) kstats().compact_index_builds++;
        return true;
    }
    // a probe ran past what the tag can hold: 16-byte slots; their overflow list ran
    // out: the atomic build
    if (again) *again = true;
    const bool was_compact = ix.ch.on != 0;
    ix.ch = CompactHash{};
    ix.kind = INDEX_BISECT;
    if (was_compact && g_region_build && ix.n >= (1u << 16) && ix.n <= (1u << 28))
        return begin_regions(ix, vbytes, st, c, s) && index_finish(ix, vbytes, st, c, s);
    return begin_atomic(ix, vbytes, st, c, s);
}

bool build_index(LayerIndex &ix, int kind, int vbytes, IndexStorage &st, int bucket_bits, Counters &c,
                 cudaStream_t s)
{
    return index_begin(ix, kind, vbytes, st, bucket_bits, c, s) && index_finish(ix, vbytes, st, c, s);
}

template <typename V>
static DevTable<V> dev_table(const LayerIndex &ix)
{
    DevTable<V> t;
    t.kind = ix.kind;
    t.keys = ix.keys;
    t.vals = (const V *)ix.vals;
    t.n = ix.n;
    t.bucket = ix.bucket;
    t.prefix = ix.prefix;
    t.bits = ix.bits;
    t.prefix_value = ix.prefix_value;
    t.slots = (const ulonglong2 *)ix.slots;
    t.cap = ix.kind == INDEX_HASH ? ix.cap : 0;
    t.ch = ix.ch;
    return t;
}

// layers of up to so many boards per warp of the chip give a pair four lanes: the solves
// of the 149 layers of a 2x4 table 3.06 -> 2.49 ms; limits of 1, 4 and 8 measured alike
constexpr u64 VIEWS_PER = 2;
int g_solve_variant = 1;  // 0: direct (one thread per board), 1: (board, cell) pairs per warp

template <typename V, int FORM>
static bool items_attr_one()
{
    const auto smem = cudaFuncAttributeMaxDynamicSharedMemorySize;
    return CGB_CUDA(cudaFuncSetAttribute(solve_items_kernel<V, FORM, false>, smem, item_smem<V>())) &&
           CGB_CUDA(cudaFuncSetAttribute(solve_items_kernel<V, FORM, true>, smem, item_smem<V>()));
}
template <typename V, bool VIEWS>
static auto items_kernel(int form)
{
    return form == CANON_ONE        ? solve_items_kernel<V, CANON_ONE, VIEWS>
           : form == CANON_DIAGONAL ? solve_items_kernel<V, CANON_DIAGONAL, VIEWS>
           : form == CANON_MIRROR   ? solve_items_kernel<V, CANON_MIRROR, VIEWS>
                                    : solve_items_kernel<V, CANON_LIST, VIEWS>;
}
template <typename V>
static bool items_attr()
{
    return items_attr_one<V, CANON_LIST>() && items_attr_one<V, CANON_ONE>() && items_attr_one<V, CANON_DIAGONAL>() &&
           items_attr_one<V, CANON_MIRROR>();
}

static bool solve_attrs()
{
    static bool attr = false;
    if (!attr) {
        if (!items_attr<double>() || !items_attr<float>() ||
            !CGB_CUDA(cudaFuncSetAttribute(solve_direct_kernel<double>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, TABLE_BYTES_S)) ||
            !CGB_CUDA(cudaFuncSetAttribute(solve_direct_kernel<float>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, TABLE_BYTES_S)))
            return false;
        attr = true;
    }
    return true;
}

// the kernel launch alone: no host round trip, so it may be captured in a graph
template <class V>
static void enqueue_solve(const u64 *keys, u64 n, V *out, const LayerIndex &t2, const LayerIndex &t4,
                          const SolveRules &r, const DeviceRowTable &rt, u64 *probes, cudaStream_t s,
                          const CanonPlan &plan, const IndexFill &fill = IndexFill{})
{
    if (g_solve_variant == 1) {
        // a warp takes `per` boards at a time: 32, fewer where the layer does not
        // give every warp of the chip that many, so that it spreads over the SMs and
        // one round of pairs serves a warp (2600 2x4 boards: 27 -> 18 us)
        const u64 warps = (u64)ITEM_WARPS * NUM_SMS_B200;
        const bool views = n <= VIEWS_PER * warps;
        u32 per = views ? 1 : 4;
        while (per < 32 && per * warps < n) per *= 2;
        const auto kernel = views ? items_kernel<V, true>(plan.form) : items_kernel<V, false>(plan.form);
        kernel<<<grid_for((n + per - 1) / per * 32, ITEM_THREADS, 1), ITEM_THREADS, item_smem<V>(), s>>>(
            keys, n, out, dev_table<V>(t2), dev_table<V>(t4), r, rt.move, probes, plan, per, fill);
    } else {
        solve_direct_kernel<V><<<grid_for(n, DIRECT_THREADS, 1), DIRECT_THREADS, TABLE_BYTES_S, s>>>(
            keys, n, out, dev_table<V>(t2), dev_table<V>(t4), r, rt.move, probes, plan);
    }
}

// An index is filled by the solve itself, a thread inserting the board whose value it
// has just formed: the insertions hide under the probes' latency, where a build of
// its own reads keys and values again and, for a small layer, costs a launch as
// long as the solve.  8-byte slots always; 16-byte slots up to so many keys: above,
// the table is far larger than L2, an insertion costs a sector read and written,
// and the build by regions wins.  Solve and index of a sweep, apart / filled: 149
// layers of 2x4 3.93 / 2.97 ms, dpdf FP32 (0.9M boards a layer) 5.17 / 4.17, LL to
// 120 (5M) 12.5 / 10.8, to 240 (12M) 95.2 / 94.5, to 330 (22M) 221 / 230; LL to
// 330 in 8-byte slots 220 / 205.
constexpr u64 FILL_KEYS = 1ull << 23;
static bool fills_wide(u64 n) { return g_solve_variant == 1 && n <= FILL_KEYS; }

constexpr int PROBES_AT = 12;  // counter word of the probes not collected yet

static bool solve_layer_launch(const u64 *keys, u64 n, void *out, int vbytes, const LayerIndex &t2, const LayerIndex &t4,
                               const SolveRules &r, const DeviceRowTable &rt, Counters &c, cudaStream_t s,
                               const CanonPlan &plan, const IndexFill &fill)
{
    if (n == 0) return true;
    if (!solve_attrs()) return false;
    kclock().begin(s, &kstats().solve_ms);
    if (vbytes == 4) enqueue_solve<float>(keys, n, (float *)out, t2, t4, r, rt, c.d + PROBES_AT, s, plan, fill);
    else enqueue_solve<double>(keys, n, (double *)out, t2, t4, r, rt, c.d + PROBES_AT, s, plan, fill);
    kclock().end(s);
    if (!CGB_CUDA(cudaGetLastError())) return false;
    KernelStats &k = kstats();
    k.solve_launches++;
    k.solve_boards += n;
    k.solve_bytes += (8 + vbytes) * n;  // keys in, values out; the probes' sectors follow
    return true;
}

bool solve_layer_launch(const u64 *keys, u64 n, void *out, int vbytes, const LayerIndex &t2, const LayerIndex &t4,
                        const SolveRules &r, const DeviceRowTable &rt, Counters &c, cudaStream_t s,
                        const CanonPlan &plan)
{
    return solve_layer_launch(keys, n, out, vbytes, t2, t4, r, rt, c, s, plan, IndexFill{});
}

bool solve_index_launch(LayerIndex &ix, int kind, int vbytes, IndexStorage &st, const LayerIndex &t2, const LayerIndex &t4,
                        const SolveRules &r, const DeviceRowTable &rt, Counters &c, cudaStream_t s, const CanonPlan &plan,
                        const KeyBits &bits, bool *indexed)
{
    *indexed = false;
    IndexFill fill;
    if (!reset_index(ix, 0)) return false;
    if (ix.n && kind == INDEX_HASH && g_solve_variant == 1) {
        if (vbytes == 4 && g_hash_compact && ix.n >= 64 && bits.known && !start_compact(ix, st, c, s, bits)) return false;
        if (ix.kind != INDEX_HASH && fills_wide(ix.n) && !start_atomic(ix, st, s)) return false;
        if (ix.kind == INDEX_HASH)
            fill = IndexFill{ix.ch.on ? FILL_COMPACT : FILL_WIDE, st.p, ix.cap, ix.ch, index_err(ix, c)};
    }
    if (!solve_layer_launch(ix.keys, ix.n, const_cast<void *>(ix.vals), vbytes, t2, t4, r, rt, c, s, plan, fill)) return false;
    if (fill.kind == FILL_NONE) return true;
    *indexed = true;
    if (fill.kind == FILL_WIDE) {
        kstats().index_builds++;
        return true;
    }
    ix.unchecked = true;
    return words_to_host(h_index_err + ix.slot, index_err(ix, c), 1, s);
}

bool solve_collect(Counters &c, cudaStream_t s)
{
    u64 &probes = c.host[Counters::HEAD];
    if (!words_to_host((u32 *)&probes, (const u32 *)(c.d + PROBES_AT), 2, s) ||
        !CGB_CUDA(cudaMemsetAsync(c.d + PROBES_AT, 0, sizeof(u64), s)) || !CGB_CUDA(cudaStreamSynchronize(s)))
        return false;
    kclock().flush();
    KernelStats &k = kstats();
    k.lookups += probes;
    k.solve_bytes += 64 * probes;  // one key sector and one value sector per probe
    return true;
}


bool solve_prepare() { return solve_attrs(); }

// target load factor of the hash index, percent; 0 = by size: 25 % (64 bytes
// of slots per board: fewer probes, measured 10 % faster solve + build on LL
// layers than 45 %) up to 2^27 keys, 45 % above, where table memory counts
int g_hash_load_pct = 0;

u64 hash_capacity(u64 n)
{
    const u64 pct = g_hash_load_pct ? (u64)g_hash_load_pct : (n <= (1ull << 27) ? 25 : 45);
    return hash_capacity_for(n, pct);
}

bool solve_index_enqueue(LayerIndex &ix, int vbytes, const LayerIndex &t2, const LayerIndex &t4, const SolveRules &r,
                         const DeviceRowTable &rt, u64 *probes, void *slots, u64 cap, u32 *err, cudaStream_t s)
{
    ix.ch = CompactHash{};
    ix.kind = INDEX_BISECT;
    ix.bucket = nullptr;
    ix.slots = nullptr;
    ix.cap = 0;
    if (ix.n == 0) return true;
    if (!solve_attrs() || !CGB_CUDA(cudaMemsetAsync(slots, 0, cap * 16, s))) return false;
    IndexFill fill;
    if (fills_wide(ix.n)) fill = IndexFill{FILL_WIDE, slots, cap, CompactHash{}, err};
    void *out = const_cast<void *>(ix.vals);
    if (vbytes == 4) enqueue_solve<float>(ix.keys, ix.n, (float *)out, t2, t4, r, rt, probes, s, CanonPlan{}, fill);
    else enqueue_solve<double>(ix.keys, ix.n, (double *)out, t2, t4, r, rt, probes, s, CanonPlan{}, fill);
    KernelStats &k = kstats();
    k.solve_launches++;
    k.solve_boards += ix.n;
    k.launches += fill.kind == FILL_NONE ? 2 : 1;
    if (fill.kind == FILL_NONE && vbytes == 8)
        hash_build_kernel<double><<<grid_for(ix.n, 256, 16), 256, 0, s>>>(ix.keys, (const double *)ix.vals, ix.n,
                                                                         (ulonglong2 *)slots, cap, err);
    else if (fill.kind == FILL_NONE)
        hash_build_kernel<float><<<grid_for(ix.n, 256, 16), 256, 0, s>>>(ix.keys, (const float *)ix.vals, ix.n,
                                                                        (ulonglong2 *)slots, cap, err);
    ix.kind = INDEX_HASH;
    ix.slots = slots;
    ix.cap = cap;
    return CGB_CUDA(cudaGetLastError());
}

bool solve_layer_f64(const u64 *keys, u64 n, double *out, const LayerIndex &t2, const LayerIndex &t4,
                     const SolveRules &r, const DeviceRowTable &rt, Counters &c, cudaStream_t s, const CanonPlan &plan)
{
    return n == 0 || (solve_layer_launch(keys, n, out, 8, t2, t4, r, rt, c, s, plan) && solve_collect(c, s));
}

bool solve_layer_f32(const u64 *keys, u64 n, float *out, const LayerIndex &t2, const LayerIndex &t4,
                     const SolveRules &r, const DeviceRowTable &rt, Counters &c, cudaStream_t s, const CanonPlan &plan)
{
    return n == 0 || (solve_layer_launch(keys, n, out, 4, t2, t4, r, rt, c, s, plan) && solve_collect(c, s));
}

// ---- batch lookup (lookup(), src/solve.c:108-164, for many boards) --------
constexpr u64 LOOKUP_FEW = 4096;  // boards up to which a warp takes each: every warp is resident at once

template <typename V>
__global__ void __launch_bounds__(256) lookup_batch_kernel(DevTable<V> t, const u64 *__restrict__ boards, u64 m,
                                                           int canon, double *__restrict__ out)
{
    for (u64 i = (u64)blockIdx.x * 256 + threadIdx.x; i < m; i += (u64)gridDim.x * 256) {
        const u64 b = boards[i];
        out[i] = (double)table_value(t, canon ? canonical(b) : b);
    }
}

// The same lookups by search in the sorted layer, without an index.
//
// A few boards: a warp per board, 31 keys probed at once, so that a layer of a
// million keys takes four dependent loads instead of twenty.
template <typename V>
__global__ void __launch_bounds__(256) lookup_few_kernel(const u64 *__restrict__ keys, const V *__restrict__ vals, u64 n,
                                                         const u64 *__restrict__ boards, u64 m, int canon,
                                                         double *__restrict__ out)
{
    const u32 lane = threadIdx.x & 31;
    const u64 warps = (u64)gridDim.x * (256 / 32);
    for (u64 i = ((u64)blockIdx.x * 256 + threadIdx.x) >> 5; i < m; i += warps) {
        const u64 b = boards[i], key = canon ? canonical(b) : b;
        u64 lo = 0, len = n;
        while (len > 32) {
            // 32 stretches; the last keys of the first 31 decide
            const u64 step = (len + 31) / 32, at = (lane + 1) * step - 1;
            const bool below = lane < 31 && at < len && __ldg(keys + lo + at) < key;
            const u64 skip = __popc(__ballot_sync(0xffffffffu, below)) * step;
            lo += skip;
            len = min(step, len - skip);
        }
        const u32 hit = __ballot_sync(0xffffffffu, lane < len && __ldg(keys + lo + lane) == key);
        if (lane == 0) out[i] = hit ? (double)__ldg(vals + lo + __ffs(hit) - 1) : 0.0;
    }
}

// Many boards: a thread per board; the first ten halvings run over 1024 evenly
// spaced keys in shared memory.
constexpr u32 LOOKUP_TOP = 1024;
template <typename V>
__global__ void __launch_bounds__(256) lookup_search_kernel(const u64 *__restrict__ keys, const V *__restrict__ vals,
                                                            u64 n, const u64 *__restrict__ boards, u64 m, int canon,
                                                            double *__restrict__ out)
{
    __shared__ u64 top[LOOKUP_TOP];
    const u64 step = (n + LOOKUP_TOP - 1) / LOOKUP_TOP;  // top[j] = the first key of stretch j
    for (u32 j = threadIdx.x; j < LOOKUP_TOP; j += 256) top[j] = j * step < n ? __ldg(keys + j * step) : ~0ull;
    __syncthreads();
    const u32 stretches = (u32)((n + step - 1) / step);
    for (u64 i = (u64)blockIdx.x * 256 + threadIdx.x; i < m; i += (u64)gridDim.x * 256) {
        const u64 b = boards[i], key = canon ? canonical(b) : b;
        u32 j = 0;
#pragma unroll
        for (u32 w = LOOKUP_TOP / 2; w; w >>= 1)
            if (j + w < stretches && top[j + w] <= key) j += w;
        u64 lo = j * step, len = min(step, n - lo);
        while (len > 1) {
            const u64 half = len >> 1;
            lo = __ldg(keys + lo + half) <= key ? lo + half : lo;
            len -= half;
        }
        out[i] = __ldg(keys + lo) == key ? (double)__ldg(vals + lo) : 0.0;
    }
}

template <typename V>
static void launch_search(const LayerIndex &ix, const u64 *boards, u64 m, bool canon, double *out, cudaStream_t s)
{
    const V *vals = (const V *)ix.vals;
    if (m <= LOOKUP_FEW)
        lookup_few_kernel<V><<<grid_for(m * 32, 256, 8), 256, 0, s>>>(ix.keys, vals, ix.n, boards, m, canon ? 1 : 0, out);
    else
        lookup_search_kernel<V><<<grid_for(m, 256, 8), 256, 0, s>>>(ix.keys, vals, ix.n, boards, m, canon ? 1 : 0, out);
}

bool lookup_sorted(const LayerIndex &ix, int vbytes, const u64 *boards, u64 m, bool canon, double *out, cudaStream_t s)
{
    if (m == 0) return true;
    if (ix.n == 0) return CGB_CUDA(cudaMemsetAsync(out, 0, m * sizeof(double), s));
    if (vbytes == 4) launch_search<float>(ix, boards, m, canon, out, s);
    else launch_search<double>(ix, boards, m, canon, out, s);
    kstats().launches++;
    return CGB_CUDA(cudaGetLastError());
}

bool lookup_batch(const LayerIndex &ix, int vbytes, const u64 *boards, u64 m, bool canon, double *out,
                  cudaStream_t s)
{
    if (m == 0) return true;
    const int grid = grid_for(m, 256, 8);
    if (vbytes == 4)
        lookup_batch_kernel<float><<<grid, 256, 0, s>>>(dev_table<float>(ix), boards, m, canon ? 1 : 0, out);
    else
        lookup_batch_kernel<double><<<grid, 256, 0, s>>>(dev_table<double>(ix), boards, m, canon ? 1 : 0, out);
    kstats().launches++;
    return CGB_CUDA(cudaGetLastError());
}

}  // namespace cgb
