// engine.h -- internal interfaces of the CUDA engine (not part of the C ABI).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <string>
#include <vector>
#include "common.cuh"
#include "board.cuh"
#include "bucketplan.h"
#include "hashidx.cuh"

namespace cgb {

// ---- device memory --------------------------------------------------------
template <typename T>
struct DevBuf {
    T *p = nullptr;
    u64 n = 0;     // elements in use
    u64 cap = 0;   // elements allocated
};

// a few words from the device to pinned memory, visible once the stream has been
// waited for.  A kernel writes them: a copy would queue in the copy engine behind
// whatever layers and tables other streams are sending to the host
bool words_to_host(u32 *pinned, const u32 *dev, int words, cudaStream_t s, u64 *started = nullptr);

constexpr u64 LARGE_BLOCK = 16ull << 20;  // freed blocks from this size up are kept for the next allocation
bool dev_alloc(void **p, u64 bytes, cudaStream_t s);
u64 failed_allocs();  // how many dev_alloc calls have found no memory
void dev_free(void *p, cudaStream_t s);
template <typename T>
bool grow(DevBuf<T> &b, u64 n, cudaStream_t s)
{
    if (b.cap >= n && b.p) return true;
    if (b.p) dev_free(b.p, s);
    b.p = nullptr;
    b.cap = 0;
    u64 want = n < 64 ? 64 : n;
    if (!dev_alloc((void **)&b.p, want * sizeof(T), s)) return false;
    b.cap = want;
    return true;
}
template <typename T>
void drop(DevBuf<T> &b, cudaStream_t s)
{
    if (b.p) dev_free(b.p, s);
    b.p = nullptr;
    b.n = b.cap = 0;
}

// ---- bucket sort (bucketsort.cu) ------------------------------------------
// AND and OR over a set of keys
struct KeyBits {
    u64 all = 0, any = 0;
    bool known = false;
};
constexpr u32 BUCKET_HEADS = 3, BUCKET_HEAD_WORDS = 16;  // heads: two sorts, and words of the caller's own
struct BucketWorkspace {
    DevBuf<u32> ctl;           // the heads, then each sort's bucket counts and look-back words
    DevBuf<u64> bounds;        // bucket boundaries
    DevBuf<u64> coarse, fine;  // the buckets
    u64 used_words = 0;
    u32 *host = nullptr;       // pinned copy of the heads
    bool growing = false;      // bucket_prepare is at work on it
    void release(cudaStream_t s);
};
constexpr u32 BUCKET_COUNT_AT = 4;  // head word of the 64-bit number of keys written
constexpr u32 BUCKET_STAMP_AT = 12; // head word of the time (ns) at which the sort started
struct BucketResult {
    u64 count = 0, empties = 0;
    u64 started = 0;        // device time in ns
    KeyBits bits;           // of the keys (unique sorts)
    u32 error = 0;
    bool overflow = false;  // nothing was written: the digit passes take the input
};
// The parts of bucket_sort, for callers that put several sorts into one stream
// without a wait: plans and room for `calls` sorts of at most n[i] keys (false:
// too many keys or no memory; likely[i], if given: the number to expect, an
// overflow being reported where a sort was launched for far fewer), one clear of all control words, the launches of
// one sort (the number of keys read from *counted where that is not null;
// returns the passes), and, once the heads have been copied to w.host, the result.
bool bucket_prepare(const u64 *n, int calls, BucketPlan *plans, BucketWorkspace &w, cudaStream_t s,
                    const u64 *likely = nullptr);
bool bucket_clear(BucketWorkspace &w, cudaStream_t s);
int bucket_enqueue(const BucketPlan &p, int slot, const u64 *keys, const u64 *counted, u64 *out, bool unique, bool empties,
                   BucketWorkspace &w, cudaStream_t s);
BucketResult bucket_result(const u32 *heads, int slot);
// out[0, *n_out) = keys[0, n) ascending, without repeats when `unique`; out must
// not alias keys, which are only read.  empties (optional): the empty cells over
// the keys kept.  *done = false (and nothing written) where the sort by buckets
// does not apply: too many keys, no memory for the buckets, or keys that repeat
// too often.
bool bucket_sort(const u64 *keys, u64 n, u64 *out, bool unique, u64 *n_out, u64 *empties, int *passes,
                 BucketWorkspace &w, cudaStream_t s, bool *done, KeyBits *bits = nullptr);

// ---- sort / unique / merge (sort.cu) ------------------------------------
struct SortWorkspace {
    // histograms, bin offsets, tile counters, error word, counts; the decoupled
    // look-back state follows in the same allocation, so one clear covers both
    static constexpr int SMALL_WORDS = 4128;
    u32 *small = nullptr;
    u32 *lookback = nullptr;
    u64 lookback_words = 0;
    u32 *host = nullptr;        // pinned copy of the small words
    bool err_dirty = false;     // a sort left its errors in the word for unique to report
    BucketWorkspace buckets;
    bool reserve(u64 words, cudaStream_t s);
    void release(cudaStream_t s);
};

struct SortStats {
    int passes = 0;
    u64 n = 0;
};

int sort_plan(const u32 *hist_host, u64 n, int *digits);
// sorts keys[0,n) ascending using tmp[0,n); *sorted points at keys or tmp
bool sort_keys(u64 *keys, u64 *tmp, u64 n, u64 **sorted, SortWorkspace &ws, cudaStream_t s,
               SortStats *stats = nullptr);
bool bucket_sorts();  // whether the "sort_variant" option lets the bucket sort run
// reports device errors a sort left behind (when no unique_keys follows)
bool sort_check(SortWorkspace &ws, cudaStream_t s);
// sort_keys then unique_keys, in one pass over the buckets where they apply:
// *out points at keys or tmp
bool sort_unique_keys(u64 *keys, u64 *tmp, u64 n, u64 **out, u64 *n_out, SortWorkspace &ws, cudaStream_t s,
                      SortStats *stats = nullptr, u64 *empties = nullptr, KeyBits *bits = nullptr);
// out must not alias in
// empties (optional): the number of empty cells over the kept keys
bool unique_keys(const u64 *in, u64 n, u64 *out, u64 *n_out, SortWorkspace &ws, cudaStream_t s,
                 u64 *empties = nullptr);
// sorted union of two sorted runs, without repeats (repeats inside a run are
// dropped as well)
bool merge_unique(const u64 *a, u64 na, const u64 *b, u64 nb, u64 *out, u64 *n_out, SortWorkspace &ws,
                  cudaStream_t s);

// ---- row table and expansion (expand.cu) ---------------------------------
struct DeviceRowTable {
    unsigned short *move = nullptr;  // 65536 rows, left move; ROW_LOCKED where a 0xf cell would move
    int free_formation = -1, ignore_f = -1;
};

// the left-move row table of the reference (src/board.c:62-132), host side
void build_row_table(int free_formation, int ignore_f, unsigned short *move, u32 *ok);
bool upload_row_table(DeviceRowTable &t, int free_formation, int ignore_f, cudaStream_t s);

struct Counters {
    // device words: [0] output count, [1] spawn total, [5] raw moves, [6] error word,
    // [12] probes, [16..20] key bits, [40..] indexes' error words
    static constexpr int ERR = 6, HEAD = 7;
    u64 *d = nullptr;
    u32 *err = nullptr;   // d + ERR
    u64 *host = nullptr;  // pinned copy of the first HEAD words, then the probes'
};

// move + prune + canonicalise every board; out needs room for 4n boards
// batched sweeps: stable partition by formation id (fid table of 65536
// entries, see fixed_pattern); counts[f] = boards of formation f
bool partition_by_formation(const u64 *in, u64 n, u64 *out, const unsigned char *fid, u32 counts[256],
                            SortWorkspace &ws, cudaStream_t s);
bool expand_moves(const u64 *in, u64 n, u64 *out, u64 cap, u64 *n_out, const DeviceRowTable &t,
                  const PruneParams &p, Counters &c, cudaStream_t s, FormationFilter ff = FormationFilter{},
                  const CanonPlan &plan = CanonPlan{});
// its launch alone: the counts (results, and legal unpruned moves before the
// repeats went) and errors are added to *count, *raw and *err
bool expand_moves_enqueue(const u64 *in, u64 n, u64 *out, u64 cap, const DeviceRowTable &t, const PruneParams &p,
                          u64 *count, u64 *raw, u32 *err, u64 *started, cudaStream_t s, FormationFilter ff,
                          const CanonPlan &plan);
// number of empty cells over all boards (exact size of the spawn streams)
bool count_spawns(const u64 *in, u64 n, u64 *total, Counters &c, cudaStream_t s);
// one spawn stream: every empty cell of a set of boards filled with `value`
struct SpawnSource {
    const u64 *boards = nullptr;
    u64 n = 0;
    u32 value = 1;  // 1: a 2 tile, 2: a 4 tile
    u64 total = 0;  // empty cells over the boards
    const u64 *counted = nullptr;  // where a kernel before this one left the number of boards (n at most)
};
// the launch of expand_next alone: the count and errors are added to *count and
// *err; nothing is written beyond cap
bool expand_next_enqueue(const SpawnSource &a, const SpawnSource &b, u64 *out, u64 cap, u64 *count, u32 *err,
                         u64 *started, cudaStream_t s, const CanonPlan &plan);
// the canonical spawns of both sources, a.total + b.total of them, in one array
// and without a wait: the counters land in c.host, for check_spawns once the
// stream has been waited for
bool expand_next(const SpawnSource &a, const SpawnSource &b, u64 *out, Counters &c, cudaStream_t s,
                 const CanonPlan &plan);
bool check_spawns(const Counters &c, u64 expect);
// canonical 2-spawn and 4-spawn of every empty cell of every board
bool expand_spawns(const u64 *in, u64 n, u64 *out2, u64 *out4, u64 cap, u64 *n_out, Counters &c,
                   cudaStream_t s, const CanonPlan &plan = CanonPlan{});

// ---- solve (solve.cu) ------------------------------------------------------
struct SolveRules {
    int nox = 0;       // char semantics already applied
    int score = 0;
    const u64 *winstates = nullptr;  // device, expanded x8
    int n_winstates = 0;
    // batched sweeps: formation f's winstates are winstates[ws_begin[f] ..
    // ws_begin[f+1]), f = fid[fixed_pattern(board)]
    const unsigned char *fid = nullptr;
    const u32 *ws_begin = nullptr;
};

// Lookup index over one solved layer (replaces the bisection of lookup(),
// src/solve.c:108-164; every kind returns the value of the key or 0.0).
enum IndexKind : int {
    INDEX_BISECT = 0,  // bisection over the sorted keys (the reference's search)
    INDEX_BUCKET = 1,  // top-bits bucket offsets after the common prefix, then bisection
    INDEX_HASH = 2,    // open addressing, key and value in one 16-byte slot
};

struct LayerIndex {
    int kind = INDEX_BISECT;
    const u64 *keys = nullptr;
    const void *vals = nullptr;   // double or float, aligned with keys
    u64 n = 0;
    // INDEX_BUCKET
    const u32 *bucket = nullptr;  // 2^bits + 1 offsets
    int prefix = 0;               // bucket = (key << prefix) >> (64 - bits)
    int bits = 0;
    u64 prefix_value = 0;         // the shared high bits (key >> (64 - prefix))
    // INDEX_HASH
    const void *slots = nullptr;  // cap slots of {u64 key, u64 value bits}; key 0 = empty
    u64 cap = 0;
    CompactHash ch;               // ch.on: cap (a power of two) 8-byte slots instead
    bool unchecked = false;       // begun, its error word not looked at yet
    int slot = 0;                 // which error word
};

// device storage owned by one index (reused across layers)
struct IndexStorage {
    void *p = nullptr;
    u64 bytes = 0;
};

// at least `bytes` bytes (what was there is not kept)
bool ensure_storage(IndexStorage &st, u64 bytes, cudaStream_t s);
// gives back the scratch that index builds keep for the next
void index_release_scratch(cudaStream_t s);

// graph-capturable form (no host round trip) of a layer's solve, ix.keys into
// ix.vals, counting probes into *probes, and of its hash index in caller-owned slots
// (hash_capacity(n) slots of 16 bytes); device errors accumulate in *err
bool solve_index_enqueue(LayerIndex &ix, int vbytes, const LayerIndex &t2, const LayerIndex &t4, const SolveRules &r,
                         const DeviceRowTable &rt, u64 *probes, void *slots, u64 cap, u32 *err, cudaStream_t s);
u64 hash_capacity(u64 n);
bool solve_prepare();  // one-time kernel attributes (call before a capture)

// builds ix (keys/vals/n already set) of the requested kind; vbytes = 8 or 4.
// index_begin launches the build: kernels behind it on the stream may use ix;
// index_finish waits for it and, where a build gave up (an overflow list or a
// probe distance ran out), builds the index another way (*again, if given: what
// used ix since has to run once more).  Indexes between the two have slots of
// their own.  bits: AND and OR of the keys, or unknown
constexpr int INDEX_SLOTS = 2;
bool index_begin(LayerIndex &ix, int kind, int vbytes, IndexStorage &st, int bucket_bits, Counters &c, cudaStream_t s,
                 const KeyBits &bits = KeyBits{}, int slot = 0);
bool index_finish(LayerIndex &ix, int vbytes, IndexStorage &st, Counters &c, cudaStream_t s, bool *again = nullptr);
// AND and OR of two sets of keys (bits[0], bits[1]) and a key to be read with them
// (into bits[2].any; first may be null), behind one wait
struct KeySet {
    const u64 *keys = nullptr;
    u64 n = 0;
};
bool key_bits(const KeySet &a, const KeySet &b, KeyBits *bits, const u64 *first, Counters &c, cudaStream_t s);
bool build_index(LayerIndex &ix, int kind, int vbytes, IndexStorage &st, int bucket_bits, Counters &c,
                 cudaStream_t s);
// the value of each of m boards (canonicalised first when canon) in an indexed
// layer, widened to double; 0.0 for a board not in it
bool lookup_batch(const LayerIndex &ix, int vbytes, const u64 *boards, u64 m, bool canon, double *out,
                  cudaStream_t s);
// the same by search in the sorted layer: ix needs keys, vals and n only
bool lookup_sorted(const LayerIndex &ix, int vbytes, const u64 *boards, u64 m, bool canon, double *out, cudaStream_t s);

// plan: images that can be canonical for the layer's 0xf mask (CanonPlan{}: all eight)
bool solve_layer_f64(const u64 *keys, u64 n, double *out, const LayerIndex &t2, const LayerIndex &t4,
                     const SolveRules &r, const DeviceRowTable &rt, Counters &c, cudaStream_t s,
                     const CanonPlan &plan = CanonPlan{});
bool solve_layer_f32(const u64 *keys, u64 n, float *out, const LayerIndex &t2, const LayerIndex &t4,
                     const SolveRules &r, const DeviceRowTable &rt, Counters &c, cudaStream_t s,
                     const CanonPlan &plan = CanonPlan{});

// the same without a wait; the probes are counted on the device until
// solve_collect (after which the stream is idle) adds them to the statistics
bool solve_layer_launch(const u64 *keys, u64 n, void *out, int vbytes, const LayerIndex &t2, const LayerIndex &t4,
                        const SolveRules &r, const DeviceRowTable &rt, Counters &c, cudaStream_t s,
                        const CanonPlan &plan);
// solves the layer ix.keys into ix.vals, and where *indexed is true on return the
// solve also fills ix's index, which index_finish then has to look at
bool solve_index_launch(LayerIndex &ix, int kind, int vbytes, IndexStorage &st, const LayerIndex &t2, const LayerIndex &t4,
                        const SolveRules &r, const DeviceRowTable &rt, Counters &c, cudaStream_t s, const CanonPlan &plan,
                        const KeyBits &bits, bool *indexed);
bool solve_collect(Counters &c, cudaStream_t s);

// ---- resident layers ------------------------------------------------------
// Resident layers of a sweep.  Layers are appended during generation and
// released top-down during the solve (last in, first out), so they are packed
// into a few large chunks instead of one allocation per layer; nothing is
// fragmented by the short-lived working buffers of each layer step.  When the
// device runs short, whole chunks of the oldest layers (the lowest tile sums,
// which the top-down solve needs last) are spilled to pinned host memory and
// brought back when a layer in them is needed again.  A spill copies on the
// I/O stream and frees the device chunk there, stream-ordered after the copy,
// so the layer loop on the main stream never waits for it.
u64 device_available_bytes(int dev);

class LayerStore {
  public:
    u64 chunk_bytes = 4ull << 30;   // device allocation unit of the store
    struct Handle {
        int chunk = -1;
        u64 off = 0, n = 0;
    };
    u64 total = 0;                  // boards that all chunks taken so far have room for
    // whether a chunk of full size has been taken since the last call: before that
    // there is nothing worth spilling, and the device query that decides costs 2.5 ms
    bool grown()
    {
        const bool yes = total * 8 >= chunk_bytes && chunks_.size() != checked_;
        if (yes) checked_ = chunks_.size();
        return yes;
    }
    bool push(u64 n, cudaStream_t s, Handle *h);      // room for n boards
    u64 *ptr(const Handle &h, cudaStream_t s);         // device address (restores a spilled chunk)
    void release(const Handle &h, cudaStream_t s);     // frees a pushed block
    // spills oldest chunks (never the last) until `bytes` are on their way to
    // the host; false when nothing could be spilled
    bool spill(u64 bytes, cudaStream_t s, cudaStream_t io);
    void clear(cudaStream_t s);
    u64 spills = 0, restores = 0;
  private:
    struct Block { u64 off, n; bool live; };
    struct Chunk {
        u64 *base = nullptr;   // device memory (null while spilled)
        void *host = nullptr;  // pinned copy while spilled
        cudaEvent_t copied = nullptr;  // the device-to-host copy of the spill is complete
        u64 cap = 0, top = 0;
        std::vector<Block> blocks;
    };
    std::vector<Chunk> chunks_;
    size_t checked_ = 0;
    void drop_chunk(Chunk &c, cudaStream_t s);
};

}  // namespace cgb
