// engine.cu -- device runtime: memory, the generation sweep and the solve sweep.
//
// Generation (src/generate.c:409-615) keeps the rolling sets on the device:
//   S_s    boards of tile sum s still to move (the reference's n)
//   L_s-2  the layer before (its 4-spawns are the reference's n4)
// and per layer runs
//   L_s   = unique(sort(expand_moves(S_s)))            -> the layer s.boards
//   S_s+2 = unique(sort(spawn2(L_s) ++ spawn4(L_s-2))) (src/generate.c:530-544)
// The reference sorts the two spawn streams apart, carries one of them to the
// next layer and merges; the set is the same, and one sort of both streams
// takes the place of two sorts and a merge.  The unique pass of the move step
// also counts the spawns the next steps will make.
// Layers go to a LayerSink: it keeps them in HBM (the resident gen+solve
// run) or copies them out (files through the C API).
//
// Solve (src/solve.c:172-224) walks the layers top-down with the s+2 and s+4
// tables resident.
#include "engine.h"
#include "cgb_engine.h"
#include <algorithm>
#include <cstring>
#include <mutex>
#include <unordered_map>

namespace cgb {

// ---- errors -----------------------------------------------------------------
static std::string g_last_error;
static std::mutex g_err_mu;

void set_error(const std::string &msg)
{
    std::lock_guard<std::mutex> g(g_err_mu);
    g_last_error = msg;
}
const char *last_error()
{
    std::lock_guard<std::mutex> g(g_err_mu);
    return g_last_error.c_str();
}
bool cuda_ok(cudaError_t e, const char *what, const char *file, int line)
{
    if (e == cudaSuccess) return true;
    char buf[512];
    snprintf(buf, sizeof buf, "%s:%d: %s failed: %s", file, line, what, cudaGetErrorString(e));
    set_error(buf);
    return false;
}
std::string err_string(u32 err)
{
    std::string s;
    if (err & ERR_LOOKBACK_TIMEOUT) s += "[look-back wait timed out]";
    if (err & ERR_CAPACITY) s += "[output capacity exceeded]";
    if (err & ERR_UNSORTED) s += "[input not sorted]";
    if (err & ERR_TOO_LARGE) s += "[size beyond 32-bit counters]";
    if (err & ERR_COPY_TIMEOUT) s += "[bulk copy wait timed out]";
    return s.empty() ? "[none]" : s;
}

// ---- kernel clocks ----------------------------------------------------------
KernelStats &kstats()
{
    static KernelStats k;
    return k;
}
KClock &kclock()
{
    static KClock c;
    return c;
}
cudaEvent_t KClock::take()
{
    if (free_.empty()) {
        cudaEvent_t e;
        cudaEventCreate(&e);
        return e;
    }
    cudaEvent_t e = free_.back();
    free_.pop_back();
    return e;
}
void KClock::begin(cudaStream_t s, double *acc)
{
    open_ = take();
    open_acc_ = acc;
    cudaEventRecord(open_, s);
    kstats().launches++;
}
void KClock::end(cudaStream_t s)
{
    if (!open_) return;
    cudaEvent_t b = take();
    cudaEventRecord(b, s);
    pend_.push_back({open_, b, open_acc_});
    open_ = nullptr;
}
void KClock::flush(size_t first)
{
    first = std::min(first, pend_.size());
    for (size_t i = 0; i < first; i++) {
        const Pending &p = pend_[i];
        float ms = 0;
        if (cudaEventElapsedTime(&ms, p.a, p.b) == cudaSuccess && p.acc) *p.acc += ms;
        free_.push_back(p.a);
        free_.push_back(p.b);
    }
    pend_.erase(pend_.begin(), pend_.begin() + first);
}

// ---- memory -----------------------------------------------------------------
// Every engine allocation goes through dev_alloc/dev_free, which count the
// bytes held, so that a cap (option device_mem_cap_mb: a host whose allocator
// gives this library a fixed budget) turns into a clean allocation failure.
u64 g_dev_mem_cap = 0;
static std::mutex g_mem_mu;
static std::unordered_map<void *, u64> g_mem_blocks;
static u64 g_mem_held = 0, g_mem_failed = 0;
u64 failed_allocs()
{
    std::lock_guard<std::mutex> g(g_mem_mu);
    return g_mem_failed;
}

// Large blocks that were freed, for the next allocation of about their size on
// the same stream.  The stream-ordered pool under them splits a large free block
// for any smaller request, so a sweep that frees and allocates blocks of hundreds
// of MB left it in pieces and made it map new memory, at 1 to 25 ms a time.
// Bounded in bytes (the solve of LL to 200, 10M boards a layer: 53.0 to 54.0 ms with
// none kept, 53.8 to 57.0 with 1 GB, 52.4 with 8, 52.5 with 32); everything goes back
// to the pool when an allocation fails and when a memory cap is set, under which
// nothing is kept.
struct FreeBlock {
    void *p;
    u64 bytes;
    cudaStream_t s;
};
static std::vector<FreeBlock> g_free_blocks;
static u64 g_free_bytes = 0;
static constexpr u64 FREE_BLOCK_BYTES = 8ull << 30;

void release_blocks()
{
    std::lock_guard<std::mutex> g(g_mem_mu);
    for (auto &b : g_free_blocks) cudaFreeAsync(b.p, b.s);
    g_free_blocks.clear();
    g_free_bytes = 0;
}
// a kept block of bytes .. 1.25 bytes; its size in *bytes
static void *take_block(u64 *bytes, cudaStream_t s)
{
    if (*bytes < LARGE_BLOCK) return nullptr;
    std::lock_guard<std::mutex> g(g_mem_mu);
    size_t best = g_free_blocks.size();
    for (size_t i = 0; i < g_free_blocks.size(); i++) {
        const FreeBlock &b = g_free_blocks[i];
        if (b.s == s && b.bytes >= *bytes && b.bytes <= *bytes + *bytes / 4 &&
            (best == g_free_blocks.size() || b.bytes < g_free_blocks[best].bytes))
            best = i;
    }
    if (best == g_free_blocks.size()) return nullptr;
    const FreeBlock b = g_free_blocks[best];
    g_free_blocks.erase(g_free_blocks.begin() + best);
    g_free_bytes -= b.bytes;
    *bytes = b.bytes;
    return b.p;
}

bool dev_alloc(void **p, u64 bytes, cudaStream_t s)
{
    *p = nullptr;
    if (bytes == 0) bytes = 256;
    auto over_cap = [&] {
        std::lock_guard<std::mutex> g(g_mem_mu);
        return g_dev_mem_cap && g_mem_held + bytes > g_dev_mem_cap;
    };
    if (over_cap()) Engine::get().drop_kept();
    {
        std::lock_guard<std::mutex> g(g_mem_mu);
        if (g_dev_mem_cap && g_mem_held + bytes > g_dev_mem_cap) {
            char buf[200];
            snprintf(buf, sizeof buf, "device allocation of %.3f GB failed: over the cap of %.3f GB (%.3f GB held)",
                     bytes / 1e9, g_dev_mem_cap / 1e9, g_mem_held / 1e9);
            set_error(buf);
            g_mem_failed++;
            return false;
        }
    }
    if ((*p = take_block(&bytes, s))) {
        std::lock_guard<std::mutex> g(g_mem_mu);
        g_mem_blocks[*p] = bytes;
        g_mem_held += bytes;
        return true;
    }
    cudaError_t e = cudaMallocAsync(p, bytes, s);
    if (e == cudaErrorMemoryAllocation) {
        // freed blocks of other sizes may still sit in the pool: return them
        // to the device and retry once
        cudaGetLastError();
        Engine::get().drop_kept();
        release_blocks();
        cudaStreamSynchronize(s);
        int dev = 0;
        cudaGetDevice(&dev);
        cudaMemPool_t pool;
        if (cudaDeviceGetDefaultMemPool(&pool, dev) == cudaSuccess) cudaMemPoolTrimTo(pool, 0);
        kstats().pool_trims++;
        e = cudaMallocAsync(p, bytes, s);
    }
    if (e != cudaSuccess) {
        char buf[160];
        snprintf(buf, sizeof buf, "device allocation of %.3f GB failed: %s", bytes / 1e9, cudaGetErrorString(e));
        set_error(buf);
        cudaGetLastError();
        *p = nullptr;
        std::lock_guard<std::mutex> g(g_mem_mu);
        g_mem_failed++;
        return false;
    }
    std::lock_guard<std::mutex> g(g_mem_mu);
    g_mem_blocks[*p] = bytes;
    g_mem_held += bytes;
    return true;
}
void dev_free(void *p, cudaStream_t s)
{
    if (!p) return;
    {
        std::lock_guard<std::mutex> g(g_mem_mu);
        auto it = g_mem_blocks.find(p);
        if (it != g_mem_blocks.end()) {
            const u64 bytes = it->second;
            g_mem_held -= bytes;
            g_mem_blocks.erase(it);
            // (blocks freed on another stream than the engine's are not allocated there)
            if (bytes >= LARGE_BLOCK && !g_dev_mem_cap && g_free_bytes + bytes <= FREE_BLOCK_BYTES &&
                s == Engine::get().stream) {
                g_free_blocks.push_back({p, bytes, s});
                g_free_bytes += bytes;
                return;
            }
        }
    }
    cudaFreeAsync(p, s);
}

__global__ void words_kernel(u32 *dst, const u32 *src, int words, u64 *started)
{
    after_previous();
    stamp(started);
    for (int i = threadIdx.x; i < words; i += blockDim.x) dst[i] = src[i];
}
bool words_to_host(u32 *pinned, const u32 *dev, int words, cudaStream_t s, u64 *started)
{
    if (started) launch_after(words_kernel, 1, 64, 0, s, pinned, dev, words, started);
    else words_kernel<<<1, 64, 0, s>>>(pinned, dev, words, started);
    return CGB_CUDA(cudaGetLastError());
}

// free device memory plus what the stream-ordered pool and the kept blocks hold unused
u64 device_available_bytes(int dev)
{
    size_t free_b = 0, total_b = 0;
    cudaMemGetInfo(&free_b, &total_b);
    cudaMemPool_t pool;
    u64 reserved = 0, used = 0;
    if (cudaDeviceGetDefaultMemPool(&pool, dev) == cudaSuccess) {
        cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &reserved);
        cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used);
    }
    std::lock_guard<std::mutex> g(g_mem_mu);
    return (u64)free_b + (reserved > used ? reserved - used : 0) + g_free_bytes;
}

// ---- resident layer store ---------------------------------------------------
bool LayerStore::push(u64 n, cudaStream_t s, Handle *h)
{
    const u64 need = n ? n : 1;
    if (chunks_.empty() || !chunks_.back().base || chunks_.back().top + need > chunks_.back().cap) {
        Chunk c;
        // the first chunk 64 MB (a small sweep needs no more, and mapping 4 GB takes
        // 25 ms), each further one as large as all before it, up to chunk_bytes
        c.cap = std::max<u64>(need, std::min<u64>(chunk_bytes / 8, std::max<u64>(8ull << 20, total)));
        if (!dev_alloc((void **)&c.base, c.cap * 8, s)) return false;
        total += c.cap;
        chunks_.push_back(std::move(c));
    }
    Chunk &c = chunks_.back();
    h->chunk = (int)chunks_.size() - 1;
    h->off = c.top;
    h->n = n;
    c.blocks.push_back({c.top, need, true});
    c.top += need;
    return true;
}

u64 *LayerStore::ptr(const Handle &h, cudaStream_t s)
{
    if (h.chunk < 0) return nullptr;
    Chunk &c = chunks_[h.chunk];
    if (!c.base) {  // spilled: bring the chunk back
        if (!dev_alloc((void **)&c.base, c.cap * 8, s)) return nullptr;
        if (!CGB_CUDA(cudaStreamWaitEvent(s, c.copied, 0))) return nullptr;
        if (c.top && !CGB_CUDA(cudaMemcpyAsync(c.base, c.host, c.top * 8, cudaMemcpyHostToDevice, s))) return nullptr;
        if (!CGB_CUDA(cudaStreamSynchronize(s))) return nullptr;
        cudaFreeHost(c.host);
        c.host = nullptr;
        restores++;
    }
    return c.base + h.off;
}

bool LayerStore::spill(u64 bytes, cudaStream_t s, cudaStream_t io)
{
    u64 done = 0;
    // never the last chunk: the generation appends to it
    for (size_t i = 0; i + 1 < chunks_.size() && done < bytes; i++) {
        Chunk &c = chunks_[i];
        if (!c.base || c.top == 0) continue;
        if (!CGB_CUDA(cudaMallocHost(&c.host, c.top * 8))) return false;
        if (!c.copied && !CGB_CUDA(cudaEventCreateWithFlags(&c.copied, cudaEventDisableTiming))) return false;
        cudaEvent_t written;  // the main stream's writes into the chunk
        if (!CGB_CUDA(cudaEventCreateWithFlags(&written, cudaEventDisableTiming))) return false;
        const bool ok = CGB_CUDA(cudaEventRecord(written, s)) && CGB_CUDA(cudaStreamWaitEvent(io, written, 0)) &&
                        CGB_CUDA(cudaMemcpyAsync(c.host, c.base, c.top * 8, cudaMemcpyDeviceToHost, io)) &&
                        CGB_CUDA(cudaEventRecord(c.copied, io));
        cudaEventDestroy(written);
        if (!ok) return false;
        dev_free(c.base, io);   // back to the pool once the copy has read it
        c.base = nullptr;
        done += c.cap * 8;
        spills++;
    }
    return done > 0;
}

void LayerStore::drop_chunk(Chunk &c, cudaStream_t s)
{
    if (c.base) dev_free(c.base, s);
    if (c.copied) {
        cudaEventSynchronize(c.copied);  // a spill copy may still be reading into c.host
        cudaEventDestroy(c.copied);
        c.copied = nullptr;
    }
    if (c.host) cudaFreeHost(c.host);
    c.base = nullptr;
    c.host = nullptr;
    c.blocks.clear();
    c.top = 0;
}

void LayerStore::release(const Handle &h, cudaStream_t s)
{
    if (h.chunk < 0 || h.chunk >= (int)chunks_.size()) return;
    Chunk &c = chunks_[h.chunk];
    for (auto &b : c.blocks)
        if (b.off == h.off) b.live = false;
    while (!c.blocks.empty() && !c.blocks.back().live) {
        c.top -= c.blocks.back().n;
        c.blocks.pop_back();
    }
    if (c.blocks.empty()) drop_chunk(c, s);
    // drop trailing empty chunks so push() starts a fresh one
    while (!chunks_.empty() && chunks_.back().blocks.empty()) {
        drop_chunk(chunks_.back(), s);
        chunks_.pop_back();
    }
}

void LayerStore::clear(cudaStream_t s)
{
    for (auto &c : chunks_) drop_chunk(c, s);
    chunks_.clear();
}

// ---- engine -----------------------------------------------------------------
Engine &Engine::get()
{
    static Engine e;
    return e;
}

bool Engine::init(int dev)
{
    if (ready && dev == device) return true;
    if (!CGB_CUDA(cudaSetDevice(dev))) return false;
    device = dev;
    if (!stream && !CGB_CUDA(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking))) return false;
    if (!io_stream && !CGB_CUDA(cudaStreamCreateWithFlags(&io_stream, cudaStreamNonBlocking))) return false;
    cudaMemPool_t pool;
    if (!CGB_CUDA(cudaDeviceGetDefaultMemPool(&pool, dev))) return false;
    // keep freed blocks cached in the pool between layer steps; an allocation
    // that fails returns the cache to the device and retries (dev_alloc)
    u64 keep = ~0ull;
    if (!CGB_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep))) return false;
    if (!ctr.d) {
        void *p;
        if (!CGB_CUDA(cudaMalloc(&p, 64 * sizeof(u64)))) return false;
        ctr.d = (u64 *)p;
        ctr.err = (u32 *)(ctr.d + Counters::ERR);
        if (!CGB_CUDA(cudaHostAlloc((void **)&ctr.host, (Counters::HEAD + 1) * sizeof(u64), cudaHostAllocDefault))) return false;
        if (!CGB_CUDA(cudaMemset(p, 0, 64 * sizeof(u64)))) return false;
    }
    ready = true;
    return true;
}

bool Engine::set_rules(const cgb_rules &r)
{
    rules = r;
    return upload_row_table(rt, r.free_formation ? 1 : 0, r.ignore_f ? 1 : 0, stream);
}

PruneParams Engine::prune_params() const
{
    PruneParams p;
    p.enabled = rules.prune ? 1 : 0;
    p.stsl = rules.stsl;
    p.ltc = rules.ltc;
    p.smallest_large = rules.smallest_large;
    return p;
}

bool Engine::sync() { return CGB_CUDA(cudaStreamSynchronize(stream)); }

// grow-only device buffer with 25 % headroom, so layer after layer of slowly
// growing sizes reuses the same allocation
static bool reserve(DevBuf<u64> &b, u64 n, cudaStream_t s)
{
    if (b.p && b.cap >= n) return true;
    return grow(b, n + n / 4 + 1024, s);
}

// sort + unique of n raw keys in x (y = scratch); returns the buffer holding
// the unique keys (the other one is left free)
bool Engine::sort_unique_step(DevBuf<u64> &x, DevBuf<u64> &y, u64 n, u64 *nu, DevBuf<u64> **out, GenTimes *tm,
                              u64 *empties, KeyBits *bits)
{
    cudaStream_t s = stream;
    u64 *u = x.p;
    SortStats st;
    if (!sort_unique_keys(x.p, y.p, n, &u, nu, ws, s, &st, empties, bits)) return false;
    if (tm) {
        tm->sorted_keys += n;
        tm->sort_passes += (u64)st.passes * n;
    }
    *out = (u == x.p) ? &x : &y;
    return true;
}

// acc = acc u run (both sorted and unique), through the scratch buffer t; the
// first run just changes places with acc
bool Engine::join(DevBuf<u64> &acc, DevBuf<u64> &run, u64 n)
{
    cudaStream_t s = stream;
    GenBuffers &g = gen;
    if (acc.n == 0) {
        std::swap(acc, run);
        acc.n = n;
        return true;
    }
    if (n == 0) return true;
    if (!reserve(g.t, acc.n + n, s)) return false;
    u64 nm = 0;
    if (!merge_unique(acc.p, acc.n, run.p, n, g.t.p, &nm, ws, s)) return false;
    std::swap(acc, g.t);
    acc.n = nm;
    return true;
}

// moved = unique(sort(expand_moves(S))); an input whose raw moves exceed
// max_sort_keys is cut into slices whose sorted unique moves are merged
bool Engine::move_layer(const u64 *d_in, u64 n, GenTimes *tm)
{
    cudaStream_t s = stream;
    GenBuffers &g = gen;
    const u64 slice = std::max<u64>(1, max_sort_keys / 4);
    const bool chunked = n > slice;
    const u64 m0 = chunked ? slice : n;
    if (chunked) g.moved.n = 0;
    g.moved_empties = GenBuffers::UNKNOWN;
    g.moved_bits = KeyBits{};
    for (u64 off = 0; off < n || (n == 0 && off == 0); off += m0) {
        const u64 m = std::min(m0, n - off);
        if (!reserve(g.a, 4 * m0, s) || !reserve(g.b, 4 * m0, s)) return false;
        u64 nr = 0;
        if (!expand_moves(d_in + off, m, g.a.p, 4 * m, &nr, rt, prune_params(), ctr, s, filter, plan)) return false;
        u64 nu = 0, empties = 0;
        DevBuf<u64> *u = nullptr;
        if (!sort_unique_step(g.a, g.b, nr, &nu, &u, tm, chunked ? nullptr : &empties, chunked ? nullptr : &g.moved_bits)) return false;
        if (!chunked) {
            std::swap(*u, g.moved);   // the layer; the old layer buffer becomes scratch
            g.moved.n = nu;
            g.moved_empties = empties;
            return true;
        }
        if (!join(g.moved, *u, nu)) return false;
        if (tm) tm->chunks++;
    }
    return true;
}

// acc = acc u the spawns of src, in slices of at most max_sort_keys spawns
bool Engine::spawn_into(SpawnSource src, DevBuf<u64> &acc, GenTimes *tm)
{
    cudaStream_t s = stream;
    GenBuffers &g = gen;
    const u64 total = src.total;
    const bool chunked = total > max_sort_keys;
    const u64 cap = chunked ? max_sort_keys : total;
    // first guess of a slice that fits; halved while its count does not
    const u64 step =
        chunked ? std::max<u64>(1, (u64)((double)src.n * 0.9 * (double)max_sort_keys / (double)total)) : src.n;
    for (u64 off = 0; off < src.n;) {
        SpawnSource part = src;
        part.boards = src.boards + off;
        part.n = std::min(step, src.n - off);
        if (chunked) {
            for (;;) {
                if (!count_spawns(part.boards, part.n, &part.total, ctr, s)) return false;
                if (part.total <= max_sort_keys || part.n == 1) break;
                part.n = (part.n + 1) / 2;
            }
            if (part.total > max_sort_keys) {
                set_error("spawn_into: one board spawns more keys than max_sort_keys");
                return false;
            }
        }
        for (auto &x : g.c)
            if (!reserve(x, cap, s)) return false;
        if (!expand_next(part, SpawnSource{}, g.c[0].p, ctr, s, plan)) return false;
        u64 nu = 0;
        DevBuf<u64> *u = nullptr;
        if (!sort_unique_step(g.c[0], g.c[1], part.total, &nu, &u, tm)) return false;
        if (!check_spawns(ctr, part.total)) return false;
        if (!join(acc, *u, nu)) return false;
        if (chunked && tm) tm->chunks++;
        off += part.n;
    }
    return true;
}

// the sorted unique 2- and 4-spawns of the moved layer (the cl seam's streams)
bool Engine::spawn_streams(GenTimes *tm)
{
    GenBuffers &g = gen;
    u64 total = g.moved_empties;
    if (total == GenBuffers::UNKNOWN && !count_spawns(g.moved.p, g.moved.n, &total, ctr, stream)) return false;
    g.moved_empties = GenBuffers::UNKNOWN;  // it belongs to this layer only
    g.u2.n = g.u4.n = 0;
    if (!reserve(g.u2, 1, stream) || !reserve(g.u4, 1, stream)) return false;
    return spawn_into(SpawnSource{g.moved.p, g.moved.n, 1, total}, g.u2, tm) &&
           spawn_into(SpawnSource{g.moved.p, g.moved.n, 2, total}, g.u4, tm);
}

// S = the 2-spawns of the moved layer and the 4-spawns of the one before it
// (and a resumed sweep's carried 4-spawns): one sort of both streams, or, where
// they are too long for one, their slices sorted apart and merged
bool Engine::next_inputs(GenTimes *tm)
{
    cudaStream_t s = stream;
    GenBuffers &g = gen;
    if (g.moved_empties == GenBuffers::UNKNOWN && !count_spawns(g.moved.p, g.moved.n, &g.moved_empties, ctr, s))
        return false;
    const SpawnSource two{g.moved.p, g.moved.n, 1, g.moved_empties}, four{g.prev.p, g.prev.n, 2, g.prev_empties};
    const u64 total = two.total + four.total;
    if (g.S.n) g.spawn_ratio = std::max(1.0, (double)total / (double)g.S.n);
    g.S.n = 0;
    if (total <= std::min(max_sort_keys, BUCKET_SORT_KEYS)) {
        for (auto &x : g.c)
            if (!reserve(x, total, s)) return false;
        if (!expand_next(two, four, g.c[0].p, ctr, s, plan)) return false;
        u64 nu = 0;
        DevBuf<u64> *u = nullptr;
        if (!sort_unique_step(g.c[0], g.c[1], total, &nu, &u, tm)) return false;
        if (total && !check_spawns(ctr, total)) return false;
        std::swap(g.S, *u);
        g.S.n = nu;
    } else if (!spawn_into(two, g.S, tm) || !spawn_into(four, g.S, tm)) {
        return false;
    }
    if (g.u4.n) {  // carried in from a checkpoint
        if (!join(g.S, g.u4, g.u4.n)) return false;
        g.u4.n = 0;
    }
    return true;
}

// One layer step without a wait inside: every size but |S| stays on the device,
// where the next kernel reads it, and the sizes come back in one copy at the end.
// A small layer's kernels take 10-20 us each, and three waits with their launches
// behind them cost as much again.  The spawns' room is a guess from the last layer;
// where it or a bucket overflows, quick_take leaves *done false or takes only the
// moved layer, and the step with waits does the rest.  After the last layer no
// input set is wanted.
//
// quick_launch leaves quick.on false where the step with waits is to be taken.
bool Engine::quick_launch(bool last)
{
    cudaStream_t s = stream;
    GenBuffers &g = gen;
    const u64 n = g.S.n;
    quick.on = false;
    if (n == 0 || n > QUICK_BOARDS || g.u4.n || !bucket_sorts() || 4 * n > max_sort_keys) return true;
    // the last layer's ratio and half as much again: it changes by a few per cent from
    // layer to layer, and factors of 1.1, 1.5 and 2.5 measured alike
    const u64 room = last ? 1 : std::max<u64>(1 << 14, (u64)(1.5 * (double)n * g.spawn_ratio));
    if (room > max_sort_keys) return true;
    const u64 sizes[2] = {4 * n, room};
    BucketPlan plans[2];
    // without memory for the guess the step with waits, which knows its sizes, takes
    // the layer, and what the guess has got of it goes back
    if (!reserve(g.a, 4 * n, s) || !reserve(g.b, 4 * n, s) || !reserve(g.c[0], room, s) || !reserve(g.c[1], room, s)) {
        for (auto &x : g.c) drop(x, s);
        return true;
    }
    BucketWorkspace &w = ws.buckets;
    // a quarter more than the last ratios give decides whether one CTA will do; where it
    // does not, the step with waits repeats what overflowed
    const u64 likely[2] = {(u64)(1.25 * (double)n * g.move_ratio), (u64)(1.25 * (double)n * g.spawn_ratio)};
    if (!bucket_prepare(sizes, last ? 1 : 2, plans, w, s, likely)) return true;
    // its own copy: what runs between launch and take may sort too
    if (!quick.host &&
        !CGB_CUDA(cudaHostAlloc((void **)&quick.host, BUCKET_HEADS * BUCKET_HEAD_WORDS * 4 + 8, cudaHostAllocDefault)))
        return false;
    // the third head: counts of moves, raw moves and spawns, error word, and the
    // times at which the expansions started (events between the kernels would keep
    // them from following one another as programmatic dependents)
    constexpr u32 OWN = 2 * BUCKET_HEAD_WORDS;
    u64 *own = (u64 *)(w.ctl.p + OWN);
    u32 *err = w.ctl.p + OWN + 6;
    u32 *const h0 = w.ctl.p;
    SpawnSource two{g.b.p, 4 * n, 1, 0, (u64 *)(h0 + BUCKET_COUNT_AT)}, four{g.prev.p, g.prev.n, 2, 0};
    if (!bucket_clear(w, s)) return false;
    if (!expand_moves_enqueue(g.S.p, n, g.a.p, 4 * n, rt, prune_params(), own, own + 1, err, own + QuickStep::EXPAND, s,
                              filter, plan))
        return false;
    quick.passes[0] = bucket_enqueue(plans[0], 0, g.a.p, own, g.b.p, true, true, w, s);
    if (!last) {
        if (!expand_next_enqueue(two, four, g.c[0].p, room, own + 2, err, own + QuickStep::SPAWN, s, plan)) return false;
        quick.passes[1] = bucket_enqueue(plans[1], 1, g.c[0].p, own + 2, g.c[1].p, true, false, w, s);
    }
    constexpr u32 WORDS = BUCKET_HEADS * BUCKET_HEAD_WORDS;  // the end's time lands behind them
    if (!CGB_CUDA(cudaGetLastError()) || !words_to_host(quick.host, w.ctl.p, WORDS, s, (u64 *)(quick.host + WORDS)))
        return false;
    quick.room = room;
    quick.on = true;
    return true;
}

bool Engine::quick_take(GenTimes *tm, bool last, bool *moved_done, bool *done)
{
    quick.on = false;
    if (!sync()) return false;
    GenBuffers &g = gen;
    const u64 n = g.S.n;
    const BucketResult moves = bucket_result(quick.host, 0), next = bucket_result(quick.host, 1);
    const u32 *own = quick.host + 2 * BUCKET_HEAD_WORDS;
    u64 counts[3];
    memcpy(counts, own, sizeof counts);
    const u32 e = own[6] & ~ERR_CAPACITY, bad = e | moves.error | next.error;
    if (bad) {
        set_error("layer step: device error " + err_string(bad));
        return false;
    }
    g.move_ratio = std::max(0.25, (double)counts[0] / (double)n);
    KernelStats &k = kstats();
    u64 at[2], end;  // the expansions' times and the end's
    memcpy(at, own + 2 * QuickStep::EXPAND, sizeof at);
    memcpy(&end, quick.host + BUCKET_HEADS * BUCKET_HEAD_WORDS, 8);
    const double ms = 1e-6;
    k.launches += last ? 2 : 4;
    k.expand_ms += ms * (double)(moves.started - at[0]);
    k.onesweep_ms += ms * (double)((last ? end : at[1]) - moves.started);
    if (!last) {
        k.spawn_ms += ms * (double)(next.started - at[1]);
        k.onesweep_ms += ms * (double)(end - next.started);
    }
    if (moves.overflow) return true;
    auto sorted = [&](u64 keys, int passes) {
        k.onesweep_bytes += 16 * keys * passes;
        k.onesweep_launches += passes;
        if (tm) {
            tm->sorted_keys += keys;
            tm->sort_passes += (u64)passes * keys;
        }
    };
    k.expand_bytes += 8 * (n + counts[0]);
    k.moves_raw += counts[1];
    k.moves_kept += counts[0];
    sorted(counts[0], quick.passes[0]);
    std::swap(g.b, g.moved);
    g.moved.n = moves.count;
    g.moved_empties = moves.empties;
    g.moved_bits = moves.bits;
    *moved_done = true;
    if (last) return *done = true;
    const u64 total = g.moved_empties + g.prev_empties;
    g.spawn_ratio = std::max(1.0, (double)total / (double)n);
    if (total > quick.room || next.overflow) return true;
    if (counts[2] != total) {
        set_error("layer step: " + std::to_string(counts[2]) + " spawns written, " + std::to_string(total) + " expected");
        return false;
    }
    k.spawn_bytes += 8 * (g.moved.n + g.prev.n + total);
    sorted(total, quick.passes[1]);
    std::swap(g.S, g.c[1]);
    g.S.n = next.count;
    *done = true;
    return true;
}

bool Engine::generate(const u64 *h_initial, u64 n_init, int start, int end, LayerSink &sink, GenTimes *tm,
                      const u64 *h_carry, u64 n_carry)
{
    cudaStream_t s = stream;
    GenBuffers &g = gen;
    if (!reserve(g.S, n_init, s) || !reserve(g.u4, n_carry, s)) return false;
    if (n_init && !CGB_CUDA(cudaMemcpyAsync(g.S.p, h_initial, n_init * 8, cudaMemcpyHostToDevice, s))) return false;
    if (n_carry && !CGB_CUDA(cudaMemcpyAsync(g.u4.p, h_carry, n_carry * 8, cudaMemcpyHostToDevice, s))) return false;
    g.S.n = n_init;
    g.u4.n = n_carry;
    g.prev.n = g.prev_empties = 0;
    g.spawn_ratio = 16;
    g.move_ratio = 4;
    // canonical layer boards share the 0xf mask of the canonical first board (fixed
    // formation cells); the kernels check every board against it
    plan = (n_init && !filter.fid) ? make_canon_plan(canonical(h_initial[0]), rules.free_formation != 0) : CanonPlan{};
    bool ok = true;
    for (int layer = start; layer <= end && ok; layer += 2) {
        // the input set of the layer after the last is made for a checkpoint only
        const bool carry = sink.wants_carry(), last = layer + 2 > end && !carry;
        bool moved = false, next = false;
        if (!quick.on) ok = sink.before(layer, s) && quick_launch(last);
        if (ok && quick.on) ok = quick_take(tm, last, &moved, &next);
        ok = ok && (moved || move_layer(g.S.p, g.S.n, tm)) && (next || last || next_inputs(tm));
        if (!ok) break;
        if (tm) tm->boards += g.moved.n;
        if (carry) {
            ok = reserve(g.u4, 1, s) && spawn_into(SpawnSource{g.moved.p, g.moved.n, 2, g.moved_empties}, g.u4, tm) &&
                 sink.layer(layer, g.moved.p, g.moved.n, s);
        }
        g.u4.n = 0;  // the next input set takes the 4-spawns from the layer itself
        std::swap(g.moved, g.prev);
        g.prev_empties = g.moved_empties;
        if (carry) continue;
        // The device goes on with the next layer while this one is handed on and the
        // spans of its kernels are read: 11 us less between two steps (the 2x4 table of
        // 149 layers 19.9 -> 18.2 ms).
        // Where memory is short the launch is tried again once the layer is stored.
        const size_t over = kclock().pending();
        if (layer + 2 <= end && !(sink.before(layer + 2, s) && quick_launch(layer + 4 > end))) quick.on = false;
        kclock().flush(over);
        ok = sink.layer(layer, g.prev.p, g.prev.n, s);
    }
    quick.on = false;
    ok = sync() && ok;
    kclock().flush();
    return ok;
}

bool OneShot::drop(cudaStream_t s)
{
    if (busy || !(ws.p || index[0].p || index[1].p)) return false;
    cgb::drop(ws, s);
    for (IndexStorage &x : index) {
        dev_free(x.p, s);
        x = IndexStorage{};
    }
    return true;
}

void Engine::end_one_shot()
{
    one_shot.busy = false;
    for (IndexStorage &x : one_shot.index)
        if (x.bytes > OneShot::KEEP) {
            dev_free(x.p, stream);
            x = IndexStorage{};
        }
    index_release_scratch(stream);
}

void Engine::drop_kept()
{
    one_shot.drop(stream);
    if (!ws.buckets.growing) ws.buckets.release(stream);
    index_release_scratch(stream);
}

bool Engine::give_back()
{
    drop_kept();
    release_blocks();
    if (!sync()) return false;
    cudaMemPool_t pool;
    return CGB_CUDA(cudaDeviceGetDefaultMemPool(&pool, device)) && CGB_CUDA(cudaMemPoolTrimTo(pool, 0));
}

void Engine::release_buffers()
{
    GenBuffers &g = gen;
    for (DevBuf<u64> *b : {&g.a, &g.b, &g.c[0], &g.c[1], &g.S, &g.u2, &g.u4, &g.moved, &g.prev, &g.t})
        drop(*b, stream);
    drop_kept();
    release_blocks();
}

}  // namespace cgb
