// Copies between the caller's host memory and the device.  Every entry point of the C ABI takes plain host pointers, so what a caller
// waits for is mostly this file: page-locked memory goes to the copy engine as it is, everything else through page-locked memory here.
//
//   tiny uploads             (<= TINY bytes) as they are: the driver puts the bytes into its command stream (1.9 us, against 3.6 us of
//                            a copy from page-locked memory).
//   small (<= SMALL bytes)   through the context's bounce area: one memcpy and one asynchronous copy.  Results come back at the next
//                            synchronisation (`sync` hands them out), so a call with several small results waits once.  The driver's
//                            own path for pageable memory stages and waits inside every single call.
//   large, pageable          through a ring of page-locked slots, filled and emptied by a few host threads beside the copy engine.
//                            One core moves about 18 GB/s (and far less into fresh pages, which it has to fault in), the bus 55 GB/s.
//   page-locked or managed   one asynchronous copy.
//
// A line that a helper's core still holds when it has gone to sleep again costs whoever touches it next a wake-up of that core: the
// copy engine (1 MB into slots that helpers had read: 45 us instead of 18), and the caller, who reads the result or makes the next input
// in the same memory (4 MB: 0.76 ms to read instead of 0.27, 0.83 ms to rewrite instead of 0.24).  So a helper leaves nothing
// behind: it writes past its caches and hands what it has read to the cache that all cores share.
#include <atomic>
#include <condition_variable>
#include <cstring>
#include <exception>
#include <functional>
#include <thread>
#if defined(__x86_64__)
#include <emmintrin.h>
#endif

#include "api_internal.h"

namespace hlapi {

namespace {

constexpr size_t ARENA_BYTES = (size_t)4 << 20;
constexpr size_t TINY = (size_t)16 << 10;
constexpr size_t SMALL = (size_t)512 << 10;  // a memcpy of this size costs about what waking the helper threads does (10 - 20 us)

inline void relax() {
#if defined(__x86_64__)
    __builtin_ia32_pause();
#endif
}

#if defined(__x86_64__)
// CLDEMOTE: moves a line to the cache that all cores share; a no-op where the processor has no such hint
inline void demote_line(const char* p) { asm volatile(".byte 0x0f, 0x1c, 0x00" ::"a"(p) : "memory"); }
#endif

// Past the caches, 16 bytes at a time.  `demote`: what has been read goes to the shared cache, a few lines behind the copy.
inline void copy_past_caches(char* d, const char* h, size_t bytes, bool demote = false) {
#if defined(__x86_64__)
    const size_t head = -(uintptr_t)d & 15, lead = head < bytes ? head : bytes, whole = (bytes - lead) & ~(size_t)63;
    constexpr size_t BEHIND = 256;
    memcpy(d, h, lead);
    for (size_t i = lead; i < lead + whole; i += 64) {
        const __m128i x0 = _mm_loadu_si128((const __m128i*)(h + i)), x1 = _mm_loadu_si128((const __m128i*)(h + i + 16));
        const __m128i x2 = _mm_loadu_si128((const __m128i*)(h + i + 32)), x3 = _mm_loadu_si128((const __m128i*)(h + i + 48));
        _mm_stream_si128((__m128i*)(d + i), x0);
        _mm_stream_si128((__m128i*)(d + i + 16), x1);
        _mm_stream_si128((__m128i*)(d + i + 32), x2);
        _mm_stream_si128((__m128i*)(d + i + 48), x3);
        if (demote && i >= lead + BEHIND) demote_line(h + i - BEHIND);
    }
    _mm_sfence();
    memcpy(d + lead + whole, h + lead + whole, bytes - lead - whole);
    if (demote && bytes)
        for (size_t i = bytes > 2 * BEHIND ? bytes - 2 * BEHIND : 0; i < bytes; i += 64) demote_line(h + i);
#else
    memcpy(d, h, bytes);
#endif
}
// a share of an upload and of a result, by a helper
inline void helper_up(char* slot, const char* h, size_t bytes) { copy_past_caches(slot, h, bytes, true); }
inline void helper_down(char* h, const char* slot, size_t bytes) {
    copy_past_caches(h, slot, bytes);
#if defined(__x86_64__)
    for (size_t i = 0; i < bytes; i += 64) demote_line(slot + i);
#endif
}

// The helper threads: one set per process, made at the first large copy and joined when the last context is shut down.  One copy has
// them at a time; a copy that finds them taken (another context's thread) does its work alone.
class Helpers {
  public:
    // runs fn on the caller's thread and on the helpers that get to it in time.  A helper that is still waking up when the caller's
    // thread is done is not waited for: an idle core of a virtual machine can take 300 us to come back.
    void run(const std::function<void()>& fn) {
        if (!busy_.try_lock()) { fn(); return; }
        start();
        {
            std::lock_guard<std::mutex> g(mu_);
            job_ = &fn;
            epoch_++;
        }
        wake_.notify_all();
        fn();
        {
            std::lock_guard<std::mutex> g(mu_);
            job_ = nullptr;
        }
        while (active_.load(std::memory_order_acquire)) relax();
        busy_.unlock();
    }
    void stop() {
        std::lock_guard<std::mutex> b(busy_);
        {
            std::lock_guard<std::mutex> g(mu_);
            quit_ = true;
        }
        wake_.notify_all();
        for (auto& t : threads_) t.join();
        threads_.clear();
        quit_ = false;
    }

  private:
    void start() {
        if (!threads_.empty()) return;
        const unsigned hw = std::thread::hardware_concurrency();
        // half the cores at most, the caller's among them (16 MB up and down in us: five helpers 509 and 515, seven 476 and 452)
        const int n = hw >= 16 ? 7 : hw >= 4 ? (int)hw / 2 - 1 : 0;
        // a process that may not make (all of) them, under a limit on threads or memory, copies with those there are
        try {
            for (int i = 0; i < n; i++) threads_.emplace_back([this, e = epoch_] { loop(e); });
        } catch (const std::exception&) {
        }
    }
    void loop(u64 seen) {
        std::unique_lock<std::mutex> g(mu_);
        for (;;) {
            wake_.wait(g, [&] { return quit_ || epoch_ != seen; });
            if (quit_) return;
            seen = epoch_;
            if (!job_) continue;
            const std::function<void()>* fn = job_;
            active_.fetch_add(1);
            g.unlock();
            (*fn)();
            active_.fetch_sub(1, std::memory_order_release);
            g.lock();
        }
    }
    std::mutex busy_, mu_;
    std::condition_variable wake_;
    std::vector<std::thread> threads_;
    const std::function<void()>* job_ = nullptr;
    std::atomic<int> active_{0};
    u64 epoch_ = 0;
    bool quit_ = false;
};

Helpers& helpers() {
    static Helpers* h = new Helpers();  // never destroyed: a forked child's exit must not wait for threads that it does not have
    return *h;
}
std::mutex g_ctx_mu;
int g_contexts = 0;

bool pageable(const void* h) {
    cudaPointerAttributes attr;
    const bool yes = cudaPointerGetAttributes(&attr, h) != cudaSuccess || attr.type == cudaMemoryTypeUnregistered;
    cudaGetLastError();  // an unregistered pointer is not an error here
    return yes;
}

}  // namespace

// A ring of page-locked slots.  Use number i of the ring takes slot i % SLOTS.  The host's side of a use (an upload: fill the slot; a
// download: empty it) is SHARES shares of the slot, so that several threads work on the piece that the copy engine or the caller is
// waiting for (one thread takes 58 us for 1 MB: that long stood before the first piece of every upload and behind the last of every
// download); `host[slot]` counts them, over all uses.  `ev[slot]` is the copy engine's side.  Only the calling thread talks
// to CUDA: eight threads that all did spent their time on the driver's lock (16 MB up: 1.2 ms; now 0.35 ms; the bus alone 0.31 ms).
struct CopyRing {
    static constexpr u32 SLOTS = 16;
    static constexpr size_t SLOT_BYTES = (size_t)1 << 20;
    static constexpr u32 SHARES = 4;
    char* mem = nullptr;
    cudaEvent_t ev[SLOTS] = {};
    std::atomic<u64> host[SLOTS];
    u64 next = 0;  // uses of the ring so far
    CopyRing() {
        for (auto& u : host) u.store(0);
    }
};

static CopyRing* ring_of(hl_ctx* c) {
    if (c->ring) return c->ring;
    CopyRing* r = new CopyRing();
    bool ok = cudaHostAlloc((void**)&r->mem, CopyRing::SLOTS * CopyRing::SLOT_BYTES, cudaHostAllocDefault) == cudaSuccess;
    for (u32 i = 0; i < CopyRing::SLOTS && ok; i++) ok = cudaEventCreateWithFlags(&r->ev[i], cudaEventDisableTiming) == cudaSuccess;
    cudaGetLastError();
    c->ring = r;
    if (!ok) host_copy_release(c);
    return c->ring;
}

void host_copy_retain() {
    std::lock_guard<std::mutex> g(g_ctx_mu);
    g_contexts++;
}

void host_copy_release(hl_ctx* c) {
    if (!c->ring) return;
    for (auto& e : c->ring->ev)
        if (e) cudaEventDestroy(e);
    if (c->ring->mem) cudaFreeHost(c->ring->mem);
    delete c->ring;
    c->ring = nullptr;
}

void host_copy_drop() {
    std::lock_guard<std::mutex> g(g_ctx_mu);
    if (--g_contexts == 0) helpers().stop();
}

// One large copy in pieces: enough of them that filling, copying and emptying overlap, none so small that its own overheads show.
struct Pieces {
    size_t bytes, each;
    u64 n, base;
    std::atomic<u64> claim{0}, open{0};  // the next share to copy on the host; how many pieces may be copied now
    Pieces(CopyRing* r, size_t b) : bytes(b) {
        const size_t p = (b / 8 + 65535) & ~(size_t)65535, least = (size_t)512 << 10;
        each = p < least ? least : p > CopyRing::SLOT_BYTES ? CopyRing::SLOT_BYTES : p;
        n = (b + each - 1) / each;
        base = r->next;
        r->next += n;
    }
    size_t off(u64 k) const { return k * each; }
    size_t len(u64 k) const { return bytes - k * each < each ? bytes - k * each : each; }
    u32 slot(u64 k) const { return (u32)((base + k) % CopyRing::SLOTS); }
    // the bytes [from, to) of share g's piece: a short last piece has short and empty shares
    void share(u64 g, size_t* from, size_t* to) const {
        const size_t part = each / CopyRing::SHARES, n_k = len(g / CopyRing::SHARES), at = g % CopyRing::SHARES * part;
        *from = at < n_k ? at : n_k;
        *to = at + part < n_k ? at + part : n_k;
    }
    void done(CopyRing* r, u64 g) const { r->host[slot(g / CopyRing::SHARES)].fetch_add(1, std::memory_order_release); }
    bool all_done(CopyRing* r, u64 k) const {
        return r->host[slot(k)].load(std::memory_order_acquire) == ((base + k) / CopyRing::SLOTS + 1) * CopyRing::SHARES;
    }
    // the next share of an open piece, or false; helpers take one ahead of its opening and wait
    bool claim_open(u64* g) {
        u64 v = claim.load();
        while (v < open.load(std::memory_order_acquire) * CopyRing::SHARES)
            if (claim.compare_exchange_weak(v, v + 1)) { *g = v; return true; }
        return false;
    }
};

// copy(g, helper) does share g of the host's side; engine() one step of the copy engine's side, true once all of it is done.  The helpers
// only copy, the calling thread does whatever is there to do.
template <class Copy, class Engine>
static void run_pieces(Pieces& pc, Copy copy, Engine engine) {
    const std::thread::id me = std::this_thread::get_id();
    helpers().run([&] {
        u64 g;
        if (std::this_thread::get_id() != me) {
            while ((g = pc.claim.fetch_add(1)) < pc.n * CopyRing::SHARES) {
                while (pc.open.load(std::memory_order_acquire) <= g / CopyRing::SHARES) relax();
                copy(g, true);
            }
            return;
        }
        while (!engine())
            if (pc.claim_open(&g)) copy(g, false);
    });
}

static cudaError_t ring_up(CopyRing* r, char* d, const char* h, size_t bytes, cudaStream_t s) {
    Pieces pc(r, bytes);
    cudaError_t err = cudaSuccess;
    u64 issued = 0;
    run_pieces(
        pc,
        [&](u64 g, bool helper) {
            const u64 k = g / CopyRing::SHARES;
            size_t from, to;
            pc.share(g, &from, &to);
            char* slot = r->mem + pc.slot(k) * CopyRing::SLOT_BYTES + from;
            if (helper) helper_up(slot, h + pc.off(k) + from, to - from);
            else copy_past_caches(slot, h + pc.off(k) + from, to - from);
            pc.done(r, g);
        },
        [&] {
            // a slot opens when the engine has read its last piece
            for (u64 o = pc.open.load(); o < pc.n && (o < CopyRing::SLOTS || o - CopyRing::SLOTS < issued); o++) {
                if (pc.base + o >= CopyRing::SLOTS && err == cudaSuccess) {
                    const cudaError_t e = cudaEventQuery(r->ev[pc.slot(o)]);
                    if (e == cudaErrorNotReady) break;
                    if (e != cudaSuccess) err = e;
                }
                pc.open.store(o + 1, std::memory_order_release);
            }
            while (issued < pc.n && issued < pc.open.load() && pc.all_done(r, issued)) {
                const u32 slot = pc.slot(issued);
                if (err == cudaSuccess) err = cudaMemcpyAsync(d + pc.off(issued), r->mem + slot * CopyRing::SLOT_BYTES, pc.len(issued), cudaMemcpyHostToDevice, s);
                if (err == cudaSuccess) err = cudaEventRecord(r->ev[slot], s);
                issued++;
            }
            return issued == pc.n;
        });
    return err;
}

static cudaError_t ring_down(CopyRing* r, char* h, const char* d, size_t bytes, cudaStream_t s) {
    Pieces pc(r, bytes);
    cudaError_t err = cudaSuccess;
    u64 posted = 0, emptied = 0;
    auto post = [&] {
        while (posted < pc.n && (posted < CopyRing::SLOTS || posted - CopyRing::SLOTS < emptied)) {
            const u32 slot = pc.slot(posted);
            if (err == cudaSuccess && posted < CopyRing::SLOTS && pc.base + posted >= CopyRing::SLOTS) err = cudaEventSynchronize(r->ev[slot]);  // an earlier upload
            if (err == cudaSuccess) err = cudaMemcpyAsync(r->mem + slot * CopyRing::SLOT_BYTES, d + pc.off(posted), pc.len(posted), cudaMemcpyDeviceToHost, s);
            if (err == cudaSuccess) err = cudaEventRecord(r->ev[slot], s);
            posted++;
        }
    };
    // the kernels ahead of the copy may take long: one thread waits for them, then the helpers join
    post();
    if (err == cudaSuccess) err = cudaEventSynchronize(r->ev[pc.slot(0)]);
    run_pieces(
        pc,
        [&](u64 g, bool helper) {
            const u64 k = g / CopyRing::SHARES;
            size_t from, to;
            pc.share(g, &from, &to);
            const char* slot = r->mem + pc.slot(k) * CopyRing::SLOT_BYTES + from;
            if (helper) helper_down(h + pc.off(k) + from, slot, to - from);
            else memcpy(h + pc.off(k) + from, slot, to - from);
            pc.done(r, g);
        },
        [&] {
            while (emptied < posted && pc.all_done(r, emptied)) emptied++;
            post();
            for (u64 o = pc.open.load(); o < posted; o++) {  // a piece opens when it has arrived
                if (err == cudaSuccess) {
                    const cudaError_t e = cudaEventQuery(r->ev[pc.slot(o)]);
                    if (e == cudaErrorNotReady) break;
                    if (e != cudaSuccess) err = e;
                }
                pc.open.store(o + 1, std::memory_order_release);
            }
            return emptied == pc.n;
        });
    return err;
}

static char* arena_slot(hl_ctx* c, size_t bytes) {
    if (!c->arena && cudaHostAlloc((void**)&c->arena, ARENA_BYTES, cudaHostAllocDefault) != cudaSuccess) {
        cudaGetLastError();
        c->arena = nullptr;
        return nullptr;
    }
    const size_t need = (bytes + 63) & ~(size_t)63;
    if (c->arena_off + need > ARENA_BYTES && sync(c, "bounce area") != HL_B200_OK) return nullptr;  // a synchronisation empties the area
    char* slot = c->arena + c->arena_off;
    c->arena_off += need;
    return slot;
}

// On return the caller's bytes are no longer needed, unless they are page-locked (then they are read by the end of the call that the
// copy is part of).
int h2d_on(hl_ctx* c, void* d, const void* h, size_t bytes, cudaStream_t s) {
    if (!bytes) return HL_B200_OK;
    const void* from = h;
    cudaError_t e;
    CopyRing* r;
    if (bytes <= TINY && pageable(h)) {
        e = cudaMemcpyAsync(d, h, bytes, cudaMemcpyHostToDevice, s);
    } else if (bytes <= SMALL) {
        char* slot = arena_slot(c, bytes);
        if (slot) { copy_past_caches(slot, (const char*)h, bytes); from = slot; }
        e = cudaMemcpyAsync(d, from, bytes, cudaMemcpyHostToDevice, s);
    } else if (pageable(h) && (r = ring_of(c)) != nullptr) {
        e = ring_up(r, (char*)d, (const char*)h, bytes, s);
    } else {
        e = cudaMemcpyAsync(d, from, bytes, cudaMemcpyHostToDevice, s);
    }
    if (e != cudaSuccess) return fail(c, HL_B200_ERR_DEVICE, "copy to device", e);
    c->stats.bytes_h2d += bytes;
    return HL_B200_OK;
}

int h2d(hl_ctx* c, void* d, const void* h, size_t bytes) { return h2d_on(c, d, h, bytes, c->stream); }

// The same for calls that return before the stream has been waited for: page-locked bytes are waited for here.
int h2d_owned(hl_ctx* c, void* d, const void* h, size_t bytes) {
    int rc = h2d(c, d, h, bytes);
    if (!rc && bytes > SMALL && !pageable(h)) rc = sync(c, "copy to device");
    return rc;
}

// The bytes are in the caller's memory after the next `sync`.
int d2h_on(hl_ctx* c, void* h, const void* d, size_t bytes, cudaStream_t s) {
    if (!bytes) return HL_B200_OK;
    cudaError_t e;
    CopyRing* r;
    char* slot;
    if (bytes <= SMALL && (slot = arena_slot(c, bytes)) != nullptr) {
        e = cudaMemcpyAsync(slot, d, bytes, cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) c->pending.push_back({h, slot, bytes});
    } else if (pageable(h) && (r = ring_of(c)) != nullptr) {
        e = ring_down(r, (char*)h, (const char*)d, bytes, s);
    } else {
        e = cudaMemcpyAsync(h, d, bytes, cudaMemcpyDeviceToHost, s);
    }
    if (e == cudaSuccess && s != c->stream) {
        e = cudaEventRecord(c->ev_main, s);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(c->stream, c->ev_main, 0);
    }
    if (e != cudaSuccess) return fail(c, HL_B200_ERR_DEVICE, "copy from device", e);
    c->stats.bytes_d2h += bytes;
    return HL_B200_OK;
}

int d2h(hl_ctx* c, void* h, const void* d, size_t bytes) { return d2h_on(c, h, d, bytes, c->stream); }

int sync(hl_ctx* c, const char* what) {
    cudaError_t e = cudaStreamSynchronize(c->stream);
    if (e == cudaSuccess)
        for (const auto& p : c->pending) memcpy(p.to, p.from, p.bytes);
    c->pending.clear();
    c->arena_off = 0;
    if (e != cudaSuccess) return fail(c, HL_B200_ERR_DEVICE, what, e);
    return HL_B200_OK;
}

}  // namespace hlapi
