// Copies between the caller's host memory and the device.  Every entry point of the C ABI takes plain host pointers, so what a caller
// waits for is mostly this file: page-locked memory goes to the copy engine as it is, everything else through page-locked memory here.
//
//   tiny uploads             (<= TINY bytes) as they are: the driver puts the bytes into its command stream, and a kernel that reads them
//                            need not wait for the copy engine (an int8 fold of 48 KB: 39 us a call, through the bounce area 52).
//   small (<= SMALL_UP and   through the context's bounce areas: pieces that the host copies while the engine moves the one before.  Results
//   SMALL_DOWN bytes)        come back at the next synchronisation (`sync` hands them out), so a call with several small results waits
//                            once.  The driver's own path for pageable memory stages and waits inside every single call.
//   large, pageable          through a ring of page-locked slots, filled and emptied by a few host threads beside the copy engine.
//                            One core moves about 18 GB/s (and far less into fresh pages, which it has to fault in), the bus 55 GB/s.
//   page-locked or managed   one asynchronous copy above SMALL_UP.
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

constexpr size_t AREA_BYTES = (size_t)4 << 20;
// Up to here the driver's own copy, of pageable bytes, stays out of the copy engine's queue (its limit is 64 KB)
constexpr size_t TINY = (size_t)64 << 10;
// Up to here one thread, from here on it and the helpers, which have to be woken.  Calls of one upload from memory that is not in the
// caller's caches, and of one result, in us, one thread against the helpers: up 330 KB 73 .. 77 against 73 .. 84, 400 KB 91 .. 97 against
// 76 .. 83, 500 KB 98 .. 101 against 78 .. 86; down 544 KB 134 .. 143 against 149 .. 155, 768 KB 154 .. 165 against 161 .. 163, 896 KB
// 171 .. 179 against 163 .. 168 (straight after the call before, and half a millisecond later).
constexpr size_t SMALL_UP = (size_t)384 << 10, SMALL_DOWN = (size_t)768 << 10;
constexpr size_t PIECE_UP = (size_t)128 << 10, PIECE_DOWN = (size_t)256 << 10;

inline void relax() {
#if defined(__x86_64__)
    __builtin_ia32_pause();
#endif
}

#if defined(__x86_64__)
// CLDEMOTE: moves a line to the cache that all cores share; a no-op where the processor has no such hint
inline void demote_line(const char* p) { asm volatile(".byte 0x0f, 0x1c, 0x00" ::"a"(p) : "memory"); }
#endif

// Past the caches, 16 bytes at a time.  `demote`: what has been read goes to the shared cache, BEHIND bytes behind the copy.
inline void copy_past_caches(char* d, const char* h, size_t bytes, bool demote = false) {
#if defined(__x86_64__)
    const size_t head = -(uintptr_t)d & 15, lead = head < bytes ? head : bytes, whole = (bytes - lead) & ~(size_t)63;
    constexpr size_t BEHIND = 4096;  // a demotion waits for its line: 16 MB up 488 us at 256 bytes, 480 at 4 KB
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

}  // namespace

bool pageable(const void* h) {
    cudaPointerAttributes attr;
    const bool yes = cudaPointerGetAttributes(&attr, h) != cudaSuccess || attr.type == cudaMemoryTypeUnregistered;
    cudaGetLastError();  // an unregistered pointer is not an error here
    return yes;
}

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

// The bounce areas: one for uploads, which the host only writes, past its caches, and one for results, which the host only reads.  (One
// area for both had the uploads write over lines that the results before had left in the caches: 512 KB 84 us instead of 50.)
static char* bounce(hl_ctx* c, hl_ctx::Bounce& b, size_t bytes) {
    if (!b.mem && cudaHostAlloc((void**)&b.mem, AREA_BYTES, cudaHostAllocDefault) != cudaSuccess) {
        cudaGetLastError();
        b.mem = nullptr;
        return nullptr;
    }
    const size_t need = (bytes + 63) & ~(size_t)63;
    if (b.off + need > AREA_BYTES && sync(c, "bounce area") != HL_B200_OK) return nullptr;  // a synchronisation empties both
    char* slot = b.mem + b.off;
    b.off += need;
    return slot;
}

static cudaError_t bounce_up(char* slot, char* d, const char* h, size_t bytes, cudaStream_t s) {
    cudaError_t e = cudaSuccess;
    for (size_t at = 0; at < bytes && e == cudaSuccess; at += PIECE_UP) {
        const size_t n = bytes - at < PIECE_UP ? bytes - at : PIECE_UP;
        copy_past_caches(slot + at, h + at, n);
        e = cudaMemcpyAsync(d + at, slot + at, n, cudaMemcpyHostToDevice, s);
    }
    return e;
}

// a result's pieces, each but the last with an event (that one comes with the stream)
static cudaError_t bounce_down(hl_ctx* c, char* slot, char* h, const char* d, size_t bytes, cudaStream_t s) {
    cudaError_t e = cudaSuccess;
    for (size_t at = 0; at < bytes && e == cudaSuccess; at += PIECE_DOWN) {
        const size_t n = bytes - at < PIECE_DOWN ? bytes - at : PIECE_DOWN;
        cudaEvent_t ev = nullptr;
        e = cudaMemcpyAsync(slot + at, d + at, n, cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess && at + n < bytes) {
            if (c->ev_spare.empty()) e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
            else { ev = c->ev_spare.back(); c->ev_spare.pop_back(); }
        }
        if (e != cudaSuccess) break;
        c->pending.push_back({h + at, slot + at, n, ev});
        if (ev) e = cudaEventRecord(ev, s);
    }
    return e;
}

// On return the caller's bytes are no longer needed, unless they are page-locked (then they are read by the end of the call that the
// copy is part of).
int h2d_on(hl_ctx* c, void* d, const void* h, size_t bytes, cudaStream_t s) {
    if (!bytes) return HL_B200_OK;
    cudaError_t e;
    char* slot;
    CopyRing* r;
    if (bytes <= TINY && pageable(h)) {
        e = cudaMemcpyAsync(d, h, bytes, cudaMemcpyHostToDevice, s);
    } else if (bytes <= SMALL_UP && (slot = bounce(c, c->up, bytes)) != nullptr) {
        c->up_elsewhere |= s != c->stream;
        e = bounce_up(slot, (char*)d, (const char*)h, bytes, s);
    } else if (pageable(h) && (r = ring_of(c)) != nullptr) {
        e = ring_up(r, (char*)d, (const char*)h, bytes, s);
    } else {
        e = cudaMemcpyAsync(d, h, bytes, cudaMemcpyHostToDevice, s);
    }
    if (e != cudaSuccess) return fail(c, HL_B200_ERR_DEVICE, "copy to device", e);
    c->stats.bytes_h2d += bytes;
    return HL_B200_OK;
}

int h2d(hl_ctx* c, void* d, const void* h, size_t bytes) { return h2d_on(c, d, h, bytes, c->stream); }

// The same for calls that return before the stream has been waited for: page-locked bytes are waited for here.
int h2d_owned(hl_ctx* c, void* d, const void* h, size_t bytes) {
    int rc = h2d(c, d, h, bytes);
    if (!rc && bytes > SMALL_UP && !pageable(h)) rc = sync(c, "copy to device");
    return rc;
}

// The bytes are in the caller's memory after the next `sync`.
int d2h_on(hl_ctx* c, void* h, const void* d, size_t bytes, cudaStream_t s) {
    if (!bytes) return HL_B200_OK;
    cudaError_t e;
    CopyRing* r;
    char* slot;
    if (bytes <= SMALL_DOWN && (bytes <= SMALL_UP || pageable(h)) && (slot = bounce(c, c->down, bytes)) != nullptr) {
        e = bounce_down(c, slot, (char*)h, (const char*)d, bytes, s);
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

// hands the results in the bounce area out, each piece when it has arrived, and waits for the stream
int sync(hl_ctx* c, const char* what) {
    cudaError_t e = cudaSuccess;
    bool through = false;  // the stream has been waited for
    for (const auto& p : c->pending) {
        if (!through) {
            e = p.ev ? cudaEventSynchronize(p.ev) : cudaStreamSynchronize(c->stream);
            through = !p.ev;
        }
        if (e != cudaSuccess) break;
        memcpy(p.to, p.from, p.bytes);
    }
    if (!through && e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    if (c->up_elsewhere && e == cudaSuccess) e = cudaStreamSynchronize(c->copy_stream);  // it reads the upload area too
    c->up_elsewhere = false;
    drop_pending(c);
    c->up.off = c->down.off = 0;
    if (e != cudaSuccess) return fail(c, HL_B200_ERR_DEVICE, what, e);
    return HL_B200_OK;
}

void drop_pending(hl_ctx* c) {
    for (const auto& p : c->pending)
        if (p.ev) c->ev_spare.push_back(p.ev);
    c->pending.clear();
}

}  // namespace hlapi
