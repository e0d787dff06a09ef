// Host-side objects behind the opaque handles of include/hl_b200.h.
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <map>
#include <set>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/hl_b200.h"
#include "kernels.h"
#include "sumcheck.h"

namespace hlapi { struct CopyRing; }

struct hl_ctx {
    int device = 0;
    int sm_count = 0;
    cudaStream_t own_stream = nullptr;
    cudaStream_t stream = nullptr;
    cudaStream_t copy_stream = nullptr;     // uploads that overlap the encoder
    cudaEvent_t ev_main = nullptr;
    std::vector<cudaEvent_t> ev_chunks;
    bool fast_encoder = true;
    bool slot_kernels = false;  // run a slot program whose graph is known through its generated kernel instead of its program (measured slower: off)
    std::mutex mu;
    std::mutex err_mu;       // guards last_error and stats.declines: a decline may be recorded before `mu` is taken, from any thread
    std::map<u32, u64*> tw;  // log2 nn -> nn powers of the nn-th root
    std::map<u32, u64*> enc_tables;  // log2 n + 64 log2 rate -> the tensor-core encoder's constants
    // Where the tensor-core encoder tells that a bounded wait ran out: a page-locked word for each of its stores, into which the store's own
    // mark is written, so that a word can go on to the next store while the last one's kernels are still queued; and one that asynchronous
    // commitments set as well, which hl_b200_sync reads
    std::vector<u32*> enc_blocks, enc_words;  // 1,024 words each; those that no store has
    u32* enc_later = nullptr;
    u32 enc_mark = 0, enc_limit = 1u << 22;
    std::string label, last_error;
    hl_stats stats{};
    bool timing = false;
    hlk::ScWaits waits;      // of the sumchecks' resident CTAs
    struct Span { cudaEvent_t a, b; int cls; };
    std::vector<Span> spans;          // recorded, not yet read
    std::vector<cudaEvent_t> ev_pool;  // events ready for reuse
    hl_timing timing_acc{};
    hlapi::CopyRing* ring = nullptr;  // page-locked slots for large copies of pageable host memory (host_copy.cu, made on first use)
    // page-locked bounce areas for small copies (host_copy.cu), empty after every synchronisation
    struct Bounce { char* mem = nullptr; size_t off = 0; } up, down;
    bool up_elsewhere = false;  // a copy from the upload area went to the copy stream
    struct Pending { void* to; const char* from; size_t bytes; cudaEvent_t ev; };  // ev: when the piece has arrived (none: with the stream)
    std::vector<Pending> pending;  // pieces of results on their way through the bounce area, handed out by the next `sync`
    std::vector<cudaEvent_t> ev_spare;
    int* wp_flag = nullptr;  // page-locked: the witness products' status word: zero between calls
    bool wp_attr = false;      // the product kernel's shared-memory size has been raised on this device
    std::set<const struct hl_store*> stores;  // the live commitment stores (a planned slot table that reads one checks it is still there when it is built)
    // something of the present call has failed: its copies may still be under way, on either stream (`settle`)
    std::atomic<bool> failed{false};
    size_t alloc_live = 0;   // bytes handed out and not yet returned
    size_t alloc_cap = 0;    // 0 = none; a host-side failure-injection cap (mod.rs:121 set_alloc_cap_for_test)
};

struct hl_store {
    hl_ctx* ctx = nullptr;
    u32 rows = 0, logn = 0, logr = 0, q = 0;
    bool zk = false;
    bool owns_inputs = true;      // false: d_data / d_pads belong to the caller
    bool fold_data = false;       // a plain store whose row fold reads d_data (a masking commitment's coefficient rows)
    u64* d_data = nullptr;        // rows x n
    u64* d_pads = nullptr;        // rows x q
    u64* d_enc = nullptr;         // rows x nn, the words of a row in `order`
    ColOrder order;
    uint32_t* d_leaves = nullptr; // nn x 8 words, unsalted
    int encoder_path = -1;
    u32* enc_word = nullptr;      // holds enc_mark: the encoder gave up, nothing of the encoding is valid (encoded_ok)
    u32 enc_mark = 0;
    size_t n() const { return (size_t)1 << logn; }
    size_t nn() const { return (size_t)1 << (logn + logr); }
};

namespace hlapi {
int fail(hl_ctx* c, int code, const char* what, cudaError_t e = cudaSuccess);
int dev_alloc(hl_ctx* c, void** p, size_t bytes);
bool dev_try(hl_ctx* c, void** p, size_t bytes, cudaError_t* why = nullptr);
void dev_free(hl_ctx* c, void* p, size_t bytes);
void settle(hl_ctx* c);  // waits for both streams if something of the present call has failed
// host_copy.cu: uploads on the context's stream (h2d_on: on another one that the context's stream waits for before the call ends);
// h2d_owned: the caller's bytes are no longer needed when it returns, whatever kind of host memory they live in;
// d2h: the bytes are in place after the next `sync`
bool pageable(const void* h);
int h2d(hl_ctx* c, void* d, const void* h, size_t bytes);
int h2d_on(hl_ctx* c, void* d, const void* h, size_t bytes, cudaStream_t s);
int h2d_owned(hl_ctx* c, void* d, const void* h, size_t bytes);
int d2h(hl_ctx* c, void* h, const void* d, size_t bytes);
// the same on a second stream; the context's stream waits for it
int d2h_on(hl_ctx* c, void* h, const void* d, size_t bytes, cudaStream_t s);
int sync(hl_ctx* c, const char* what);
void drop_pending(hl_ctx* c);
void host_copy_retain();
void host_copy_release(hl_ctx* c);
void host_copy_drop();

// What every entry point that works on a context holds: its lock and its device.  A call that succeeds has waited for what it queued, or
// keeps it on the context's stream.  One that fails on the way has not, and `dev_free` orders what it gives back after the context's stream
// alone: so a failed call settles before it frees anything and before it returns.  Results that it left in the bounce area go with it:
// nothing may write to that caller's memory later.
struct Call {
    hl_ctx* c;
    std::lock_guard<std::mutex> g;
    explicit Call(hl_ctx* ctx) : c(ctx), g(ctx->mu) {
        cudaSetDevice(c->device);
        c->failed = false;
    }
    ~Call() {
        settle(c);
        drop_pending(c);
    }
};
int root_powers(hl_ctx* c, u32 lognn, const u64** out);
int encoder_tables(hl_ctx* c, u32 logn, u32 logr, const u64** out);
int encoder_word(hl_ctx* c, hl_store* st);
int encoded_ok(hl_ctx* c, const hl_store* st);  // asked once the encoding has been waited for: HL_B200_ERR_TIMEOUT if the encoder gave up
int upload_key(hl_ctx* c, const uint8_t* key32, uint32_t** d_key);
int log2_exact(size_t v);
void store_release(hl_store* st);  // frees a store; the caller holds the context's lock
// a hiding commitment of rows that are on the device already (hl_b200_commit_zk_dev); the caller holds the context's lock.
// leaves false: the encoding alone is wanted, its columns are not hashed
int commit_resident(hl_ctx* c, u32 log_cols, u32 inv_rate, const u64* d_data, size_t rows, const u64* d_pads, size_t q, const u64* d_pows,
                    const uint8_t* key32, hl_store** store, uint8_t* d_leaves32, bool leaves = true);

// rho^T [M | pads] for k host vectors over a device matrix, each by the kernel for its support
struct FoldSource {
    const u64* d = nullptr;   // element (i, j) at d[i ld + j ir]
    const u64* pads = nullptr;
    size_t ld = 0;
    u32 rows = 0, n = 0, q = 0, ir = 1;
};
struct FoldPlan {
    hl_ctx* c = nullptr;
    FoldSource src;
    u32 kd = 0, ks = 0, few = 0, splits = 1;
    std::vector<u32> sparse_map;
    char* blk = nullptr;
    size_t blk_bytes = 0, part_bytes = 0;
    u64 *d_rhos = nullptr, *d_sw = nullptr, *d_part = nullptr;
    u32 *d_soff = nullptr, *d_srows = nullptr, *d_dmap = nullptr, *d_smap = nullptr;
    int make(hl_ctx* c, const FoldSource& src, const uint64_t* rhos, size_t k);
    bool sparse_span(u32* first) const;  // whether the sparse vectors are neighbours, and where they start
    int launch_sparse(u64* d_out);
    int launch_dense(u64* d_out);
    void release();
};

// Brackets the launches of one kernel family with two events when the context's timing is on.
struct Timed {
    hl_ctx* c;
    hl_ctx::Span s;
    bool on;
    Timed(hl_ctx* c, int cls);
    ~Timed();
};
}  // namespace hlapi
