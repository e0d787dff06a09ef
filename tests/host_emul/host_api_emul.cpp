// The library's host code over a runtime without a device (fake_cuda.h).
//   host_api_emul failures     every entry point below with every fallible call of it failing in turn: whatever happens, no memory goes while
//                              a copy uses it, no copy uses the caller's memory once the call is over, and nothing is lost
//   host_api_emul copies       the bytes of copies of all sizes and alignments
//   host_api_emul threads N    the same where the process can make only N threads
//   host_api_emul timeouts     who is told that a row encoder's bounded wait ran out
//   host_api_emul pieces       the row pieces of uploads
//   host_api_emul reorder      the encoding's way into the columns' order: once, whatever fails, and with little memory
#include "fake_cuda.h"

#include <dlfcn.h>
#include <pthread.h>

#include <cerrno>
#include <cstdio>
#include <functional>

#include "../../intelligenceregulation_b200/csrc/api_internal.h"

static long g_threads = -1;  // how many more threads may be made (-1: any number)
extern "C" int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* x) noexcept {
    static auto real = (int (*)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*))dlsym(RTLD_NEXT, "pthread_create");
    if (g_threads == 0) return EAGAIN;
    if (g_threads > 0) g_threads--;
    return real(t, a, f, x);
}

namespace hlk {
static cudaError_t launch() { return fake::fails() ? cudaErrorUnknown : cudaSuccess; }
size_t encode_scratch_words(u32, u32, int, u32) { return 64; }
bool encode_split_pays(u32, u32, u32, int) { return false; }
static std::vector<u32> g_pieces;  // the rows of every encoder launch
cudaError_t encode_rows(const enc::RowArgs& a, u32, bool, int, size_t, cudaStream_t, int*) { g_pieces.push_back(a.rows); return launch(); }
size_t encode_tc_table_words(u32, u32) { return 8; }
void encode_tc_build(u32, u32, u64* out) { for (int i = 0; i < 8; i++) out[i] = 0; }
bool encode_tc_takes(u32 logn, u32, u32, int) { return logn >= 10; }
size_t encode_tc_scratch_words(u32, u32, u32, u32, int) { return 64; }
size_t encode_tc_least_words(u32, u32, u32, u32, int) { return 32; }
static bool g_gives_up = false;  // the encoder's waits run out
cudaError_t encode_rows_tc(enc::RowArgs a, u32, const u64*, int, size_t, TcReport r, cudaStream_t, int*) {
    g_pieces.push_back(a.rows);
    if (g_gives_up) {
        *r.word = r.mark;
        if (r.also) *r.also = 1;
    }
    return launch();
}
u32 natural_order_rows(u32 rows, int sms) { return rows < 2u * sms ? rows : 2u * sms; }
static u32 g_reorders = 0, g_reorder_ctas = 0;
cudaError_t natural_order(u64*, u32, size_t, ColOrder, u64*, u32 ctas, cudaStream_t) {
    if (fake::fails()) return cudaErrorUnknown;
    g_reorders++;
    g_reorder_ctas = ctas;
    return cudaSuccess;
}
cudaError_t widen_rows(const unsigned char*, const u64*, const unsigned char*, u64*, u32, u32, int, cudaStream_t) { return launch(); }
u32 hash_chunks(u32 rows) { return (rows + 127) / 128; }
cudaError_t hash_column_chunks(const u64*, u32, u32, const uint32_t*, u32, u32, uint32_t*, uint32_t*, cudaStream_t, ColOrder) { return launch(); }
cudaError_t hash_column_merge(u32, u32, const uint32_t*, const uint32_t*, uint32_t*, cudaStream_t, ColOrder) { return launch(); }
cudaError_t hash_columns(const u64*, u32, u32, const uint32_t*, uint32_t*, uint32_t*, cudaStream_t, ColOrder) { return launch(); }
cudaError_t merkle_tree(const uint32_t*, const uint32_t*, u32, const uint32_t*, const uint32_t*, uint32_t*, cudaStream_t, int* n) { *n = 1; return launch(); }
u32 fold_row_splits(u32, u32, u32, u32, int) { return 1; }
u32 fold_few_ranges(u32, u32, u32, u32, u32, int) { return 0; }
cudaError_t fold_rows_few(const u64*, u32, u32, size_t, const u64*, u32, size_t, const u64*, u32, const u32*, u64*, u32, u32, u64*, cudaStream_t) { return launch(); }
cudaError_t fold_rows(const u64*, u32, u32, size_t, u32, const u64*, u32, size_t, const u64*, u32, const u32*, u64*, u32, cudaStream_t, u32, u64*) { return launch(); }
cudaError_t fold_rows_sparse(const u64*, u32, size_t, u32, const u64*, u32, size_t, const u32*, const u32*, const u64*, u32, const u32*, u64*, u32, cudaStream_t) { return launch(); }
cudaError_t gather_columns(const u64*, u32, size_t, const u64*, u32, u64*, cudaStream_t, ColOrder) { return launch(); }
// out: a + b, a - b, a b, three words a pair.  Here: a, b, 0, which shows that both arrays arrived and the results came back
cudaError_t probe_field(const u64* a, const u64* b, size_t n, u64* out, cudaStream_t st) {
    cudaStreamSynchronize(st);
    for (size_t i = 0; i < n; i++) { out[3 * i] = a[i]; out[3 * i + 1] = b[i]; out[3 * i + 2] = 0; }
    return launch();
}
cudaError_t butterfly_peak(const u64*, u64*, u32, int, cudaStream_t) { return launch(); }
cudaError_t compress_peak(const u64*, u64*, u32, int, cudaStream_t) { return launch(); }
}  // namespace hlk

// memory of the caller, page-locked or not
struct Host {
    std::vector<std::vector<uint64_t>> all;
    bool lock;
    explicit Host(bool l) : lock(l) {}
    uint64_t* words(size_t n) {
        all.emplace_back(n, 1);
        if (lock) fake::locked[(const char*)all.back().data()] = n * 8;
        return all.back().data();
    }
    uint8_t* bytes(size_t n) { return (uint8_t*)words((n + 7) / 8); }
    bool busy() const {
        for (auto& v : all)
            if (fake::busy(v.data(), v.size() * 8)) return true;
        return false;
    }
    ~Host() {
        if (lock)
            for (auto& v : all) fake::locked.erase((const char*)v.data());
    }
};

static int g_bad = 0;
static void bad(const char* what, const std::string& how) {
    if (g_bad++ < 200) printf("%s: %s\n", what, how.c_str());
}

static void sweep(const char* what, hl_ctx* c, Host& h, const std::function<int()>& call) {
    fake::fail_at = -1;
    if (call()) bad(what, "fails with nothing failing");
    const size_t blocks = fake::device.size(), live = c->alloc_live;
    for (long at = 0;; at++) {
        fake::calls = 0;
        fake::fail_at = at;
        const int rc = call();
        const bool past = fake::calls <= at;
        fake::fail_at = -1;
        const std::string where = " (call " + std::to_string(at) + ", rc " + std::to_string(rc) + ")";
        if (h.busy()) bad(what, "a copy uses the caller's memory after the call" + where);
        for (auto& f : fake::faults) bad(what, f + where);
        fake::faults.clear();
        cudaStreamSynchronize(c->stream);
        cudaStreamSynchronize(c->copy_stream);
        for (auto& f : fake::faults) bad(what, f + ", later" + where);
        fake::faults.clear();
        if (fake::device.size() != blocks || c->alloc_live != live) bad(what, "device memory lost" + where);
        if (past) break;
    }
    if (call()) bad(what, "does not recover");
}

static void failures(bool lock) {
    hl_ctx* c = nullptr;
    hl_b200_init(0, &c);
    const uint8_t key[32] = {1};
    for (const u32 rows : {6u, 300u}) {  // whole, and in pieces (32 MiB and more than four waves of the encoder)
        const u32 lc = rows == 6 ? 12 : 14, q = 40;
        const size_t n = (size_t)1 << lc, nn = 2 * n;
        Host h(lock);
        uint64_t *data = h.words(rows * n), *pads = h.words(rows * q), *pows = h.words(nn);
        uint8_t *salts = h.bytes(nn * 32), *levels = h.bytes((2 * nn - 1) * 32), *leaves = h.bytes(nn * 32), *widths = h.bytes(rows);
        memset(widths, 8, rows);
        const char* names[2] = {"commit_zk_packed", "commit_zk_tree"};
        for (int form = 0; form < (rows == 6 ? 2 : 1); form++)
            sweep(names[form], c, h, [&] {
                hl_store* st = nullptr;
                const int rc = form ? hl_b200_commit_zk_tree(c, lc, 2, data, rows, pads, q, pows, lc + 1, key, salts, key, key, &st, leaves, levels)
                                    : hl_b200_commit_zk_packed(c, lc, 2, data, widths, rows, pads, q, pows, lc + 1, key, salts, key, key, &st, leaves, levels);
                hl_b200_store_free(st);
                return rc;
            });
        hl_store* st = nullptr;
        hl_b200_commit_zk(c, lc, 2, data, rows, pads, q, pows, lc + 1, key, &st, leaves);
        if (rows == 6) sweep("store_merkle", c, h, [&] { return hl_b200_store_merkle(st, salts, key, key, levels); });
        if (rows == 6) sweep("merkle", c, h, [&] { return hl_b200_merkle(c, leaves, salts, nn, key, key, levels); });
        const size_t k = 9, cols = 70;  // eight vectors that live on one row, together, and a dense one: their results go back on both streams
        uint64_t *rhos = h.words(k * rows * 2), *out = h.words(k * (n + q) * 2), *idx = h.words(cols), *got = h.words(cols * rows);
        for (size_t g = 0; g + 1 < k; g++) memset(rhos + (g * rows + 1) * 2, 0, (rows - 1) * 16);
        sweep("store_fold", c, h, [&] { return hl_b200_store_fold(st, rhos, k, 1, out); });
        sweep("store_columns", c, h, [&] { return hl_b200_store_columns(st, idx, cols, got); });
        hl_b200_store_free(st);
    }
    hl_b200_shutdown(c);
}

// every size class of the copies and both sides of its limits, at every alignment that words have
static void sizes(bool lock) {
    hl_ctx* c = nullptr;
    hl_b200_init(0, &c);
    for (const size_t n : {1, 7, 8191, 8192, 8193, 16384, 16385, 21845, 32768, 32769, 43691, 49152, 49153, 65537, 100001, 3000001}) {
        std::vector<uint64_t> a(n + 8), b(n + 8), out(3 * n + 8);
        for (size_t i = 0; i < n + 8; i++) { a[i] = i * 0x9E3779B97F4A7C15ull; b[i] = ~a[i]; }
        if (lock)
            for (auto* v : {&a, &b, &out}) fake::locked[(const char*)v->data()] = v->size() * 8;
        for (size_t off = 0; off < (n > 1000000 ? 2u : 8u); off++) {
            std::fill(out.begin(), out.end(), 7);
            if (hl_b200_probe_field(c, a.data() + off, b.data() + off, n, out.data() + off)) bad("probe_field", "refused");
            const uint64_t* o = out.data() + off;
            bool ok = true;
            for (size_t i = 0; i < n && ok; i++) ok = o[3 * i] == a[off + i] && o[3 * i + 1] == b[off + i] && !o[3 * i + 2];
            for (size_t i = 0; i < off; i++) ok = ok && out[i] == 7;
            for (size_t i = 3 * n + off; i < out.size(); i++) ok = ok && out[i] == 7;
            if (!ok) bad("probe_field", "wrong bytes at " + std::to_string(n) + " words, offset " + std::to_string(off));
        }
        if (lock)
            for (auto* v : {&a, &b, &out}) fake::locked.erase((const char*)v->data());
    }
    hl_b200_shutdown(c);
}

// more small copies in one call than the bounce areas hold, on both streams in turn
static void areas() {
    hl_ctx* c = nullptr;
    hl_b200_init(0, &c);
    const size_t n = 40000, count = 50;
    std::vector<uint64_t> a(n * count), out(n * count);
    for (size_t i = 0; i < a.size(); i++) a[i] = i * 0x9E3779B97F4A7C15ull;
    {
        hlapi::Call g(c);
        u64* d = nullptr;
        int rc = hlapi::dev_alloc(c, (void**)&d, a.size() * 8);
        for (size_t i = 0; i < count && !rc; i++) rc = hlapi::h2d_on(c, d + i * n, a.data() + i * n, n * 8, i % 3 ? c->copy_stream : c->stream);
        cudaEventRecord(c->ev_main, c->copy_stream);
        cudaStreamWaitEvent(c->stream, c->ev_main, 0);
        for (size_t i = 0; i < count && !rc; i++) rc = hlapi::d2h_on(c, out.data() + i * n, d + i * n, n * 8, i % 3 ? c->stream : c->copy_stream);
        if (!rc) rc = hlapi::sync(c, "areas");
        hlapi::dev_free(c, d, a.size() * 8);
        if (rc || a != out) bad("areas", "wrong bytes");
    }
    hl_b200_shutdown(c);
}

// A wait of the encoder that runs out is told to the calls on that store, and for an asynchronous commitment to hl_b200_sync, once; never to
// another call.
static void timeouts() {
    hl_ctx* c = nullptr;
    hl_b200_init(0, &c);
    const u32 rows = 6, lc = 12, q = 40;
    const size_t n = (size_t)1 << lc, nn = 2 * n;
    Host h(false);
    uint64_t *data = h.words(rows * n), *pads = h.words(rows * q), *pows = h.words(nn), *idx = h.words(1), *got = h.words(rows), *rhos = h.words(rows * 2);
    uint64_t *out = h.words((n + q) * 2);
    uint8_t *leaves = h.bytes(nn * 32), *levels = h.bytes((2 * nn - 1) * 32);
    idx[0] = 1;
    auto host = [&](bool gives_up, hl_store** st) {
        hlk::g_gives_up = gives_up;
        return hl_b200_commit_zk(c, lc, 2, data, rows, pads, q, pows, lc + 1, nullptr, st, leaves);
    };
    auto dev = [&](bool gives_up, hl_store** st) {
        hlk::g_gives_up = gives_up;
        return hl_b200_commit_zk_dev(c, lc, 2, data, rows, pads, q, pows, nullptr, st, nullptr);
    };
    auto is = [&](int rc, int want, const char* what) {
        if (rc != want) bad("timeouts", std::string(what) + " answers " + std::to_string(rc));
    };
    hl_store *lost = nullptr, *fine = nullptr, *none = nullptr;
    is(dev(true, &lost), 0, "an asynchronous commitment that will give up");
    is(host(false, &fine), 0, "another commitment");
    is(hl_b200_store_columns(fine, idx, 1, got), 0, "the other store's columns");
    for (int again = 0; again < 2; again++) {
        is(hl_b200_store_columns(lost, idx, 1, got), HL_B200_ERR_TIMEOUT, "columns");
        is(hl_b200_store_fold(lost, rhos, 1, 1, out), HL_B200_ERR_TIMEOUT, "fold");
        is(hl_b200_store_merkle(lost, nullptr, nullptr, nullptr, levels), HL_B200_ERR_TIMEOUT, "tree");
        if (hl_b200_store_encoded_dev(lost)) bad("timeouts", "the encoding is given out");
    }
    is(hl_b200_sync(c), HL_B200_ERR_TIMEOUT, "sync");
    is(hl_b200_sync(c), 0, "sync, later");
    hl_b200_store_free(lost);
    is(dev(true, &lost), 0, "an asynchronous commitment that will give up");
    hl_b200_store_free(lost);
    is(host(false, &lost), 0, "a commitment after it");
    is(hl_b200_store_columns(lost, idx, 1, got), 0, "its columns");
    is(hl_b200_sync(c), HL_B200_ERR_TIMEOUT, "sync for a store that is gone");
    hl_b200_store_free(lost);
    is(host(true, &none), HL_B200_ERR_TIMEOUT, "a commitment that gives up");
    if (none) bad("timeouts", "a failed commitment left a store");
    is(hl_b200_sync(c), 0, "sync after a commitment that told it itself");
    for (long at = 0; at < 200; at++) {  // whatever else fails in a call whose encoder gives up, the next call does not hear of it
        fake::calls = 0;
        fake::fail_at = at;
        hl_store* st = nullptr;
        host(true, &st);
        fake::fail_at = -1;
        is(hl_b200_store_columns(fine, idx, 1, got), 0, "another store's columns after a call that failed");
        is(hl_b200_sync(c), 0, "sync after a call that failed");
    }
    for (int i = 0; i < 3000; i++) {  // more words than a block holds, given back in between
        hl_store* st = nullptr;
        is(dev(false, &st), 0, "a commitment");
        hl_b200_store_free(st);
    }
    std::vector<hl_store*> many(2500);
    for (auto& st : many) is(dev(false, &st), 0, "a commitment");
    is(hl_b200_sync(c), 0, "sync");
    for (auto& st : many) hl_b200_store_free(st);
    hl_b200_store_free(fine);
    hlk::g_gives_up = false;
    hl_b200_shutdown(c);
}

static void reorder() {
    hl_ctx* c = nullptr;
    hl_b200_init(0, &c);
    const u32 rows = 6, lc = 12, q = 40;
    const size_t n = (size_t)1 << lc, nn = 2 * n;
    Host h(false);
    uint64_t *data = h.words(rows * n), *pads = h.words(rows * q), *pows = h.words(nn);
    uint8_t* leaves = h.bytes(nn * 32);
    hl_store* st = nullptr;
    auto commit = [&] { return hl_b200_commit_zk(c, lc, 2, data, rows, pads, q, pows, lc + 1, nullptr, &st, leaves); };
    // every fallible call of it in turn: the rows are never put in order a second time, and where they have not been the store says so
    for (long at = 0;; at++) {
        commit();
        hlk::g_reorders = 0;
        fake::calls = 0;
        fake::fail_at = at;
        hl_b200_store_encoded_dev(st);
        fake::fail_at = -1;
        const bool past = fake::calls <= at;
        if ((st->order.logr == 0) != (hlk::g_reorders == 1)) bad("reorder", "the store's order is not that of its rows, call " + std::to_string(at));
        if (!hl_b200_store_encoded_dev(st)) bad("reorder", "does not recover");
        if (hlk::g_reorders != 1) bad("reorder", "the rows were put in order " + std::to_string(hlk::g_reorders) + " times, call " + std::to_string(at));
        hl_b200_store_free(st);
        if (past) break;
    }
    commit();
    hlk::g_reorders = 0;
    fake::next_wait_fails = true;  // behind the launch
    if (hl_b200_store_encoded_dev(st)) bad("reorder", "a failed wait is not told");
    if (!hl_b200_store_encoded_dev(st) || hlk::g_reorders != 1 || st->order.logr) bad("reorder", "after a failed wait the rows are put in order again");
    hl_b200_store_free(st);
    for (u32 fit = 0; fit <= 6; fit++) {  // memory for so many rows
        commit();
        const u64 declines = c->stats.declines;
        hl_b200_set_alloc_cap(c, c->alloc_live + fit * nn * 8 + (fit ? 0 : 1));
        hlk::g_reorder_ctas = 0;
        const uint64_t* p = hl_b200_store_encoded_dev(st);
        hl_b200_set_alloc_cap(c, 0);
        const u32 want = fit >= 6 ? 6 : fit >= 3 ? 3 : fit >= 1 ? 1 : 0;
        if ((p != nullptr) != (fit > 0) || hlk::g_reorder_ctas != want || (c->stats.declines != declines) != (fit == 0))
            bad("reorder", "with memory for " + std::to_string(fit) + " rows " + std::to_string(hlk::g_reorder_ctas) + " at once");
        hl_b200_store_free(st);
    }
    hl_b200_shutdown(c);
}

// Every row in one piece, whole batches but for the last; 64-bit rows of every length come in pieces from 32 MB on, no more than two turns of
// the machine each and no more than one at the end, and small or resident ones whole.
static void pieces() {
    hl_ctx* c = nullptr;
    hl_b200_init(0, &c);
    struct { u32 lc, rows, bytes; bool lock; u32 last; } all[] = {  // last: batches of 2^14 words behind which nothing is on the bus
        {14, 300, 8, true, 74}, {14, 1000, 8, false, 74}, {13, 520, 8, true, 74}, {13, 1000, 8, true, 74}, {13, 1001, 8, true, 74}, {12, 1500, 8, false, 74},
        {12, 2301, 8, true, 74}, {11, 3001, 8, true, 74}, {10, 4097, 8, true, 74}, {9, 9000, 8, true, 74}, {8, 20001, 8, true, 74}, {14, 600, 4, true, 74}, {12, 4500, 2, true, 148},
        {14, 1100, 2, false, 148}, {14, 1100, 2, true, 296}, {10, 34000, 1, true, 296}, {14, 2605, 1, true, 296}, {15, 161, 8, true, 74}, {14, 255, 8, true, 0}, {12, 900, 8, true, 0}};
    for (auto& k : all) {
        const size_t n = (size_t)1 << k.lc, nn = 2 * n;
        const u32 batch = k.lc < 14 ? 16384u >> k.lc : 1u;
        Host h(k.lock);
        uint64_t *data = h.words(k.rows * n * k.bytes / 8), *pads = h.words(k.rows), *pows = h.words(nn);
        uint8_t *leaves = h.bytes(nn * 32), *widths = h.bytes(k.rows);
        memset(widths, k.bytes, k.rows);
        hlk::g_pieces.clear();
        hl_store* st = nullptr;
        if (hl_b200_commit_zk_packed(c, k.lc, 2, data, widths, k.rows, pads, 1, pows, 0, nullptr, nullptr, nullptr, nullptr, &st, leaves, nullptr)) bad("pieces", "refused");
        hl_b200_store_free(st);
        const std::vector<u32> p = hlk::g_pieces;
        std::string how = "2^" + std::to_string(k.lc) + ":";
        u32 sum = 0;
        bool ok = !p.empty() && (p.size() > 1) == (k.last > 0);
        for (size_t i = 0; i < p.size(); i++) {
            how += " " + std::to_string(p[i]);
            sum += p[i];
            ok = ok && p[i] > 0 && (i + 1 == p.size() || p[i] % batch == 0) && (p.size() == 1 || p[i] <= 3 * 148 * batch);
        }
        if (!ok || sum != k.rows || (k.last && (p.back() + batch - 1) / batch > k.last)) bad("pieces", how);
    }
    hl_b200_shutdown(c);
}

int main(int argc, char** argv) {
    if (argc == 3 && !strcmp(argv[1], "threads")) {
        g_threads = atol(argv[2]);
        sizes(false);
    } else if (argc == 2 && !strcmp(argv[1], "copies")) {
        sizes(false);
        sizes(true);
        areas();
    } else if (argc == 2 && !strcmp(argv[1], "timeouts")) {
        timeouts();
    } else if (argc == 2 && !strcmp(argv[1], "reorder")) {
        reorder();
    } else if (argc == 2 && !strcmp(argv[1], "pieces")) {
        pieces();
    } else {
        failures(false);
        failures(true);
    }
    if (!g_bad) printf("ok\n");
    return g_bad != 0;
}
