// C ABI: commitments (Backend::try_commit*), stores (EncodedStore), Merkle trees.
#include <algorithm>
#include <cstring>

#include "api_internal.h"

using namespace hlapi;

namespace hlapi {

// An opening's group vectors are zero outside their claims' rows (pcs.rs:851-891), its proximity vector is dense.  Vectors with few
// non-zero rows go to the list kernel, the others to the dense ones; all write the caller's order.
int FoldPlan::make(hl_ctx* ctx, const FoldSource& source, const uint64_t* rhos, size_t k) {
    c = ctx;
    src = source;
    const u32 rows = src.rows;
    std::vector<u32> dense, s_off{0}, s_rows;
    std::vector<u64> s_w;
    for (size_t g = 0; g < k; g++) {
        const uint64_t* r = rhos + g * (size_t)rows * 2;
        const size_t from = s_rows.size();
        bool is_sparse = true;
        for (u32 i0 = 0; i0 < rows && is_sparse; i0 += 8) {
            const u32 i1 = i0 + 8 < rows ? i0 + 8 : rows;
            u64 any = 0;
            for (u32 i = 2 * i0; i < 2 * i1; i++) any |= r[i];
            if (!any) continue;
            for (u32 i = i0; i < i1; i++)
                if (r[2 * i] | r[2 * i + 1]) { s_rows.push_back(i); s_w.push_back(r[2 * i]); s_w.push_back(r[2 * i + 1]); }
            is_sparse = (s_rows.size() - from) * 8u <= rows;
        }
        if (is_sparse) {
            s_off.push_back((u32)s_rows.size());
            sparse_map.push_back((u32)g);
        } else {
            s_rows.resize(from);
            s_w.resize(2 * from);
            dense.push_back((u32)g);
        }
    }
    kd = (u32)dense.size();
    ks = (u32)sparse_map.size();
    // one upload: 64-bit words first
    const size_t wd = (size_t)kd * rows * 2, words = wd + s_w.size(), ints = s_rows.size() + s_off.size() + kd + ks;
    std::vector<u64> up(words + (ints + 1) / 2);
    for (u32 i = 0; i < kd; i++) memcpy(up.data() + (size_t)i * rows * 2, rhos + dense[i] * (size_t)rows * 2, (size_t)rows * 16);
    if (s_w.size()) memcpy(up.data() + wd, s_w.data(), s_w.size() * 8);
    u32* ip = reinterpret_cast<u32*>(up.data() + words);
    const size_t o_rows = s_off.size(), o_dmap = o_rows + s_rows.size(), o_smap = o_dmap + kd;
    memcpy(ip, s_off.data(), s_off.size() * 4);
    if (s_rows.size()) memcpy(ip + o_rows, s_rows.data(), s_rows.size() * 4);
    if (kd) memcpy(ip + o_dmap, dense.data(), kd * 4);
    if (ks) memcpy(ip + o_smap, sparse_map.data(), ks * 4);
    few = kd ? hlk::fold_few_ranges(rows, src.n, src.q, kd, src.ir, c->sm_count) : 0;
    splits = kd && !few ? hlk::fold_row_splits(rows, src.n, src.q, kd, c->sm_count) : 1;
    const size_t w = (size_t)src.n + src.q;
    part_bytes = few ? (size_t)few * kd * w * 16 : splits > 1 ? (size_t)splits * kd * w * 16 : 0;
    blk_bytes = ((up.size() * 8 + 15) & ~(size_t)15) + part_bytes;
    int rc = dev_alloc(c, (void**)&blk, blk_bytes);
    if (!rc) rc = h2d(c, blk, up.data(), up.size() * 8);
    if (rc) return rc;
    d_rhos = (u64*)blk;
    d_sw = d_rhos + wd;
    d_soff = (u32*)(d_rhos + words);
    d_srows = d_soff + o_rows;
    d_dmap = d_soff + o_dmap;
    d_smap = d_soff + o_smap;
    d_part = part_bytes ? (u64*)(blk + blk_bytes - part_bytes) : nullptr;
    return HL_B200_OK;
}

bool FoldPlan::sparse_span(u32* first) const {
    if (!ks || sparse_map.back() - sparse_map.front() + 1 != ks) return false;  // the map is increasing
    *first = sparse_map.front();
    return true;
}

int FoldPlan::launch_sparse(u64* d_out) {
    if (!ks) return HL_B200_OK;
    cudaError_t e = hlk::fold_rows_sparse(src.d, src.n, src.ld, src.ir, src.pads, src.q, src.q, d_soff, d_srows, d_sw, ks, d_smap, d_out, src.n + src.q, c->stream);
    c->stats.kernel_launches++;
    return e == cudaSuccess ? HL_B200_OK : fail(c, HL_B200_ERR_DEVICE, "fold launch", e);
}

int FoldPlan::launch_dense(u64* d_out) {
    if (!kd) return HL_B200_OK;
    const u32 w = src.n + src.q;
    cudaError_t e = few ? hlk::fold_rows_few(src.d, src.rows, src.n, src.ld, src.pads, src.q, src.q, d_rhos, kd, d_dmap, d_out, w, few, d_part, c->stream)
                        : hlk::fold_rows(src.d, src.rows, src.n, src.ld, src.ir, src.pads, src.q, src.q, d_rhos, kd, d_dmap, d_out, w, c->stream, splits, d_part);
    c->stats.kernel_launches += few || splits > 1 ? 2 : 1;
    return e == cudaSuccess ? HL_B200_OK : fail(c, HL_B200_ERR_DEVICE, "fold launch", e);
}

void FoldPlan::release() {
    if (blk) dev_free(c, blk, blk_bytes);
    blk = nullptr;
}

}  // namespace hlapi

static int merkle_on_device(hl_ctx* c, const uint32_t* d_leaves, const uint32_t* d_salts, size_t nn, const uint8_t* leaf_key32,
                            const uint8_t* node_key32, uint32_t* d_levels) {
    uint32_t *d_lk = nullptr, *d_nk = nullptr;
    int rc = upload_key(c, leaf_key32, &d_lk);
    if (!rc) rc = upload_key(c, node_key32, &d_nk);
    if (!rc) {
        Timed t(c, HL_T_MERKLE);
        int launches = 0;
        const cudaError_t e = hlk::merkle_tree(d_leaves, d_salts, (u32)nn, d_lk, d_nk, d_levels, c->stream, &launches);
        c->stats.kernel_launches += launches;
        if (e != cudaSuccess) rc = fail(c, HL_B200_ERR_DEVICE, "merkle launch", e);
    }
    if (d_lk) dev_free(c, d_lk, 32);
    if (d_nk) dev_free(c, d_nk, 32);
    return rc;
}

namespace {

struct Shape {
    u32 logn, logr, rows, q;
    bool zk;
};

// Where the data rows come from: NULL base = already in st->d_data; otherwise host memory, either 64-bit words (row_w NULL) or
// packed rows of 1-, 2-, 4- or 8-byte two's-complement words (row r at byte off[r], width row_w[r]).
struct HostRows {
    const void* base = nullptr;
    const uint8_t* row_w = nullptr;
    std::vector<u64> off;  // packed form only: rows + 1 byte offsets
    // what else the call brings from the host.  When the rows go up in pieces these ride with them instead of ahead of them: the
    // pads of a piece's rows behind the piece (st->d_pads is their place), `tail` (the salts: nothing reads them before the
    // tree) behind the last piece.  Otherwise both are copied before the rows.
    const u64* pads = nullptr;
    const void* tail_src = nullptr;
    void* tail_dst = nullptr;
    size_t tail_bytes = 0;
};

// The pieces of rows that come from the host: a piece is encoded and its complete 1 KiB hash chunks (128 rows) are hashed while the next one
// is on the bus.  Sizes are turns of the machine, `sms` batches of 2^14 words; `bus` and `device` are what a turn takes on either side, in
// us: 44 a byte of a word from page-locked memory and 58 from pageable (55 and 42 GB/s), 35 a transform with its share of the hash, 29 for
// rows of 2^10 .. 2^13 words.
// Where the bus is the slower side little must follow its last byte: pieces of two turns, one turn at the end, and where it is much slower half
// a turn behind that, whose rows are split by residue.  1,000 rows of 2^13 64-bit words 1,741 us with no pieces below four turns, 1,469
// now; 600 of 2^14 1,869 -> 1,737 (two turns and one); 9,000 of 2^9 1,597 -> 996 and 20,000 of 2^8 3,247 -> 1,276 (pieces of 296 rows);
// 32-bit rows, 1,300 of 2^14 2,089 -> 1,987; 16-bit ones, 9,000 of 2^12 2,296 -> 2,177 (the growing pieces below), pageable ones, 1,777 of
// 2^14 2,188 -> 2,023.
// Where the device is (16-bit rows of 2^14 words from page-locked memory, 8-bit rows, lower rates) it should start early and have few
// launches: 1, 1, 2, 2, 3, 3, .. turns and two at the end.  Twos ending in one: 2,504 rows of 2^14 2,304 -> 2,379 us, 2,000 of them 1,949 -> 1,979; the other
// way round below ten turns, 1,200 of them 1,393 -> 1,324.  One turn at the end instead of two: between 2 % faster and 2 % slower over nineteen
// shapes of this kind, 0.3 % faster on average, 2,504 rows of 2^14 1 % slower.  Rows written just before (their lines in the host's caches) keep these
// differences and take 30 to 60 us more.
std::vector<u32> row_pieces(u32 rows, u32 sms, u32 batch, double bus, double device) {
    std::vector<u32> sizes;  // in batches
    u32 left = (rows + batch - 1) / batch;
    if (bus >= device) {
        auto take = [&](u32 b) {
            if (!left) return;
            if (b > left) b = left;
            if (b < sms / 4 && !sizes.empty()) sizes.back() += b;  // not worth a launch
            else sizes.push_back(b);
            left -= b;
        };
        if (bus >= 1.5 * device) take(sms / 2);
        take(sms);
        while (left) take(2 * sms);
        std::reverse(sizes.begin(), sizes.end());
    } else {
        u32 turns = (left + sms - 1) / sms;
        auto take = [&](u32 t) {
            sizes.push_back(t * sms < left ? t * sms : left);
            left -= sizes.back();
            turns -= t;
        };
        for (u32 k = 0; turns > 2; k++) take(std::min(k < 2 ? 1u : k < 4 ? 2u : 3u, turns - 2));
        if (turns) take(turns);
    }
    u32 at = 0;
    for (u32& s : sizes) {
        s = std::min(s * batch, rows - at);
        at += s;
    }
    return sizes;
}

// Encode + column-hash.  With no host rows the data rows are already in st->d_data; otherwise they are
// uploaded here in row chunks on the context's copy stream while the encoder works on the chunks that
// have arrived (the upload of a block-sized matrix takes longer than its encoding).  Packed rows travel as
// their narrow bytes and are widened into st->d_data by the encoder's first pass.  Leaves stay in st->d_leaves.
int commit_on_device(hl_ctx* c, hl_store* st, const u64* d_pows, const uint8_t* key32, const HostRows& hr, bool leaves = true) {
    const u32 logn = st->logn, lognn = st->logn + st->logr;
    const size_t n = st->n(), nn = st->nn();
    // rows above 2^14 words run as 2 or 4 shared-memory transforms of 2^14 (encode_core.cuh)
    const u32 logb = logn > 14 ? 14u : logn, loga = logn - logb;
    const size_t nb = (size_t)1 << logb;
    const u32 T = st->zk ? (u32)((n + st->q + nb - 1) / nb) : (u32)(n / nb);
    const u64* tw = nullptr;
    int rc = root_powers(c, lognn, &tw);
    if (rc) return rc;
    const void* h_data = hr.base;
    const bool packed = h_data && hr.row_w;
    const bool fused_widen = packed && loga == 0 && logb >= 8 && c->fast_encoder;  // else a widening pass of its own per piece
    uint32_t* d_key = nullptr;
    u64* scratch = nullptr;
    uint32_t* cvs = nullptr;
    unsigned char *d_narrow = nullptr, *d_row_w = nullptr;
    u64* d_row_off = nullptr;
    size_t scratch_words = 0;
    const bool tc = c->fast_encoder && hlk::encode_tc_takes(logn, st->logr, st->rows, c->sm_count);
    const u64* tc_tab = nullptr;
    hlk::TcReport report;
    const bool later = !h_data && leaves;  // hl_b200_commit_zk_dev, which returns before its kernels have run
    st->order = ColOrder();
    if (tc) {
        st->order.logn = logn;
        st->order.logr = st->logr;
        rc = encoder_tables(c, logn, st->logr, &tc_tab);
        if (!rc) rc = encoder_word(c, st);
        if (rc) return rc;
        report = {st->enc_word, st->enc_mark, later ? c->enc_later : nullptr, c->enc_limit};
    }
    const u32 nchunks = hlk::hash_chunks(st->rows);
    const size_t cvs_bytes = nchunks > 1 && leaves ? (size_t)nchunks * nn * 32 : 0;
    const size_t total_bytes = packed ? (size_t)hr.off[st->rows] : (size_t)st->rows * n * 8;
    rc = upload_key(c, key32, &d_key);
    if (!rc && cvs_bytes) rc = dev_alloc(c, (void**)&cvs, cvs_bytes);
    if (!rc && packed) rc = dev_alloc(c, (void**)&d_narrow, total_bytes + 16);
    if (!rc && packed) rc = dev_alloc(c, (void**)&d_row_off, (size_t)st->rows * 8);
    if (!rc && packed) rc = dev_alloc(c, (void**)&d_row_w, st->rows);
    if (!rc && packed) rc = h2d_owned(c, d_row_off, hr.off.data(), (size_t)st->rows * 8);
    if (!rc && packed) rc = h2d_owned(c, d_row_w, hr.row_w, st->rows);
    auto byte_at = [&](u32 r) { return packed ? (size_t)hr.off[r] : (size_t)r * n * 8; };
    const u32 batch = logn < 14 ? 16384u >> logn : 1u;
    const bool pieces = h_data && total_bytes >= ((size_t)32 << 20) && st->rows > (u32)c->sm_count * batch;
    std::vector<u32> piece_rows{st->rows};
    if (pieces) {
        const double bus = (double)total_bytes / ((double)st->rows * n) * (pageable(h_data) ? 58 : 44), device = (1 + (1u << st->logr)) * (tc && logn < 14 ? 29 : 35);
        piece_rows = row_pieces(st->rows, (u32)c->sm_count, batch, bus, device);
    }
    if (!rc && tc) {
        for (const u32 nr : piece_rows) {
            const size_t w = hlk::encode_tc_scratch_words(logn, st->logr, st->q, nr, c->sm_count);
            if (w > scratch_words) scratch_words = w;
        }
        if (!dev_try(c, (void**)&scratch, scratch_words * 8)) scratch_words = hlk::encode_tc_least_words(logn, st->logr, st->q, st->rows, c->sm_count);
    } else if (!rc) {
        scratch_words = hlk::encode_scratch_words(logb, T, c->sm_count, st->rows);
    }
    if (!rc && !scratch) rc = dev_alloc(c, (void**)&scratch, scratch_words * 8);
    if (!rc && pieces) {
        // the copy stream may touch the fresh allocations only after the main stream has made them
        cudaError_t e = cudaEventRecord(c->ev_main, c->stream);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(c->copy_stream, c->ev_main, 0);
        if (e != cudaSuccess) rc = fail(c, HL_B200_ERR_DEVICE, "stream ordering", e);
    }
    if (!rc && !pieces && hr.pads) rc = h2d(c, st->d_pads, hr.pads, (size_t)st->rows * st->q * 8);
    if (!rc && !pieces && hr.tail_bytes) rc = h2d(c, hr.tail_dst, hr.tail_src, hr.tail_bytes);
    if (!rc) {
        Timed t(c, HL_T_ENCODE);
        size_t ev_i = 0;
        u32 nr = 0, chunks_done = 0;
        size_t pk = 0;
        for (u32 r0 = 0; r0 < st->rows && !rc; r0 += nr) {
            nr = piece_rows[pk++];
            if (h_data) {
                cudaStream_t cs = pieces ? c->copy_stream : c->stream;
                const size_t b0 = byte_at(r0), bytes = byte_at(r0 + nr) - b0;
                void* to = packed ? (void*)(d_narrow + b0) : (void*)(st->d_data + (size_t)r0 * n);
                rc = h2d_on(c, to, (const char*)h_data + b0, bytes, cs);
                if (!rc && pieces && hr.pads) rc = h2d_on(c, st->d_pads + (size_t)r0 * st->q, hr.pads + (size_t)r0 * st->q, (size_t)nr * st->q * 8, cs);
                if (!rc && pieces && hr.tail_bytes && r0 + nr == st->rows) rc = h2d_on(c, hr.tail_dst, hr.tail_src, hr.tail_bytes, cs);
                if (rc) break;
                cudaError_t e = cudaSuccess;
                if (e == cudaSuccess && cs != c->stream) {
                    if (ev_i == c->ev_chunks.size()) {
                        cudaEvent_t ev = nullptr;
                        e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
                        if (e == cudaSuccess) c->ev_chunks.push_back(ev);
                    }
                    if (e == cudaSuccess) e = cudaEventRecord(c->ev_chunks[ev_i], cs);
                    if (e == cudaSuccess) e = cudaStreamWaitEvent(c->stream, c->ev_chunks[ev_i], 0);
                    ev_i++;
                }
                if (e != cudaSuccess) { rc = fail(c, HL_B200_ERR_DEVICE, "row upload", e); break; }
            }
            if (packed && !fused_widen) {
                cudaError_t e = hlk::widen_rows(d_narrow, d_row_off + r0, d_row_w + r0, st->d_data + (size_t)r0 * n, nr, (u32)n, c->sm_count, c->stream);
                c->stats.kernel_launches += 1;
                if (e != cudaSuccess) { rc = fail(c, HL_B200_ERR_DEVICE, "row widening launch", e); break; }
            }
            enc::RowArgs a;
            a.data = st->d_data + (size_t)r0 * n;
            a.pads = st->d_pads ? st->d_pads + (size_t)r0 * st->q : nullptr;
            a.pows = d_pows; a.tw_nn = tw; a.enc = st->d_enc + (size_t)r0 * nn; a.scratch = scratch;
            a.rows = nr; a.q = st->zk ? st->q : 0; a.T = T; a.logr = st->logr + loga; a.loga = loga; a.zk = st->zk ? 1 : 0;
            a.ninv = gl_inv((u64)n); a.coef_out = nullptr;
            if (fused_widen) { a.narrow = d_narrow; a.row_off = d_row_off + r0; a.row_w = d_row_w + r0; }
            // a handful of rows (a boundary commitment, the last piece of an upload): one CTA per (row, residue)
            a.split = hlk::encode_split_pays(logb, st->logr, nr, c->sm_count) ? 1 : 0;
            cudaError_t e = tc ? hlk::encode_rows_tc(a, logn, tc_tab, c->sm_count, scratch_words, report, c->stream, &st->encoder_path)
                               : hlk::encode_rows(a, logb, c->fast_encoder || loga, c->sm_count, scratch_words, c->stream, &st->encoder_path);
            c->stats.kernel_launches += 1;
            if (e != cudaSuccess) rc = fail(c, HL_B200_ERR_DEVICE, "row encoder launch", e);
            if (!rc && pieces) {  // the 128-row hash chunks that are complete now
                const u32 c1 = r0 + nr == st->rows ? nchunks : (r0 + nr) / 128u;
                if (c1 > chunks_done) {
                    e = hlk::hash_column_chunks(st->d_enc, st->rows, (u32)nn, d_key, chunks_done, c1 - chunks_done, cvs, st->d_leaves, c->stream, st->order);
                    c->stats.kernel_launches += 1;
                    if (e != cudaSuccess) rc = fail(c, HL_B200_ERR_DEVICE, "column hash launch", e);
                    chunks_done = c1;
                }
            }
        }
    }
    if (!rc && pieces) {
        Timed t(c, HL_T_HASH);
        cudaError_t e = hlk::hash_column_merge(st->rows, (u32)nn, d_key, cvs, st->d_leaves, c->stream, st->order);
        c->stats.kernel_launches += 1;
        if (e != cudaSuccess) rc = fail(c, HL_B200_ERR_DEVICE, "column hash merge launch", e);
    }
    if (!rc && !pieces && leaves) {
        Timed t(c, HL_T_HASH);
        cudaError_t e = hlk::hash_columns(st->d_enc, st->rows, (u32)nn, d_key, cvs, st->d_leaves, c->stream, st->order);
        c->stats.kernel_launches += nchunks > 1 ? 2 : 1;
        if (e != cudaSuccess) rc = fail(c, HL_B200_ERR_DEVICE, "column hash launch", e);
    }
    dev_free(c, scratch, scratch_words * 8);
    if (cvs) dev_free(c, cvs, cvs_bytes);
    if (d_key) dev_free(c, d_key, 32);
    if (d_narrow) dev_free(c, d_narrow, total_bytes + 16);
    if (d_row_off) dev_free(c, d_row_off, (size_t)st->rows * 8);
    if (d_row_w) dev_free(c, d_row_w, st->rows);
    return rc;
}

int check_shape(hl_ctx* c, uint32_t log_cols, uint32_t inv_rate, size_t rows, size_t q, bool zk, uint32_t max_log, Shape* s) {
    int logr = log2_exact(inv_rate);
    if (logr < 0 || rows == 0 || rows > 0x7FFFFFFFu) return fail(c, HL_B200_ERR_ARG, "commit: rows or inv_rate");
    if (log_cols < 1) return fail(c, HL_B200_ERR_UNSUPPORTED, "commit: fewer than 2 columns");
    if (log_cols > 16) return fail(c, HL_B200_ERR_UNSUPPORTED, "commit: more than 2^16 columns per row");
    if (max_log && log_cols + (uint32_t)logr > max_log) return fail(c, HL_B200_ERR_ARG, "commit: transform exceeds the caller's NTT tables");
    size_t n = (size_t)1 << log_cols, nn = n << logr;
    if (zk && (q == 0 || n + q > nn)) return fail(c, HL_B200_ERR_ARG, "commit_zk: pad count (need 0 < q and n + q <= nn)");
    if (rows * nn > ((size_t)1 << 36)) return fail(c, HL_B200_ERR_UNSUPPORTED, "commit: encoding above 512 GiB");
    s->logn = log_cols; s->logr = (u32)logr; s->rows = (u32)rows; s->q = zk ? (u32)q : 0; s->zk = zk;
    return HL_B200_OK;
}

void free_store(hl_store* st) {
    hl_ctx* c = st->ctx;
    c->stores.erase(st);
    if (st->enc_word) c->enc_words.push_back(st->enc_word);
    if (st->owns_inputs) {
        dev_free(c, st->d_data, (size_t)st->rows * st->n() * 8);
        dev_free(c, st->d_pads, (size_t)st->rows * st->q * 8);
    }
    dev_free(c, st->d_enc, (size_t)st->rows * st->nn() * 8);
    dev_free(c, st->d_leaves, st->nn() * 32);
    delete st;
}

// the salted tree to build in the same call (commit_zk_owned_with_tag draws the salts before it offers the commitment, pcs.rs:788-792)
struct TreeAsk {
    const uint8_t *salts32, *leaf_key32, *node_key32;
    uint8_t* levels_out;
};

int commit_host(hl_ctx* c, const Shape& s, const HostRows& data, const uint64_t* pads, const uint64_t* pows,
                const uint8_t* key32, hl_store** store, uint8_t* leaves32, const TreeAsk* tree = nullptr) {
    hl_store* st = new hl_store();
    st->ctx = c; st->rows = s.rows; st->logn = s.logn; st->logr = s.logr; st->q = s.q; st->zk = s.zk;
    const size_t n = st->n(), nn = st->nn();
    u64* d_pows = nullptr;
    uint32_t *d_salts = nullptr, *d_levels = nullptr;
    int rc = dev_alloc(c, (void**)&st->d_data, (size_t)s.rows * n * 8);
    if (!rc && tree) rc = dev_alloc(c, (void**)&d_salts, nn * 32);
    if (!rc && tree) rc = dev_alloc(c, (void**)&d_levels, (2 * nn - 1) * 32);
    if (!rc && s.zk) rc = dev_alloc(c, (void**)&st->d_pads, (size_t)s.rows * s.q * 8);
    if (!rc && s.zk) rc = dev_alloc(c, (void**)&d_pows, nn * 8);
    if (!rc) rc = dev_alloc(c, (void**)&st->d_enc, (size_t)s.rows * nn * 8);
    if (!rc) rc = dev_alloc(c, (void**)&st->d_leaves, nn * 32);
    if (!rc && s.zk) rc = h2d(c, d_pows, pows, nn * 8);
    HostRows hr = data;  // the pads and the salts travel with the rows (commit_on_device)
    if (s.zk) hr.pads = reinterpret_cast<const u64*>(pads);
    if (tree) { hr.tail_src = tree->salts32; hr.tail_dst = d_salts; hr.tail_bytes = nn * 32; }
    if (!rc) rc = commit_on_device(c, st, d_pows, key32, hr);
    if (!rc && tree) rc = merkle_on_device(c, st->d_leaves, d_salts, nn, tree->leaf_key32, tree->node_key32, d_levels);
    if (!rc && leaves32) rc = d2h(c, leaves32, st->d_leaves, nn * 32);
    if (!rc && tree) rc = d2h(c, tree->levels_out, d_levels, (2 * nn - 1) * 32);
    if (!rc) rc = sync(c, "commit");
    if (!rc) rc = encoded_ok(c, st);
    if (!rc && tree) c->stats.merkles++;
    if (d_pows) dev_free(c, d_pows, nn * 8);
    if (d_salts) dev_free(c, d_salts, nn * 32);
    if (d_levels) dev_free(c, d_levels, (2 * nn - 1) * 32);
    if (rc) { free_store(st); return rc; }
    c->stats.commits++;
    c->stores.insert(st);
    *store = st;
    return HL_B200_OK;
}

}  // namespace

void hlapi::store_release(hl_store* st) { free_store(st); }

// hl_b200_commit_zk_dev without the lock: for entry points that hold it already
int hlapi::commit_resident(hl_ctx* c, u32 log_cols, u32 inv_rate, const u64* d_data, size_t rows, const u64* d_pads, size_t q, const u64* d_pows,
                           const uint8_t* key32, hl_store** store, uint8_t* d_leaves32, bool leaves) {
    Shape s;
    int rc = check_shape(c, log_cols, inv_rate, rows, q, true, 0, &s);
    if (rc) return rc;
    hl_store* st = new hl_store();
    st->ctx = c; st->rows = s.rows; st->logn = s.logn; st->logr = s.logr; st->q = s.q; st->zk = true;
    st->owns_inputs = false;
    st->d_data = const_cast<u64*>(d_data);
    st->d_pads = const_cast<u64*>(d_pads);
    const size_t nn = st->nn();
    rc = dev_alloc(c, (void**)&st->d_enc, (size_t)s.rows * nn * 8);
    if (!rc) rc = dev_alloc(c, (void**)&st->d_leaves, nn * 32);
    if (!rc) rc = commit_on_device(c, st, d_pows, key32, HostRows(), leaves);
    if (!rc && d_leaves32) {
        cudaError_t e = cudaMemcpyAsync(d_leaves32, st->d_leaves, nn * 32, cudaMemcpyDeviceToDevice, c->stream);
        if (e != cudaSuccess) rc = fail(c, HL_B200_ERR_DEVICE, "leaf copy", e);
    }
    if (rc) { free_store(st); return rc; }
    c->stats.commits++;
    c->stores.insert(st);
    *store = st;
    return HL_B200_OK;
}

extern "C" {

int hl_b200_commit(hl_ctx* c, uint32_t log_cols, uint32_t inv_rate, const uint64_t* data, size_t rows, uint32_t max_log,
                   const uint8_t* key32, hl_store** store, uint8_t* leaves32) {
    if (!c || !data || !store || !leaves32) return fail(c, HL_B200_ERR_ARG, "commit: null argument");
    Call g(c);
    Shape s;
    int rc = check_shape(c, log_cols, inv_rate, rows, 0, false, max_log, &s);
    if (rc) return rc;
    HostRows hr;
    hr.base = data;
    return commit_host(c, s, hr, nullptr, nullptr, key32, store, leaves32);
}

int hl_b200_commit_zk(hl_ctx* c, uint32_t log_cols, uint32_t inv_rate, const uint64_t* data, size_t rows,
                      const uint64_t* pads, size_t q, const uint64_t* pows, uint32_t max_log, const uint8_t* key32,
                      hl_store** store, uint8_t* leaves32) {
    if (!c || !data || !pads || !pows || !store || !leaves32) return fail(c, HL_B200_ERR_ARG, "commit_zk: null argument");
    Call g(c);
    Shape s;
    int rc = check_shape(c, log_cols, inv_rate, rows, q, true, max_log, &s);
    if (rc) return rc;
    HostRows hr;
    hr.base = data;
    return commit_host(c, s, hr, pads, pows, key32, store, leaves32);
}

int hl_b200_commit_zk_tree(hl_ctx* c, uint32_t log_cols, uint32_t inv_rate, const uint64_t* data, size_t rows, const uint64_t* pads, size_t q,
                           const uint64_t* pows, uint32_t max_log, const uint8_t* key32, const uint8_t* salts32, const uint8_t* leaf_key32,
                           const uint8_t* node_key32, hl_store** store, uint8_t* leaves32, uint8_t* levels_out) {
    if (!c || !data || !pads || !pows || !salts32 || !store || !levels_out) return fail(c, HL_B200_ERR_ARG, "commit_zk_tree: null argument");
    Call g(c);
    Shape s;
    int rc = check_shape(c, log_cols, inv_rate, rows, q, true, max_log, &s);
    if (rc) return rc;
    const TreeAsk tree{salts32, leaf_key32, node_key32, levels_out};
    HostRows hr;
    hr.base = data;
    return commit_host(c, s, hr, pads, pows, key32, store, leaves32, &tree);
}

int hl_b200_commit_zk_packed(hl_ctx* c, uint32_t log_cols, uint32_t inv_rate, const void* packed, const uint8_t* row_width, size_t rows,
                             const uint64_t* pads, size_t q, const uint64_t* pows, uint32_t max_log, const uint8_t* key32, const uint8_t* salts32,
                             const uint8_t* leaf_key32, const uint8_t* node_key32, hl_store** store, uint8_t* leaves32, uint8_t* levels_out) {
    if (!c || !packed || !row_width || !pads || !pows || !store || (salts32 && !levels_out) || (!salts32 && !leaves32))
        return fail(c, HL_B200_ERR_ARG, "commit_zk_packed: null argument");
    Shape s;
    HostRows hr;
    if (int rc = check_shape(c, log_cols, inv_rate, rows, q, true, max_log, &s)) return rc;
    if (log_cols < 3) return fail(c, HL_B200_ERR_UNSUPPORTED, "commit_zk_packed: rows of fewer than 8 words");  // keeps every row 8-byte aligned
    hr.base = packed;
    hr.row_w = row_width;
    hr.off.resize(rows + 1);
    u64 at = 0;
    for (size_t r = 0; r < rows; r++) {
        const uint8_t w = row_width[r];
        if (w != 1 && w != 2 && w != 4 && w != 8) return fail(c, HL_B200_ERR_ARG, "commit_zk_packed: a row width other than 1, 2, 4 or 8 bytes");
        hr.off[r] = at;
        at += (u64)w << log_cols;
    }
    hr.off[rows] = at;
    Call g(c);
    if (salts32) {
        const TreeAsk tree{salts32, leaf_key32, node_key32, levels_out};
        return commit_host(c, s, hr, pads, pows, key32, store, leaves32, &tree);
    }
    return commit_host(c, s, hr, pads, pows, key32, store, leaves32);
}

int hl_b200_commit_zk_dev(hl_ctx* c, uint32_t log_cols, uint32_t inv_rate, const uint64_t* d_data, size_t rows,
                          const uint64_t* d_pads, size_t q, const uint64_t* d_pows, const uint8_t* key32,
                          hl_store** store, uint8_t* d_leaves32) {
    if (!c || !d_data || !d_pads || !d_pows || !store) return fail(c, HL_B200_ERR_ARG, "commit_zk_dev: null argument");
    Call g(c);
    return commit_resident(c, log_cols, inv_rate, (const u64*)d_data, rows, (const u64*)d_pads, q, (const u64*)d_pows, key32, store, d_leaves32);
}

int hl_b200_store_shape(hl_store* st, size_t* rows, size_t* n, size_t* nn, size_t* q) {
    if (!st) return HL_B200_ERR_ARG;
    if (rows) *rows = st->rows;
    if (n) *n = st->n();
    if (nn) *nn = st->nn();
    if (q) *q = st->q;
    return HL_B200_OK;
}

// the words as the header promises them: an encoding that lies residue by residue is put into the columns' own order first, and stays in it
const uint64_t* hl_b200_store_encoded_dev(hl_store* st) {
    if (!st) return nullptr;
    hl_ctx* c = st->ctx;
    Call g(c);
    int rc = HL_B200_OK;
    if (st->order.logr) {
        // a CTA needs a row of scratch: fewer of them where memory is short, one at the least
        u32 ctas = hlk::natural_order_rows(st->rows, c->sm_count);
        u64* d_rows = nullptr;
        while (ctas > 1 && !dev_try(c, (void**)&d_rows, (size_t)ctas * st->nn() * 8)) ctas /= 2;
        if (!d_rows) rc = dev_alloc(c, (void**)&d_rows, st->nn() * 8);
        if (!rc) {
            const cudaError_t e = hlk::natural_order(st->d_enc, st->rows, st->nn(), st->order, d_rows, ctas, c->stream);
            c->stats.kernel_launches++;
            if (e == cudaSuccess) st->order = ColOrder();  // for what is queued behind it, whatever becomes of this call
            else rc = fail(c, HL_B200_ERR_DEVICE, "column order launch", e);
        }
        if (!rc) rc = sync(c, "store_encoded_dev");
        dev_free(c, d_rows, (size_t)ctas * st->nn() * 8);
    }
    if (!rc) rc = encoded_ok(c, st);  // where that is known already
    return rc ? nullptr : (const uint64_t*)st->d_enc;
}
const uint8_t* hl_b200_store_leaves_dev(hl_store* st) { return st ? (const uint8_t*)st->d_leaves : nullptr; }

void hl_b200_store_free(hl_store* st) {
    if (!st) return;
    hl_ctx* c = st->ctx;
    Call g(c);
    free_store(st);
}

int hl_b200_store_fold(hl_store* st, const uint64_t* rhos, size_t k, int with_pads, uint64_t* out) {
    if (!st) return HL_B200_ERR_ARG;
    hl_ctx* c = st->ctx;
    if (k && (!rhos || !out)) return fail(c, HL_B200_ERR_ARG, "store_fold: null argument");
    if (with_pads && !st->zk) return fail(c, HL_B200_ERR_ARG, "store_fold: pads asked of a plain store");
    if (k == 0) return HL_B200_OK;
    if (k > 0xFFFFu * 8u) return fail(c, HL_B200_ERR_ARG, "store_fold: too many vectors");
    Call g(c);
    const u32 n = (u32)st->n(), q = with_pads ? st->q : 0, w = n + q, rows = st->rows;
    const size_t row_bytes = (size_t)w * 16, ob = k * row_bytes;
    // hiding form: the message is the resident data (the encoding is not systematic, pcs.rs:985-987);
    // plain form: the systematic positions of the encoding (pcs.rs:332-340)
    FoldSource src;
    const bool from_data = st->zk || st->fold_data;
    src.rows = rows; src.n = n; src.q = q;
    src.d = from_data ? st->d_data : st->d_enc;
    src.ld = from_data ? n : st->nn();
    src.ir = from_data || st->order.logr ? 1u : 1u << st->logr;  // the systematic positions are residue 0
    src.pads = st->zk && q ? st->d_pads : nullptr;
    u64* d_out = nullptr;
    FoldPlan plan;
    int rc = dev_alloc(c, (void**)&d_out, ob);
    if (!rc) rc = plan.make(c, src, rhos, k);
    u32 first = 0, sparse_done = 0;  // the sparse vectors' results, when they lie together, go back while the dense ones are computed
    if (!rc) {
        Timed t(c, HL_T_FOLD);
        rc = plan.launch_sparse(d_out);
        if (!rc && plan.kd && plan.sparse_span(&first)) {
            cudaError_t e = cudaEventRecord(c->ev_main, c->stream);
            if (e == cudaSuccess) e = cudaStreamWaitEvent(c->copy_stream, c->ev_main, 0);
            if (e != cudaSuccess) rc = fail(c, HL_B200_ERR_DEVICE, "stream ordering", e);
            sparse_done = plan.ks;
        }
        if (!rc) rc = plan.launch_dense(d_out);
    }
    auto back = [&](u32 g0, u32 g1, cudaStream_t s) {
        return g1 > g0 ? d2h_on(c, (char*)out + g0 * row_bytes, (char*)d_out + g0 * row_bytes, (g1 - g0) * row_bytes, s) : HL_B200_OK;
    };
    if (!rc) rc = back(first, first + sparse_done, c->copy_stream);
    if (!rc) rc = back(0, first, c->stream);
    if (!rc) rc = back(first + sparse_done, (u32)k, c->stream);
    if (!rc) rc = sync(c, "store_fold");
    if (!rc) rc = encoded_ok(c, st);
    plan.release();
    if (d_out) dev_free(c, d_out, ob);
    if (!rc) c->stats.folds++;
    return rc;
}

int hl_b200_store_columns(hl_store* st, const uint64_t* idx, size_t nidx, uint64_t* out) {
    if (!st) return HL_B200_ERR_ARG;
    hl_ctx* c = st->ctx;
    if (nidx && (!idx || !out)) return fail(c, HL_B200_ERR_ARG, "store_columns: null argument");
    if (nidx == 0) return HL_B200_OK;
    if (nidx > 65535) return fail(c, HL_B200_ERR_ARG, "store_columns: more than 65535 columns in one call");
    for (size_t i = 0; i < nidx; i++)
        if (idx[i] >= st->nn()) return fail(c, HL_B200_ERR_ARG, "store_columns: index out of range");
    Call g(c);
    u64 *d_idx = nullptr, *d_out = nullptr;
    const size_t ob = nidx * (size_t)st->rows * 8;
    int rc = dev_alloc(c, (void**)&d_idx, nidx * 8);
    if (!rc) rc = dev_alloc(c, (void**)&d_out, ob);
    if (!rc) rc = h2d(c, d_idx, idx, nidx * 8);
    if (!rc) {
        Timed t(c, HL_T_GATHER);
        cudaError_t e = hlk::gather_columns(st->d_enc, st->rows, st->nn(), d_idx, (u32)nidx, d_out, c->stream, st->order);
        c->stats.kernel_launches++;
        if (e != cudaSuccess) rc = fail(c, HL_B200_ERR_DEVICE, "gather launch", e);
    }
    if (!rc) rc = d2h(c, out, d_out, ob);
    if (!rc) rc = sync(c, "store_columns");
    if (!rc) rc = encoded_ok(c, st);
    dev_free(c, d_idx, nidx * 8); dev_free(c, d_out, ob);
    if (!rc) c->stats.gathers++;
    return rc;
}

// salted leaves + all levels into d_levels, from device leaves (and device salts, or none)
static int merkle_common(hl_ctx* c, const uint32_t* d_leaves_in, const uint8_t* h_leaves, const uint8_t* salts32, size_t nn,
                         const uint8_t* leaf_key32, const uint8_t* node_key32, uint8_t* levels_out) {
    if (log2_exact(nn) < 0 || nn > ((size_t)1 << 26)) return fail(c, HL_B200_ERR_ARG, "merkle: leaf count must be a power of two");
    const size_t lv_bytes = (2 * nn - 1) * 32;
    uint32_t *d_levels = nullptr, *d_in = nullptr, *d_salts = nullptr;
    int rc = dev_alloc(c, (void**)&d_levels, lv_bytes);
    const uint32_t* leaves = d_leaves_in;
    if (!rc && !leaves) {
        rc = dev_alloc(c, (void**)&d_in, nn * 32);
        if (!rc) rc = h2d(c, d_in, h_leaves, nn * 32);
        leaves = d_in;
    }
    if (!rc && salts32) {
        rc = dev_alloc(c, (void**)&d_salts, nn * 32);
        if (!rc) rc = h2d(c, d_salts, salts32, nn * 32);
    }
    if (!rc) rc = merkle_on_device(c, leaves, d_salts, nn, leaf_key32, node_key32, d_levels);
    if (!rc) rc = d2h(c, levels_out, d_levels, lv_bytes);
    if (!rc) rc = sync(c, "merkle");
    dev_free(c, d_levels, lv_bytes);
    if (d_in) dev_free(c, d_in, nn * 32);
    if (d_salts) dev_free(c, d_salts, nn * 32);
    if (!rc) c->stats.merkles++;
    return rc;
}

int hl_b200_merkle(hl_ctx* c, const uint8_t* leaves32, const uint8_t* salts32, size_t nn, const uint8_t* leaf_key32,
                   const uint8_t* node_key32, uint8_t* levels_out) {
    if (!c || !leaves32 || !levels_out) return fail(c, HL_B200_ERR_ARG, "merkle: null argument");
    Call g(c);
    return merkle_common(c, nullptr, leaves32, salts32, nn, leaf_key32, node_key32, levels_out);
}

int hl_b200_store_merkle(hl_store* st, const uint8_t* salts32, const uint8_t* leaf_key32, const uint8_t* node_key32,
                         uint8_t* levels_out) {
    if (!st || !levels_out) return HL_B200_ERR_ARG;
    hl_ctx* c = st->ctx;
    Call g(c);
    const int rc = merkle_common(c, st->d_leaves, nullptr, salts32, st->nn(), leaf_key32, node_key32, levels_out);
    return rc ? rc : encoded_ok(c, st);
}

int hl_b200_store_merkle_dev(hl_store* st, const uint8_t* d_salts32, const uint8_t* leaf_key32, const uint8_t* node_key32,
                             uint8_t* d_levels_out) {
    if (!st || !d_levels_out) return HL_B200_ERR_ARG;
    hl_ctx* c = st->ctx;
    // the tree kernels move digests as 16-byte vectors: a misaligned caller pointer would be a device fault, not a status
    if (((uintptr_t)d_levels_out & 15) || ((uintptr_t)d_salts32 & 15)) return fail(c, HL_B200_ERR_ARG, "store_merkle_dev: device pointers must be 16-byte aligned");
    Call g(c);
    int rc = encoded_ok(c, st);  // where that is known already
    if (!rc) rc = merkle_on_device(c, st->d_leaves, (const uint32_t*)d_salts32, st->nn(), leaf_key32, node_key32, (uint32_t*)d_levels_out);
    if (!rc) c->stats.merkles++;
    return rc;
}

}  // extern "C"
