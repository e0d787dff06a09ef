// A slot's sumcheck tables built where they are used (private_block/argument.rs:907 build_tables_device; the reference's
// Metal form: gpu/metal.rs MetalTables::{new, plan_eq, plan_plane, build_planned, flush, to_vecs}).
//
// Two table kinds are written by kernels, from small host-made maps, instead of being built on the host and uploaded
// (the 8B block's tables are 1.3 GB per block):
//
//   eq cube      out[x] = hi[y >> p_lo] * lo[y & (2^p_lo - 1)],  y = (x >> shift) & (2^p - 1)
//                with hi, lo the eq tables of the two halves of the point (argument.rs:643-660 eq_cube_split_into);
//   plane        out[x] = sum_z eqf[z] * v(inv(x & used) | zbits[z]),   v(idx) = sum_s coef_s * rows[off_s + idx]
//                a committed witness plane read through the inverse of its index bit map, partially evaluated at the
//                plane's fixed coordinates (argument.rs:386-577 priv_table_fill; the per-output form of :470-540).
//                The rows are the commitment's own resident copy (gpu/metal.rs:3105 MetalCommit::resident_rows).
//
// Every word is the canonical representative of the element the host builder writes: same formula, exact arithmetic,
// only the order of exact additions differs.  A table the caller declares base-valued is checked as it is written
// (imaginary word zero); a violation surfaces at flush as HL_B200_ERR_MISMATCH (metal.rs:2649-2665 refuses the same way).
#include <cstring>
#include <vector>

#include "api_internal.h"
#include "gl_field.cuh"

using namespace hlapi;

// One planned table: what the kernel needs to write it, with its maps as offsets into the two pools of the set's plan.
struct TabDesc {
    u32 kind, table;           // 0 eq cube, 1 plane; the table it fills
    u32 shift, p, p_lo;        // eq
    u32 xlo, nz, ns;           // plane
    int one_slice, base_check;
    u64 used;
    u32 ident, split2;         // plane: its index is x itself (under `used`); two slices with coefficients 1 and u, the two words of the entry
    u64 off_pt;                // eq planned from its point: the point's place in the 64-bit pool (hi / lo are then computed on the device)
    u64 off_a, off_b;          // 64-bit pool: eq hi / lo, or plane eqf / slices
    u64 off_lo, off_hi, off_zb;  // 32-bit pool: plane inv_lo / inv_hi / zbits
    const u64* rows;           // plane: the committed data, flat
    const hl_store* store;     // plane: the commitment those rows belong to, or NULL for caller-owned device rows (host use only)
};

// The eq and plane calls only PLAN a table (MetalTables::plan_eq / plan_plane do the same, gpu/metal.rs): the maps are copied
// into the set's host pools at once, so the caller's arrays are free when the call returns, and everything planned is written by
// one upload and one launch when the set is flushed, read or handed to an evaluator (MetalTables::build_planned).  A slot with
// sixty small tables was sixty launches and some two hundred small copies before.
struct hl_tables {
    hl_ctx* ctx = nullptr;
    u32 k = 0, n_vars = 0;
    u64* d_tables = nullptr;   // k x 2^n_vars Fp2, table-major
    u32* d_flag = nullptr;
    std::vector<TabDesc> plan;
    std::vector<u64> pool64;
    std::vector<u32> pool32;
    u64 eq_words = 0;          // words of device-made eq halves, behind the 64-bit pool
    u64 eq_most = 0;           // entries of the largest pair of them
    u32 eq_points = 0;         // planned tables that have them
    bool checked = false;      // a table was declared base-valued: the flush has to ask
    size_t len() const { return (size_t)1 << n_vars; }
    size_t bytes() const { return (size_t)k * len() * 16; }
};

namespace {

__device__ __forceinline__ fp2 ld2(const u64* p) {
    ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
    return f2(v.x, v.y);
}
__device__ __forceinline__ void st2(u64* p, fp2 v) { *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(v.c0, v.c1); }

struct PlaneArgs {
    const u64* rows;       // the committed data, flat
    const u32 *inv_lo, *inv_hi, *zbits;
    const u64* eqf;        // nz Fp2 (unused when nz == 0)
    const u64* slices;     // ns x (offset, c0, c1)
    u64 used;
    u32 xlo, nz, ns, ident;
    int one_slice;         // one slice with coefficient 1
};

__device__ __forceinline__ fp2 plane_value(const PlaneArgs& a, size_t idx) {
    if (a.one_slice) return f2(a.rows[a.slices[0] + idx], 0);
    fp2 v = f2(0, 0);
    for (u32 s = 0; s < a.ns; s++) {
        const u64* sl = a.slices + 3 * (size_t)s;
        v = f2_add(v, f2_mul_base(f2(sl[1], sl[2]), a.rows[sl[0] + idx]));
    }
    return v;
}

__device__ __forceinline__ fp2 plane_entry(const PlaneArgs& a, size_t x) {
    const u64 xu = x & a.used;
    const size_t im = a.ident ? xu : (size_t)a.inv_hi[xu >> a.xlo] | a.inv_lo[xu & (((u64)1 << a.xlo) - 1)];
    if (a.nz == 0) return plane_value(a, im);
    if (a.one_slice) {
        // sum_z eqf[z] * word: the products are summed as integers and reduced once per component
        // (argument.rs:349-384 does the same on the host); 2^128 = -2^32 (mod p) per wrap
        u64 lo0 = 0, hi0 = 0, w0 = 0, lo1 = 0, hi1 = 0, w1 = 0;
        for (u32 z = 0; z < a.nz; z++) {
            const fp2 e = ld2(a.eqf + 2 * (size_t)z);
            const u64 d = a.rows[a.slices[0] + (im | a.zbits[z])];
            const gl_wide p0 = gl_mulw(e.c0, d), p1 = gl_mulw(e.c1, d);
            u64 t = lo0 + p0.lo, c = t < lo0; lo0 = t;
            t = hi0 + p0.hi; u64 c2 = t < hi0; hi0 = t + c; c2 += hi0 < t; w0 += c2;
            t = lo1 + p1.lo; c = t < lo1; lo1 = t;
            t = hi1 + p1.hi; c2 = t < hi1; hi1 = t + c; c2 += hi1 < t; w1 += c2;
        }
        const u64 two128 = 0xFFFFFFFE00000001ull;  // 2^128 mod p
        return f2(gl_add(gl_reduce128(lo0, hi0), gl_mul(w0, two128)), gl_add(gl_reduce128(lo1, hi1), gl_mul(w1, two128)));
    }
    fp2 v = f2(0, 0);
    for (u32 z = 0; z < a.nz; z++) v = f2_add(v, f2_mul(ld2(a.eqf + 2 * (size_t)z), plane_value(a, im | a.zbits[z])));
    return v;
}

// The two half tables of every eq cube planned from its point: entry e of a half over m coordinates is prod_j (bit ? r_j : 1 - r_j),
// first coordinate = most significant bit.  A few thousand entries of some ten products each: 4 us on the device, where the host took
// 80 us for a 2^21 cube and then had them to upload.
__global__ void __launch_bounds__(128) k_tab_eq_halves(const TabDesc* __restrict__ descs, u32 n_desc, u64* __restrict__ p64) {
    u32 seen = 0, t = 0;  // the blockIdx.y-th eq entry planned from a point
    for (; t < n_desc; t++)
        if (descs[t].kind == 0 && descs[t].off_pt != ~0ull && seen++ == blockIdx.y) break;
    if (t == n_desc) return;
    const TabDesc& d = descs[t];
    const u32 p_hi = d.p - d.p_lo, n_hi = 1u << p_hi, e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n_hi + (1u << d.p_lo)) return;
    const bool hi = e < n_hi;
    const u32 m = hi ? p_hi : d.p_lo, at = hi ? e : e - n_hi;
    const u64* pt = p64 + d.off_pt + (hi ? 0 : 2 * (size_t)p_hi);
    fp2 v = f2(1, 0);
    for (u32 j = 0; j < m; j++) {
        fp2 r = ld2(pt + 2 * j);
        if (!((at >> (m - 1 - j)) & 1)) r = f2_sub(f2(1, 0), r);
        v = f2_mul(v, r);
    }
    st2(p64 + (hi ? d.off_a : d.off_b) + 2 * (size_t)at, v);
}

// Every planned table of a set in one launch: blockIdx.y = the plan entry, blockIdx.x over spans of TAB_SPAN entries.  HBM is what it
// has to wait for (16 bytes written per entry, 8 or 16 read), so a thread has its TAB_PER loads under way before its first store.
constexpr u32 TAB_T = 256, TAB_PER = 4, TAB_SPAN = TAB_T * TAB_PER;
__global__ void __launch_bounds__(TAB_T) k_tab_batch(u64* __restrict__ tables, size_t len, const TabDesc* __restrict__ descs, const u64* __restrict__ p64,
                                                     const u32* __restrict__ p32, u32* __restrict__ flag) {
    __shared__ TabDesc d;
    if (threadIdx.x < sizeof(TabDesc) / 4) reinterpret_cast<u32*>(&d)[threadIdx.x] = reinterpret_cast<const u32*>(descs + blockIdx.y)[threadIdx.x];
    __syncthreads();
    const size_t x0 = (size_t)blockIdx.x * TAB_SPAN + threadIdx.x;
    u64* out = tables + 2 * (size_t)d.table * len;
    u64 odd = 0;  // any second word, for a table declared base-valued
    if (d.kind == 0) {
        const u64 *hi = p64 + d.off_a, *lo = p64 + d.off_b;
#pragma unroll
        for (u32 k = 0; k < TAB_PER; k++) {
            const size_t x = x0 + k * TAB_T;
            if (x >= len) break;
            const size_t y = (x >> d.shift) & (((size_t)1 << d.p) - 1);
            const fp2 v = f2_mul(ld2(hi + 2 * (y >> d.p_lo)), ld2(lo + 2 * (y & (((size_t)1 << d.p_lo) - 1))));
            st2(out + 2 * x, v);
            odd |= v.c1;
        }
    } else if (d.ident && d.nz == 0 && (d.one_slice || d.split2)) {
        const u64 *re = d.rows + p64[d.off_b], *im = d.split2 ? d.rows + p64[d.off_b + 3] : nullptr;
        u64 a[TAB_PER], b[TAB_PER];
#pragma unroll
        for (u32 k = 0; k < TAB_PER; k++) {
            const size_t x = x0 + k * TAB_T, at = x & d.used;
            a[k] = x < len ? re[at] : 0;
            b[k] = im && x < len ? im[at] : 0;
        }
#pragma unroll
        for (u32 k = 0; k < TAB_PER; k++) {
            const size_t x = x0 + k * TAB_T;
            if (x >= len) break;
            st2(out + 2 * x, f2(a[k], b[k]));
            odd |= b[k];
        }
    } else {
        PlaneArgs a;
        a.rows = d.rows; a.inv_lo = p32 + d.off_lo; a.inv_hi = p32 + d.off_hi; a.zbits = p32 + d.off_zb; a.eqf = p64 + d.off_a; a.slices = p64 + d.off_b;
        a.used = d.used; a.xlo = d.xlo; a.nz = d.nz; a.ns = d.ns; a.one_slice = d.one_slice; a.ident = d.ident;
        for (u32 k = 0; k < TAB_PER; k++) {
            const size_t x = x0 + k * TAB_T;
            if (x >= len) break;
            const fp2 v = plane_entry(a, x);
            st2(out + 2 * x, v);
            odd |= v.c1;
        }
    }
    if (d.base_check && odd) atomicOr(flag, 1u);
}

}  // namespace

u64* hl_tables_adopt(hl_tables* t) {  // rounds_api.cu takes the device tables over
    u64* p = t->d_tables;
    t->d_tables = nullptr;
    return p;
}

const u64* hl_tables_peek(hl_tables* t) { return t->d_tables; }

void hl_tables_shape(hl_tables* t, hl_ctx** c, size_t* k, uint32_t* n_vars) {
    *c = t->ctx;
    *k = t->d_tables ? t->k : 0;
    *n_vars = t->n_vars;
}

static void drop_plan(hl_tables* t) {
    t->plan.clear();
    t->pool64.clear();
    t->pool32.clear();
    t->eq_words = t->eq_most = 0;
    t->eq_points = 0;
}

// writes every planned table: one upload of the descriptors and the two pools, one launch; the caller holds the context's lock
static int launch_planned(hl_tables* t) {
    if (t->plan.empty()) return HL_B200_OK;
    hl_ctx* c = t->ctx;
    for (const TabDesc& d : t->plan)
        if (d.kind == 1 && d.store && !c->stores.count(d.store)) {  // the rows are gone: nothing is launched over them
            drop_plan(t);
            return fail(c, HL_B200_ERR_ARG, "tables: a planned plane's commitment was freed before the set was built");
        }
    if (t->pool64.size() & 1) t->pool64.push_back(0);
    for (TabDesc& d : t->plan)
        if (d.kind == 0 && d.off_pt != ~0ull) { d.off_a += t->pool64.size(); d.off_b += t->pool64.size(); }  // the halves lie behind the pool
    // one block: descriptors, the 32-bit pool, the 64-bit pool, then the eq halves; the first three in one upload
    const size_t nd = t->plan.size(), b_desc = (nd * sizeof(TabDesc) + 15) & ~(size_t)15, b32 = (t->pool32.size() * 4 + 15) & ~(size_t)15,
                 b64 = t->pool64.size() * 8, up = b_desc + b32 + b64, total = up + t->eq_words * 8;
    std::vector<char> h(up);
    memcpy(h.data(), t->plan.data(), nd * sizeof(TabDesc));
    if (b32) memcpy(h.data() + b_desc, t->pool32.data(), t->pool32.size() * 4);
    if (b64) memcpy(h.data() + b_desc + b32, t->pool64.data(), b64);
    char* blk = nullptr;
    int rc;
    {
        Timed tm(c, HL_T_TABLES);  // the span takes the maps' upload with it: it is part of what building the tables costs
        rc = dev_alloc(c, (void**)&blk, total);
        if (!rc) rc = h2d_owned(c, blk, h.data(), up);
        if (!rc) {
            const TabDesc* d_desc = (const TabDesc*)blk;
            const u32* d_p32 = (const u32*)(blk + b_desc);
            u64* d_p64 = (u64*)(blk + b_desc + b32);
            const size_t len = t->len();
            if (t->eq_points) {
                k_tab_eq_halves<<<dim3((unsigned)((t->eq_most + 127) / 128), t->eq_points), 128, 0, c->stream>>>(d_desc, (u32)nd, d_p64);
                c->stats.kernel_launches++;
            }
            k_tab_batch<<<dim3((unsigned)((len + TAB_SPAN - 1) / TAB_SPAN), (unsigned)nd), TAB_T, 0, c->stream>>>(t->d_tables, len, d_desc, d_p64, d_p32, t->d_flag);
            c->stats.kernel_launches++;
            cudaError_t e = cudaGetLastError();
            if (e != cudaSuccess) rc = fail(c, HL_B200_ERR_DEVICE, "planned tables launch", e);
        }
    }
    if (blk) dev_free(c, blk, total);
    drop_plan(t);
    return rc;
}

int hl_tables_flush_locked(hl_tables* t) {
    hl_ctx* c = t->ctx;
    u32 flag = 0;
    int rc = launch_planned(t);
    if (!t->checked) return rc;
    if (!rc) rc = d2h(c, &flag, t->d_flag, 4);
    if (!rc) rc = sync(c, "tables_flush");
    if (!rc && flag) rc = fail(c, HL_B200_ERR_MISMATCH, "tables: a table declared base-valued holds an extension word");
    if (!rc) t->checked = false;  // asked and answered: the next plan asks again
    return rc;
}

static TabDesc eq_desc(hl_tables* t, size_t i, u32 start, u32 p, int base_check) {
    TabDesc d;
    memset(&d, 0, sizeof d);
    d.kind = 0; d.table = (u32)i; d.shift = t->n_vars - start - p; d.p = p; d.p_lo = p / 2; d.base_check = base_check; d.off_pt = ~0ull;
    t->checked |= base_check != 0;
    return d;
}

// A plane's descriptor without its maps; `all`: the OR of everything its index can be.  Every address the kernel can form stays inside
// the rows: the index is an OR of map entries.
static int plane_desc(hl_tables* t, size_t i, const hl_store* store, const uint64_t* d_rows, size_t n_words, u64 all, const uint64_t* slices, u32 ns, int base_check,
                      TabDesc* d) {
    hl_ctx* c = t->ctx;
    if (store) {
        if (store->ctx != c) return fail(c, HL_B200_ERR_ARG, "tables_plane: the commitment belongs to another context");
        d_rows = reinterpret_cast<const uint64_t*>(store->d_data);
        n_words = (size_t)store->rows * store->n();
    }
    if (!d_rows) return fail(c, HL_B200_ERR_ARG, "tables_plane: no rows");
    u64 max_off = 0;
    for (u32 s = 0; s < ns; s++) max_off = slices[3 * (size_t)s] > max_off ? slices[3 * (size_t)s] : max_off;
    if (max_off >= n_words || all >= n_words - max_off) return fail(c, HL_B200_ERR_ARG, "tables_plane: a slice reaches past the committed rows");
    memset(d, 0, sizeof *d);
    d->kind = 1; d->table = (u32)i; d->ns = ns; d->base_check = base_check; d->off_pt = ~0ull;
    d->one_slice = ns == 1 && slices[1] == 1 && slices[2] == 0;
    d->split2 = ns == 2 && slices[1] == 1 && slices[2] == 0 && slices[4] == 0 && slices[5] == 1;
    d->rows = reinterpret_cast<const u64*>(d_rows);
    d->store = store;
    t->checked |= base_check != 0;
    return HL_B200_OK;
}

static void plane_pools(hl_tables* t, TabDesc* d, const uint32_t* zbits, const uint64_t* eqf, const uint64_t* slices) {
    d->off_zb = t->pool32.size();
    if (d->nz) t->pool32.insert(t->pool32.end(), zbits, zbits + d->nz);
    if (t->pool64.size() & 1) t->pool64.push_back(0);  // every 64-bit array read as Fp2 starts on a 16-byte boundary
    d->off_a = t->pool64.size();
    if (d->nz) t->pool64.insert(t->pool64.end(), eqf, eqf + (size_t)d->nz * 2);
    d->off_b = t->pool64.size();
    t->pool64.insert(t->pool64.end(), slices, slices + (size_t)d->ns * 3);
    if (t->pool64.size() & 1) t->pool64.push_back(0);
    t->plan.push_back(*d);
}

extern "C" {

int hl_b200_tables_new(hl_ctx* c, size_t k, uint32_t n_vars, hl_tables** out) {
    if (!c || !out || k == 0) return fail(c, HL_B200_ERR_ARG, "tables_new: null argument or no table");
    if (n_vars > 30 || k > 64) return fail(c, HL_B200_ERR_UNSUPPORTED, "tables_new: more than 30 variables or 64 tables");
    Call g(c);
    hl_tables* t = new hl_tables();
    t->ctx = c; t->k = (u32)k; t->n_vars = n_vars;
    int rc = dev_alloc(c, (void**)&t->d_tables, t->bytes());
    if (!rc) rc = dev_alloc(c, (void**)&t->d_flag, 4);
    if (!rc) {
        cudaError_t e = cudaMemsetAsync(t->d_flag, 0, 4, c->stream);
        if (e != cudaSuccess) rc = fail(c, HL_B200_ERR_DEVICE, "tables_new", e);
    }
    if (rc) {
        if (t->d_tables) dev_free(c, t->d_tables, t->bytes());
        if (t->d_flag) dev_free(c, t->d_flag, 4);
        delete t;
        return rc;
    }
    *out = t;
    return HL_B200_OK;
}

void hl_b200_tables_free(hl_tables* t) {
    if (!t) return;
    hl_ctx* c = t->ctx;
    Call g(c);
    if (t->d_tables) dev_free(c, t->d_tables, t->bytes());
    dev_free(c, t->d_flag, 4);
    delete t;
}

int hl_b200_tables_put(hl_tables* t, size_t i, const uint64_t* words) {
    if (!t || !words || !t->d_tables || i >= t->k) return HL_B200_ERR_ARG;
    hl_ctx* c = t->ctx;
    Call g(c);
    if (int rc = launch_planned(t)) return rc;  // a planned table may be the one overwritten here: keep the caller's order
    return h2d_owned(c, t->d_tables + 2 * i * t->len(), words, t->len() * 16);
}

int hl_b200_tables_eq(hl_tables* t, size_t i, uint32_t start, uint32_t p, const uint64_t* hi, const uint64_t* lo, int base_check) {
    if (!t || !t->d_tables || i >= t->k || !hi || !lo) return HL_B200_ERR_ARG;
    hl_ctx* c = t->ctx;
    if (start + p > t->n_vars) return fail(c, HL_B200_ERR_ARG, "tables_eq: start + |point| exceeds the cube");  // argument.rs:604-607
    std::lock_guard<std::mutex> g(c->mu);
    TabDesc d = eq_desc(t, i, start, p, base_check);
    d.off_a = t->pool64.size();
    t->pool64.insert(t->pool64.end(), hi, hi + ((size_t)2 << (p - d.p_lo)));
    d.off_b = t->pool64.size();
    t->pool64.insert(t->pool64.end(), lo, lo + ((size_t)2 << d.p_lo));
    t->plan.push_back(d);
    return HL_B200_OK;
}

int hl_b200_tables_eq_point(hl_tables* t, size_t i, uint32_t start, uint32_t p, const uint64_t* point, int base_check) {
    if (!t || !t->d_tables || i >= t->k || (p && !point)) return HL_B200_ERR_ARG;
    hl_ctx* c = t->ctx;
    if (start + p > t->n_vars) return fail(c, HL_B200_ERR_ARG, "tables_eq_point: start + |point| exceeds the cube");
    std::lock_guard<std::mutex> g(c->mu);
    TabDesc d = eq_desc(t, i, start, p, base_check);
    if (t->pool64.size() & 1) t->pool64.push_back(0);
    d.off_pt = t->pool64.size();
    if (p) t->pool64.insert(t->pool64.end(), point, point + 2 * (size_t)p);
    const u64 n_hi = (u64)1 << (p - d.p_lo), n_lo = (u64)1 << d.p_lo;
    d.off_a = t->eq_words;  // from the end of the pool, whose size is known at the launch
    d.off_b = t->eq_words + 2 * n_hi;
    t->eq_words += 2 * (n_hi + n_lo);
    if (n_hi + n_lo > t->eq_most) t->eq_most = n_hi + n_lo;
    t->eq_points++;
    t->plan.push_back(d);
    return HL_B200_OK;
}

int hl_b200_tables_plane(hl_tables* t, size_t i, const hl_store* store, const uint64_t* d_rows, size_t n_words, uint64_t used, uint32_t xlo,
                         const uint32_t* inv_lo, const uint32_t* inv_hi, const uint32_t* zbits, uint32_t nz, const uint64_t* eqf,
                         const uint64_t* slices, uint32_t ns, int base_check) {
    if (!t || !t->d_tables || i >= t->k || !inv_lo || !inv_hi || !slices || ns == 0) return HL_B200_ERR_ARG;
    hl_ctx* c = t->ctx;
    if (nz && (!zbits || !eqf)) return fail(c, HL_B200_ERR_ARG, "tables_plane: fixed coordinates without their maps");
    if (xlo > t->n_vars || t->n_vars - xlo > 24 || xlo > 24 || nz > (1u << 16)) return fail(c, HL_B200_ERR_UNSUPPORTED, "tables_plane: map sizes");
    const size_t nlo = (size_t)1 << xlo, nhi = (size_t)1 << (t->n_vars - xlo);
    u64 all = 0;
    bool ident = true;  // on the entries that `used` lets through, the map is the index itself: the kernel then needs no map
    for (size_t j = 0; j < nlo; j++) { all |= inv_lo[j]; ident &= (j & ~used) || inv_lo[j] == j; }
    for (size_t j = 0; j < nhi; j++) { all |= inv_hi[j]; ident &= ((j << xlo) & ~used) || inv_hi[j] == j << xlo; }
    for (u32 z = 0; z < nz; z++) all |= zbits[z];
    std::lock_guard<std::mutex> g(c->mu);
    TabDesc d;
    if (int rc = plane_desc(t, i, store, d_rows, n_words, all, slices, ns, base_check, &d)) return rc;
    d.xlo = xlo; d.nz = nz; d.used = used; d.ident = ident;
    if (!ident) {
        d.off_lo = t->pool32.size();
        t->pool32.insert(t->pool32.end(), inv_lo, inv_lo + nlo);
        d.off_hi = t->pool32.size();
        t->pool32.insert(t->pool32.end(), inv_hi, inv_hi + nhi);
    }
    plane_pools(t, &d, zbits, eqf, slices);
    return HL_B200_OK;
}

int hl_b200_tables_plane_coords(hl_tables* t, size_t i, const hl_store* store, const uint64_t* d_rows, size_t n_words, const int32_t* coords, uint32_t n_coords,
                                const uint64_t* fixed, const uint64_t* slices, uint32_t ns, int base_check) {
    if (!t || !t->d_tables || i >= t->k || (n_coords && !coords) || !slices || ns == 0) return HL_B200_ERR_ARG;
    hl_ctx* c = t->ctx;
    const u32 n = t->n_vars, xlo = n / 2;
    if (n_coords > 32 || n - xlo > 24) return fail(c, HL_B200_ERR_UNSUPPORTED, "tables_plane_coords: map sizes");
    // argument.rs:486-512: coordinate j reads bit n_coords - 1 - j of the plane's index, from a cube variable or (fixed) from the point
    u64 used = 0, zall = 0;
    u32 to[32] = {0}, fpos[32], nf = 0;
    bool flip[32] = {false}, ident = true;
    for (u32 j = 0; j < n_coords; j++) {
        const u32 ib = n_coords - 1 - j;
        if (coords[j] == HL_COORD_FIXED) { fpos[nf++] = ib; zall |= (u64)1 << ib; continue; }
        const u32 k = (u32)(coords[j] < 0 ? -1 - coords[j] : coords[j]);
        if (k >= n || ((used >> (n - 1 - k)) & 1)) return fail(c, HL_B200_ERR_ARG, "tables_plane_coords: a cube variable outside the cube or read twice");
        const u32 b = n - 1 - k;
        used |= (u64)1 << b;
        to[b] = ib; flip[b] = coords[j] < 0;
        ident &= ib == b && coords[j] >= 0;
    }
    if (nf > 16) return fail(c, HL_B200_ERR_UNSUPPORTED, "tables_plane_coords: more than 16 fixed coordinates");
    if (nf && !fixed) return HL_B200_ERR_ARG;
    u64 all = zall;
    for (u32 b = 0; b < n; b++)
        if ((used >> b) & 1) all |= (u64)1 << to[b];
    std::lock_guard<std::mutex> g(c->mu);
    TabDesc d;
    if (int rc = plane_desc(t, i, store, d_rows, n_words, all, slices, ns, base_check, &d)) return rc;
    d.xlo = xlo; d.nz = nf ? 1u << nf : 0; d.used = used; d.ident = ident;
    if (!ident) {
        // each half by doubling: an entry is the one without its top bit, with that bit's image toggled
        auto half = [&](u32 first, u32 bits) {
            const size_t at = t->pool32.size();
            t->pool32.resize(at + ((size_t)1 << bits));
            u32* o = t->pool32.data() + at;
            o[0] = 0;
            for (u32 b = 0; b < bits; b++)
                if (flip[first + b]) o[0] |= 1u << to[first + b];
            for (u32 b = 0; b < bits; b++) {
                const u32 img = ((used >> (first + b)) & 1) ? 1u << to[first + b] : 0u;
                for (size_t v = 0; v < ((size_t)1 << b); v++) o[((size_t)1 << b) + v] = o[v] ^ img;
            }
            return (u64)at;
        };
        d.off_lo = half(0, xlo);
        d.off_hi = half(xlo, n - xlo);
    }
    std::vector<u32> zbits(d.nz);
    std::vector<fp2> eqf(d.nz);
    if (nf) {  // first fixed coordinate = most significant bit of z, and of the eq table
        for (u32 z = 0; z < d.nz; z++)
            for (u32 f = 0; f < nf; f++) zbits[z] |= ((z >> (nf - 1 - f)) & 1) << fpos[f];
        eqf[0] = f2(1, 0);
        for (u32 f = 0; f < nf; f++) {
            const fp2 r = f2(fixed[2 * f], fixed[2 * f + 1]);
            for (size_t e = (size_t)1 << f; e-- > 0;) {
                const fp2 hi = f2_mul(eqf[e], r);
                eqf[2 * e + 1] = hi;
                eqf[2 * e] = f2_sub(eqf[e], hi);
            }
        }
    }
    plane_pools(t, &d, zbits.data(), reinterpret_cast<const uint64_t*>(eqf.data()), slices);
    return HL_B200_OK;
}

int hl_b200_tables_flush(hl_tables* t) {
    if (!t || !t->d_tables) return HL_B200_ERR_ARG;
    hl_ctx* c = t->ctx;
    Call g(c);
    return hl_tables_flush_locked(t);
}

int hl_b200_tables_read(hl_tables* t, size_t i, uint64_t* out) {
    if (!t || !t->d_tables || i >= t->k || !out) return HL_B200_ERR_ARG;
    hl_ctx* c = t->ctx;
    Call g(c);
    int rc = launch_planned(t);
    if (!rc) rc = d2h(c, out, t->d_tables + 2 * i * t->len(), t->len() * 16);
    if (!rc) rc = sync(c, "tables_read");
    return rc;
}

}  // extern "C"
