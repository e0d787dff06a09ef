// Row encoder on the tensor cores (encode_tc.cuh has the arithmetic and the layouts).
#define GL_PLAIN_CANONICAL_FORMS 1  // as the shared-memory encoder: the lazy forms are used where it counts
#include "encode_tc.cuh"
#include "kernels.h"
#include "umma.cuh"

namespace {

using namespace enc;

constexpr u32 TC_WORKERS = 16, TC_THREADS = 32 * (TC_WORKERS + 4);  // a warpgroup for the issuing warp: it gives its registers to the workers
// shared memory: the words, the two matrices, the small twiddles
constexpr u32 TC_S_B = TC_WORDS * 8, TC_S_B3 = TC_S_B + 65536, TC_S_SMALL = TC_S_B3 + 16384, TC_SMEM = TC_S_SMALL + TC_SMALL_WORDS * 8;

enum { BAR_FULL = 0, BAR_FREE = 2, BAR_READY = 4, BAR_DONE = 16, BAR_COUNT = 17 };

__device__ __forceinline__ void tc_sts(u32 addr, u64 v) { asm volatile("st.shared.b64 [%0], %1;\n" ::"r"(addr), "l"(v) : "memory"); }
__device__ __forceinline__ void tc_sts2(u32 addr, u64 v, u64 w) { asm volatile("st.shared.v2.b64 [%0], {%1, %2};\n" ::"r"(addr), "l"(v), "l"(w) : "memory"); }
__device__ __forceinline__ u64 tc_lds(u32 addr) {
    u64 v;
    asm volatile("ld.shared.b64 %0, [%1];\n" : "=l"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ u64 tc_ldg(const u64* p) {
    u64 v;
    asm volatile("ld.global.nc.b64 %0, [%1];\n" : "=l"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ void tc_arrive(u32 bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory"); }

// A batch of rows is a chain of transforms, the inverse one and one for each residue; a transform is twelve products (encode_tc.cuh: I1, I2,
// I3 or F1, F2, F3, four of each) of 128 rows by a 256 x 256 byte matrix, or of 256 rows by the 128 x 128 one, two accumulators of 256 TMEM
// columns in turn.  Warp 16 issues them; the sixteen others are the workers: each takes the 32 lanes of the accumulator that it can reach
// (warp mod 4) and a quarter of its columns, eight words a lane, which a thread makes into words, twists and puts where the next pass wants
// them.  I2's and F1's results move everywhere, so they wait in registers until the pass's last product has read its tile.  What follows a
// residue (the next residue's words, the next batch's message) is brought before the last product's results are taken out, and its first
// product runs beside them.
// Barriers: FULL[2] an accumulator holds its product; FREE[2] the workers have read it; READY[j] the operand of product j is in place, once a
// transform each.
// What bounds it: a row of 2^14 words at rate 1/2 takes some 140 k cycles, 65 k of them instructions of each scheduler (a third of them moves
// and addresses around the 8 products and 9 joins of a word), the rest waits of its four workers on each other's passes (20 k), stores (8,192
// sectors, which the L2 takes in bursts) and the twiddles' way from L2; the tensor pipe is busy 22 %.  2,606 rows: 1,326 us, the
// shared-memory encoder 1,901.  Steps that brought it there, 2,606 rows each time: both transforms through a scratch row and one order of passes
// 2,105; the forward transform's passes reversed, so that its words stay where they are 1,674; the pads worked out ahead, no branches among
// the words 1,498; the later residues' words by asynchronous copies, twiddles asked for half a product ahead 1,479; residues apart in the output
// 1,338; a shorter test in the polling loop 1,326.  Montgomery's reduction saves a seventh of the products' instructions and 0.6 % of the time, and is
// not worth a second product and tables in its form.  96 registers a thread, with 96 to 156 bytes of them spilled (`-Xptxas -v`).
// Every wait is bounded: one that runs out sets `gave_up`, after which nobody waits and no product is issued; the CTA walks to its
// end (all addresses are the same), waits for the products in flight and frees TMEM, and leaves the store's mark where the host reads it.
template <int LOGN, bool NARROW>
__global__ void __launch_bounds__(TC_THREADS, 1) k_encode_tc(RowArgs a, const u64* __restrict__ tab, const hlk::TcReport report) {
    using T = Tc<LOGN>;
    extern __shared__ __align__(16) unsigned char raw[];
    __shared__ __align__(8) u64 bars[BAR_COUNT];
    __shared__ u32 tmem_slot;
    __shared__ volatile u32 gave_up;
    const u32 tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const u32 S = ((u32)__cvta_generic_to_shared(raw) + 1023u) & ~1023u, bar0 = (u32)__cvta_generic_to_shared(bars);
    auto bar = [&](u32 i) { return bar0 + 8 * i; };
    if (tid == 0) {
        gave_up = 0;
        for (u32 i = 0; i < BAR_COUNT; i++) {
            const u32 count = i < BAR_FREE || i == BAR_DONE ? 1u : TC_WORKERS;
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar(i)), "r"(count));
        }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::);
    }
    if (warp == TC_WORKERS) {
        // all 512 columns: the allocation cannot wait on another CTA, because this kernel's shared memory lets no second CTA that holds TMEM
        // live on an SM (the witness product's has 192 KB)
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"((u32)__cvta_generic_to_shared(&tmem_slot)), "r"(512u));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
    }
    {
        const uint4* from = reinterpret_cast<const uint4*>(tab + TC_B);
        for (u32 i = tid; i < (65536 + 16384) / 16; i += TC_THREADS) {
            const uint4 v = from[i];
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};\n" ::"r"(S + TC_S_B + 16 * i), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
        }
        for (u32 i = tid; i < TC_SMALL_WORDS; i += TC_THREADS) tc_sts(S + TC_S_SMALL + 8 * i, tab[TC_SMALL + i]);
    }
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::);
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::);
    const u32 tmem = tmem_slot;
    auto wait = [&](u32 i, u32 parity) {
        for (u32 spin = 0; spin < UM_SPIN_LIMIT; spin++) {
            if (um_try_wait(bar(i), parity)) return;
            if ((spin & 63) == 63 && (gave_up || spin >= report.limit)) break;  // (looked at less often: with the limit in the loop's own condition 1 to 4 % slower)
        }
        gave_up = 1;
    };

    // a unit of work: a batch of rows, or (split) one output residue of a batch with the batch's inverse transform before it
    const u32 R = 1u << a.logr, nn = T::N << a.logr;
    const u32 batches = (a.rows + T::ROWS - 1) / T::ROWS, units = a.split ? batches << a.logr : batches;
    const u32 residues = a.split ? 1u : R;

    if (warp >= TC_WORKERS) {
        // 96 registers a thread at launch; 4 x 112 + 24 = 472 of 5 x 96
        asm volatile("setmaxnreg.dec.sync.aligned.u32 24;\n" ::);
        if (warp == TC_WORKERS && lane == 0) {
            const u32 mine = (units - blockIdx.x + gridDim.x - 1) / gridDim.x;
            u32 count = 0;  // transforms so far
            for (u32 u = 0; u < mine && !gave_up && report.limit; u++)  // a limit of 0: no product is issued, all waits for one run out
                for (u32 f = 0; f <= residues && !gave_up; f++, count++) {
#pragma unroll 1
                    for (u32 j = 0; j < 12; j++) {
                        const u32 acc = j & 1u;
                        wait(BAR_READY + j, count & 1u);
                        if (count || j >= 2) wait(BAR_FREE + acc, ((j >> 1) + 1) & 1u);
                        if (gave_up) break;
                        asm volatile("tcgen05.fence::after_thread_sync;\n" ::);
                        const u32 d = tmem + acc * 256, at = S + (j & 3u) * 32768;
                        if (f ? j >= 4 : j < 8) {
#pragma unroll
                            for (u32 k = 0; k < 8; k++)
                                um_mma(d, um_desc(at + (k >> 2) * 16384 + (k & 3) * 32), um_desc(S + TC_S_B + (k >> 2) * 32768 + (k & 3) * 32),
                                       um_idesc(false, false, 128, 256), k ? 1u : 0u);
                        } else {
#pragma unroll
                            for (u32 k = 0; k < 8; k++)
                                um_mma(d + (k >> 2) * 128, um_desc(at + (k >> 2) * 16384 + (k & 3) * 32), um_desc(S + TC_S_B3 + (k & 3) * 32),
                                       um_idesc(false, false, 128, 128), k & 3 ? 1u : 0u);
                        }
                        um_commit(bar(BAR_FULL + acc));
                    }
                }
        }
        __syncwarp();
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 112;\n" ::);
        const u32 q = warp & 3u, g = warp >> 2, m = lane + 32 * q;
        const u32 tq = tmem + ((q * 32) << 16) + g * 64;
        // the CTA's scratch slot: the words of the residues after the first, in the order of the threads that make them; then what the pads bring
        // to the batch, `slot` words each of pad_below and of every residue's pad_above
        const u32 slot = tc_pad_words(LOGN, a.q), live = slot / T::ROWS;
        u64* const X0 = a.scratch + blockIdx.x * tc_slot_words(LOGN, residues, a.q);
        u64 *const X = X0 + 2 * tid, *const D = X0 + (residues - 1) * TC_WORDS;
        const bool wide = ((uintptr_t)a.data & 31) == 0;

        auto arrive = [&](u32 j, u32 count) {  // the warp's stores are visible to the tensor core's reads
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
            __syncwarp();
            if (lane == 0)
                for (u32 i = 0; i < count; i++) tc_arrive(bar(BAR_READY + j + i));
        };
        auto product_done = [&](u32 j) {
            wait(BAR_FULL + (j & 1u), (j >> 1) & 1u);
            __syncwarp();
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::);
        };
        // four of the eight words of product j: use(e, word) for e < 4
        auto half = [&](u32 j, u32 h, auto use) {
            u32 v[32];
            __syncwarp();  // what `use` did may have parted the lanes
            um_ld32(tq + (j & 1u) * 256 + h * 32, v);
            asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
            if (h) {
                asm volatile("tcgen05.fence::before_thread_sync;\n" ::);
                __syncwarp();
                if (lane == 0) tc_arrive(bar(BAR_FREE + (j & 1u)));
            }
#pragma unroll
            for (u32 e = 0; e < 4; e++) use(e, tc_join(v + 8 * e));
        };
        // four twiddles `step` words apart, asked for half a product before they are used
        auto ask = [&](const u64* p, u32 step, u64 (&w)[4]) {
#pragma unroll
            for (u32 e = 0; e < 4; e++) w[e] = tc_ldg(p + e * step);
        };
        auto first_row = [&](u32 unit) { return (a.split ? unit >> a.logr : unit) * T::ROWS; };
        // A batch's message.  A lane takes (a0, b0 .. b3), which spreads its stores over the banks, and four neighbouring c' at a time: a 32-byte
        // sector of a row of 2^12 words and more.
        auto fetch = [&](u32 row0) {
#pragma unroll 1
            for (u32 o = 0; o < 2; o++) {
                const u32 x = warp + 16 * o, av = ((lane >> 3) & 1u) + ((x & 15u) << 1), b = (lane & 7u) + ((lane >> 4) << 3) + ((x >> 4) << 4);
                const u32 m0 = (av << (LOGN - 5)) + (b << T::G);
                u64 y[16];
                if constexpr (NARROW) {
                    u64 rw[16 / T::VEC];
                    u32 w[16 / T::VEC];
#pragma unroll
                    for (u32 c = 0; c < 16; c += T::VEC) {
                        const u32 row = row0 + (c >> T::G);
                        w[c / T::VEC] = row < a.rows ? a.row_w[row] : 0u;
                        rw[c / T::VEC] = row < a.rows ? T::narrow_raw(a, row, m0 + (c & T::CMASK), w[c / T::VEC]) : 0u;
                    }
#pragma unroll
                    for (u32 c = 0; c < 16; c += T::VEC) {
                        if (w[c / T::VEC]) T::fill_narrow(a, row0 + (c >> T::G), m0 + (c & T::CMASK), w[c / T::VEC], rw[c / T::VEC], y + c);
                        else
                            for (u32 e = 0; e < T::VEC; e++) y[c + e] = 0;
                    }
                } else {
#pragma unroll
                    for (u32 c = 0; c < 16; c += T::VEC) {
                        const u32 row = row0 + (c >> T::G);
                        if (row < a.rows) T::fill_message(a, row, m0 + (c & T::CMASK), wide, y + c);
                        else
                            for (u32 e = 0; e < T::VEC; e++) y[c + e] = 0;
                    }
                }
                const u32 to = S + at_i1(0, b, av);  // at_i1(c, b, a) = at_i1(0, b, a) + 2^12 (c & 3) + 2^15 (c >> 2)
#pragma unroll
                for (u32 c = 0; c < 16; c++) tc_sts(to + ((c & 3u) << 12) + ((c >> 2) << 15), y[c]);
            }
            arrive(0, 4);
        };
        auto pads = [&](u32 row0, u32 s0) {
            for (u32 x = tid; x < slot; x += 32 * TC_WORKERS) {
                const u32 r = x / live, i = x - r * live;
                if (row0 + r >= a.rows) break;
                D[x] = T::pad_below(a, row0 + r, i);
                for (u32 f = 0; f < residues; f++) D[(f + 1) * slot + x] = T::pad_above(a, row0 + r, i, s0 + f);
            }
        };
        // I3's and F1's places: eight words c' = 8 (g & 1) + r of row m of tile 2 t + (g >> 1)
        const u32 o0 = 8 * (g & 1u);
        auto place = [&](u32 t, u32 pair) { return S + ((2 * t + (g >> 1)) << 14) + tc_swizzled(m, (o0 + 2 * pair) * 8); };
        // the coefficient's index i of word r there
        auto index = [&](u32 t, u32 r) { return (T::N - tc_k_of(2 * t + (g >> 1), m) - 1024 * ((o0 + r) & T::CMASK)) & (T::N - 1); };
        // what the pads bring to the words 4 h + e there (part 0: pad_below, 1 + f: pad_above); false where no word of the warp has any
        auto pad_words = [&](u32 t, u32 h, u32 part, u64 (&d)[4]) {
            bool any = false;
#pragma unroll
            for (u32 e = 0; e < 4; e++) any |= index(t, 4 * h + e) < live;
            if (!__any_sync(0xFFFFFFFFu, any)) return false;
#pragma unroll
            for (u32 e = 0; e < 4; e++) {
                const u32 i = index(t, 4 * h + e);
                d[e] = 0;
                if (i < live) d[e] = D[part * slot + ((o0 + 4 * h + e) >> T::G) * live + i];
            }
            return true;
        };

        fetch(first_row(blockIdx.x));
        for (u32 unit = blockIdx.x; unit < units; unit += gridDim.x) {
            const u32 row0 = first_row(unit), s0 = a.split ? unit & (R - 1u) : 0u;
            pads(row0, s0);  // beside the batch's first products
            // ---- I1 ----
            {
                const u64* w1 = tab + TC_I1 + (8 * g * 16 + q) * 32 + lane;
                u64 wa[4], wb[4];
                ask(w1, 512, wa);
#pragma unroll 1
                for (u32 t = 0; t < 4; t++) {
                    const u32 to = S + at_i2(4 * t + q, 8 * g, lane);
                    ask(w1 + t * 128 + 2048, 512, wb);
                    product_done(t);
                    half(t, 0, [&](u32 e, u64 v) { tc_sts(go_i2(to, e), gl_mul_lazy(v, wa[e])); });
                    if (t < 3) ask(w1 + (t + 1) * 128, 512, wa);
                    half(t, 1, [&](u32 e, u64 v) { tc_sts(go_i2(to, 4 + e), gl_mul_lazy(v, wb[e])); });
                    arrive(4 + t, 1);
                }
            }
            // ---- I2 ----
            {
                // the next batch's message, on its way to L2: a thread asks for every 512th line
                if (const u32 next = unit + gridDim.x; next < units) {
                    const u32 nrow = first_row(next);
                    if constexpr (NARROW) {
                        for (u32 r = 0; r < T::ROWS && nrow + r < a.rows; r++) {
                            const unsigned char* from = a.narrow + a.row_off[nrow + r];
                            for (u32 x = tid * 128; x < T::N * a.row_w[nrow + r]; x += 32 * TC_WORKERS * 128)
                                asm volatile("prefetch.global.L2 [%0];\n" ::"l"(from + x));
                        }
                    } else {
                        const u64 *from = a.data + (size_t)nrow * T::N, *end = a.data + (size_t)a.rows * T::N;
                        for (u32 x = tid * 16; x < TC_WORDS; x += 32 * TC_WORKERS * 16)
                            if (from + x < end) asm volatile("prefetch.global.L2 [%0];\n" ::"l"(from + x));
                    }
                }
                const u32 ka = (m >> 1) & 31u, c0 = (m & 1u) + ((m >> 6) << 1);
                const u32 tw = S + TC_S_SMALL + (8 * g * 16 + c0) * 8, to = S + at_c(ka, 8 * g, c0);
                u64 hold[24];
#pragma unroll
                for (u32 t = 0; t < 4; t++) {
                    product_done(4 + t);
                    if (t == 3) {
#pragma unroll
                        for (u32 i = 0; i < 24; i++) tc_sts(go_c(tile_i2(to, i >> 3), i & 7), hold[i]);
                    }
#pragma unroll
                    for (u32 h = 0; h < 2; h++)
                        half(4 + t, h, [&](u32 e, u64 v) {
                            const u32 r = 4 * h + e;
                            v = gl_mul_lazy(v, tc_lds(tw + r * 128 + t * 32));
                            if (t == 3) tc_sts(go_c(tile_i2(to, 3), r), v);
                            else hold[8 * (t % 3) + r] = v;
                        });
                }
                arrive(8, 4);
            }
            // ---- I3 ----
            // the coset's words, then every residue's: the first one's stay here, the others' go to the scratch slot
            {
                u64 wa[4], wb[4];
                auto powers = [&](u32 t, u32 h, u64 (&w)[4]) {
#pragma unroll
                    for (u32 e = 0; e < 4; e++) w[e] = a.zk ? tc_ldg(a.pows + index(t, 4 * h + e)) : 1;
                };
                auto finish = [&](u32 t, u32 h, const u64 (&w)[4]) {
                    u64 x[4], y[4], z[4], d[4];
                    const bool later = residues > 1;
                    auto twists = [&](u32 s) {
#pragma unroll
                        for (u32 e = 0; e < 4; e++) z[e] = tc_ldg(tab + TC_TWIST + ((index(t, 4 * h + e) * s) & (nn - 1)));
                    };
                    if (later || s0) twists(later ? 1u : s0);
                    half(8 + t, h, [&](u32 e, u64 v) { x[e] = gl_mul_lazy(v, w[e]); });
                    const bool padded = pad_words(t, h, 0, d);
                    if (padded) {
#pragma unroll
                        for (u32 e = 0; e < 4; e++) x[e] = gl_add_lazy(x[e], d[e]);
                    }
#pragma unroll 1
                    for (u32 f = later ? 1u : 0u;;) {
                        const u32 s = s0 + f;
#pragma unroll
                        for (u32 e = 0; e < 4; e++) y[e] = x[e];
                        if (padded) {
                            pad_words(t, h, 1 + f, d);
#pragma unroll
                            for (u32 e = 0; e < 4; e++) y[e] = gl_add_lazy(y[e], d[e]);
                        }
                        if (s) {
#pragma unroll
                            for (u32 e = 0; e < 4; e++) y[e] = gl_mul_lazy(y[e], z[e]);
                        }
                        if (f == 0) break;
#pragma unroll
                        for (u32 e = 0; e < 4; e += 2)
                            asm volatile("st.global.v2.b64 [%0], {%1, %2};\n" ::"l"(X + (f - 1) * TC_WORDS + (t * 4 + 2 * h + e / 2) * 1024), "l"(y[e]), "l"(y[e + 1]) : "memory");
                        f = f + 1 < residues ? f + 1 : 0;
                        if (f) twists(f);
                    }
#pragma unroll
                    for (u32 e = 0; e < 4; e += 2) tc_sts2(place(t, 2 * h + e / 2), y[e], y[e + 1]);
                };
                powers(0, 0, wa);
                asm volatile("bar.sync 1, %0;\n" ::"r"(32 * TC_WORKERS) : "memory");  // the pads' words are there
#pragma unroll 1
                for (u32 t = 0; t < 4; t++) {
                    powers(t, 1, wb);
                    product_done(8 + t);
                    finish(t, 0, wa);
                    if (t < 3) powers(t + 1, 0, wa);
                    finish(t, 1, wb);
                    arrive(t, 1);
                }
            }
#pragma unroll 1
            for (u32 f = 0; f < residues; f++) {
                const u32 s = s0 + f;
                // ---- F1 ----
                {
                    const u32 k0 = tc_k_of(g >> 1, m);
                    const u32 to = S + at_f2(o0, k0 & 31u, k0 >> 5);
                    const u64* tw = tab + TC_F1 + (o0 * 8 + (g >> 1)) * 128 + m;
                    u64 hold[24], wa[4], wb[4];
                    ask(tw, 1024, wa);
#pragma unroll
                    for (u32 t = 0; t < 4; t++) {
                        ask(tw + t * 256 + 4096, 1024, wb);
                        product_done(t);
                        if (t == 3) {
#pragma unroll
                            for (u32 i = 0; i < 24; i++) tc_sts(go_f2(tile_f1(to, i >> 3), i & 7), hold[i]);
                        }
#pragma unroll
                        for (u32 h = 0; h < 2; h++) {
                            half(t, h, [&](u32 e, u64 v) {
                                const u32 r = 4 * h + e;
                                v = gl_mul_lazy(v, h ? wb[e] : wa[e]);
                                if (t == 3) tc_sts(go_f2(tile_f1(to, 3), r), v);
                                else hold[8 * (t % 3) + r] = v;
                            });
                            if (h == 0 && t < 3) ask(tw + (t + 1) * 256, 1024, wa);
                        }
                    }
                    arrive(4, 4);
                }
                // ---- F2 ----
#pragma unroll 1
                for (u32 t = 0; t < 4; t++) {
                    const u32 tw = S + TC_S_SMALL + (TC_F2 + 8 * g * 32 + lane) * 8, to = S + at_f3(4 * t + q, 8 * g, lane);
                    product_done(4 + t);
#pragma unroll
                    for (u32 h = 0; h < 2; h++) half(4 + t, h, [&](u32 e, u64 v) { tc_sts(go_f3(to, 4 * h + e), gl_mul_lazy(v, tc_lds(tw + (4 * h + e) * 256))); });
                    arrive(8 + t, 1);
                }
                // ---- F3 ----
#pragma unroll 1
                for (u32 t = 0; t < 4; t++) {
                    if (t == 3) {
                        const u32 next = unit + gridDim.x;
                        product_done(11);  // every operand has been read
                        if (f + 1 < residues) {
                            for (u32 p = 0; p < 16; p++)
                                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(place(p >> 2, p & 3u)), "l"(X + f * TC_WORDS + p * 1024) : "memory");
                        } else if (next < units) {
                            fetch(first_row(next));
                        }
                    }
                    const u32 c = 4 * t + (m & 3u), row = row0 + (c >> T::G), j0 = (c & T::CMASK) + ((m >> 2) << T::G) + 8 * g * (T::N / 32);
                    u64* out = a.enc + (((size_t)row << a.logr) + s) * T::N;  // residue by residue (ColOrder)
                    product_done(8 + t);
#pragma unroll
                    for (u32 h = 0; h < 2; h++) {
                        half(8 + t, h, [&](u32 e, u64 v) {
                            if (row < a.rows) out[(T::N - j0 - (4 * h + e) * (T::N / 32)) & (T::N - 1)] = gl_canon_fast(v);
                        });
                        if (h == 0 && t == 3 && f + 1 < residues) {
                            asm volatile("cp.async.wait_all;\n" ::: "memory");
                            arrive(0, 4);
                        }
                    }
                }
            }
        }
    }
    // the products in flight, then TMEM
    if (tid == 32 * TC_WORKERS) {
        um_commit(bar(BAR_DONE));
        if (!um_wait(bar(BAR_DONE), 0)) gave_up = 1;
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::);
    __syncthreads();
    if (tid == 0 && gave_up) {  // behind every wait of every warp
        *reinterpret_cast<volatile u32*>(report.word) = report.mark;
        if (report.also) *reinterpret_cast<volatile u32*>(report.also) = 1;
    }
    if (warp == TC_WORKERS) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512u));
}

template <int LOGN, bool NARROW>
cudaError_t launch_tc(const RowArgs& a, const u64* tab, unsigned grid, const hlk::TcReport& report, cudaStream_t st) {
    auto kern = k_encode_tc<LOGN, NARROW>;
    const int smem = (int)TC_SMEM + 1024;
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    kern<<<grid, TC_THREADS, smem, st>>>(a, tab, report);
    return cudaGetLastError();
}

u32 tc_batches(u32 logn, u32 rows) {
    const u32 per = TC_WORDS >> logn;
    return (rows + per - 1) / per;
}
// whether one residue a CTA, with the inverse transform before it, takes fewer turns of the machine than all of them after one inverse transform
bool tc_splits(u32 logr, u64 batches, u64 sms) {
    return logr >= 1 && ((batches << logr) + sms - 1) / sms * 2 < (batches + sms - 1) / sms * (1 + ((u64)1 << logr));
}

}  // namespace

namespace hlk {

size_t encode_tc_table_words(u32 logn, u32 logr) { return tc_table_words(logn, logr); }
void encode_tc_build(u32 logn, u32 logr, u64* out) { tc_build(logn, logr, out); }

// Rows of 2^14 words always: 2,606 of them 1,901 -> 1,326 us, 74 of them 74 -> 56, 4 of them 72 -> 55; at rate 1/4 1,184 rows 1,625 -> 1,146.
// Shorter rows where a CTA that takes 2^14 words' worth of them is not the longer chain: a transform takes one 26 us and a machine full of
// them no longer.  The shared-memory encoder gives rows of 2^13 words a CTA each per residue (44 us) while they fit the SMs, and
// takes 12 us + 0.195 us for each 2^14 words and transform of shorter ones (both fitted to rows of 2^10 .. 2^13 words, 4 to 2,606 times 2^14
// words, rates 1/2 and 1/4): 592 rows of 2^11 56 -> 52, 1,184 of them 95 -> 74, 720 of them 65 (72 here); 2,368 of 2^12 346 -> 283, 800 of them
// 131 (142 here); 148 of 2^13 63 -> 56, 74 of them 47 (54 here).
// Measured at rates down to 1/64, 1 to 444 times 2^14 words (rows of 2^14: rate 1/8 38 rows 221 -> 143, 1,036 of them 3,204 -> 1,903; rate 1/16
// 148 rows 1,121 -> 596; rate 1/64 4 rows 179 -> 119, 38 of them 1,407 -> 866; rows of 2^13 alike): what the line gives to this encoder is never
// more than 3 % slower here (400 rows of 2^13 at 1/2 142, 146 here).  It is a cautious one: the other encoder's scratch leaves L2 at rates of
// 1/16 and less, where its 0.195 us become 0.4 and more, and rows of 2^10 .. 2^12 that it keeps would take half the time here (592 rows of
// 2^11 at 1/64 2,885, 1,301 here).
bool encode_tc_takes(u32 logn, u32 logr, u32 rows, int sm_count) {
    if (logn < 10 || logn > 14) return false;
    if (logn == 14) return true;
    const u64 sms = (u64)sm_count;
    if (logn == 13) return ((u64)rows << logr) > sms;
    const u64 batches = tc_batches(logn, rows), whole = (batches + sms - 1) / sms * (1 + ((u64)1 << logr)), split = ((batches << logr) + sms - 1) / sms * 2;
    return (whole < split ? whole : split) * 26000 < 12000 + 195 * (1 + ((u64)1 << logr)) * batches * 148 / sms;
}

// A slot for each CTA, never more CTAs than SMs.  Whole batches keep the words of all residues but one, so their slots come near the
// encoding's own size where the machine holds every batch at once; split ones keep the pads' words alone.
size_t encode_tc_scratch_words(u32 logn, u32 logr, u32 q, u32 rows, int sm_count) {
    const u64 batches = tc_batches(logn, rows), sms = (u64)sm_count;
    if (tc_splits(logr, batches, sms)) return encode_tc_least_words(logn, logr, q, rows, sm_count);
    return (size_t)(batches < sms ? batches : sms) * tc_slot_words(logn, 1u << logr, q);
}
size_t encode_tc_least_words(u32 logn, u32 logr, u32 q, u32 rows, int sm_count) {
    const u64 units = (u64)tc_batches(logn, rows) << logr, sms = (u64)sm_count;
    return (size_t)(units < sms ? units : sms) * tc_slot_words(logn, 1u, q);
}

cudaError_t encode_rows_tc(RowArgs a, u32 logn, const u64* tab, int sm_count, size_t scratch_words, TcReport report, cudaStream_t st, int* path_out) {
    const u64 batches = tc_batches(logn, a.rows), sms = (u64)sm_count;
    // split as well where the scratch is not what whole batches take: at rate 1/64 148 rows of 2^14 words would keep 1.2 GB
    a.split = tc_splits(a.logr, batches, sms) || (a.logr && scratch_words < encode_tc_scratch_words(logn, a.logr, a.q, a.rows, sm_count));
    u64 grid = a.split ? batches << a.logr : batches;
    if (grid > sms) grid = sms;
    const u64 per = tc_slot_words(logn, a.split ? 1u : 1u << a.logr, a.q);  // none for one residue without pads
    if (per && grid > scratch_words / per) grid = scratch_words / per;
    if (grid < 1 || a.loga) return cudaErrorInvalidValue;
    if (path_out) *path_out = a.narrow ? 2 : 1;
    const unsigned gr = (unsigned)grid;
    switch (logn) {
        case 10: return a.narrow ? launch_tc<10, true>(a, tab, gr, report, st) : launch_tc<10, false>(a, tab, gr, report, st);
        case 11: return a.narrow ? launch_tc<11, true>(a, tab, gr, report, st) : launch_tc<11, false>(a, tab, gr, report, st);
        case 12: return a.narrow ? launch_tc<12, true>(a, tab, gr, report, st) : launch_tc<12, false>(a, tab, gr, report, st);
        case 13: return a.narrow ? launch_tc<13, true>(a, tab, gr, report, st) : launch_tc<13, false>(a, tab, gr, report, st);
        case 14: return a.narrow ? launch_tc<14, true>(a, tab, gr, report, st) : launch_tc<14, false>(a, tab, gr, report, st);
    }
    return cudaErrorInvalidValue;
}

}  // namespace hlk
