// Host-side execution of the row encoder's phase functions (csrc/encode_core.cuh), one
// emulated thread at a time.  Test infrastructure: it checks the kernels' index arithmetic
// (windows, swizzle, twiddle indexing, pad placement) on a machine without a GPU.  A phase is
// run for every thread before the next phase starts, which is what the barriers guarantee.
#include <cstdlib>
#include <cstring>
#include <utility>
#include <vector>
#include "../../intelligenceregulation_b200/csrc/encode_core.cuh"

using namespace enc;

static std::vector<u64> make_tw(u32 lognn) {
    u64 r32 = gl_pow(7, (GL_P - 1) >> 32), w = gl_pow(r32, 1ULL << (32 - lognn));
    std::vector<u64> tw((size_t)1 << lognn);
    u64 c = 1;
    for (auto& x : tw) { x = c; c = gl_mul(c, w); }
    return tw;
}

struct NoSync { void operator()() const {} };

template <int LOGN>
static void run_fast(RowArgs a, u32 nt) {
    using F = Fast<LOGN>;
    std::vector<u64> S(F::N + 16), TW(F::TW_WORDS + 16);
    for (u32 t = 0; t < nt; t++) F::load_twiddles(a, TW.data(), t, nt);
    // one emulated thread owning every group keeps the pass order of the device code
    for (u32 row = 0; row < a.rows; row++) {
        F::row_coeffs(a, row, S.data(), TW.data(), a.scratch, 0, 1, NoSync());
        for (u32 s = 0; s < (1u << a.logr); s++) F::row_residue(a, row, s, S.data(), TW.data(), a.scratch, 0, 1, NoSync());
    }
}

extern "C" int emul_encode(int fast, const u64* data, u32 rows, u32 logn, u32 logr, const u64* pads, u32 q,
                           const u64* pows, int zk, u32 nt, u64* out) {
    u32 n = 1u << logn;
    std::vector<u64> tw = make_tw(logn + logr);
    // rows above 2^14 words run as 2 or 4 transforms of 2^14, exactly as the library's commit sets them up
    const u32 logb = logn > 14 ? 14 : logn, loga = logn - logb, nb = 1u << logb;
    RowArgs a;
    a.data = data; a.pads = pads; a.pows = pows; a.tw_nn = tw.data(); a.enc = out;
    a.rows = rows; a.q = zk ? q : 0; a.logr = logr + loga; a.loga = loga; a.zk = zk;
    a.T = zk ? (n + q + nb - 1) / nb : n / nb;
    a.ninv = gl_inv(n); a.coef_out = nullptr; a.split = 0;
    std::vector<u64> X((size_t)a.T * nb, 0xA5A5A5A5A5A5A5A5ULL);  // poisoned: unwritten words must never be read
    a.scratch = X.data();
    if (fast) {
        switch (logb) {
            case 8: run_fast<8>(a, nt); break;
            case 9: run_fast<9>(a, nt); break;
            case 10: run_fast<10>(a, nt); break;
            case 11: run_fast<11>(a, nt); break;
            case 12: run_fast<12>(a, nt); break;
            case 13: run_fast<13>(a, nt); break;
            case 14: run_fast<14>(a, nt); break;
            default: return -1;
        }
        return 0;
    }
    std::vector<u64> S(n);
    for (u32 row = 0; row < rows; row++) {
        for (u32 t = 0; t < nt; t++) Generic::load(a, row, logn, S.data(), t, nt);
        for (u32 ln = logn; ln >= 1; ln--)
            for (u32 t = 0; t < nt; t++) Generic::dif_stage(a, logn, ln, S.data(), t, nt);
        for (u32 t = 0; t < nt; t++) Generic::coeffs(a, row, logn, S.data(), a.scratch, t, nt);
        for (u32 s = 0; s < (1u << logr); s++) {
            for (u32 t = 0; t < nt; t++) Generic::twist(a, logn, s, a.scratch, S.data(), t, nt);
            for (u32 ln = 1; ln <= logn; ln++)
                for (u32 t = 0; t < nt; t++) Generic::dit_stage(a, logn, ln, S.data(), t, nt);
            for (u32 t = 0; t < nt; t++) Generic::store(a, row, logn, s, S.data(), t, nt);
        }
    }
    return 0;
}

// The tensor-core path (csrc/encode_tc.cuh): its layouts, tables and twiddles, with the matrix products done byte by byte on operands
// addressed as the instruction's descriptors address them (rows of 128 bytes, swizzled pieces, K halves and tiles apart).
#include "../../intelligenceregulation_b200/csrc/encode_tc.cuh"

static void sums8(const unsigned char* A, u32 a_half, u32 m, const unsigned char* B, u32 b_half, u32 slot, u32 kbytes, u32* s) {
    for (u32 d = 0; d < 8; d++) {
        u32 t = 0;
        for (u32 kb = 0; kb < kbytes; kb++)
            t += (u32)A[(kb >> 7) * a_half + tc_swizzled(m, kb & 127)] * B[(kb >> 7) * b_half + tc_swizzled(8 * slot + d, kb & 127)];
        s[d] = t;
    }
}

template <int LOGN>
static int run_tc(const RowArgs& a) {
    using T = Tc<LOGN>;
    std::vector<u64> tab(tc_table_words(LOGN, a.logr));
    tc_build(LOGN, a.logr, tab.data());
    const unsigned char *B = (const unsigned char*)(tab.data() + TC_B), *B3 = (const unsigned char*)(tab.data() + TC_B3);
    std::vector<u64> Sw(TC_WORDS), keep(TC_WORDS);
    if (tc_slot_words(LOGN, 1u << a.logr, a.q) % 2 || tc_slot_words(LOGN, 1, a.q) % 2) return -3;
    unsigned char* S = (unsigned char*)Sw.data();
    const u32 nn = T::N << a.logr;
    auto word = [&](u32 at) -> u64& { return *(u64*)(S + at); };
    bool bad = false;
    // one product of a pass over 32 points (tile t) or over c' (tile t of eight): put(row, slot, word) for all its results
    auto product = [&](bool c16, u32 t, auto put) {
        for (u32 m = 0; m < 128; m++)
            for (u32 k = 0; k < (c16 ? 16u : 32u); k++) {
                u32 sum[8];
                if (c16) sums8(S + t * 16384, 0, m, B3, 0, k, 128, sum);
                else sums8(S + t * 32768, 16384, m, B, 32768, k, 256, sum);
                put(m, k, tc_join(sum));
            }
    };
    std::vector<std::pair<u32, u64>> hold;
    auto flush = [&](int tile) {  // tile >= 0: the results stay within that tile of 32 KB
        for (auto& h : hold) {
            bad |= tile >= 0 && (int)(h.first >> 15) != tile;
            word(h.first) = h.second;
        }
        hold.clear();
    };
    // the kernel's way to an address, from an operand that lies at any multiple of 1,024
    constexpr u32 S0 = 0x2C00;
    auto to = [&](u32 at, u32 same, u64 v) {
        bad |= at != S0 + same || same >= 8 * TC_WORDS;
        hold.push_back({same, v});
    };
    for (u32 row0 = 0; row0 < a.rows; row0 += T::ROWS) {
        for (u32 i = 0; i < TC_WORDS; i++) word(8 * i) = 0;
        for (u32 a0 = 0; a0 < 32; a0++)
            for (u32 b = 0; b < 32; b++)
                for (u32 c = 0; c < 16; c += T::VEC) {
                    u64 y[4];
                    if (row0 + (c >> T::G) >= a.rows) continue;
                    T::fill_message(a, row0 + (c >> T::G), (a0 << (LOGN - 5)) + (b << T::G) + (c & T::CMASK), true, y);
                    for (u32 e = 0; e < T::VEC; e++) word(at_i1(c + e, b, a0)) = y[e];
                }
        for (u32 t = 0; t < 4; t++) {
            product(false, t, [&](u32 m, u32 k, u64 v) {
                const u32 b = m & 31, c = 4 * t + (m >> 5);
                to(go_i2(S0 + at_i2(c, k & ~7u, b), k & 7), at_i2(c, k, b), gl_mul_lazy(v, tab[TC_I1 + (k * 16 + c) * 32 + b]));
            });
            flush(t);
        }
        for (u32 t = 0; t < 4; t++)
            product(false, t, [&](u32 m, u32 k, u64 v) {
                const u32 ka = (m >> 1) & 31, c = 4 * t + (m & 1) + ((m >> 6) << 1);
                to(go_c(tile_i2(S0 + at_c(ka, k & ~7u, c & 3), t), k & 7), at_c(ka, k, c), gl_mul_lazy(v, tab[TC_SMALL + k * 16 + c]));
            });
        flush(-1);
        for (u32 s = 0; s < (1u << a.logr); s++) {
            if (s == 0) {
                for (u32 t = 0; t < 8; t++) {
                    product(true, t, [&](u32 m, u32 o, u64 v) {
                        const u32 i = (T::N - tc_k_of(t, m) - 1024 * (o & T::CMASK)) & (T::N - 1), row = row0 + (o >> T::G), at = t * 16384 + tc_swizzled(m, 8 * o);
                        const bool pad = row < a.rows && i < tc_pad_words(LOGN, a.q) / T::ROWS;
                        u64 x = gl_mul_lazy(v, a.zk ? a.pows[i] : 1);
                        if (pad) x = gl_add_lazy(x, T::pad_below(a, row, i));
                        keep[at / 8] = x;
                        if (pad) x = gl_add_lazy(x, T::pad_above(a, row, i, 0));
                        to(S0 + at, at_c(tc_k_of(t, m) & 31, tc_k_of(t, m) >> 5, o), x);
                    });
                    flush(t >> 1);
                }
            } else {
                for (u32 t = 0; t < 8; t++)
                    for (u32 m = 0; m < 128; m++)
                        for (u32 o = 0; o < 16; o++) {
                            const u32 i = (T::N - tc_k_of(t, m) - 1024 * (o & T::CMASK)) & (T::N - 1), row = row0 + (o >> T::G), at = t * 16384 + tc_swizzled(m, 8 * o);
                            u64 x = keep[at / 8];
                            if (row < a.rows && i < tc_pad_words(LOGN, a.q) / T::ROWS) x = gl_add_lazy(x, T::pad_above(a, row, i, s));
                            word(at) = gl_mul_lazy(x, tab[TC_TWIST + ((i * s) & (nn - 1))]);
                        }
            }
            for (u32 t = 0; t < 8; t++)
                product(true, t, [&](u32 m, u32 c, u64 v) {
                    const u32 ka = tc_k_of(t, m) & 31, kb = tc_k_of(t, m) >> 5;
                    to(go_f2(tile_f1(S0 + at_f2(c & ~7u, ka, kb & 7), t >> 1), c & 7), at_f2(c, ka, kb), gl_mul_lazy(v, tab[TC_F1 + (c * 8 + t) * 128 + m]));
                });
            flush(-1);
            for (u32 t = 0; t < 4; t++) {
                product(false, t, [&](u32 m, u32 k, u64 v) {
                    const u32 ka = m & 31, c = 4 * t + (m >> 5);
                    to(go_f3(S0 + at_f3(c, k & ~7u, ka), k & 7), at_f3(c, k, ka), gl_mul_lazy(v, tab[TC_SMALL + TC_F2 + k * 32 + ka]));
                });
                flush(t);
            }
            for (u32 t = 0; t < 4; t++)
                product(false, t, [&](u32 m, u32 k, u64 v) {
                    const u32 c = 4 * t + (m & 3), jb = m >> 2, row = row0 + (c >> T::G), j = (c & T::CMASK) + (jb << T::G) + k * (T::N / 32);
                    if (row < a.rows) a.enc[(((size_t)row << a.logr) + s) * T::N + ((T::N - j) & (T::N - 1))] = gl_canon_fast(v);
                });
        }
    }
    return bad ? -2 : 0;
}

extern "C" int emul_encode_tc(const u64* data, u32 rows, u32 logn, u32 logr, const u64* pads, u32 q, const u64* pows, int zk, u64* out) {
    std::vector<u64> tw = make_tw(logn + logr);
    RowArgs a;
    a.data = data; a.pads = pads; a.pows = pows; a.tw_nn = tw.data(); a.enc = out; a.scratch = nullptr;
    a.rows = rows; a.q = zk ? q : 0; a.logr = logr; a.loga = 0; a.zk = zk; a.T = 1;
    a.ninv = 0; a.coef_out = nullptr; a.split = 0;
    switch (logn) {
        case 10: return run_tc<10>(a);
        case 11: return run_tc<11>(a);
        case 12: return run_tc<12>(a);
        case 13: return run_tc<13>(a);
        case 14: return run_tc<14>(a);
    }
    return -1;
}

// eight sums at their largest and around every carry of the join
extern "C" int emul_join(const u32* sums, u32 count, u64* out) {
    for (u32 i = 0; i < count; i++) out[i] = gl_canon(tc_join(sums + 8 * i));
    return 0;
}
