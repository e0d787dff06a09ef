// Row encoder on the tensor cores: what one thread does, and where everything lies.
//
// A DFT of r <= 32 points over the Goldilocks field is a matrix product over BYTES.  With x_j = sum_b 2^(8b) x_jb,
//
//     y_i = sum_j w^(ij) x_j = sum_(j,b) x_jb (2^(8b) w^(ij) mod p) = sum_d 2^(8d) sum_(j,b) x_jb C[(j,b)][(i,d)],
//
// C[(j,b)][(i,d)] being byte d of the constant: u8 x u8 sums of at most 256 terms, below 2^24, exact in the int32 accumulators of
// tcgen05.mma kind::i8.  The eight bytes of a word ARE the limbs: any word congruent mod p is an operand as it lies in memory.
// What is left to the integer pipes is to put eight sums together into a word (`tc_join`) and the twiddles between passes.
//
// One CTA takes 2^14 words at a time: 2^(14 - LOGN) rows of n = 2^LOGN words, G = LOGN - 10.  A row's message index is
// i = a (n / 32) + b 2^G + c, a, b < 32, c < 2^G, and a four-bit c' = (row in the batch) 2^G + c stands for both: the DFT over c' is
// one of 2^G points beside the identity over the batch's rows, a 16-point matrix whatever G is.
//
//     inverse   F[k] = sum_i msg[i] w_n^(ik), k = ka + 32 kb + 1024 kc:
//               I1 over a, times w_n^(ka (b 2^G + c));  I2 over b, times w_(n/32)^(kb c) / n;  I3 over c'
//               F[k] / n is the coefficient of x^(n - k); I3 makes the twisted coefficient y_s[k] of it where it stands
//     forward   H[j] = sum_k y_s[k] w_n^(jk), j = jc + 2^G jb + (n / 32) ja, is the codeword's word n - j of residue s:
//               F1 over kc, times w_n^(jc (ka + 32 kb));  F2 over kb, times w_1024^(jb ka);  F3 over ka
//
// So a row's words stay in shared memory from its message to its first residue; the coefficients wait in a scratch slot (L2) for the other
// residues only, each in the place of the thread that made it.  Shared memory holds the 2^14 words as the A operand of the product to
// come: K-major rows of 128 bytes (16 words) with the 128-byte swizzle, tiles of 128 rows.  The five layouts below are chosen so that
// the stores of a half-warp fall into 16 different banks, and so that I1, I3 and F2 write a tile's results over that tile.
//
// The functions compile for the host too, where a test runs whole rows through them against the oracle.
#pragma once
#include "encode_core.cuh"

namespace enc {

// ---- the constants of a transform size, made once on the host (`tc_build`) and kept on the device ----
constexpr u32 TC_WORDS = 1u << 14;           // words in flight per CTA
constexpr u32 TC_I1 = 0;                     // 32 x 16 x 32: [ka][c'][b]
constexpr u32 TC_F1 = TC_I1 + 16384;         // 16 x 8 x 128: [jc'][tile of (ka, kb)][row of the tile]
constexpr u32 TC_SMALL = TC_F1 + 16384;      // I2's 32 x 16 [kb][c'], F2's 32 x 32 [jb][ka]
constexpr u32 TC_F2 = 512;                   // (within the small ones)
constexpr u32 TC_SMALL_WORDS = 512 + 1024;
constexpr u32 TC_B = TC_SMALL + TC_SMALL_WORDS;  // the 32-point matrix, 256 x 256 bytes in the order shared memory holds it
constexpr u32 TC_B3 = TC_B + 8192;           // the matrix over c', 128 x 128 bytes
constexpr u32 TC_TABLE_WORDS = TC_B3 + 2048;

// byte `kb` of row `r` of a K-major operand of 128-byte rows: 16-byte pieces XORed with the row within its group of eight
GL_HD u32 tc_swizzled(u32 r, u32 kb) { return r * 128 + ((((kb >> 4) & 7u) ^ (r & 7u)) << 4) + (kb & 15u); }

// ---- byte addresses of a word before each product ----
// A 32-point operand: tile = c' >> 2 of 32 KB, K halves of 16 KB.  Rows: I1 b + 32 (c' & 3); I2 (c' & 1) + 2 ka + 64 (c' >> 1 & 1);
// F2 ka + 32 (c' & 3); F3 (c' & 3) + 4 jb.
GL_HD u32 tc_at32(u32 c, u32 row, u32 k) { return ((c >> 2) << 15) + ((k >> 4) << 14) + tc_swizzled(row, (k & 15u) * 8); }
GL_HD u32 at_i1(u32 c, u32 b, u32 a) { return tc_at32(c, b + ((c & 3u) << 5), a); }
GL_HD u32 at_i2(u32 c, u32 ka, u32 b) { return tc_at32(c, (c & 1u) + 2 * ka + ((c & 2u) << 5), b); }
GL_HD u32 at_f2(u32 c, u32 ka, u32 kb) { return tc_at32(c, ka + ((c & 3u) << 5), kb); }
GL_HD u32 at_f3(u32 c, u32 jb, u32 ka) { return tc_at32(c, (c & 3u) + 4 * jb, ka); }
// I3 and F1: eight tiles of 16 KB, tile = kb >> 2, rows (ka & 7) + 8 (kb & 1) + 16 (ka >> 3) + 64 (kb >> 1 & 1)
GL_HDC u32 tc_row(u32 ka, u32 kb) { return (ka & 7u) + ((kb & 1u) << 3) + ((ka >> 3) << 4) + ((kb & 2u) << 5); }
GL_HD u32 at_c(u32 ka, u32 kb, u32 c) { return ((kb >> 2) << 14) + tc_swizzled(tc_row(ka, kb), c * 8); }
// and back: the k = ka + 32 kb of a row of a tile
GL_HD u32 tc_k_of(u32 tile, u32 row) { return (row & 7u) + (((row >> 4) & 3u) << 3) + (((row >> 3) & 1u) << 5) + ((row >> 6) << 6) + (tile << 7); }
// From the address of a thread's first word to that of word r < 8: of at_i2(c, 8 g, b) to at_i2(c, 8 g + r, b), and so on.  `base` may
// hold the operand's own address, a multiple of 1,024: what is XORed lies below that, the rest is added.
GL_HD u32 go_i2(u32 base, u32 r) { return (base ^ ((r & 3u) << 5)) + (r << 8); }                           // ka
GL_HD u32 go_c(u32 base, u32 r) { return base + ((r & 1u) << 10) + ((r & 2u) << 12) + ((r >> 2) << 14); }  // kb
GL_HD u32 go_f2(u32 base, u32 r) { return base + ((r & 3u) << 12) + ((r >> 2) << 15); }                    // c'
GL_HD u32 go_f3(u32 base, u32 r) { return (base ^ ((r & 1u) << 6)) + (r << 9); }                           // jb
// and from I2's tile 0 to tile t (c' + 4 t), from F1's tiles 0 and 1 to 2 t and 2 t + 1 (kb + 8 t)
GL_HD u32 tile_i2(u32 base, u32 t) { return base ^ (t << 5); }
GL_HD u32 tile_f1(u32 base, u32 t) { return (base ^ ((t & 1u) << 6)) + ((t >> 1) << 14); }

// Words of a CTA's scratch slot: the words of every residue but the first that the CTA makes, in pairs on 16-byte boundaries (so the slot is a
// multiple of two words), then what the pads bring, a part below the message and one above it for each residue
GL_HD u32 tc_pad_words(u32 logn, u32 q) { return (q < (1u << logn) ? q : 1u << logn) * (TC_WORDS >> logn); }
GL_HD size_t tc_slot_words(u32 logn, u32 residues, u32 q) { return (size_t)(residues - 1) * TC_WORDS + ((((size_t)residues + 1) * tc_pad_words(logn, q) + 1) & ~(size_t)1); }

// ---- arithmetic ----
// sum_d 2^(8d) s[d] as a word (lazy), s[d] <= 256 * 255 * 255.  Neighbours fit 32 bits together (0xFE0100 * 257 = 0xFEFF0100); with
// e0 .. e3 the pairs, V = e0 + 2^16 e1 + 2^32 e2 + 2^48 e3 < 2^81 and 2^64 = 2^32 - 1.
GL_HD u64 tc_join(const u32* s) {
    const u32 e0 = s[0] + (s[1] << 8), e1 = s[2] + (s[3] << 8), e2 = s[4] + (s[5] << 8), e3 = s[6] + (s[7] << 8);
#ifdef __CUDA_ARCH__
    u64 w, g;
    u32 r0, r1;
    asm("mad.wide.u32 %0, %1, 0x10000, %2;" : "=l"(w) : "r"(e1), "l"(((u64)e2 << 32) | e0));  // e0 + 2^16 e1 + 2^32 e2 < 2^64
    asm("mad.wide.u32 %0, %1, 0x10000, %2;" : "=l"(g) : "r"(e3), "l"(w >> 32));
    asm("{\n\t"
        ".reg .u32 m;\n\t"
        "mad.lo.cc.u32 %0, %4, 0xFFFFFFFF, %2;\n\t"  // the third word's (2^32 - 1), itself below 2^17
        "madc.hi.cc.u32 %1, %4, 0xFFFFFFFF, %3;\n\t"
        "addc.u32 m, 0, 0;\n\t"                      // a carry out leaves less than 2^49: its own 2^32 - 1 does not carry again
        "neg.s32 m, m;\n\t"
        "add.cc.u32 %0, %0, m;\n\t"
        "addc.u32 %1, %1, 0;\n\t"
        "}"
        : "=&r"(r0), "=&r"(r1)
        : "r"((u32)w), "r"((u32)g), "r"((u32)(g >> 32)));
    return ((u64)r1 << 32) | r0;
#else
    const u64 w = (u64)e0 + ((u64)e1 << 16) + ((u64)e2 << 32), g = (w >> 32) + ((u64)e3 << 16);
    const u64 v = (g << 32) | (u32)w, add = (g >> 32) * GL_EPS;
    u64 r = v + add;
    if (r < v) r += GL_EPS;
    return r;
#endif
}

template <int LOGN>
struct Tc {
    static_assert(LOGN >= 10 && LOGN <= 14, "tensor-core path sizes");
    static constexpr int G = LOGN - 10;
    static constexpr u32 N = 1u << LOGN, ROWS = TC_WORDS / N, CMASK = (1u << G) - 1u;
    static constexpr u32 VEC = G >= 2 ? 4u : 1u << G;  // words of a row that lie together among four neighbouring c'

    // VEC words of a row's message from index m on; packed ones are widened and written back.  `wide`: the rows start on 32-byte boundaries
    GL_HD static void fill_message(const RowArgs& a, u32 row, u32 m, bool wide, u64* y) {
        const u64* src = a.data + (size_t)row * N + m;
#ifdef __CUDA_ARCH__
        if (wide) {
            if constexpr (VEC == 4) asm volatile("ld.global.v4.b64 {%0, %1, %2, %3}, [%4];" : "=l"(y[0]), "=l"(y[1]), "=l"(y[2]), "=l"(y[3]) : "l"(src) : "memory");
            else if constexpr (VEC == 2) asm volatile("ld.global.v2.b64 {%0, %1}, [%2];" : "=l"(y[0]), "=l"(y[1]) : "l"(src) : "memory");
            else y[0] = *src;
            return;
        }
#endif
        for (u32 e = 0; e < VEC; e++) y[e] = src[e];
    }
    // Packed rows in two steps, so that the loads of several places are in flight together: `raw` is what one load brings for widths 1 and
    // 2 (a row starts on a multiple of n bytes); the wider words are read in the second step, which also leaves the widened words in `data`.
    GL_HD static u64 narrow_raw(const RowArgs& a, u32 row, u32 m, u32 w) {
        const unsigned char* p = a.narrow + a.row_off[row] + (size_t)m * w;
        const u32 bytes = VEC * w;
        if (w > 2) return 0;
        if (bytes == 8) return *reinterpret_cast<const u64*>(p);
        if (bytes == 4) return *reinterpret_cast<const u32*>(p);
        if (bytes == 2) return *reinterpret_cast<const unsigned short*>(p);
        return *p;
    }
    GL_HD static void fill_narrow(const RowArgs& a, u32 row, u32 m, u32 w, u64 raw, u64* y) {
        u64* dst = const_cast<u64*>(a.data) + (size_t)row * N + m;
        for (u32 e = 0; e < VEC; e++) {
            if (w <= 2) {
                const long long x = w == 2 ? (long long)(short)(raw >> (16 * e)) : (long long)(signed char)(raw >> (8 * e));
                y[e] = (u64)x + (x < 0 ? GL_P : 0);
            } else {
                y[e] = widen_word(a.narrow + a.row_off[row], m + e, w);
            }
        }
#ifdef __CUDA_ARCH__
        if constexpr (VEC == 4) {
            asm volatile("st.global.v4.b64 [%0], {%1, %2, %3, %4};\n" ::"l"(dst), "l"(y[0]), "l"(y[1]), "l"(y[2]), "l"(y[3]) : "memory");
        } else
#endif
        {
            for (u32 e = 0; e < VEC; e++) dst[e] = y[e];
        }
    }

    // Residue s transforms y_s[i] = w_nn^(i s) (x[i] + sum_t w_R^(t s) x[i + t n]), x[i] = (c[i] - pad[i]) h^i the coefficients on the coset and
    // x[n + i] = (pad[i] - pad[n + i]) h^(n + i) the pads' copies above the message.  What the pads bring, at i < q, is worked out ahead
    // (canonical): `pad_below` is added to c[i] h^i, `pad_above` to that before it is twisted.
    GL_HD static u64 pad_below(const RowArgs& a, u32 row, u32 i) { return gl_neg(gl_mul_fast(a.pads[(size_t)row * a.q + i], a.pows[i])); }
    GL_HD static u64 pad_above(const RowArgs& a, u32 row, u32 i, u32 s) {
        const u64* pad = a.pads + (size_t)row * a.q;
        const u32 nn = N << a.logr;
        u64 sum = 0;
#pragma unroll 1
        for (u32 k = i; k < a.q; k += N) {
            u64 u = pad[k];
            if (k + N < a.q) u = gl_sub(u, pad[k + N]);
            u = gl_mul_fast(u, a.pows[k + N]);
            if (s) u = gl_mul_fast(u, a.tw_nn[((k + N - i) * s) & (nn - 1)]);
            sum = gl_add(sum, u);
        }
        return sum;
    }
};

// The tables of rows of 2^logn words at rate 2^-logr; `out` holds tc_table_words words: those above, and then the residues' twists
// w_nn^j, j < nn.  I2's twiddles carry 1 / n.
constexpr u32 TC_TWIST = TC_TABLE_WORDS;
inline size_t tc_table_words(u32 logn, u32 logr) { return TC_TABLE_WORDS + ((size_t)1 << (logn + logr)); }
inline void tc_build(u32 logn, u32 logr, u64* out) {
    const u32 g = logn - 10, cm = (1u << g) - 1u, N = 1u << logn;
    const u64 root = gl_pow(gl_pow(7, (GL_P - 1) >> 32), 1ull << (32 - logn)), ninv = gl_inv(N);
    u64* w = new u64[N];
    u64 x = 1;
    for (u32 i = 0; i < N; i++) { w[i] = x; x = gl_mul(x, root); }
    const u64 root_nn = gl_pow(gl_pow(7, (GL_P - 1) >> 32), 1ull << (32 - logn - logr));
    x = 1;
    for (size_t j = 0; j < (size_t)1 << (logn + logr); j++) { out[TC_TWIST + j] = x; x = gl_mul(x, root_nn); }
    for (u32 k = 0; k < 32; k++) {
        for (u32 c = 0; c < 16; c++) {
            for (u32 b = 0; b < 32; b++) out[TC_I1 + (k * 16 + c) * 32 + b] = w[(k * ((b << g) + (c & cm))) & (N - 1)];
            out[TC_SMALL + k * 16 + c] = gl_mul(w[(32 * k * (c & cm)) & (N - 1)], ninv);
        }
        for (u32 b = 0; b < 32; b++) out[TC_SMALL + TC_F2 + k * 32 + b] = w[(k * b * (N / 1024)) & (N - 1)];
    }
    for (u32 c = 0; c < 16; c++)
        for (u32 tile = 0; tile < 8; tile++)
            for (u32 row = 0; row < 128; row++) out[TC_F1 + (c * 8 + tile) * 128 + row] = w[((c & cm) * tc_k_of(tile, row)) & (N - 1)];
    unsigned char* bm = reinterpret_cast<unsigned char*>(out + TC_B);
    for (u32 i = 0; i < 32; i++)
        for (u32 j = 0; j < 32; j++)
            for (u32 b = 0; b < 8; b++) {
                const u64 v = gl_mul(w[(i * j * (N / 32)) & (N - 1)], 1ull << (8 * b));
                for (u32 d = 0; d < 8; d++) bm[(j >> 4) * 32768 + tc_swizzled(8 * i + d, (j & 15) * 8 + b)] = (unsigned char)(v >> (8 * d));
            }
    unsigned char* b3 = reinterpret_cast<unsigned char*>(out + TC_B3);
    for (u32 i = 0; i < 16; i++)
        for (u32 j = 0; j < 16; j++)
            for (u32 b = 0; b < 8; b++) {
                const u64 v = (i >> g) != (j >> g) ? 0 : gl_mul(w[((i & cm) * (j & cm) * (N >> g)) & (N - 1)], 1ull << (8 * b));
                for (u32 d = 0; d < 8; d++) b3[tc_swizzled(8 * i + d, j * 8 + b)] = (unsigned char)(v >> (8 * d));
            }
    delete[] w;
}

}  // namespace enc
