// A slot polynomial given as data: the expression graph of private_block/slot_ir.rs:57-345 flattened
// into 32-bit words, and what the host checks of such a stream.  The kernels run it as a program (slot_vm.cuh).
//
//   polynomial = sum over terms of    coef * prod(factors)
//   factor     = a table's value at the point, or a node's value
//   node       = affine:  konst + sum_i coef_i * table_i
//                sum:     sum over subterms of coef * prod(factors)      (nodes only refer back)
//
// Word stream: the node records in order, then the term records.
//   affine node   [IR_AFFINE | count << 8] [konst coef] count x ([coef] [table])
//   sum node      [IR_SUM    | count << 8] count x ( [coef] [nf] nf x [factor] )
//   term          [coef] [nf] nf x [factor]          (wrapper tables first, then the inner factors)
//   factor        table id, or IR_NODE | node id
//   coef          index into the Fp2 coefficient array, or IR_ONE / IR_NEG_ONE / IR_ZERO
//
// Field arithmetic is exact and results are canonical words, so the order of the additions and
// multiplications is free: any evaluator of the same graph returns the reference's words.
#pragma once
#include <cstddef>
#include <vector>

#include "gl_field.cuh"

namespace ir {

constexpr u32 IR_AFFINE = 0, IR_SUM = 1;
constexpr u32 IR_NODE = 0x80000000u;
constexpr u32 IR_ONE = 0xFFFFFFFFu, IR_NEG_ONE = 0xFFFFFFFEu, IR_ZERO = 0xFFFFFFFDu;
constexpr u32 MAX_DEGREE = 1u << 20;  // degrees are counted up to here (64 factors of it do not wrap)
constexpr u32 MAX_TABLES = 64, MAX_NODES = 128, MAX_WORDS = 4096, MAX_COEFS = 512;

struct Shape {
    u32 n_tables, n_nodes, n_terms, n_coefs, n_words;
};

GL_HD fp2 coef_value(u32 ci, const fp2* cf) {
    if (ci == IR_ONE) return f2(1, 0);
    if (ci == IR_NEG_ONE) return f2(GL_P - 1, 0);
    if (ci == IR_ZERO) return f2(0, 0);
    return cf[ci];
}

// Host-side check of a word stream before it reaches a kernel: every id in range, nodes refer back only,
// the stream ends exactly at n_words (the invariant of slot_ir.rs:445-489).  Returns 0 when well formed.
inline int validate(const Shape& s, const u32* w) {
    if (s.n_tables == 0 || s.n_tables > MAX_TABLES || s.n_nodes > MAX_NODES || s.n_words > MAX_WORDS || s.n_coefs > MAX_COEFS) return 1;
    u32 pc = 0;
    auto coef_ok = [&](u32 ci) { return ci == IR_ONE || ci == IR_NEG_ONE || ci == IR_ZERO || ci < s.n_coefs; };
    auto prod_ok = [&](u32 upto) {
        if (pc + 2 > s.n_words) return false;
        const u32 ci = w[pc++], nf = w[pc++];
        if (!coef_ok(ci) || nf > 64 || pc + nf > s.n_words) return false;
        for (u32 i = 0; i < nf; i++) {
            const u32 f = w[pc++];
            if (f & IR_NODE) { if ((f & ~IR_NODE) >= upto) return false; }
            else if (f >= s.n_tables) return false;
        }
        return true;
    };
    for (u32 n = 0; n < s.n_nodes; n++) {
        if (pc >= s.n_words) return 2;
        const u32 head = w[pc++], cnt = head >> 8, kind = head & 0xFFu;
        if (kind == IR_AFFINE) {
            if (pc + 1 + 2 * (size_t)cnt > s.n_words || !coef_ok(w[pc])) return 3;
            pc++;
            for (u32 i = 0; i < cnt; i++) {
                if (!coef_ok(w[pc]) || w[pc + 1] >= s.n_tables) return 4;
                pc += 2;
            }
        } else if (kind == IR_SUM) {
            for (u32 i = 0; i < cnt; i++)
                if (!prod_ok(n)) return 5;
        } else {
            return 6;
        }
    }
    for (u32 t = 0; t < s.n_terms; t++)
        if (!prod_ok(s.n_nodes)) return 7;
    return pc == s.n_words ? 0 : 8;
}

// The SIGNATURE of a well-formed stream: FNV-1a over (n_tables, n_nodes, n_terms) and the stream's words with every
// coefficient word replaced by the coefficient's class (the special words as they are; a general coefficient by whether
// its value lies in the base field), so that a graph is recognised whatever its challenges are.  The generated kernels
// (slot_gen.cuh) are keyed by it and read their coefficients by OCCURRENCE: `by_occurrence` receives the value of the
// j-th coefficient word of the stream.
constexpr u32 IR_CLASS_BASE = 0xFFFFFFF0u, IR_CLASS_EXT = 0xFFFFFFF1u;
inline u64 signature(const Shape& s, const u32* w, const fp2* cf, std::vector<fp2>* by_occurrence) {
    u64 h = 0xCBF29CE484222325ull;
    auto mix = [&](u32 word) {
        for (int b = 0; b < 4; b++) h = (h ^ ((word >> (8 * b)) & 0xFFu)) * 0x100000001B3ull;
    };
    auto coef = [&](u32 ci) {
        const fp2 v = coef_value(ci, cf);
        if (by_occurrence) by_occurrence->push_back(v);
        mix((ci == IR_ONE || ci == IR_NEG_ONE || ci == IR_ZERO) ? ci : (v.c1 == 0 ? IR_CLASS_BASE : IR_CLASS_EXT));
    };
    mix(s.n_tables); mix(s.n_nodes); mix(s.n_terms);
    u32 pc = 0;
    auto product = [&]() {
        coef(w[pc++]);
        const u32 nf = w[pc++];
        mix(nf);
        for (u32 i = 0; i < nf; i++) mix(w[pc++]);
    };
    for (u32 n = 0; n < s.n_nodes; n++) {
        const u32 head = w[pc++], cnt = head >> 8;
        mix(head);
        if ((head & 0xFFu) == IR_AFFINE) {
            coef(w[pc++]);
            for (u32 i = 0; i < cnt; i++) { coef(w[pc++]); mix(w[pc++]); }
        } else {
            for (u32 i = 0; i < cnt; i++) product();
        }
    }
    for (u32 t = 0; t < s.n_terms; t++) product();
    return h;
}

// the degree a well-formed stream attains along one variable
inline u32 attained_degree(const Shape& s, const u32* w) {
    std::vector<u32> deg(s.n_nodes, 0);
    u32 pc = 0, top = 0;
    auto prod_deg = [&]() {
        const u32 nf = w[pc + 1];
        u32 d = 0;
        for (u32 i = 0; i < nf; i++) d += (w[pc + 2 + i] & IR_NODE) ? deg[w[pc + 2 + i] & ~IR_NODE] : 1u;
        if (d > MAX_DEGREE) d = MAX_DEGREE;  // a chain of products of the node before with itself doubles it per node
        pc += 2 + nf;
        return d;
    };
    for (u32 n = 0; n < s.n_nodes; n++) {
        const u32 head = w[pc++], cnt = head >> 8;
        u32 d = 0;
        if ((head & 0xFFu) == IR_AFFINE) {
            d = cnt ? 1u : 0u;
            pc += 1 + 2 * cnt;
        } else {
            for (u32 i = 0; i < cnt; i++) { const u32 x = prod_deg(); d = x > d ? x : d; }
        }
        deg[n] = d;
    }
    for (u32 t = 0; t < s.n_terms; t++) { const u32 x = prod_deg(); top = x > top ? x : top; }
    return top;
}

}  // namespace ir
