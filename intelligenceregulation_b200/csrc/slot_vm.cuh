// A slot polynomial as a straight-line program for a machine of one value and two kinds of slots: what the sumcheck kernels run.
//
// The graph of slot_ir.cuh names up to 128 nodes; an evaluator that keeps them all per thread keeps kilobytes, which spill into local
// memory and from there past L2 (the block's width check: 3.5 ns per pair, five times its arithmetic).  Along an order in which a value
// is used as soon as it exists, few live at a time.  The program is that order:
//
//   X        the running product, at every evaluation point of the thread, in registers
//   R        a linear combination of tables (lo, difference along the round's variable) in registers: every table is affine in the
//            evaluation point, so a linear node costs two values whatever the number of points
//   P[q]     slots of the size of X, in shared memory: partial sums, and nodes that are used more than once
//   A[a]     slots of the size of R, in shared memory: linear nodes that are used more than once
//
// An instruction is one 64-bit word (op, source, class and index of a coefficient, slot or table), the same for all threads of a CTA.
// Exact arithmetic on canonical words: any order of the sums and products gives the graph's value.
#pragma once
#include <algorithm>
#include <functional>
#include <utility>
#include <vector>

#include "slot_ir.cuh"

namespace vm {

enum Op : u32 { INIT, MUL, R_SET, R_ADD, R_CONST, A_SET, P_SET, P_ACC, X_ADDP, X_MULC, X_CONST, END };
enum Src : u32 { TABLE, ASLOT, PSLOT, REG };
enum Class : u32 { ONE, NEG, BASE, EXT };  // of the coefficient: 1, -1, a base-field word, an extension word

constexpr int MAX_NPT = 5;  // evaluation points per thread in the long rounds (more points: more threads per pair)

GL_HD u64 ins(u32 op, u32 src, u32 cls, u32 idx, u32 coef) { return (u64)op | ((u64)src << 4) | ((u64)cls << 6) | ((u64)idx << 16) | ((u64)coef << 32); }
GL_HD u32 op_of(u64 w) { return (u32)w & 15u; }
GL_HD u32 src_of(u64 w) { return ((u32)w >> 4) & 3u; }
GL_HD u32 cls_of(u64 w) { return ((u32)w >> 6) & 3u; }
GL_HD u32 idx_of(u64 w) { return (u32)w >> 16; }
GL_HD u32 coef_of(u64 w) { return (u32)(w >> 32); }

// `parts` programs whose values sum to the polynomial's: part w starts at code[start[w]].  One part is the whole; where a round has fewer
// pairs than the device has threads, several threads take a pair's parts.
constexpr u32 MAX_PARTS = 8;
struct Program {
    std::vector<u64> code;
    std::vector<fp2> coefs;   // the general ones, in the order of their first use
    u32 parts = 1;
    u32 start[MAX_PARTS + 1] = {0};  // [parts]: the end
    u32 p_slots = 0, a_slots = 0;
    u32 degree = 0;           // attained along one variable
};

class Compiler {
  public:
    Program out;
    // the whole, at code[0]
    void run(const ir::Shape& s, const u32* w, const fp2* cf) {
        parse(s, w, cf);
        out.degree = ir::attained_degree(s, w);
        const std::vector<Node> graph = nodes_;
        part(graph.back().units);
        out.start[1] = (u32)out.code.size();
    }
    // behind it, the same in `parts` parts of about equal cost (fewer where there is less to share out)
    void split(const ir::Shape& s, const u32* w, const fp2* cf, u32 parts) {
        parse(s, w, cf);
        const std::vector<Node> graph = nodes_;
        // a unit whose one non-linear factor is a sum that only it uses: the sum's units, each under the unit's other factors
        struct Item { size_t prefix; Unit u; u32 cost; };
        std::vector<Unit> prefixes;
        std::vector<Item> items;
        count_uses();
        count_costs();
        std::function<void(const Unit&, const std::vector<Unit>&)> flatten = [&](const Unit& pre, const std::vector<Unit>& units) {
            prefixes.push_back(pre);
            const size_t here = prefixes.size() - 1;
            for (auto& u : units) {
                Unit deeper{f2_mul(pre.c, u.c), pre.f};
                u32 non = 0, inner = 0;
                for (u32 f : u.f) {
                    if (is_linear(f)) deeper.f.push_back(f);
                    else { non++; inner = f & ~ir::IR_NODE; }
                }
                if (non == 1 && nodes_[inner].uses == 1 && nodes_[inner].units.size() > 1 && deeper.f.size() <= 2) flatten(deeper, nodes_[inner].units);
                else items.push_back({here, u, unit_cost(u)});
            }
        };
        flatten(Unit{f2(1, 0), {}}, nodes_.back().units);
        std::sort(items.begin(), items.end(), [](const Item& x, const Item& y) { return x.cost > y.cost; });
        if (parts > items.size()) parts = (u32)items.size();
        if (parts < 2) return;
        std::vector<std::vector<const Item*>> bins(parts);
        std::vector<u32> load(parts, 0);
        for (auto& it : items) {  // the largest first, each to the lightest part
            const size_t w0 = std::min_element(load.begin(), load.end()) - load.begin();
            bins[w0].push_back(&it);
            load[w0] += it.cost + 1;
        }
        out.parts = parts;
        for (u32 k = 0; k < parts; k++) {
            nodes_ = graph;
            std::vector<Unit> top;
            for (size_t p = 0; p < prefixes.size(); p++) {
                Node sum;
                for (auto* it : bins[k])
                    if (it->prefix == p) sum.units.push_back(it->u);
                if (sum.units.empty()) continue;
                const Unit& pre = prefixes[p];
                if (pre.f.empty() && pre.c.c0 == 1 && pre.c.c1 == 0) { top.insert(top.end(), sum.units.begin(), sum.units.end()); continue; }
                Unit u = pre;
                u.f.push_back(ir::IR_NODE | (u32)nodes_.size());
                nodes_.push_back(sum);
                top.push_back(u);
            }
            out.start[k] = (u32)out.code.size();
            part(top);
        }
        out.start[parts] = (u32)out.code.size();
    }

  private:
    struct Unit { fp2 c; std::vector<u32> f; };
    struct Node { std::vector<Unit> units; bool linear = true; u32 uses = 0, cost = 0; int slot = -1; };
    static constexpr u32 COST_CAP = 4096;
    std::vector<Node> nodes_;
    std::vector<u32> p_free_, a_free_;

    void parse(const ir::Shape& s, const u32* w, const fp2* cf) {
        nodes_.assign(s.n_nodes + 1, Node());
        u32 pc = 0;
        auto product = [&](Node& nd) {
            Unit u;
            u.c = ir::coef_value(w[pc], cf);
            const u32 nf = w[pc + 1];
            u.f.assign(w + pc + 2, w + pc + 2 + nf);
            pc += 2 + nf;
            if (!f2_is_zero(u.c)) nd.units.push_back(u);
        };
        for (u32 n = 0; n < s.n_nodes; n++) {
            const u32 head = w[pc++], cnt = head >> 8;
            if ((head & 0xFFu) == ir::IR_AFFINE) {
                const fp2 k = ir::coef_value(w[pc++], cf);
                if (!f2_is_zero(k)) nodes_[n].units.push_back({k, {}});
                for (u32 i = 0; i < cnt; i++, pc += 2) {
                    const fp2 c = ir::coef_value(w[pc], cf);
                    if (!f2_is_zero(c)) nodes_[n].units.push_back({c, {w[pc + 1]}});
                }
            } else {
                for (u32 i = 0; i < cnt; i++) product(nodes_[n]);
            }
        }
        for (u32 t = 0; t < s.n_terms; t++) product(nodes_[s.n_nodes]);
        mark_linear();
    }
    void mark_linear() {  // nodes refer to earlier ones only
        for (auto& nd : nodes_)
            for (auto& u : nd.units)
                if (u.f.size() > 1 || (u.f.size() == 1 && !is_linear(u.f[0]))) nd.linear = false;
    }
    void count_uses() {  // what the last node needs, and how often
        std::vector<bool> live(nodes_.size(), false);
        live.back() = true;
        for (auto& nd : nodes_) nd.uses = 0;
        for (size_t n = nodes_.size(); n-- > 0;) {
            if (!live[n]) continue;
            for (auto& u : nodes_[n].units)
                for (u32 f : u.f)
                    if (f & ir::IR_NODE) { live[f & ~ir::IR_NODE] = true; nodes_[f & ~ir::IR_NODE].uses++; }
        }
    }
    // instructions, about; a shared node counts with everyone who uses it, since it may end up in several parts.  Nodes refer to earlier
    // ones only: each is counted once, in their order (a chain of nodes that use the one before twice would be 2^nodes visits), up to a cap.
    u32 unit_cost(const Unit& u) const {
        u32 c = 2;
        for (u32 f : u.f) c += f & ir::IR_NODE ? nodes_[f & ~ir::IR_NODE].cost : 1;
        return c;
    }
    void count_costs() {
        for (auto& nd : nodes_) {
            nd.cost = 1;
            for (auto& u : nd.units) nd.cost = std::min(nd.cost + unit_cost(u), COST_CAP);
        }
    }
    void part(const std::vector<Unit>& top) {
        Node root;
        root.units = top;
        nodes_.push_back(root);
        mark_linear();
        count_uses();
        p_free_.clear();
        a_free_.clear();
        // slot numbers start over in every part; the counts are the largest
        const u32 p_most = out.p_slots, a_most = out.a_slots;
        out.p_slots = out.a_slots = 0;
        const std::vector<Unit> units = nodes_.back().units;
        sum(units);
        out.code.push_back(ins(END, 0, 0, 0, 0));
        out.p_slots = std::max(out.p_slots, p_most);
        out.a_slots = std::max(out.a_slots, a_most);
    }
    static u32 take(std::vector<u32>& free_list, u32& high) {
        if (!free_list.empty()) { const u32 q = free_list.back(); free_list.pop_back(); return q; }
        return high++;
    }
    u32 cls(fp2 c, u32* index) {
        *index = 0;
        if (c.c1 == 0 && c.c0 == 1) return ONE;
        if (c.c1 == 0 && c.c0 == GL_P - 1) return NEG;
        for (size_t i = 0; i < out.coefs.size(); i++)
            if (out.coefs[i].c0 == c.c0 && out.coefs[i].c1 == c.c1) { *index = (u32)i; return c.c1 ? EXT : BASE; }
        *index = (u32)out.coefs.size();
        out.coefs.push_back(c);
        return c.c1 ? EXT : BASE;
    }
    void emit(u32 op, u32 src, u32 idx, fp2 c) {
        u32 ci;
        const u32 k = cls(c, &ci);
        out.code.push_back(ins(op, src, k, idx, ci));
    }
    void emit(u32 op, u32 src, u32 idx) { emit(op, src, idx, f2(1, 0)); }

    // ---- linear parts: R = sum of c * (table or linear node), and constants ----
    struct Lin { fp2 konst = f2(0, 0); std::vector<std::pair<fp2, u32>> terms; };  // factor words: tables, or multi-use linear nodes
    void gather(const std::vector<Unit>& units, fp2 scale, Lin& l) {
        for (auto& u : units) gather(u, scale, l);
    }
    void gather(const Unit& u, fp2 scale, Lin& l) {
        const fp2 c = f2_mul(scale, u.c);
        if (u.f.empty()) {
            l.konst = f2_add(l.konst, c);
        } else {
            const u32 f = u.f[0];
            if (!(f & ir::IR_NODE) || nodes_[f & ~ir::IR_NODE].uses > 1 || nodes_[f & ~ir::IR_NODE].slot >= 0) l.terms.push_back({c, f});
            else gather(nodes_[f & ~ir::IR_NODE].units, c, l);  // used here only: its terms directly
        }
    }
    void prepare(const Lin& l) {  // the multi-use nodes it reads, while R is free
        for (auto& t : l.terms)
            if (t.second & ir::IR_NODE) linear_slot(t.second & ~ir::IR_NODE);
    }
    void linear_slot(u32 n) {
        Node& nd = nodes_[n];
        if (nd.slot >= 0) return;
        Lin l;
        gather(nd.units, f2(1, 0), l);
        to_r(l);
        nd.slot = (int)take(a_free_, out.a_slots);
        emit(A_SET, REG, (u32)nd.slot);
    }
    void used(u32 n) {
        Node& nd = nodes_[n];
        if (--nd.uses == 0 && nd.slot >= 0) (nd.linear ? a_free_ : p_free_).push_back((u32)nd.slot);
    }
    // the operand of a factor word, which must be a table or a multi-use linear node in its slot
    void operand(u32 f, u32* src, u32* idx) {
        if (f & ir::IR_NODE) { *src = ASLOT; *idx = (u32)nodes_[f & ~ir::IR_NODE].slot; }
        else { *src = TABLE; *idx = f; }
    }
    void to_r(const Lin& l) {
        prepare(l);
        bool have = false;
        if (!f2_is_zero(l.konst) || l.terms.empty()) { emit(R_CONST, REG, 0, l.konst); have = true; }
        for (auto& t : l.terms) {
            u32 src, idx;
            operand(t.second, &src, &idx);
            emit(have ? R_ADD : R_SET, src, idx, t.first);
            have = true;
            if (t.second & ir::IR_NODE) used(t.second & ~ir::IR_NODE);
        }
    }
    bool is_linear(u32 f) const { return !(f & ir::IR_NODE) || nodes_[f & ~ir::IR_NODE].linear; }

    // X = c * f or X *= c * f for a linear factor
    void linear_factor(u32 op, u32 f, fp2 c) {
        if (!(f & ir::IR_NODE)) { emit(op, TABLE, f, c); return; }
        const u32 n = f & ~ir::IR_NODE;
        if (nodes_[n].uses > 1 || nodes_[n].slot >= 0) {
            linear_slot(n);
            emit(op, ASLOT, (u32)nodes_[n].slot, c);
        } else {
            Lin l;
            gather(nodes_[n].units, c, l);  // the coefficient goes into the combination
            to_r(l);
            emit(op, REG, 0);
        }
        used(n);
    }
    // X = the value of a non-linear node
    void node(u32 n) {
        Node& nd = nodes_[n];
        if (nd.slot >= 0) {
            emit(INIT, PSLOT, (u32)nd.slot);
        } else {
            sum(nd.units);
            if (nd.uses > 1) {
                nd.slot = (int)take(p_free_, out.p_slots);
                emit(P_SET, PSLOT, (u32)nd.slot);
            }
        }
        used(n);
    }
    void unit(const Unit& u) {
        std::vector<u32> lin, non;
        for (u32 f : u.f) (is_linear(f) ? lin : non).push_back(f);
        fp2 c = u.c;
        bool have = false;
        for (u32 f : non) {
            const u32 n = f & ~ir::IR_NODE;
            if (!have) { node(n); have = true; continue; }
            if (nodes_[n].slot >= 0) {
                emit(MUL, PSLOT, (u32)nodes_[n].slot);
                used(n);
            } else {
                const u32 q = take(p_free_, out.p_slots);
                emit(P_SET, PSLOT, q);
                node(n);
                emit(MUL, PSLOT, q);
                p_free_.push_back(q);
            }
        }
        for (u32 f : lin) {
            linear_factor(have ? MUL : INIT, f, c);  // the coefficient rides on the first linear factor
            c = f2(1, 0);
            have = true;
        }
        if (!have) emit(X_CONST, REG, 0, c);
        else if (!(c.c0 == 1 && c.c1 == 0)) emit(X_MULC, REG, 0, c);
    }
    // X = the sum of the units: the linear ones together, the others after them, partial sums in a P slot
    void sum(const std::vector<Unit>& units) {
        std::vector<const Unit*> linear, rest;
        for (auto& u : units) (u.f.empty() || (u.f.size() == 1 && is_linear(u.f[0])) ? linear : rest).push_back(&u);
        bool have = false;
        if (!linear.empty() || rest.empty()) {
            Lin l;
            for (const Unit* u : linear) gather(*u, f2(1, 0), l);
            to_r(l);
            emit(INIT, REG, 0);
            have = true;
        }
        u32 q = 0;
        bool slot = false;
        for (size_t i = 0; i < rest.size(); i++) {
            if (have) {
                if (!slot) { q = take(p_free_, out.p_slots); emit(P_SET, PSLOT, q); slot = true; }
                else emit(P_ACC, PSLOT, q);
            }
            unit(*rest[i]);
            have = true;
        }
        if (slot) {
            emit(X_ADDP, PSLOT, q);
            p_free_.push_back(q);
        }
    }
};

// Fp2 entries of one thread's slots; with one point per thread R and A are values at that point
GL_HD u32 slot_entries(u32 p_slots, u32 a_slots, int npt) { return p_slots * (u32)npt + a_slots * (npt == 1 ? 1u : 2u); }

// a coefficient times any word; the result is lazy
GL_HD fp2 apply(u32 cls, const fp2* cf, u32 ci, fp2 x) {
    if (cls == ONE) return x;
    if (cls == NEG) return f2_neg(f2_canon(x));
    if (cls == BASE) return f2_mul_base_lazy(x, cf[ci].c0);
    return x.c1 == 0 ? f2_mul_base_lazy(cf[ci], x.c0) : f2_mul_lazy(cf[ci], x);
}
GL_HD fp2 constant(u32 cls, const fp2* cf, u32 ci) { return cls == ONE ? f2(1, 0) : cls == NEG ? f2(GL_P - 1, 0) : cf[ci]; }

// The program at NPT >= 2 evaluation points p_first, p_first + 1, .. (after the point 0 comes the point 2 when `skip` is set: the point 1 is
// known from the claim).  table(t, lo, hi): the two ends of a table's pair; slots: this thread's entries, entry e at slots[e * stride].
// The ends of the next instruction's table are fetched before this one's arithmetic.  X is lazy throughout (so is the result), R and the
// slots are canonical: a sum then has one canonical operand, and a product takes anything.
template <int NPT, class Table>
GL_HD void eval(const u64* code, const fp2* cf, Table table, fp2* slots, u32 stride, u32 a_base, u32 p_first, bool skip, fp2 (&X)[NPT]) {
    fp2 rv = f2(0, 0), rd = f2(0, 0), lo = f2(0, 0), hi = f2(0, 0);
    u64 w = code[0];
    if (src_of(w) == TABLE && op_of(w) <= R_ADD) table(idx_of(w), lo, hi);
    for (u32 pc = 0;; pc++) {
        const u32 op = op_of(w), src = src_of(w), cls = cls_of(w), idx = idx_of(w), ci = coef_of(w);
        if (op == END) return;
        const u64 nw = code[pc + 1];
        fp2 nlo = f2(0, 0), nhi = f2(0, 0);
        if (src_of(nw) == TABLE && op_of(nw) <= R_ADD) table(idx_of(nw), nlo, nhi);
        if (op <= R_ADD) {
            fp2 v, d = f2(0, 0);
            if (src == TABLE) {
                v = lo;
                d = f2_sub(hi, lo);
            } else if (src == ASLOT) {
                v = slots[(a_base + 2 * idx) * stride];
                d = slots[(a_base + 2 * idx + 1) * stride];
            } else {
                v = rv;
                d = rd;
            }
            if (src != PSLOT && cls != ONE) {
                v = apply(cls, cf, ci, v);
                d = f2_canon(apply(cls, cf, ci, d));
            }
            if (op >= R_SET) {
                if (op == R_SET) { rv = f2_canon(v); rd = d; }
                else { rv = f2_canon(f2_add_lazy(v, rv)); rd = f2_add(rd, d); }
            } else {
                fp2 y[NPT];
                bool base = false;
                if (src == PSLOT) {
#pragma unroll
                    for (int j = 0; j < NPT; j++) y[j] = slots[(idx * NPT + j) * stride];
                } else {
                    base = (v.c1 | d.c1) == 0;
                    for (u32 p = 0; p < p_first; p++) v = f2_add_lazy(v, d);
                    y[0] = v;
#pragma unroll
                    for (int j = 1; j < NPT; j++) {
                        v = f2_add_lazy(v, d);
                        if (j == 1 && skip && p_first == 0) v = f2_add_lazy(v, d);
                        y[j] = v;
                    }
                }
                if (op == INIT) {
#pragma unroll
                    for (int j = 0; j < NPT; j++) X[j] = y[j];
                } else if (base) {
#pragma unroll
                    for (int j = 0; j < NPT; j++) X[j] = f2_mul_base_lazy(X[j], y[j].c0);
                } else {
#pragma unroll
                    for (int j = 0; j < NPT; j++) X[j] = f2_mul_lazy(X[j], y[j]);
                }
            }
        } else {
            switch (op) {
                case R_CONST: rv = constant(cls, cf, ci); rd = f2(0, 0); break;
                case A_SET:
                    slots[(a_base + 2 * idx) * stride] = rv;
                    slots[(a_base + 2 * idx + 1) * stride] = rd;
                    break;
                case P_SET:
#pragma unroll
                    for (int j = 0; j < NPT; j++) slots[(idx * NPT + j) * stride] = f2_canon(X[j]);
                    break;
                case P_ACC:
#pragma unroll
                    for (int j = 0; j < NPT; j++) slots[(idx * NPT + j) * stride] = f2_canon(f2_add_lazy(X[j], slots[(idx * NPT + j) * stride]));
                    break;
                case X_ADDP:
#pragma unroll
                    for (int j = 0; j < NPT; j++) X[j] = f2_add_lazy(X[j], slots[(idx * NPT + j) * stride]);
                    break;
                case X_MULC:
#pragma unroll
                    for (int j = 0; j < NPT; j++) X[j] = apply(cls, cf, ci, X[j]);
                    break;
                default: {
                    const fp2 c = constant(cls, cf, ci);
#pragma unroll
                    for (int j = 0; j < NPT; j++) X[j] = c;
                }
            }
        }
        w = nw;
        lo = nlo;
        hi = nhi;
    }
}

// The program at ONE point, where a round waits for its chain and not for its instructions: table(t) is the table's value at the point.
template <class Table>
GL_HD fp2 eval_one(const u64* code, const fp2* cf, Table table, fp2* slots, u32 stride, u32 a_base) {
    fp2 X = f2(0, 0), R = f2(0, 0), next = f2(0, 0);
    u64 w = code[0];
    if (src_of(w) == TABLE && op_of(w) <= R_ADD) next = table(idx_of(w));
    for (u32 pc = 0;; pc++) {
        const u32 op = op_of(w), src = src_of(w), cls = cls_of(w), idx = idx_of(w), ci = coef_of(w);
        if (op == END) return X;
        const u64 nw = code[pc + 1];
        fp2 y = next;
        if (src_of(nw) == TABLE && op_of(nw) <= R_ADD) next = table(idx_of(nw));
        if (op <= R_ADD) {
            if (src == ASLOT) y = slots[(a_base + idx) * stride];
            else if (src == PSLOT) y = slots[idx * stride];
            else if (src == REG) y = R;
            if (src != PSLOT) y = apply(cls, cf, ci, y);
            if (op == MUL) X = y.c1 == 0 ? f2_mul_base_lazy(X, y.c0) : f2_mul_lazy(X, y);
            else if (op == R_ADD) R = f2_canon(f2_add_lazy(y, R));
            else if (op == INIT) X = y;
            else R = f2_canon(y);
        } else {
            switch (op) {
                case R_CONST: R = constant(cls, cf, ci); break;
                case A_SET: slots[(a_base + idx) * stride] = R; break;
                case P_SET: slots[idx * stride] = f2_canon(X); break;
                case P_ACC: slots[idx * stride] = f2_canon(f2_add_lazy(X, slots[idx * stride])); break;
                case X_ADDP: X = f2_add_lazy(X, slots[idx * stride]); break;
                case X_MULC: X = apply(cls, cf, ci, X); break;
                default: X = constant(cls, cf, ci);
            }
        }
        w = nw;
    }
}

}  // namespace vm
