// Compiles a slot polynomial to the sumcheck kernels' straight-line program (csrc/slot_vm.cuh) and runs it on the host.
#include "../../intelligenceregulation_b200/csrc/slot_vm.cuh"

static std::vector<fp2> poisoned(const vm::Program& p, int npt) {
    return std::vector<fp2>(vm::slot_entries(p.p_slots, p.a_slots, npt) + 1, f2(0xA5A5A5A5A5A5A5A5ull, 0x5A5A5A5A5A5A5A5Aull));
}

template <int NPT>
static void run(const vm::Program& p, const fp2* lo, const fp2* hi, u32 first, bool skip, u64* out) {
    std::vector<fp2> slots = poisoned(p, NPT);
    fp2 x[NPT];
    vm::eval<NPT>(p.code.data(), p.coefs.data(), [&](u32 t, fp2& a, fp2& b) { a = lo[t]; b = hi[t]; }, slots.data(), 1, p.p_slots * NPT, first, skip, x);
    for (int j = 0; j < NPT; j++) { const fp2 v = f2_canon(x[j]); out[2 * j] = v.c0; out[2 * j + 1] = v.c1; }
}

// parts 1: the whole program; above: the sum of that many parts' values, one point
extern "C" void emul_vm(const u32* words, u32 n_words, u32 n_tables, u32 n_nodes, u32 n_terms, const u64* coefs, u32 n_coefs, const u64* lo, const u64* hi,
                        int npt, u32 first, int skip, u32 parts, u64* out, u32* info) {
    ir::Shape s{n_tables, n_nodes, n_terms, n_coefs, n_words};
    vm::Compiler c;
    c.run(s, words, reinterpret_cast<const fp2*>(coefs));
    if (parts > 1) c.split(s, words, reinterpret_cast<const fp2*>(coefs), parts);
    const vm::Program& p = c.out;
    info[0] = p.parts; info[1] = p.p_slots; info[2] = p.a_slots; info[3] = p.degree;
    const fp2 *l = reinterpret_cast<const fp2*>(lo), *h = reinterpret_cast<const fp2*>(hi);
    switch (npt) {
        case 1: {
            fp2 sum = f2(0, 0);
            for (u32 k = 0; k < p.parts; k++) {
                std::vector<fp2> slots = poisoned(p, 1);
                auto table = [&](u32 t) { fp2 v = l[t]; for (u32 d = 0; d < first; d++) v = f2_add(v, f2_sub(h[t], l[t])); return v; };
                sum = f2_add(sum, f2_canon(vm::eval_one(p.code.data() + (p.parts > 1 ? p.start[k] : 0), p.coefs.data(), table, slots.data(), 1, p.p_slots)));
            }
            out[0] = sum.c0; out[1] = sum.c1;
            break;
        }
        case 2: run<2>(p, l, h, first, skip, out); break;
        case 3: run<3>(p, l, h, first, skip, out); break;
        case 4: run<4>(p, l, h, first, skip, out); break;
        case 5: run<5>(p, l, h, first, skip, out); break;
    }
}
