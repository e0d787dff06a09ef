// Compiles a slot polynomial to the sumcheck kernels' straight-line program (csrc/slot_vm.cuh) and runs it on the host.
#include "../../intelligenceregulation_b200/csrc/slot_vm.cuh"

template <int NPT>
static void run(const vm::Program& p, const fp2* lo, const fp2* hi, u32 first, bool skip, u64* out) {
    std::vector<fp2> slots(vm::slot_entries(p.p_slots, p.a_slots, NPT) + 1, f2(0xA5A5A5A5A5A5A5A5ull, 0x5A5A5A5A5A5A5A5Aull));  // poisoned
    fp2 x[NPT];
    vm::eval<NPT>(p.code.data(), p.coefs.data(), [&](u32 t, fp2& a, fp2& b) { a = lo[t]; b = hi[t]; }, slots.data(), 1, p.p_slots * NPT, first, skip, x);
    for (int j = 0; j < NPT; j++) { out[2 * j] = x[j].c0; out[2 * j + 1] = x[j].c1; }
}

extern "C" void emul_vm(const u32* words, u32 n_words, u32 n_tables, u32 n_nodes, u32 n_terms, const u64* coefs, u32 n_coefs, const u64* lo, const u64* hi,
                        int npt, u32 first, int skip, u64* out, u32* info) {
    ir::Shape s{n_tables, n_nodes, n_terms, n_coefs, n_words};
    vm::Compiler c;
    c.run(s, words, reinterpret_cast<const fp2*>(coefs));
    info[0] = (u32)c.out.code.size(); info[1] = c.out.p_slots; info[2] = c.out.a_slots; info[3] = c.out.degree;
    const fp2 *l = reinterpret_cast<const fp2*>(lo), *h = reinterpret_cast<const fp2*>(hi);
    switch (npt) {
        case 1: run<1>(c.out, l, h, first, skip, out); break;
        case 2: run<2>(c.out, l, h, first, skip, out); break;
        case 3: run<3>(c.out, l, h, first, skip, out); break;
        case 4: run<4>(c.out, l, h, first, skip, out); break;
        case 5: run<5>(c.out, l, h, first, skip, out); break;
    }
}
