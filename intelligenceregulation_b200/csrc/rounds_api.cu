// C ABI: the sumcheck evaluator (`impl SumcheckRounds`, sumcheck/rounds.rs:22-28) and its
// device-side batch of rounds with the Fiat-Shamir step (the reference's Metal form:
// metal.rs:3509-3669 MetalRounds, :4141-4192 TailedRounds::masked_prove).
#include <cstring>

#include "api_internal.h"
#include "../../include/hl_b200_bench.h"
#include "slot_gen.cuh"
#include "slot_vm.cuh"
#include "sumcheck.h"

using namespace hlapi;

struct hl_tables;
u64* hl_tables_adopt(hl_tables* t);        // tables.cu: hands the device tables over (the set is empty afterwards)
const u64* hl_tables_peek(hl_tables* t);   // the device tables, still owned by the set
int hl_tables_flush_locked(hl_tables* t);  // waits for the builders; refuses a base-declared table with an extension word
void hl_tables_shape(hl_tables* t, hl_ctx** c, size_t* k, uint32_t* n_vars);

struct hl_rounds {
    hl_ctx* ctx = nullptr;
    int poly = 0;
    u32 k = 0, n_vars = 0, degree = 0, next = 0;
    size_t stride = 0, len = 0, ncoefs = 0;
    u32 max_blocks = 0;
    u64* d_tables = nullptr;
    // one device block of everything else: [inverse denominators, extrapolation weights, coefficients, plan] as uploaded at the start,
    // then [mask rows and table | state | what the resident CTAs share] as uploaded by a batch (the mask ends where the state begins), then [rows of the output,
    // finals], which a batch reads back together with the state, then the CTA partials
    char* blk = nullptr;
    size_t blk_bytes = 0, mask_cap = 0;
    u64* d_coefs = nullptr;
    u64* d_partials = nullptr;
    u64* d_slots = nullptr;    // slots of a slot program that shared memory does not hold
    size_t slot_bytes = 0;
    hlk::ScSync* d_sync = nullptr;
    u64* d_other = nullptr;    // the one-launch rounds' second table buffer
    u64* d_out = nullptr;      // n_vars rows of (2 (degree+1) + 1) Fp2
    u64* d_finals = nullptr;   // k Fp2 behind them
    u64* d_inv_den = nullptr;
    u64* d_extrap = nullptr;   // weights of the points above the evaluated degree (data-form polynomials only)
    std::vector<u64> finals;   // the finals, once a batch has brought them along with its last round
    u32 eval_degree = 0;
    hlk::ScState* d_state = nullptr;
    hlk::IrDev ir{};           // poly == POLY_IR: the polynomial as data
    const sg::Entry* gen = nullptr;  // the generated kernel of this program's graph, when there is one
    u64* d_cfo = nullptr;      // its coefficients by occurrence
    u64* d_nonbase = nullptr;  // one word: bit t set when table t is extension-valued before the first fold
    u64 nonbase = ~0ull;
    int failed = 0;            // the status of a batch that failed on the way: the tables are between two rounds, nothing goes on from there
    size_t out_row() const { return (2 * ((size_t)degree + 1) + 1) * 2; }
};

namespace {

void free_rounds(hl_rounds* r) {
    hl_ctx* c = r->ctx;
    if (r->d_tables) dev_free(c, r->d_tables, r->k * r->stride * 16);
    dev_free(c, r->blk, r->blk_bytes);
    if (r->d_cfo) dev_free(c, r->d_cfo, (size_t)(r->gen ? r->gen->n_cfo : 1) * 16);
    if (r->d_nonbase) dev_free(c, r->d_nonbase, 8);
    delete r;
}

int spent(hl_rounds* r) { return fail(r->ctx, r->failed, "rounds: an earlier batch of this evaluator failed"); }

// What every round of a batch takes its step with; a plain round() leaves it as it is made.
struct StepPlan {
    int fs = 0, recover = 0, mask_vars = 0, between = 0;
    const u64 *mask = nullptr, *mask_tab = nullptr;
};

hlk::ScStep step_of(const hl_rounds* r, u32 round, u32 nb, int use_claim, const StepPlan& p) {
    hlk::ScStep a;
    a.partials = r->d_partials; a.nblocks = nb; a.degree = (int)r->degree; a.round = (int)round;
    a.use_claim = use_claim; a.recover = p.recover; a.fs = p.fs; a.mask = p.mask; a.mask_tab = p.mask_tab; a.mask_vars = p.mask_vars;
    a.inv_den = r->d_inv_den; a.state = r->d_state; a.out = r->d_out;
    a.eval_degree = (int)r->eval_degree; a.extrap = r->d_extrap; a.between = p.between;
    return a;
}

// launches round r->next, its sums and its step; the caller holds the context lock
int launch_round(hl_rounds* r, int eval_one, int use_claim, const StepPlan& plan) {
    hl_ctx* c = r->ctx;
    const u32 half = (u32)(r->len / 2);
    const bool is_ir = r->poly == hlk::POLY_IR;
    const u32 nb = hlk::sc_round_blocks(half, c->sm_count);
    const hlk::ScStep step = step_of(r, r->next, nb, use_claim, plan);
    cudaError_t e;
    if (is_ir && r->gen && c->slot_kernels) {
        // the generated kernel of this graph: the first-round typing while the tables it reads as base words are base-valued
        const u32 skip = (!eval_one && r->eval_degree >= 1) ? 1u : 0u, npe = r->eval_degree + 1 - skip;
        const bool r0 = r->next == 0 && (r->gen->base_mask & r->nonbase) == 0;
        const bool per_point = (u64)half < (u64)c->sm_count * sg::GT * 2;
        u32 bx = (half + sg::GT - 1) / sg::GT, cap = (u32)c->sm_count * 4;
        if (bx > cap) bx = cap;
        if (bx > r->max_blocks) bx = r->max_blocks;
        if (bx < 1) bx = 1;
        c->stats.generated_rounds++;
        e = r->gen->launch(r0, per_point, bx, r->d_tables, r->stride, half, r->d_cfo, (int)r->degree, npe, skip, r->d_partials, c->stream);
        c->stats.kernel_launches++;
        if (e == cudaSuccess) e = hlk::sc_step(step_of(r, r->next, bx, use_claim, plan), c->stream);
    } else {
        e = is_ir ? hlk::sc_round_ir(r->ir, r->d_tables, r->stride, half, (int)r->degree, eval_one, r->d_slots, c->sm_count, step, r->d_sync, c->stream)
                  : hlk::sc_round(r->poly, (int)r->k, r->d_tables, r->stride, half, r->d_coefs, eval_one, step, r->d_sync, c->stream);
    }
    c->stats.kernel_launches++;
    if (e != cudaSuccess) return fail(c, HL_B200_ERR_DEVICE, "round launch", e);
    return HL_B200_OK;
}

int launch_fold(hl_rounds* r) {
    hl_ctx* c = r->ctx;
    cudaError_t e = hlk::sc_fold(r->d_tables, r->stride, (u32)(r->len / 2), r->k, r->d_state, c->stream);
    c->stats.kernel_launches++;
    if (e != cudaSuccess) return fail(c, HL_B200_ERR_DEVICE, "fold launch", e);
    r->len /= 2;
    r->next++;
    return HL_B200_OK;
}

// A program of more than a dozen instructions is also cut into parts of about that many, for the rounds with few pairs.
void compile(vm::Compiler& prog, const ir::Shape& sh, const uint32_t* words, const uint64_t* coefs) {
    const fp2* cf = reinterpret_cast<const fp2*>(coefs);
    prog.run(sh, words, cf);
    const u32 parts = ((u32)prog.out.code.size() + 11) / 12;
    if (parts > 1) prog.split(sh, words, cf, parts < vm::MAX_PARTS ? parts : vm::MAX_PARTS);
}

struct GenAsk {  // a slot program's generated kernel, looked up by the caller
    const sg::Entry* entry = nullptr;
    std::vector<fp2> cfo;
};

// the evaluator of either kind; `program` when poly == POLY_IR
int rounds_build(hl_ctx* c, int poly, size_t k, uint32_t n_vars, uint32_t degree, const uint64_t* tables, const uint64_t* coefs,
                 size_t ncoefs, const vm::Program* program, hl_rounds** out, hl_tables* built = nullptr, const GenAsk* gen = nullptr) {
    Call g(c);
    if (built) {
        if (int rc = hl_tables_flush_locked(built)) return rc;
    }
    hl_rounds* r = new hl_rounds();
    r->ctx = c; r->poly = poly; r->k = (u32)k; r->n_vars = n_vars; r->degree = degree; r->ncoefs = ncoefs;
    r->stride = r->len = (size_t)1 << n_vars;
    r->max_blocks = hlk::sc_round_blocks((u32)(r->len / 2), c->sm_count);
    r->eval_degree = degree;
    if (poly == hlk::POLY_IR) {
        const vm::Program& pg = *program;
        r->eval_degree = r->ir.eval_degree = pg.degree < degree ? pg.degree : degree;
        r->ir.n_code = (u32)pg.code.size(); r->ir.n_coefs = (u32)pg.coefs.size(); r->ir.n_tables = (u32)k;
        r->ir.p_slots = pg.p_slots; r->ir.a_slots = pg.a_slots; r->ir.parts = pg.parts;
        for (u32 w = 0; w < pg.parts; w++) r->ir.start[w] = pg.start[w];
        r->max_blocks = (u32)c->sm_count * 4;
        const size_t long_slots = hlk::sc_ir_slot_bytes(r->ir, c->sm_count),
                     run_slots = hlk::sc_run_slot_bytes(poly, r->ir, (int)k, (int)r->eval_degree, c->sm_count);
        r->slot_bytes = long_slots > run_slots ? long_slots : run_slots;
    }
    const u32 run_len = hlk::sc_run_len(poly, r->ir) < r->len ? hlk::sc_run_len(poly, r->ir) : (u32)r->len;
    // what the kernels read and no challenge changes, in one upload
    std::vector<char> head;
    auto put = [&](size_t bytes) {
        const size_t at = head.size();
        head.resize((at + bytes + 15) & ~(size_t)15, 0);
        return at;
    };
    const size_t at_den = put(((size_t)degree + 1) * 8);
    {
        u64* inv_den = reinterpret_cast<u64*>(head.data() + at_den);
        for (u32 i = 0; i <= degree; i++) {
            u64 den = 1;
            for (u32 j = 0; j <= degree; j++)
                if (j != i) den = gl_mul(den, gl_from_i64((long long)i - (long long)j));
            inv_den[i] = gl_inv(den);
        }
    }
    const bool extrapolates = r->eval_degree < degree;
    const size_t at_ex = extrapolates ? put((size_t)hlk::SC_MAX_POINTS * hlk::SC_MAX_POINTS * 8) : 0;
    if (extrapolates) {
        // s(p) = sum_i s(i) prod_{j != i} (p - j) / (i - j) over i, j <= eval_degree, for p above it
        u64* wts = reinterpret_cast<u64*>(head.data() + at_ex);
        const u32 de = r->eval_degree;
        for (u32 pnt = de + 1; pnt <= degree; pnt++)
            for (u32 i = 0; i <= de; i++) {
                u64 num = 1, den = 1;
                for (u32 j = 0; j <= de; j++)
                    if (j != i) {
                        num = gl_mul(num, gl_from_i64((long long)pnt - (long long)j));
                        den = gl_mul(den, gl_from_i64((long long)i - (long long)j));
                    }
                wts[(pnt - de - 1) * (de + 1) + i] = gl_mul(num, gl_inv(den));
            }
    }
    const bool is_ir = poly == hlk::POLY_IR;
    const size_t n_cf = is_ir ? program->coefs.size() : ncoefs;
    const size_t at_cf = put((n_cf ? n_cf : 1) * 16);
    if (n_cf) memcpy(head.data() + at_cf, is_ir ? (const void*)program->coefs.data() : (const void*)coefs, n_cf * 16);
    const size_t at_code = is_ir ? put(program->code.size() * 8) : 0;
    if (is_ir) memcpy(head.data() + at_code, program->code.data(), program->code.size() * 8);
    r->mask_cap = ((size_t)63 * degree + 2) * 16 + (size_t)63 * (degree + 1) * 16;
    const size_t at_state = head.size() + r->mask_cap, state_bytes = (sizeof(hlk::ScState) + 15) & ~(size_t)15;
    const size_t at_sync = at_state + state_bytes, at_out = at_sync + ((sizeof(hlk::ScSync) + 15) & ~(size_t)15), at_fin = at_out + (n_vars ? n_vars : 1) * r->out_row() * 8, at_part = at_fin + k * 16;
    const size_t at_slots = at_part + (size_t)r->max_blocks * (degree + 1) * 16;
    const size_t at_other = (at_slots + r->slot_bytes + 15) & ~(size_t)15;
    r->blk_bytes = at_other + hlk::sc_run_other_bytes((int)k, run_len);
    int rc = built ? HL_B200_OK : dev_alloc(c, (void**)&r->d_tables, k * r->stride * 16);
    if (!rc) rc = dev_alloc(c, (void**)&r->blk, r->blk_bytes);
    if (!rc) {
        r->d_inv_den = (u64*)(r->blk + at_den);
        r->d_extrap = extrapolates ? (u64*)(r->blk + at_ex) : nullptr;
        r->d_coefs = (u64*)(r->blk + at_cf);
        if (is_ir) { r->ir.code = (const u64*)(r->blk + at_code); r->ir.coefs = (const u64*)(r->blk + at_cf); }
        r->d_state = (hlk::ScState*)(r->blk + at_state);
        r->d_out = (u64*)(r->blk + at_out);
        r->d_finals = (u64*)(r->blk + at_fin);
        r->d_partials = (u64*)(r->blk + at_part);
        r->d_slots = r->slot_bytes ? (u64*)(r->blk + at_slots) : nullptr;
        r->d_sync = (hlk::ScSync*)(r->blk + at_sync);
        r->d_other = (u64*)(r->blk + at_other);
    }
    if (!rc && !built) rc = h2d_owned(c, r->d_tables, tables, k * r->stride * 16);
    if (!rc) rc = h2d_owned(c, r->blk, head.data(), head.size());
    if (!rc) {
        cudaError_t e = cudaMemsetAsync(r->d_state, 0, (char*)r->d_out - (char*)r->d_state, c->stream);
        if (e != cudaSuccess) rc = fail(c, HL_B200_ERR_DEVICE, "state clear", e);
    }
    if (!rc && c->slot_kernels && gen && gen->entry && gen->entry->n_tables == k && gen->entry->n_cfo == gen->cfo.size()) {
        // the generated kernels are switched on and the graph has one: its coefficients by occurrence, and which tables are base-valued
        // right now (a scan of every table: not paid while the switch is off)
        r->gen = gen->entry;
        rc = dev_alloc(c, (void**)&r->d_cfo, (size_t)(gen->cfo.size() ? gen->cfo.size() : 1) * 16);
        if (!rc) rc = dev_alloc(c, (void**)&r->d_nonbase, 8);
        if (!rc && gen->cfo.size()) rc = h2d(c, r->d_cfo, gen->cfo.data(), gen->cfo.size() * 16);
        if (!rc && cudaMemsetAsync(r->d_nonbase, 0, 8, c->stream) != cudaSuccess) rc = fail(c, HL_B200_ERR_DEVICE, "mask clear");
        if (!rc) {
            const u64* tabs = built ? hl_tables_peek(built) : r->d_tables;
            cudaError_t e = hlk::sc_nonbase_mask(tabs, r->stride, r->len, (u32)k, r->d_nonbase, c->sm_count, c->stream);
            c->stats.kernel_launches++;
            if (e != cudaSuccess) rc = fail(c, HL_B200_ERR_DEVICE, "table typing launch", e);
        }
        if (!rc) rc = d2h(c, &r->nonbase, r->d_nonbase, 8);
        if (!rc) rc = sync(c, "rounds_new");
    }
    if (rc) { free_rounds(r); return rc; }
    if (built) r->d_tables = hl_tables_adopt(built);  // only now: a failed build leaves the set with its owner
    *out = r;
    return HL_B200_OK;
}

}  // namespace

extern "C" {

int hl_b200_rounds_new(hl_ctx* c, int poly, size_t k, uint32_t n_vars, uint32_t degree, const uint64_t* tables,
                       const uint64_t* coefs, size_t ncoefs, hl_rounds** out) {
    if (!c || !tables || !out) return fail(c, HL_B200_ERR_ARG, "rounds_new: null argument");
    if (n_vars > 30) return fail(c, HL_B200_ERR_UNSUPPORTED, "rounds_new: more than 30 variables");
    if (poly == hlk::POLY_IR) return fail(c, HL_B200_ERR_ARG, "rounds_new: a data-form polynomial goes through rounds_new_ir");
    if (!hlk::sc_supported(poly, (int)k, (int)degree)) return fail(c, HL_B200_ERR_UNSUPPORTED, "rounds_new: polynomial family / table count / degree");
    if ((poly == hlk::POLY_LOGUP_Q || poly == hlk::POLY_LOGUP_T) && (!coefs || ncoefs < 1)) return fail(c, HL_B200_ERR_ARG, "rounds_new: alpha missing");
    return rounds_build(c, poly, k, n_vars, degree, tables, coefs, ncoefs, nullptr, out);
}

int hl_b200_rounds_new_ir(hl_ctx* c, size_t k, uint32_t n_vars, uint32_t degree, const uint64_t* tables, const uint32_t* words,
                          size_t n_words, uint32_t n_nodes, uint32_t n_terms, const uint64_t* coefs, size_t ncoefs, hl_rounds** out) {
    if (!c || !tables || !words || !out || (ncoefs && !coefs)) return fail(c, HL_B200_ERR_ARG, "rounds_new_ir: null argument");
    if (n_vars > 30) return fail(c, HL_B200_ERR_UNSUPPORTED, "rounds_new_ir: more than 30 variables");
    if (!hlk::sc_supported(hlk::POLY_IR, (int)k, (int)degree) || n_words > ir::MAX_WORDS || n_nodes > ir::MAX_NODES || ncoefs > ir::MAX_COEFS)
        return fail(c, HL_B200_ERR_UNSUPPORTED, "rounds_new_ir: table count, degree or program size beyond the evaluator's limits");
    ir::Shape sh{(u32)k, n_nodes, n_terms, (u32)ncoefs, (u32)n_words};
    if (int why = ir::validate(sh, words)) {
        char buf[96];
        snprintf(buf, sizeof buf, "rounds_new_ir: malformed program (check %d)", why);
        return fail(c, HL_B200_ERR_ARG, buf);
    }
    vm::Compiler prog;
    compile(prog, sh, words, coefs);
    GenAsk gen;
    gen.entry = sg::find(ir::signature(sh, words, reinterpret_cast<const fp2*>(coefs), &gen.cfo));
    return rounds_build(c, hlk::POLY_IR, k, n_vars, degree, tables, coefs, ncoefs, &prog.out, out, nullptr, &gen);
}

int hl_b200_rounds_from_tables(hl_ctx* c, int poly, uint32_t degree, hl_tables* t, const uint64_t* coefs, size_t ncoefs, hl_rounds** out) {
    if (!c || !t || !out) return fail(c, HL_B200_ERR_ARG, "rounds_from_tables: null argument");
    hl_ctx* tc = nullptr;
    size_t k = 0;
    uint32_t n_vars = 0;
    hl_tables_shape(t, &tc, &k, &n_vars);
    if (tc != c || k == 0) return fail(c, HL_B200_ERR_ARG, "rounds_from_tables: the table set is empty or belongs to another context");
    if (poly == hlk::POLY_IR) return fail(c, HL_B200_ERR_ARG, "rounds_from_tables: a data-form polynomial goes through rounds_from_tables_ir");
    if (!hlk::sc_supported(poly, (int)k, (int)degree)) return fail(c, HL_B200_ERR_UNSUPPORTED, "rounds_from_tables: polynomial family / table count / degree");
    if ((poly == hlk::POLY_LOGUP_Q || poly == hlk::POLY_LOGUP_T) && (!coefs || ncoefs < 1)) return fail(c, HL_B200_ERR_ARG, "rounds_from_tables: alpha missing");
    return rounds_build(c, poly, k, n_vars, degree, nullptr, coefs, ncoefs, nullptr, out, t);
}

int hl_b200_rounds_from_tables_ir(hl_ctx* c, uint32_t degree, hl_tables* t, const uint32_t* words, size_t n_words, uint32_t n_nodes,
                                  uint32_t n_terms, const uint64_t* coefs, size_t ncoefs, hl_rounds** out) {
    if (!c || !t || !words || !out || (ncoefs && !coefs)) return fail(c, HL_B200_ERR_ARG, "rounds_from_tables_ir: null argument");
    hl_ctx* tc = nullptr;
    size_t k = 0;
    uint32_t n_vars = 0;
    hl_tables_shape(t, &tc, &k, &n_vars);
    if (tc != c || k == 0) return fail(c, HL_B200_ERR_ARG, "rounds_from_tables_ir: the table set is empty or belongs to another context");
    if (!hlk::sc_supported(hlk::POLY_IR, (int)k, (int)degree) || n_words > ir::MAX_WORDS || n_nodes > ir::MAX_NODES || ncoefs > ir::MAX_COEFS)
        return fail(c, HL_B200_ERR_UNSUPPORTED, "rounds_from_tables_ir: table count, degree or program size beyond the evaluator's limits");
    ir::Shape sh{(u32)k, n_nodes, n_terms, (u32)ncoefs, (u32)n_words};
    if (ir::validate(sh, words)) return fail(c, HL_B200_ERR_ARG, "rounds_from_tables_ir: malformed program");
    {
        // the tables' kernels go first: the device builds them (the width check's 37 of 2^19 entries: 90 us) while this thread compiles
        // the program (its 250 instructions and their parts: 90 us)
        Call g(c);
        if (int rc = hl_tables_flush_locked(t)) return rc;
    }
    vm::Compiler prog;
    compile(prog, sh, words, coefs);
    GenAsk gen;
    gen.entry = sg::find(ir::signature(sh, words, reinterpret_cast<const fp2*>(coefs), &gen.cfo));
    return rounds_build(c, hlk::POLY_IR, k, n_vars, degree, nullptr, coefs, ncoefs, &prog.out, out, t, &gen);
}

void hl_b200_rounds_free(hl_rounds* r) {
    if (!r) return;
    hl_ctx* c = r->ctx;
    Call g(c);
    free_rounds(r);
}

int hl_b200_rounds_round(hl_rounds* r, uint32_t j, int eval_one, uint64_t* sums) {
    if (!r || !sums) return HL_B200_ERR_ARG;
    hl_ctx* c = r->ctx;
    if (r->failed) return spent(r);
    if (j != r->next || j >= r->n_vars) return fail(c, HL_B200_ERR_ARG, "rounds_round: round order (a round needs the preceding fold)");
    Call g(c);
    int rc;
    {
        Timed t(c, HL_T_ROUNDS);
        rc = launch_round(r, eval_one, 0, StepPlan());
    }
    if (!rc) rc = d2h(c, sums, r->d_out + (size_t)j * r->out_row(), ((size_t)r->degree + 1) * 16);
    if (!rc) rc = sync(c, "rounds_round");
    return rc;
}

int hl_b200_rounds_fold(hl_rounds* r, const uint64_t rr[2]) {
    if (!r || !rr) return HL_B200_ERR_ARG;
    hl_ctx* c = r->ctx;
    if (r->failed) return spent(r);
    if (r->next >= r->n_vars) return fail(c, HL_B200_ERR_ARG, "rounds_fold: every variable is already folded");
    Call g(c);
    int rc = h2d(c, (char*)r->d_state + offsetof(hlk::ScState, r), rr, 16);
    if (!rc) {
        Timed t(c, HL_T_ROUNDS);
        rc = launch_fold(r);
    }
    if (!rc) rc = sync(c, "rounds_fold");
    return rc;
}

int hl_b200_rounds_finals(hl_rounds* r, uint64_t* out) {
    if (!r || !out) return HL_B200_ERR_ARG;
    hl_ctx* c = r->ctx;
    if (r->failed) return spent(r);
    if (r->next != r->n_vars) return fail(c, HL_B200_ERR_ARG, "rounds_finals: finals need all folds");
    Call g(c);
    if (r->finals.empty()) {
        std::vector<u64> got(2 * (size_t)r->k);
        cudaError_t e = hlk::sc_finals(r->d_tables, r->stride, r->k, r->d_finals, c->stream);
        c->stats.kernel_launches++;
        int rc = e == cudaSuccess ? d2h(c, got.data(), r->d_finals, got.size() * 8) : fail(c, HL_B200_ERR_DEVICE, "finals launch", e);
        if (!rc) rc = sync(c, "rounds_finals");
        if (rc) return rc;
        r->finals.swap(got);
    }
    memcpy(out, r->finals.data(), r->finals.size() * 8);
    return HL_B200_OK;
}

int hl_b200_set_dependent_launch(int on) {
    hlk::sc_set_dependent_launch(on != 0);
    return HL_B200_OK;
}

int hl_b200_set_wait_limits(hl_ctx* c, uint32_t sums, uint32_t challenge) {
    if (!c) return HL_B200_ERR_ARG;
    Call g(c);
    c->waits.sums = sums;
    c->waits.challenge = challenge;
    return HL_B200_OK;
}

int hl_b200_rounds_batched(hl_rounds* r, uint32_t nd, hl_fs_state* fs, const uint64_t* mask_coeffs, uint32_t mask_vars,
                           const uint64_t mask_c[2], uint64_t* out) {
    if (!r || !fs || !out) return HL_B200_ERR_ARG;
    hl_ctx* c = r->ctx;
    if (nd == 0) return HL_B200_OK;
    if (r->failed) return spent(r);
    if (r->next + nd > r->n_vars) return fail(c, HL_B200_ERR_ARG, "rounds_batched: more rounds than variables left");
    if (mask_coeffs && (r->next != 0 || !mask_c || mask_vars < r->n_vars || mask_vars > 63))
        return fail(c, HL_B200_ERR_ARG, "rounds_batched: a masked batch starts at round 0 and its mask covers every variable");
    if (fs->recover_one && r->degree < 1) return fail(c, HL_B200_ERR_ARG, "rounds_batched: claim recovery requires degree >= 1");
    Call g(c);
    hlk::ScState st;
    memset(&st, 0, sizeof st);
    memcpy(st.state, fs->state, 32);
    memcpy(st.key, fs->key, 32);
    st.counter = fs->counter;
    st.keyed = fs->keyed;
    st.claim = f2(fs->claim[0], fs->claim[1]);
    u64 *d_mask = nullptr, *d_mtab = nullptr;
    const size_t row_words = mask_coeffs ? (size_t)mask_vars * r->degree * 2 : 0, tab_words = mask_coeffs ? (size_t)mask_vars * (r->degree + 1) * 2 : 0;
    const size_t st_words = (size_t)((char*)r->d_out - (char*)r->d_state) / 8;  // the state and, zeroed, what the resident CTAs share
    std::vector<u64> up(row_words + tab_words + st_words);
    int rc = HL_B200_OK;
    if (mask_coeffs) {
        // the mask scaled by its challenge: the device then adds c g_j without a product
        const fp2 mc = f2(mask_c[0], mask_c[1]);
        std::vector<fp2> scaled((size_t)mask_vars * r->degree + 2);
        for (size_t i = 0; i < scaled.size(); i++) scaled[i] = f2_mul(mc, reinterpret_cast<const fp2*>(mask_coeffs)[i]);
        const fp2* co = scaled.data();
        st.ap = co[1];  // c a' times the empty product
        // per round j and point x: 2^(N-1-j) (a0 + sum_{i>j} u_i(1)/2 + u_j(x)) (sumcheck.rs:260-295): the part of g_j(x) no challenge enters
        const u64 half = gl_inv(2);
        u64* const mtab = up.data() + row_words;
        fp2 run = f2(0, 0);
        for (int i = (int)mask_vars - 1; i >= 0; i--) {
            const fp2* ai = co + 2 + (size_t)i * r->degree;
            const u64 scale = 1ull << (mask_vars - 1 - (u32)i);  // mask_vars <= 63: the power of two is its own canonical word
            for (u32 x = 0; x <= r->degree; x++) {
                fp2 u = f2(0, 0);
                u64 xp = 1;
                for (u32 e = 1; e <= r->degree; e++) { xp = gl_mul(xp, (u64)x); u = f2_add(u, f2_mul_base(ai[e - 1], xp)); }
                const fp2 v = f2_mul_base(f2_add(f2_add(co[0], run), u), scale);
                mtab[((size_t)i * (r->degree + 1) + x) * 2] = v.c0; mtab[((size_t)i * (r->degree + 1) + x) * 2 + 1] = v.c1;
            }
            fp2 u1 = f2(0, 0);
            for (u32 e = 0; e < r->degree; e++) u1 = f2_add(u1, ai[e]);
            run = f2_add(run, f2_mul_base(u1, half));
        }
        memcpy(up.data(), co + 2, row_words * 8);
        d_mask = (u64*)r->d_state - row_words - tab_words;
        d_mtab = (u64*)r->d_state - tab_words;
    }
    memcpy(up.data() + row_words + tab_words, &st, sizeof st);
    rc = h2d(c, (u64*)r->d_state - row_words - tab_words, up.data(), up.size() * 8);
    // with the generated kernels switched on they take the rounds down to 2^11 pairs: the switch is there to compare them
    const u32 first = r->next, run_len = r->gen && c->slot_kernels ? 1u << 12 : hlk::sc_run_len(r->poly, r->ir);
    bool have_claim = fs->recover_one && fs->have_claim;
    {
        Timed t(c, HL_T_ROUNDS);
        StepPlan plan;
        plan.fs = 1; plan.recover = fs->recover_one ? 1 : 0; plan.mask = d_mask; plan.mask_tab = d_mtab; plan.mask_vars = (int)mask_vars;
        u32 i = 0;
        for (; i < nd && !rc && r->len > run_len; i++) {
            rc = launch_round(r, have_claim ? 0 : 1, have_claim ? 1 : 0, plan);
            if (!rc) rc = launch_fold(r);
            have_claim = fs->recover_one != 0;
            plan.between = 1;
        }
        if (!rc && i == nd) {  // the batch ends here: the last challenge's claim
            cudaError_t e = hlk::sc_between(step_of(r, r->next, 0, 0, plan), c->stream);
            c->stats.kernel_launches++;
            if (e != cudaSuccess) rc = fail(c, HL_B200_ERR_DEVICE, "step launch", e);
        }
        if (!rc && i < nd) {  // the short rounds: one launch (sumcheck_run.cu)
            const u32 left = nd - i;
            cudaError_t e = hlk::sc_run(r->poly, r->ir, (int)r->k, r->d_tables, r->stride, (u32)r->len, r->d_coefs, step_of(r, r->next, 1, 0, plan), (int)left,
                                        have_claim ? 1 : 0, r->d_sync, c->waits, r->d_slots, r->d_other, c->sm_count, c->stream);
            c->stats.kernel_launches++;
            if (e != cudaSuccess) rc = fail(c, HL_B200_ERR_DEVICE, "short rounds launch", e);
            r->len >>= left;
            r->next += left;
        }
    }
    const bool last = r->next == r->n_vars;
    if (!rc && last) {  // the finals come along
        cudaError_t e = hlk::sc_finals(r->d_tables, r->stride, r->k, r->d_finals, c->stream);
        c->stats.kernel_launches++;
        if (e != cudaSuccess) rc = fail(c, HL_B200_ERR_DEVICE, "finals launch", e);
    }
    const size_t o_out = (size_t)((char*)r->d_out - (char*)r->d_state), o_fin = (size_t)((char*)r->d_finals - (char*)r->d_state);
    std::vector<char> got(o_fin + r->k * 16);
    if (!rc) rc = d2h(c, got.data(), r->d_state, last ? got.size() : o_fin);
    if (!rc) rc = sync(c, "rounds_batched");
    hlk::ScSync sync_got;
    memcpy(&sync_got, got.data() + ((char*)r->d_sync - (char*)r->d_state), sizeof sync_got);
    if (!rc && sync_got.failed) rc = fail(c, HL_B200_ERR_TIMEOUT, "rounds_batched: a device wait ran out");
    if (rc) return r->failed = rc;
    memcpy(out, got.data() + o_out + first * r->out_row() * 8, (size_t)nd * r->out_row() * 8);
    memcpy(&st, got.data(), sizeof st);
    if (last) {
        r->finals.resize(2 * (size_t)r->k);
        memcpy(r->finals.data(), got.data() + o_fin, r->k * 16);
    }
    memcpy(fs->state, st.state, 32);
    fs->counter = st.counter;
    fs->claim[0] = st.claim.c0; fs->claim[1] = st.claim.c1;
    fs->have_claim = fs->recover_one ? 1 : fs->have_claim;
    c->stats.round_batches++;
    return HL_B200_OK;
}

}  // extern "C"
