// Shared declarations of the sumcheck kernels and their C-ABI wrapper.
#pragma once
#include <cuda_runtime.h>
#include "gl_field.cuh"
#include "slot_ir.cuh"

namespace hlk {

enum { POLY_PROD = 0, POLY_ZC = 1, POLY_LOGUP_Q = 2, POLY_LOGUP_T = 3, POLY_IR = 4 };
constexpr int SC_MAX_POINTS = 8;  // degree <= 7

// Device-resident state of one evaluator: the transcript (state, counter, key), the running
// unmasked claim, the last challenge, and the CFS mask's running terms.
struct ScState {
    uint32_t state[8];
    uint32_t key[8];
    u64 counter;
    int keyed;
    int pending;    // 1 + the round whose claim and mask terms are still to be taken from `sums` and `r` (0: none)
    fp2 claim;
    fp2 r;
    fp2 acc;        // c sum_{i<j} u_i(r_i), c the mask's challenge
    fp2 ap;         // c a' prod_{i<j} r_i (the mask's linear term, sumcheck.rs:260-295)
    fp2 sums[SC_MAX_POINTS];  // of the pending round
    fp2 g[SC_MAX_POINTS];     // the mask's values for round ahead - 1
    int ahead, pad_;
};

struct ScStep {
    const u64* partials;        // nblocks x (degree+1) Fp2 (the generated kernels' rounds; the others add to ScSync)
    u32 nblocks;                // rows, or the grid of a closed form's round
    int degree, round;
    int use_claim;              // s(1) := claim - s(0)
    int recover;                // keep the running claim (rounds.rs recover_one)
    int fs;                     // 0: only reduce and write the sums (host-driven round())
    const u64* mask;            // `degree` CFS coefficients c a_{j,e} per round, or NULL
    // per round j and point x = 0..degree: c 2^(N-1-j) (a0 + sum_{i>j} u_i(1)/2 + u_j(x)), the part of the mask's round
    // polynomial c g_j(x) that no challenge enters (made by the host once per batch)
    const u64* mask_tab;
    int mask_vars;
    const u64* inv_den;         // degree+1 inverse Lagrange denominators
    int eval_degree;            // the sums arrive at the points 0..eval_degree; the points above are extrapolated
    const u64* extrap;          // (degree - eval_degree) rows of eval_degree + 1 base-field weights, or NULL
    ScState* state;
    u64* out;                   // per round: (degree+1) sums, (degree+1) masked, r  (Fp2 each)
    int between = 0;            // a CTA beside the round's takes what the round before left pending
};

// a slot polynomial as a program (slot_vm.cuh), resident on the device
struct IrDev {
    const u64* code;
    const u64* coefs;  // n_coefs Fp2
    u32 n_code, n_coefs, n_tables, p_slots, a_slots;
    u32 parts, start[8];   // the program in parts (slot_vm.cuh); code[0] starts the whole
    u32 eval_degree;   // min(declared, attained): the points the kernels evaluate are 0 .. eval_degree
};

// What the CTAs of k_sc_run share beside the tables; zero at its launch.
struct ScSync {
    u64 r[2][2];      // the last two challenges
    u32 flag;         // rounds whose challenge is published
    u32 arrived;      // sums handed in so far
    u32 failed;       // a wait ran out
    u32 done;         // CTAs of a round's own launch that have handed in their sums (back at zero with the last one)
    // A round's sums, added up by all CTAs: per point the low and high halves of the two words, as plain integers (below 2^32 CTAs they
    // do not wrap).  Two sets: the one that has been read is cleared for the round after the next.
    u64 sums[2][SC_MAX_POINTS][4];
};

// How often the CTAs of k_sc_run look for something before they give up: CTA 0 for a round's sums, the others for its challenge.
struct ScWaits {
    u32 sums = 1u << 22, challenge = 1u << 22;  // some seconds
};

void sc_set_dependent_launch(bool on);
bool sc_dependent_launch();
u32 sc_round_blocks(u32 half, int sm_count);
// the long rounds of a slot program; slots: sc_ir_slot_bytes of scratch (NULL when that is 0)
size_t sc_ir_slot_bytes(const IrDev& p, int sm_count);
cudaError_t sc_round_ir(const IrDev& p, const u64* tables, size_t stride, u32 half, int degree, int eval_one, u64* slots, int sm_count, const ScStep& step, ScSync* sync,
                        cudaStream_t s);
// all remaining rounds in one launch, from a table length of at most sc_run_len (sumcheck_run.cu).  slots: sc_run_slot_bytes of scratch (NULL when that is 0); other: sc_run_other_bytes; sync: zeroed
constexpr int SC_RUN_CTAS = 4;  // per SM, at most
u32 sc_run_len(int poly, const IrDev& p);
size_t sc_run_other_bytes(int k, u32 len);
size_t sc_run_slot_bytes(int poly, const IrDev& p, int k, int eval_degree, int sm_count);
cudaError_t sc_run(int poly, const IrDev& p, int k, u64* tables, size_t stride, u32 len, const u64* coefs, const ScStep& a, int nrounds, int have_claim,
                   ScSync* sync, const ScWaits& waits, u64* slots, u64* other, int sm_count, cudaStream_t s);
bool sc_supported(int poly, int k, int degree);
// A round's sums and, by the CTA that finishes last, its step (sync: zero, and left ready for the next round)
cudaError_t sc_round(int poly, int k, const u64* tables, size_t stride, u32 half, const u64* coefs, int eval_one, const ScStep& step, ScSync* sync,
                     cudaStream_t s);
cudaError_t sc_step(const ScStep& a, cudaStream_t s);  // the step alone
// bit t of *d_mask is set when table t holds a non-zero second word anywhere in its first `len` entries (*d_mask zeroed by the caller)
cudaError_t sc_nonbase_mask(const u64* tables, size_t stride, size_t len, u32 k, u64* d_mask, int sm_count, cudaStream_t s);
// the first entry of every table, k Fp2 in a row
cudaError_t sc_finals(const u64* d_tables, size_t stride, u32 k, u64* d_out, cudaStream_t st);
cudaError_t sc_fold(u64* tables, size_t stride, u32 half, u32 k, const ScState* st, cudaStream_t s);
// takes what the round before a.round left pending
cudaError_t sc_between(const ScStep& a, cudaStream_t s);

}  // namespace hlk
