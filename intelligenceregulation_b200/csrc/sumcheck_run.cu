// The short rounds of a sumcheck in ONE launch.
//
// Once a round has some thousands of pairs, what it waits for is not arithmetic: as separate launches (sums, Fiat-Shamir step, fold) a
// round of 2^13 pairs and one of two took the same 25 us.  k_sc_run keeps the CTAs resident (a cooperative launch) and runs all of the
// remaining rounds: per round a CTA folds its pairs with the last challenge on the way in, evaluates them one (pair, evaluation point)
// per thread, and hands its sums to CTA 0, whose first warp takes the Fiat-Shamir step and publishes the challenge.
//
//   ownership   pair i of a round belongs to one CTA.  Its two entries T[i], T[i + half] are folded from T[i], T[i + len], T[i + half],
//               T[i + half + len] of the round before: four places that no other CTA touches in this round.  So the only thing the
//               CTAs wait for is the challenge.
//   shrinking   a round of at most CHUNK pairs needs one CTA: the others leave, and CTA 0 keeps the tables in shared memory from there on
//   the step    warp 0 prepares the mask before the sums arrive and updates the claim while the other warps fold (sc_step.cuh)
// Every wait is bounded: a CTA that waits too long records it and leaves, and the call returns HL_B200_ERR_TIMEOUT.
#include "sc_poly.cuh"
#include "sc_step.cuh"
#include "slot_vm.cuh"

namespace {

// `release` / `acquire` at device scope
__device__ __forceinline__ void st_release(u32* p, u32 v) { asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory"); }
__device__ __forceinline__ u32 ld_acquire(const u32* p) {
    u32 v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
constexpr u32 POLL_LIMIT = 1u << 22;  // polls of one wait: some seconds
constexpr u32 FLAG_FAILED = 0xFFFFFFFFu;

struct RunArgs {
    u64* tables;
    size_t stride;
    u32 len;             // live entries per table at the first round
    u32 k, nrounds, chunk, planes, parts, npe_max;
    int have_claim;      // the first round's claim is known
    hlk::ScStep step;    // step.round: the first round's number
    hlk::ScSync* sync;   // zero at the launch
    u64* partials;       // one row of 2 npe_max words per CTA
};

// Shared memory: [evaluator's own][table chunk][its successor, half as long], the two swapping roles once one CTA is left.
// A chunk holds table t of pair i at point p at [(t * planes + p) * chunk + i]: the ends of the pair (the points 0 and 1) and, where
// they all fit, the points above.  An evaluator then reads a value where it would step to it, and every evaluator of the pair would.
struct TabSmem {
    const fp2* base;
    u32 chunk, planes;
    __device__ __forceinline__ fp2 at(u32 t, u32 i, u32 point) const {
        const fp2* b = base + (size_t)t * planes * chunk + i;
        if (point < planes) return b[point * chunk];
        fp2 v = b[chunk];
        const fp2 d = f2_sub(v, b[0]);
        for (u32 p = 1; p < point; p++) v = f2_add(v, d);
        return v;
    }
};

// The closed-form families (sumcheck.h), one evaluation point
template <int POLY, int K>
struct ClosedEval {
    const u64* coefs;
    __device__ u32 stage(char*, u32) { return 0; }
    __device__ fp2 at(const TabSmem& tab, u32 i, u32 point, u32, u32) const {
        fp2 v[K];
#pragma unroll
        for (int t = 0; t < K; t++) v[t] = tab.at(t, i, point);
        const fp2* cf = reinterpret_cast<const fp2*>(coefs);
        return hlk::poly_eval<POLY, K>(v, cf);
    }
};

// Any slot polynomial, as a program (slot_vm.cuh)
struct ProgramEval {
    hlk::IrDev p;
    fp2* slots_g;    // the slots of all CTAs, where they do not fit shared memory
    int code_fits;   // code and coefficients fit shared memory
    const u64* code;
    const fp2* cf;
    fp2* slots;
    __device__ u32 stage(char* mem, u32 threads) {
        u32 used = 0;
        code = p.code;
        cf = reinterpret_cast<const fp2*>(p.coefs);
        if (code_fits) {
            u64* c = reinterpret_cast<u64*>(mem);
            for (u32 x = threadIdx.x; x < p.n_code; x += threads) c[x] = p.code[x];
            used = (p.n_code * 8 + 15) & ~15u;
            fp2* f = reinterpret_cast<fp2*>(mem + used);
            for (u32 x = threadIdx.x; x < p.n_coefs; x += threads) f[x] = ld2(p.coefs + 2 * (size_t)x);
            used += p.n_coefs * 16;
            code = c;
            cf = f;
        }
        const u32 entries = vm::slot_entries(p.p_slots, p.a_slots, 1) * threads;
        slots = (slots_g ? slots_g + (size_t)blockIdx.x * entries : reinterpret_cast<fp2*>(mem + used)) + threadIdx.x;
        return slots_g ? used : used + entries * 16;
    }
    __device__ fp2 at(const TabSmem& tab, u32 i, u32 point, u32 part, u32 threads) const {
        return f2_canon(vm::eval_one(p.parts > 1 ? code + p.start[part] : code, cf, [&](u32 t) { return tab.at(t, i, point); }, slots, threads, p.p_slots));
    }
};

__device__ __forceinline__ fp2 warp_sum(fp2 v) {
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) {
        const u32 a0 = __shfl_down_sync(0xffffffffu, (u32)v.c0, off), a1 = __shfl_down_sync(0xffffffffu, (u32)(v.c0 >> 32), off);
        const u32 b0 = __shfl_down_sync(0xffffffffu, (u32)v.c1, off), b1 = __shfl_down_sync(0xffffffffu, (u32)(v.c1 >> 32), off);
        v = f2_add(v, f2(((u64)a1 << 32) | a0, ((u64)b1 << 32) | b0));
    }
    return v;
}

constexpr u32 RUN_MAX_T = 512, RUN_PASSES = 4;

template <class Eval>
__global__ void __launch_bounds__(RUN_MAX_T) k_sc_run(RunArgs a, Eval ev) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    extern __shared__ __align__(16) char smem[];
    __shared__ StepSmem sm;
    __shared__ hlk::ScState st_s;
    __shared__ __align__(16) u64 rows_s[2 * 63 * (hlk::SC_MAX_POINTS - 1)];
    __shared__ __align__(16) u64 tab_s[2 * 63 * hlk::SC_MAX_POINTS];
    __shared__ u64 invden_s[hlk::SC_MAX_POINTS], extrap_s[hlk::SC_MAX_POINTS * hlk::SC_MAX_POINTS];
    __shared__ fp2 task_s[RUN_PASSES * RUN_MAX_T / 32];  // one sum per warp and pass: [task][warp of the chunk]
    __shared__ fp2 cta_s[hlk::SC_MAX_POINTS];
    __shared__ fp2 r_s;
    __shared__ u32 failed_s;
    const u32 T = blockDim.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, cta = blockIdx.x, C = a.chunk;
    const int degree = a.step.degree, np = degree + 1;
    const u32 own = ev.stage(smem, T);
    fp2* const buf0 = reinterpret_cast<fp2*>(smem + own);
    fp2* const buf1 = buf0 + (size_t)a.k * a.planes * C;  // with half the stride: it only ever holds the rounds after the first one
    if (tid == 0) failed_s = 0;
    if (cta == 0) {
        const u32* src = reinterpret_cast<const u32*>(a.step.state);
        u32* dst = reinterpret_cast<u32*>(&st_s);
        for (u32 i = tid; i < sizeof(hlk::ScState) / 4; i += T) dst[i] = src[i];
        if (a.step.mask) {
            const u32 nr = 2u * a.step.mask_vars * degree, nt = 2u * a.step.mask_vars * np;
            for (u32 i = tid; i < nr; i += T) rows_s[i] = a.step.mask[i];
            for (u32 i = tid; i < nt; i += T) tab_s[i] = a.step.mask_tab[i];
        }
        if ((int)tid < np) invden_s[tid] = a.step.inv_den[tid];
        if (a.step.extrap && (int)tid < (degree - a.step.eval_degree) * (a.step.eval_degree + 1)) extrap_s[tid] = a.step.extrap[tid];
    }
    __syncthreads();
    StepArgs sa;
    sa.degree = degree; sa.recover = a.step.recover; sa.fs = 1; sa.mask_vars = a.step.mask_vars; sa.eval_degree = a.step.eval_degree;
    sa.rows = a.step.mask ? reinterpret_cast<const fp2*>(rows_s) : nullptr;
    sa.tab = reinterpret_cast<const fp2*>(tab_s);
    sa.row0 = 0;
    sa.inv_den = invden_s; sa.extrap = a.step.extrap ? extrap_s : nullptr; sa.state = &st_s; sa.out = a.step.out;
    fp2 g = f2(0, 0), r = f2(0, 0);
    if (cta == 0 && warp == 0) g = step_ahead(sa, sm, a.step.round, lane);

    u32 len = a.len, arrived = 0, ncta_prev = 0;
    bool resident = false, second = false;  // the tables live in a buffer (one CTA): in the second one
    for (u32 rd = 0; rd < a.nrounds; rd++) {
        const u32 half = len >> 1, ncta = min(gridDim.x, (half + C - 1) / C);
        const int j = a.step.round + (int)rd;
        // nothing of this round or a later one is ours: our entries, folded with every challenge but the last, are in the tables
        if (cta >= ncta) return;
        // the last challenge
        if (rd > 0) {
            if (cta == 0) {
                r = r_s;
            } else {
                if (tid == 0) {
                    u32 f = 0;
                    for (u32 n = 0; n < POLL_LIMIT && (f = ld_acquire(&a.sync->flag)) < rd; n++) {}
                    if (f < rd || f == FLAG_FAILED) failed_s = 1;
                    else r_s = ld2(a.sync->r[(rd - 1) & 1]);
                }
                __syncthreads();
                if (failed_s) return;
                r = r_s;
            }
        }
        const bool claim = a.step.recover && (rd > 0 || a.have_claim);
        const bool skip = claim && a.step.eval_degree >= 1;
        const u32 npe = a.step.eval_degree + (skip ? 0 : 1);
        // CTA 0's first warp is behind: it still has to bring the claim and the mask up to the challenge just published
        const u32 ft = cta == 0 && rd > 0 ? T - 32 : T, f0 = cta == 0 && rd > 0 ? tid - 32 : tid;
        // a task is one point and one part of the polynomial, for all pairs of a chunk; a warp lies within one task
        const u32 tasks = npe * a.parts, tslots = T / C, my = tid / C, ti = tid - my * C;
        fp2 acc[RUN_PASSES];
#pragma unroll
        for (u32 q = 0; q < RUN_PASSES; q++) acc[q] = f2(0, 0);
        for (u32 c0 = cta * C; c0 < half; c0 += ncta * C) {
            const u32 cn = min(C, half - c0), lcn = __ffs((int)cn) - 1;  // powers of two, all of them
            if (c0 != cta * C) __syncthreads();  // the chunk before has been evaluated
            const bool to2 = resident && !second;
            fp2* to = to2 ? buf1 : buf0;
            const u32 ts_to = to2 ? C / 2 : C, ts_from = second ? C / 2 : C;
            if (cta == 0 && rd > 0 && warp == 0 && c0 == 0) {
                step_after(sa, sm, j - 1, r, lane);
                g = step_ahead(sa, sm, j, lane);
            } else if (cta != 0 || rd == 0 || warp > 0) {
                for (u32 x = f0; x < a.k * cn; x += ft) {
                    const u32 t = x >> lcn, i = x & (cn - 1);
                    fp2 v[2];  // the pair's two entries, c0 + i and c0 + i + half of the table
                    if (resident) {
                        const fp2* from = (second ? buf1 : buf0) + (size_t)t * a.planes * ts_from + i;
#pragma unroll
                        for (u32 e = 0; e < 2; e++) {
                            const fp2 lo = from[e * half];
                            v[e] = f2_add(lo, f2_mul(r, f2_sub(from[ts_from + e * half], lo)));
                        }
                    } else {
                        u64* p = a.tables + 2 * ((size_t)t * a.stride + c0 + i);
#pragma unroll
                        for (u32 e = 0; e < 2; e++) v[e] = ld2(p + 2 * (size_t)e * half);
                        if (rd > 0) {
#pragma unroll
                            for (u32 e = 0; e < 2; e++) v[e] = f2_add(v[e], f2_mul(r, f2_sub(ld2(p + 2 * ((size_t)e * half + len)), v[e])));
                            if (half > C) {
#pragma unroll
                                for (u32 e = 0; e < 2; e++) st2(p + 2 * (size_t)e * half, v[e]);
                            }
                        }
                    }
                    fp2* o = to + (size_t)t * a.planes * ts_to + i;
                    o[0] = v[0];
                    o[ts_to] = v[1];
                    if (a.planes > 2) {
                        const fp2 d = f2_sub(v[1], v[0]);
                        fp2 y = v[1];
                        for (u32 p = 2; p < a.planes; p++) { y = f2_add(y, d); o[p * ts_to] = y; }
                    }
                }
            }
            __syncthreads();
            const TabSmem tab{to, ts_to, a.planes};
#pragma unroll
            for (u32 q = 0; q < RUN_PASSES; q++) {
                const u32 task = my + q * tslots, part = task / npe, pi = task - part * npe;
                if (task < tasks && ti < cn) acc[q] = f2_add(acc[q], ev.at(tab, ti, skip && pi ? pi + 1 : pi, part, T));
            }
        }
        if (resident) second = !second;
        else if (half <= C) resident = true;
#pragma unroll
        for (u32 q = 0; q < RUN_PASSES; q++) {
            if (q * tslots >= tasks) break;
            acc[q] = warp_sum(acc[q]);
            if (lane == 0) task_s[q * (T / 32) + warp] = acc[q];
        }
        __syncthreads();
        if (tid < npe) {
            fp2 s = f2(0, 0);
            for (u32 part = 0; part < a.parts; part++)
                for (u32 w = 0; w < C / 32; w++) s = f2_add(s, task_s[(part * npe + tid) * (C / 32) + w]);
            cta_s[tid] = s;
            if (cta != 0) st2(a.partials + 2 * ((size_t)cta * a.npe_max + tid), s);
        }
        if (cta != 0) {
            __syncthreads();
            if (tid == 0) {
                __threadfence();
                asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&a.sync->arrived) : "memory");
            }
        } else {
            arrived += ncta - 1;
            if (ncta > 1) {
                // the other CTAs' sums: warp w takes the point w
                if (tid == 0) {
                    u32 n = 0;
                    while (n < POLL_LIMIT && ld_acquire(&a.sync->arrived) < arrived) n++;
                    if (n == POLL_LIMIT) failed_s = 1;
                }
                __syncthreads();
                if (failed_s) {
                    if (tid == 0) { a.sync->failed = 1; st_release(&a.sync->flag, FLAG_FAILED); }
                    return;
                }
                for (u32 pi = warp; pi < npe; pi += T / 32) {
                    fp2 s = f2(0, 0);
                    for (u32 b = 1 + lane; b < ncta; b += 32) {
                        const ulonglong2 v = __ldcg(reinterpret_cast<const ulonglong2*>(a.partials + 2 * ((size_t)b * a.npe_max + pi)));
                        s = f2_add(s, f2(v.x, v.y));
                    }
                    s = warp_sum(s);
                    if (lane == 0) cta_s[pi] = f2_add(cta_s[pi], s);
                }
                __syncthreads();
            }
            if (warp == 0) {
                __syncwarp();
                if (lane < hlk::SC_MAX_POINTS) {
                    fp2 s = f2(0, 0);
                    const u32 pi = skip && lane > 1 ? lane - 1 : lane;
                    if (pi < npe && !(skip && lane == 1)) s = cta_s[pi];
                    reinterpret_cast<fp2*>(sm.sums)[lane] = s;
                }
                __syncwarp();
                r = step_challenge(sa, sm, j, claim, g, lane);
                if (lane == 0) {
                    r_s = r;
                    if (ncta > 1) {
                        st2(a.sync->r[rd & 1], r);
                        st_release(&a.sync->flag, rd + 1);
                    }
                }
            }
            __syncthreads();
        }
        ncta_prev = ncta;
        len = half;
    }
    // the last challenge's fold, and CTA 0's state
    if (cta != 0) {
        if (tid == 0) {
            u32 f = 0;
            for (u32 n = 0; n < POLL_LIMIT && (f = ld_acquire(&a.sync->flag)) < a.nrounds; n++) {}
            if (f < a.nrounds || f == FLAG_FAILED) failed_s = 1;
            else r_s = ld2(a.sync->r[(a.nrounds - 1) & 1]);
        }
        __syncthreads();
        if (failed_s) return;
    }
    r = r_s;
    if (cta == 0 && warp == 0) step_after(sa, sm, a.step.round + (int)a.nrounds - 1, r, lane);
    for (u32 c0 = cta * C; c0 < len; c0 += ncta_prev * C) {
        const u32 cn = min(C, len - c0), lcn = __ffs((int)cn) - 1, st = second ? C / 2 : C;
        const fp2* b = second ? buf1 : buf0;
        for (u32 x = tid; x < a.k * cn; x += T) {
            const u32 t = x >> lcn, i = x & (cn - 1);
            u64* p = a.tables + 2 * ((size_t)t * a.stride + c0 + i);
            fp2 lo, hi;
            if (resident) { lo = b[(size_t)t * a.planes * st + i]; hi = b[((size_t)t * a.planes + 1) * st + i]; }
            else { lo = ld2(p); hi = ld2(p + 2 * (size_t)len); }
            st2(p, f2_add(lo, f2_mul(r, f2_sub(hi, lo))));
        }
    }
    if (cta == 0) {
        __syncthreads();
        const u32* src = reinterpret_cast<const u32*>(&st_s);
        u32* dst = reinterpret_cast<u32*>(a.step.state);
        for (u32 i = tid; i < sizeof(hlk::ScState) / 4; i += T) dst[i] = src[i];
    }
}

constexpr size_t RUN_SMEM = 200 * 1024;
constexpr size_t RUN_CODE = 64 * 1024;

// How much of a round fits one CTA: the larger chunk with every point's values, then less of both; a task per thread group where the
// threads suffice, several passes otherwise.
struct RunShape {
    u32 chunk, planes, parts, threads;
    bool slots_global, code_fits;
    size_t smem;
};
RunShape run_shape(int poly, const hlk::IrDev& p, int k, int eval_degree) {
    RunShape s;
    const u32 points = (u32)eval_degree + 1, usual = eval_degree > 0 ? (u32)eval_degree : 1u;  // the point 1 comes from the claim
    const bool is_ir = poly == hlk::POLY_IR;
    s.parts = is_ir ? p.parts : 1u;
    const size_t fixed = is_ir ? (((size_t)p.n_code * 8 + 15) & ~(size_t)15) + (size_t)p.n_coefs * 16 : 0;
    s.code_fits = fixed <= RUN_CODE;
    for (int pass = 0; pass < 4; pass++) {
        s.chunk = pass == 0 ? 64 : 32;
        s.planes = pass < 2 && points > 2 ? points : 2;
        s.slots_global = pass == 3;
        u32 groups = usual * s.parts, most = RUN_MAX_T / s.chunk;
        if (groups > most) groups = most;
        while (groups * RUN_PASSES < points * s.parts) groups++;
        s.threads = s.chunk * groups;
        if (s.threads < 64) s.threads = 64;  // CTA 0 folds with all warps but one
        const size_t slots = is_ir && !s.slots_global ? (size_t)vm::slot_entries(p.p_slots, p.a_slots, 1) * s.threads * 16 : 0;
        s.smem = (s.code_fits ? fixed : 0) + slots + (size_t)k * s.planes * s.chunk * 24;
        if (pass == 0 && groups < usual * s.parts) continue;  // the smaller chunk has a thread group for every task
        if (s.smem <= RUN_SMEM) break;
    }
    return s;
}

template <class Eval>
cudaError_t launch_run(const RunArgs& a, const Eval& ev, const RunShape& sh, int sm_count, cudaStream_t st) {
    const u32 want = (a.len / 2 + sh.chunk - 1) / sh.chunk;
    const u32 grid = want < 1 ? 1u : want > (u32)sm_count ? (u32)sm_count : want;
    if (sh.smem > 24 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(k_sc_run<Eval>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh.smem);
        if (e != cudaSuccess) return e;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(sh.threads);
    cfg.dynamicSmemBytes = sh.smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    if (grid > 1) {  // the CTAs wait for one another: all of them resident, or the launch is refused
        at[0].id = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
    } else {
        at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[0].val.programmaticStreamSerializationAllowed = 1;
    }
    cfg.attrs = at;
    cfg.numAttrs = grid > 1 || hlk::sc_dependent_launch() ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, k_sc_run<Eval>, a, ev);
}

}  // namespace

namespace hlk {

// Where a round is down at its latencies: 2^13 pairs are one chunk for most of the SMs.  Above it the rounds are launches of their own,
// whose evaluation has every thread and register of the SM.
u32 sc_run_len(int) { return 1u << 14; }

size_t sc_run_partial_bytes(int eval_degree, int sm_count) { return (size_t)sm_count * (eval_degree + 1) * 16; }

size_t sc_run_slot_bytes(int poly, const IrDev& p, int k, int eval_degree, int sm_count) {
    if (poly != POLY_IR) return 0;
    const RunShape s = run_shape(poly, p, k, eval_degree);
    return s.slots_global ? (size_t)vm::slot_entries(p.p_slots, p.a_slots, 1) * s.threads * 16 * sm_count : 0;
}

cudaError_t sc_run(int poly, const IrDev& p, int k, u64* tables, size_t stride, u32 len, const u64* coefs, const ScStep& step, int nrounds, int have_claim,
                   ScSync* sync, u64* partials, u64* slots, int sm_count, cudaStream_t st) {
    RunArgs a;
    a.tables = tables; a.stride = stride; a.len = len; a.k = (u32)k; a.nrounds = (u32)nrounds; a.npe_max = (u32)step.eval_degree + 1;
    a.have_claim = have_claim; a.step = step; a.sync = sync; a.partials = partials;
    const RunShape sh = run_shape(poly, p, k, step.eval_degree);
    a.chunk = sh.chunk; a.planes = sh.planes; a.parts = sh.parts;
    if (poly == POLY_IR) {
        ProgramEval ev;
        ev.p = p; ev.slots_g = sh.slots_global ? reinterpret_cast<fp2*>(slots) : nullptr; ev.code_fits = sh.code_fits;
        ev.code = nullptr; ev.cf = nullptr; ev.slots = nullptr;
        return launch_run(a, ev, sh, sm_count, st);
    }
#define R(P, K) return launch_run(a, ClosedEval<P, K>{coefs}, sh, sm_count, st)
    switch (poly) {
        case POLY_PROD:
            switch (k) {
                case 1: R(POLY_PROD, 1);
                case 2: R(POLY_PROD, 2);
                case 3: R(POLY_PROD, 3);
                case 4: R(POLY_PROD, 4);
                case 5: R(POLY_PROD, 5);
                case 6: R(POLY_PROD, 6);
            }
            break;
        case POLY_ZC: R(POLY_ZC, 4);
        case POLY_LOGUP_Q: R(POLY_LOGUP_Q, 3);
        case POLY_LOGUP_T: R(POLY_LOGUP_T, 4);
    }
#undef R
    return cudaErrorInvalidValue;
}

}  // namespace hlk
