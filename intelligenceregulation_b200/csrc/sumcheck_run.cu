// The short rounds of a sumcheck in ONE launch.
//
// Once a round has some thousands of pairs, what it waits for is not arithmetic: as separate launches (sums, Fiat-Shamir step, fold) a
// round of 2^13 pairs and one of two took the same 25 us.  k_sc_run keeps the CTAs resident (a cooperative launch) and runs all of the
// remaining rounds: per round a CTA folds its pairs with the last challenge on the way in, evaluates them one (pair, evaluation point)
// per thread, and hands its sums to CTA 0, one warp of which takes the Fiat-Shamir step and publishes the challenge.
//
//   units       a CTA has a chunk of pairs and one part of the polynomial (slot_vm.cuh; a closed form is one part).  The folded tables go
//               from one buffer to the other, so that the CTAs of a chunk's parts can all fold it for themselves (part 0's CTA stores it)
//               and nothing but the challenge is waited for.
//   shrinking   a round with fewer units than CTAs lets the others go; once a single CTA is left it keeps the tables in shared memory
//   the step    has a warp of its own, which prepares the mask before the sums arrive and updates the claim while the others fold and
//               evaluate (sc_step.cuh): a round of two pairs is 5.5 k cycles of hashing and 4 k of everything else
// Every wait is bounded: a CTA that waits too long records it for the host and leaves, and the call returns HL_B200_ERR_TIMEOUT.
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
constexpr u32 FLAG_FAILED = 0xFFFFFFFFu;

struct RunArgs {
    u64* tables;         // where the tables are, and where the last fold leaves them
    u64* other;          // the other buffer: k tables of len / 2 entries
    size_t stride;
    u32 len;             // live entries per table at the first round
    u32 k, nrounds, chunk, planes, parts;
    int have_claim;      // the first round's claim is known
    hlk::ScStep step;    // step.round: the first round's number
    hlk::ScSync* sync;   // zero at the launch
    hlk::ScWaits waits;
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

constexpr u32 RUN_MAX_T = 384;  // working threads (64 pairs of the six-table product); one more warp takes the step
constexpr u32 RUN_PASSES = 2;

// the working threads alone
__device__ __forceinline__ void bar_workers(u32 threads) { asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory"); }

template <class Eval>
__global__ void __launch_bounds__(RUN_MAX_T + 32) k_sc_run(RunArgs a, Eval ev) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    extern __shared__ __align__(16) char smem[];
    __shared__ StepSmem sm;
    __shared__ hlk::ScState st_s;
    __shared__ __align__(16) u64 rows_s[2 * 63 * (hlk::SC_MAX_POINTS - 1)];
    __shared__ __align__(16) u64 tab_s[2 * 63 * hlk::SC_MAX_POINTS];
    __shared__ u64 invden_s[hlk::SC_MAX_POINTS], extrap_s[hlk::SC_MAX_POINTS * hlk::SC_MAX_POINTS];
    __shared__ fp2 task_s[RUN_PASSES * RUN_MAX_T / 32];  // one sum per warp and pass: [point][warp of the chunk]
    __shared__ fp2 cta_s[hlk::SC_MAX_POINTS];
    __shared__ fp2 r_s;
    __shared__ u32 failed_s;
    const u32 T = blockDim.x - 32, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, cta = blockIdx.x, C = a.chunk;
    const bool worker = tid < T, first = cta == 0;
    const u32 part = cta % a.parts, owner = cta / a.parts;  // this CTA's part, and its number among that part's CTAs
    const int degree = a.step.degree, np = degree + 1;
    if (!worker && !first) return;  // the step is CTA 0's
    const u32 own = ev.stage(smem, T);
    fp2* const buf0 = reinterpret_cast<fp2*>(smem + own);
    fp2* const buf1 = buf0 + (size_t)a.k * a.planes * C;  // with half the stride: it only ever holds the rounds after the first one
    StepArgs sa;
    sa.degree = degree; sa.recover = a.step.recover; sa.fs = 1; sa.mask_vars = a.step.mask_vars; sa.eval_degree = a.step.eval_degree;
    sa.rows = a.step.mask ? reinterpret_cast<const fp2*>(rows_s) : nullptr;
    sa.tab = reinterpret_cast<const fp2*>(tab_s);
    sa.row0 = 0;
    sa.inv_den = invden_s; sa.extrap = a.step.extrap ? extrap_s : nullptr; sa.state = &st_s; sa.out = a.step.out;
    if (tid == 0) failed_s = 0;
    if (first) {
        const u32 all = T + 32;
        const u32* src = reinterpret_cast<const u32*>(a.step.state);
        u32* dst = reinterpret_cast<u32*>(&st_s);
        for (u32 i = tid; i < sizeof(hlk::ScState) / 4; i += all) dst[i] = src[i];
        if (a.step.mask) {
            const u32 nr = 2u * a.step.mask_vars * degree, nt = 2u * a.step.mask_vars * np;
            for (u32 i = tid; i < nr; i += all) rows_s[i] = a.step.mask[i];
            for (u32 i = tid; i < nt; i += all) tab_s[i] = a.step.mask_tab[i];
        }
        if ((int)tid < np) invden_s[tid] = a.step.inv_den[tid];
        if (a.step.extrap && (int)tid < (degree - a.step.eval_degree) * (a.step.eval_degree + 1)) extrap_s[tid] = a.step.extrap[tid];
        __syncthreads();
    } else {
        bar_workers(T);
    }

    if (!worker) {  // ---- CTA 0's last warp: the steps
        for (u32 rd = 0; rd < a.nrounds; rd++) {
            const int j = a.step.round + (int)rd;
            const bool claim = a.step.recover && (rd > 0 || a.have_claim), skip = claim && a.step.eval_degree >= 1;
            const u32 npe = a.step.eval_degree + (skip ? 0 : 1);
            step_after(sa, lane);
            step_head(sa, sm, lane);
            const fp2 g = step_mask(sa, j, lane);
            __syncthreads();  // the sums are there
            if (failed_s) return;
            if (lane < hlk::SC_MAX_POINTS) {
                fp2 s = f2(0, 0);
                const u32 pi = skip && lane > 1 ? lane - 1 : lane;
                if (pi < npe && !(skip && lane == 1)) s = cta_s[pi];
                reinterpret_cast<fp2*>(sm.sums)[lane] = s;
            }
            __syncwarp();
            const fp2 r = step_challenge(sa, sm, j, claim, g, lane);
            if (lane == 0) {
                r_s = r;
                if (gridDim.x > 1) {
                    st2(a.sync->r[rd & 1], r);
                    st_release(&a.sync->flag, rd + 1);
                }
            }
            __syncthreads();  // the challenge is there
        }
        step_after(sa, lane);
        __syncwarp();
        const u32* src = reinterpret_cast<const u32*>(&st_s);
        u32* dst = reinterpret_cast<u32*>(a.step.state);
        for (u32 i = lane; i < sizeof(hlk::ScState) / 4; i += 32) dst[i] = src[i];
        return;
    }

    // ---- the working threads
    fp2 r = f2(0, 0);
    // the challenge of round rd; false: the wait ran out
    auto challenge = [&](u32 rd) {
        if (!first) {
            if (tid == 0) {
                u32 f = 0;
                for (u32 n = 0; n < a.waits.challenge && (f = ld_acquire(&a.sync->flag)) < rd + 1; n++) {}
                if (f < rd + 1) {  // ran out: our entries stay unfolded, also when CTA 0 has nothing more to wait for
                    failed_s = 1;
                    a.sync->failed = 1;
                    st_release(&a.sync->flag, FLAG_FAILED);
                } else if (f == FLAG_FAILED) {
                    failed_s = 1;
                } else {
                    r_s = ld2(a.sync->r[rd & 1]);
                }
            }
            bar_workers(T);
            if (failed_s) return false;
        }
        r = r_s;
        return true;
    };
    u32 len = a.len, arrived = 0, owners = 1;
    bool resident = false, second = false;  // the tables live in a shared buffer (one CTA): in the second one
    u64 *from_g = a.tables, *to_g = a.other;
    size_t from_stride = a.stride, to_stride = a.len / 2;
    for (u32 rd = 0; rd < a.nrounds; rd++) {
        const u32 half = len >> 1, chunks = (half + C - 1) / C;
        owners = min(gridDim.x / a.parts, chunks);
        const u32 ncta = owners * a.parts;
        // nothing of this round or a later one is ours: our entries, folded with every challenge but the last, are in the tables
        if (cta >= ncta) return;
        if (rd > 0 && !challenge(rd - 1)) return;
        const bool claim = a.step.recover && (rd > 0 || a.have_claim), skip = claim && a.step.eval_degree >= 1;
        const u32 npe = a.step.eval_degree + (skip ? 0 : 1);
        // one evaluation point per thread, for all pairs of a chunk; a warp lies within one point
        const u32 tslots = T / C, my = tid / C, ti = tid - my * C;
        fp2 acc[RUN_PASSES];
#pragma unroll
        for (u32 q = 0; q < RUN_PASSES; q++) acc[q] = f2(0, 0);
        for (u32 c0 = owner * C; c0 < half; c0 += owners * C) {
            const u32 cn = min(C, half - c0), lcn = __ffs((int)cn) - 1;  // powers of two, all of them
            if (c0 != owner * C) bar_workers(T);  // the chunk before has been evaluated
            const bool to2 = resident && !second;
            fp2* to = to2 ? buf1 : buf0;
            const u32 ts_to = to2 ? C / 2 : C, ts_from = second ? C / 2 : C;
            auto stage = [&](u32 t, u32 i, const fp2 (&v)[2]) {  // the pair's two entries, c0 + i and c0 + i + half of the table
                fp2* o = to + (size_t)t * a.planes * ts_to + i;
                o[0] = v[0];
                o[ts_to] = v[1];
                if (a.planes > 2) {
                    const fp2 d = f2_sub(v[1], v[0]);
                    fp2 y = v[1];
                    for (u32 p = 2; p < a.planes; p++) { y = f2_add(y, d); o[p * ts_to] = y; }
                }
            };
            const u32 items = a.k * cn;
            if (resident) {
                for (u32 x = tid; x < items; x += T) {
                    const u32 t = x >> lcn, i = x & (cn - 1);
                    const fp2* from = (second ? buf1 : buf0) + (size_t)t * a.planes * ts_from + i;
                    fp2 v[2];
#pragma unroll
                    for (u32 e = 0; e < 2; e++) {
                        const fp2 lo = from[e * half];
                        v[e] = f2_add(lo, f2_mul(r, f2_sub(from[ts_from + e * half], lo)));
                    }
                    stage(t, i, v);
                }
            } else {
                // the loads of the next item (an L2 latency each) are under way while this one is folded
                fp2 nx[4];
                auto fetch = [&](u32 x) {
                    if (x >= items) return;
                    const u64* p = from_g + 2 * ((size_t)(x >> lcn) * from_stride + c0 + (x & (cn - 1)));
                    nx[0] = ld2(p);
                    nx[1] = ld2(p + 2 * (size_t)half);
                    if (rd > 0) { nx[2] = ld2(p + 2 * (size_t)len); nx[3] = ld2(p + 2 * ((size_t)half + len)); }
                };
                fetch(tid);
                for (u32 x = tid; x < items; x += T) {
                    const u32 t = x >> lcn, i = x & (cn - 1);
                    fp2 v[2] = {nx[0], nx[1]};
                    const fp2 h0 = nx[2], h1 = nx[3];
                    fetch(x + T);
                    if (rd > 0) {
                        v[0] = f2_add(v[0], f2_mul(r, f2_sub(h0, v[0])));
                        v[1] = f2_add(v[1], f2_mul(r, f2_sub(h1, v[1])));
                        if (part == 0 && (a.parts > 1 || half > C)) {
                            u64* o = to_g + 2 * ((size_t)t * to_stride + c0 + i);
                            st2(o, v[0]);
                            st2(o + 2 * (size_t)half, v[1]);
                        }
                    }
                    stage(t, i, v);
                }
            }
            bar_workers(T);
            const TabSmem tab{to, ts_to, a.planes};
#pragma unroll
            for (u32 q = 0; q < RUN_PASSES; q++) {
                const u32 pi = my + q * tslots;
                if (pi < npe && ti < cn) acc[q] = f2_add(acc[q], ev.at(tab, ti, skip && pi ? pi + 1 : pi, part, T));
            }
        }
        if (rd > 0) {  // the folded tables are in the other buffer
            u64* t = from_g; from_g = to_g; to_g = t;
            const size_t st = from_stride; from_stride = to_stride; to_stride = st;
        }
        if (resident) second = !second;
        else if (a.parts == 1 && half <= C) resident = true;
#pragma unroll
        for (u32 q = 0; q < RUN_PASSES; q++) {
            if (q * tslots >= npe) break;
            acc[q] = warp_sum(acc[q]);
            if (lane == 0) task_s[q * (T / 32) + warp] = acc[q];
        }
        bar_workers(T);
        u64(*sums)[4] = a.sync->sums[rd & 1];  // of all CTAs, where there are several
        if (tid < 2 * npe) {
            const u32 pi = tid >> 1, word = tid & 1;
            u64 s = 0;
            for (u32 w = 0; w < C / 32; w++) s = gl_add(s, word ? task_s[pi * (C / 32) + w].c1 : task_s[pi * (C / 32) + w].c0);
            if (first) reinterpret_cast<u64*>(cta_s)[tid] = s;
            else add_word(&sums[pi][2 * word], s);
        }
        if (!first) {
            bar_workers(T);
            if (tid == 0) {
                __threadfence();
                asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&a.sync->arrived) : "memory");
            }
        } else {
            arrived += ncta - 1;
            if (ncta > 1) {
                if (tid == 0) {
                    u32 n = 0;
                    while (n < a.waits.sums && ld_acquire(&a.sync->arrived) < arrived) n++;
                    if (n == a.waits.sums) {
                        failed_s = 1;
                        a.sync->failed = 1;
                        st_release(&a.sync->flag, FLAG_FAILED);
                    }
                }
                bar_workers(T);
                if (tid < 2 * npe) {
                    u64* c = reinterpret_cast<u64*>(cta_s) + tid;
                    *c = gl_add(*c, take_word(&sums[tid >> 1][2 * (tid & 1)]));
                }
            }
            __syncthreads();  // the step takes the sums
            if (failed_s) return;
            __syncthreads();  // and leaves the challenge
        }
        len = half;
    }
    // the last challenge's fold, into `tables`
    if (part != 0 || !challenge(a.nrounds - 1)) return;
    for (u32 c0 = owner * C; c0 < len; c0 += owners * C) {
        const u32 cn = min(C, len - c0), lcn = __ffs((int)cn) - 1, st = second ? C / 2 : C;
        const fp2* b = second ? buf1 : buf0;
        for (u32 x = tid; x < a.k * cn; x += T) {
            const u32 t = x >> lcn, i = x & (cn - 1);
            const u64* p = from_g + 2 * ((size_t)t * from_stride + c0 + i);
            fp2 lo, hi;
            if (resident) { lo = b[(size_t)t * a.planes * st + i]; hi = b[((size_t)t * a.planes + 1) * st + i]; }
            else { lo = ld2(p); hi = ld2(p + 2 * (size_t)len); }
            st2(a.tables + 2 * ((size_t)t * a.stride + c0 + i), f2_add(lo, f2_mul(r, f2_sub(hi, lo))));
        }
    }
}

constexpr size_t RUN_SMEM = 200 * 1024;
constexpr size_t RUN_CODE = 64 * 1024;

// How much of a round fits one CTA.  A closed form stages every point's values; a program's CTAs share an SM, so it steps to them.
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
    // A closed form waits for its folds and hashes: 64 pairs a CTA.  A program waits for its instructions, and four warps, one per
    // scheduler, run them fastest: 32.
    for (int pass = 0; pass < 3; pass++) {
        s.chunk = is_ir ? 32 : 64;
        s.planes = pass < 1 && points > 2 && !is_ir ? points : 2;
        s.slots_global = pass == 2;
        s.threads = s.chunk * usual;
        if (s.threads < 64) s.threads = 64;
        const size_t slots = is_ir && !s.slots_global ? (size_t)vm::slot_entries(p.p_slots, p.a_slots, 1) * s.threads * 16 : 0;
        // the second buffer is for one CTA left over, which a polynomial of several parts never is
        s.smem = (s.code_fits ? fixed : 0) + slots + (size_t)k * s.planes * s.chunk * (s.parts > 1 ? 16 : 24);
        if (s.smem <= RUN_SMEM) break;
    }
    return s;
}

// the largest grid that stays resident, in whole sets of parts
template <class Eval>
cudaError_t run_grid(const RunShape& sh, u32 len, int sm_count, u32* grid) {
    if (sh.smem > 24 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(k_sc_run<Eval>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh.smem);
        if (e != cudaSuccess) return e;
    }
    int per_sm = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_sc_run<Eval>, (int)sh.threads + 32, sh.smem);
    if (e != cudaSuccess) return e;
    if (per_sm > hlk::SC_RUN_CTAS) per_sm = hlk::SC_RUN_CTAS;
    const u32 chunks = (len / 2 + sh.chunk - 1) / sh.chunk, most = (u32)(per_sm * sm_count) / sh.parts;
    *grid = (chunks < 1 ? 1u : chunks > most ? most : chunks) * sh.parts;
    return *grid ? cudaSuccess : cudaErrorInvalidConfiguration;
}

template <class Eval>
cudaError_t launch_run(const RunArgs& a, const Eval& ev, const RunShape& sh, int sm_count, cudaStream_t st) {
    u32 grid;
    cudaError_t e = run_grid<Eval>(sh, a.len, sm_count, &grid);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(sh.threads + 32);
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

// From which length on a round is better off here than with launches of its own: one evaluation point per thread costs a long program a
// third more, a launch costs a short one.  Whole sumchecks of the closed forms (products of two and six tables, the zero check, both LogUp
// checks) over 2^14 .. 2^21 entries and of the 23 recorded programs over 2^12 .. 2^20, from 2^8 .. 2^21 entries on, in us:
//   closed forms           2^18 is the best or within 2 % of it (LogUp over 2^21: 2^14 395, 2^16 376, 2^18 369, 2^20 395)
//   24 instructions        2^13 .. 2^15 within 2 % of one another (over 2^18: 2^11 377, 2^14 365, 2^16 389)
//   3 to 8 instructions    2^14 within 9 % of the best, which is 2^15 or 2^16 (5 over 2^20: 2^11 384, 2^14 372, 2^16 362; 3 over 2^18: 215, 211, 201)
//   59 and more            2^11 within 2 % of the best (59 over 2^16: 347, 2^14 381, 2^16 480; 246 over 2^18: 1,399, 1,531, 1,938)
// The code's length counts the program and its parts: 54 words for those 24 instructions, 125 for the 59.
constexpr u32 RUN_SHORT_CODE = 64;
u32 sc_run_len(int poly, const IrDev& p) { return poly != POLY_IR ? 1u << 18 : p.n_code <= RUN_SHORT_CODE ? 1u << 14 : 1u << 11; }

size_t sc_run_other_bytes(int k, u32 len) { return (size_t)k * (len / 2 ? len / 2 : 1) * 16; }

size_t sc_run_slot_bytes(int poly, const IrDev& p, int k, int eval_degree, int sm_count) {
    if (poly != POLY_IR) return 0;
    const RunShape s = run_shape(poly, p, k, eval_degree);
    return s.slots_global ? (size_t)vm::slot_entries(p.p_slots, p.a_slots, 1) * s.threads * 16 * sm_count * SC_RUN_CTAS : 0;
}

cudaError_t sc_run(int poly, const IrDev& p, int k, u64* tables, size_t stride, u32 len, const u64* coefs, const ScStep& step, int nrounds, int have_claim,
                   ScSync* sync, const ScWaits& waits, u64* slots, u64* other, int sm_count, cudaStream_t st) {
    RunArgs a;
    a.waits = waits;
    a.tables = tables; a.other = other; a.stride = stride; a.len = len; a.k = (u32)k; a.nrounds = (u32)nrounds;
    a.have_claim = have_claim; a.step = step; a.sync = sync;
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
