// Sumcheck kernels: round polynomial, Fiat-Shamir step, table fold (sumcheck/rounds.rs:94-160).
//
// Tables are k arrays of `stride` Fp2 (16 bytes each); the live part of a table is its first
// `len` entries.  Variable 0 is the most significant index bit, so round j pairs entry i with
// entry i + len/2, and the fold writes the first half in place.
//
// A round of its own launches is two of them:
// k_sc_round   one grid pass over the pairs: each thread evaluates the slot polynomial at the points 0..D by repeated addition of
//              (T(i+half) - T(i)) and keeps D+1 running sums; warp-shuffle tree, then a shared-memory tree across warps, one partial
//              row per CTA.  The CTA that finishes last adds the rows up and takes the Fiat-Shamir step (sc_step.cuh).
//              A CTA beside them brings the claim and the mask up to the challenge before.
// k_sc_fold    T[i] += r (T[i+half] - T[i]) for every table.
// The host replays the rounds through its own transcript.  The short rounds are one launch in all (sumcheck_run.cu).
#include "kernels.h"
#include "sc_poly.cuh"
#include "sc_step.cuh"
#include "slot_vm.cuh"

namespace hlk {
bool g_sc_dependent_launch = true;
void sc_set_dependent_launch(bool on) { g_sc_dependent_launch = on; }
bool sc_dependent_launch() { return g_sc_dependent_launch; }
}  // namespace hlk

namespace {

// Programmatic dependent launch: every kernel of a sumcheck is a link of one dependency chain in one stream.  A kernel waits until the
// previous link has completed and its writes are visible (`chain_wait`), and only then lets the next link be scheduled (`chain_next`; its
// CTAs take the SM slots this grid leaves free): what a link does before its own wait may rely on the link before the previous one.  The
// step makes use of that.  Launched without the attribute the two instructions do nothing.  What the chain saves is the launch latency
// between dependent kernels, a few microseconds per link.
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_enter() {
    chain_wait();
    chain_next();
}

template <class... P, class... A>
cudaError_t chain_launch(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = hlk::g_sc_dependent_launch ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, P(args)...);
}


using hlk::ScStep;

__device__ __forceinline__ u64 shfl_down64(u64 v, int d) {
    u32 lo = __shfl_down_sync(0xffffffffu, (u32)v, d), hi = __shfl_down_sync(0xffffffffu, (u32)(v >> 32), d);
    return ((u64)hi << 32) | lo;
}

constexpr int RT = 256;  // threads of a round CTA

__device__ __forceinline__ StepArgs step_args(const ScStep& a, hlk::ScState* state) {
    StepArgs x;
    x.degree = a.degree; x.recover = a.recover; x.fs = a.fs; x.mask_vars = a.mask_vars; x.eval_degree = a.eval_degree;
    x.rows = reinterpret_cast<const fp2*>(a.mask);
    x.tab = reinterpret_cast<const fp2*>(a.mask_tab);
    x.row0 = 0;
    x.inv_den = a.inv_den; x.extrap = a.extrap; x.state = state; x.out = a.out;
    return x;
}

struct FinishSmem {
    StepSmem step;
    hlk::ScState state;
    int last;
};
__device__ __forceinline__ void load_state(const ScStep& a, FinishSmem& fs) {
    for (u32 i = threadIdx.x; i < sizeof(hlk::ScState) / 4; i += blockDim.x) reinterpret_cast<u32*>(&fs.state)[i] = __ldcg(reinterpret_cast<const u32*>(a.state) + i);
}
// by one warp, the sums in fs.step and the state in fs.state
__device__ __forceinline__ void take_step(const ScStep& a, FinishSmem& fs, int lane) {
    const StepArgs x = step_args(a, &fs.state);
    step_head(x, fs.step, lane);
    const fp2 g = fs.state.ahead == a.round + 1 ? fs.state.g[lane & 7] : step_mask(x, a.round, lane);
    step_challenge(x, fs.step, a.round, a.use_claim != 0, g, lane);
    __syncwarp();
    for (u32 i = lane; i < sizeof(hlk::ScState) / 4; i += 32) reinterpret_cast<u32*>(a.state)[i] = reinterpret_cast<const u32*>(&fs.state)[i];
}

// Every CTA of a round ends here: threads w < words hold the CTA's sum of word w (point w / 2).  The last CTA to come takes the step.
// (As a launch of its own the step cost another 6 us a round, and reading a row per CTA 2 us.)
__device__ __forceinline__ void finish_round(const ScStep& a, hlk::ScSync* sync, u32 total, bool mine, u64 word) {
    __shared__ FinishSmem fs;
    const u32 w = threadIdx.x;
    u64(*sums)[4] = sync->sums[a.round & 1];
    if (mine) add_word(&sums[w >> 1][2 * (w & 1)], word);
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        fs.last = atomicAdd(&sync->done, 1u) == total - 1;
        if (fs.last) sync->done = 0;
    }
    __syncthreads();
    if (!fs.last) return;
    __threadfence();
    load_state(a, fs);
    if (w < 2 * hlk::SC_MAX_POINTS) fs.step.sums[w] = take_word(&sums[w >> 1][2 * (w & 1)]);
    __syncthreads();
    if (w < 32) take_step(a, fs, (int)w);
}

// One warp beside a round's CTAs: what the challenge before means for the claim and the mask, and this round's mask values.
__device__ __forceinline__ void step_between(const ScStep& a) {
    const int lane = (int)threadIdx.x;
    if (lane >= 32) return;
    const StepArgs x = step_args(a, a.state);
    step_after(x, lane);
    const fp2 g = step_mask(x, a.round, lane);
    if (lane < hlk::SC_MAX_POINTS) a.state->g[lane] = g;
    if (lane == 0) a.state->ahead = a.round + 1;
    __threadfence();
}

// a round whose sums came as rows from another kernel (the generated ones)
constexpr int STEP_T = 512;
__global__ void __launch_bounds__(STEP_T) k_sc_step(ScStep a) {
    __shared__ FinishSmem fs;
    __shared__ u64 red[STEP_T];
    chain_enter();
    const u32 tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, W = 2 * (a.degree + 1), w = tid & 15;  // W <= 16 words per row
    load_state(a, fs);
    u64 s = 0;
    if (w < W) {
#pragma unroll 4
        for (u32 b = tid >> 4; b < a.nblocks; b += STEP_T / 16) s = gl_add(s, a.partials[(size_t)b * W + w]);
    }
    red[tid] = s;
    __syncthreads();
    if (warp < W) {
        u64 z = red[lane * 16 + warp];
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) z = gl_add(z, shfl_down64(z, off));
        if (lane == 0) fs.step.sums[warp] = z;
    }
    __syncthreads();
    if (warp == 0) {
        step_after(step_args(a, &fs.state), (int)lane);
        take_step(a, fs, (int)lane);
    }
}

template <int POLY, int K, int D>
__global__ void __launch_bounds__(RT) k_sc_round(const u64* __restrict__ tables, size_t stride, u32 half, const u64* __restrict__ coefs,
                                                 int eval_one, ScStep step, hlk::ScSync* sync) {
    chain_enter();
    if (blockIdx.x == step.nblocks) {
        step_between(step);
        finish_round(step, sync, gridDim.x, false, 0);
        return;
    }
    fp2 acc[D + 1];
#pragma unroll
    for (int d = 0; d <= D; d++) acc[d] = f2(0, 0);
    const fp2* cf = reinterpret_cast<const fp2*>(coefs);
    for (u32 i = blockIdx.x * RT + threadIdx.x; i < half; i += step.nblocks * RT) {
        fp2 cur[K], dif[K];
#pragma unroll
        for (int t = 0; t < K; t++) {
            const u64* tb = tables + 2 * (size_t)t * stride;
            cur[t] = ld2(tb + 2 * (size_t)i);
            dif[t] = f2_sub(ld2(tb + 2 * ((size_t)i + half)), cur[t]);
        }
        acc[0] = f2_add(acc[0], hlk::poly_eval<POLY, K>(cur, cf));
#pragma unroll
        for (int d = 1; d <= D; d++) {
#pragma unroll
            for (int t = 0; t < K; t++) cur[t] = f2_add(cur[t], dif[t]);
            if (d != 1 || eval_one) acc[d] = f2_add(acc[d], hlk::poly_eval<POLY, K>(cur, cf));
        }
    }
    // warp tree
#pragma unroll
    for (int d = 0; d <= D; d++) {
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) {
            acc[d].c0 = gl_add(acc[d].c0, shfl_down64(acc[d].c0, off));
            acc[d].c1 = gl_add(acc[d].c1, shfl_down64(acc[d].c1, off));
        }
    }
    __shared__ u64 wsum[RT / 32][2 * (D + 1)];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) {
#pragma unroll
        for (int d = 0; d <= D; d++) { wsum[warp][2 * d] = acc[d].c0; wsum[warp][2 * d + 1] = acc[d].c1; }
    }
    __syncthreads();
    u64 s = 0;
    if (threadIdx.x < 2 * (D + 1)) {
#pragma unroll
        for (int w = 0; w < RT / 32; w++) s = gl_add(s, wsum[w][threadIdx.x]);
    }
    finish_round(step, sync, gridDim.x, threadIdx.x < 2 * (D + 1), s);
}


// the first entry of every table, in a row: one read-back for all of them
__global__ void __launch_bounds__(64) k_sc_finals(const u64* __restrict__ tables, size_t stride, u32 k, u64* __restrict__ out) {
    chain_enter();
    if (threadIdx.x < k) st2(out + 2 * threadIdx.x, ld2(tables + 2 * (size_t)threadIdx.x * stride));
}

// which tables are extension-valued: one CTA row per table, the second words OR-ed
__global__ void __launch_bounds__(256) k_sc_nonbase(const u64* __restrict__ tables, size_t stride, size_t len, u64* __restrict__ mask) {
    const u32 t = blockIdx.y;
    const u64* tb = tables + 2 * (size_t)t * stride;
    u64 any = 0;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < len; i += (size_t)gridDim.x * blockDim.x) any |= tb[2 * i + 1];
    if (__syncthreads_or(any != 0) && threadIdx.x == 0) atomicOr(mask, 1ull << t);
}

__global__ void __launch_bounds__(256) k_sc_fold(u64* __restrict__ tables, size_t stride, u32 half, const hlk::ScState* __restrict__ st) {
    chain_enter();
    const u32 i = blockIdx.x * blockDim.x + threadIdx.x, t = blockIdx.y;
    if (i >= half) return;
    const fp2 r = st->r;
    u64* tb = tables + 2 * (size_t)t * stride;
    fp2 a = ld2(tb + 2 * (size_t)i), b = ld2(tb + 2 * ((size_t)i + half));
    st2(tb + 2 * (size_t)i, f2_add(a, f2_mul(r, f2_sub(b, a))));
}

// the same for a batch that ends with a round of its own launches
__global__ void __launch_bounds__(32) k_sc_between(ScStep a) {
    chain_enter();
    step_between(a);
}

// ---------------------------------------------------------------------------------------------
// Slot polynomials given as data: the long rounds, one pair per thread (or NPT of its points), the polynomial as a program (slot_vm.cuh)
// ---------------------------------------------------------------------------------------------
constexpr int VMT = 128;
template <int NPT>
__global__ void __launch_bounds__(VMT) k_sc_round_vm(const u64* __restrict__ tables, size_t stride, u32 half, hlk::IrDev p, int degree, u32 npe, bool skip,
                                                     fp2* __restrict__ slots_g, ScStep step, hlk::ScSync* sync) {
    chain_enter();
    const u32 columns = gridDim.x - step.between;
    if (blockIdx.x == columns) {
        if (blockIdx.y == 0 && blockIdx.z == 0) step_between(step);
        finish_round(step, sync, gridDim.x * gridDim.y * gridDim.z, false, 0);
        return;
    }
    extern __shared__ __align__(16) char vm_smem[];
    __shared__ u64 wsum[VMT / 32][2 * NPT];
    u64* code = reinterpret_cast<u64*>(vm_smem);
    fp2* cf = reinterpret_cast<fp2*>(vm_smem + (((size_t)p.n_code * 8 + 15) & ~(size_t)15));
    for (u32 x = threadIdx.x; x < p.n_code; x += VMT) code[x] = p.code[x];
    for (u32 x = threadIdx.x; x < p.n_coefs; x += VMT) cf[x] = ld2(p.coefs + 2 * (size_t)x);
    const u32 entries = vm::slot_entries(p.p_slots, p.a_slots, NPT), row = blockIdx.z * columns + blockIdx.x;
    fp2* slots = (slots_g ? slots_g + (size_t)(blockIdx.y * columns * gridDim.z + row) * entries * VMT : cf + p.n_coefs) + threadIdx.x;
    // the whole program, or a share of its parts
    const u32 whole = gridDim.z == 1, part1 = whole ? 1u : p.parts;
    __syncthreads();
    const u32 e0 = blockIdx.y * NPT;  // this thread's first evaluated point, by its position among them
    const u32 first = skip && e0 ? e0 + 1 : e0;
    fp2 acc[NPT];
#pragma unroll
    for (int j = 0; j < NPT; j++) acc[j] = f2(0, 0);
    for (u32 i = blockIdx.x * VMT + threadIdx.x; i < half; i += columns * VMT)
    for (u32 part = blockIdx.z; part < part1; part += gridDim.z) {
        const u64* prog = whole ? code : code + p.start[part];
        fp2 x[NPT];
        if constexpr (NPT == 1) {
            x[0] = vm::eval_one(
                prog, cf,
                [&](u32 t) {
                    const u64* tb = tables + 2 * ((size_t)t * stride + i);
                    const fp2 lo = ld2(tb), d = f2_sub(ld2(tb + 2 * (size_t)half), lo);
                    fp2 v = lo;
                    for (u32 q = 0; q < first; q++) v = f2_add(v, d);
                    return v;
                },
                slots, VMT, p.p_slots);
        } else {
            vm::eval<NPT>(
                prog, cf,
                [&](u32 t, fp2& lo, fp2& hi) {
                    const u64* tb = tables + 2 * ((size_t)t * stride + i);
                    lo = ld2(tb);
                    hi = ld2(tb + 2 * (size_t)half);
                },
                slots, VMT, p.p_slots * NPT, first, skip, x);
        }
#pragma unroll
        for (int j = 0; j < NPT; j++) acc[j] = f2_canon(f2_add_lazy(x[j], acc[j]));
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int j = 0; j < NPT; j++) {
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) {
            acc[j].c0 = gl_add(acc[j].c0, shfl_down64(acc[j].c0, off));
            acc[j].c1 = gl_add(acc[j].c1, shfl_down64(acc[j].c1, off));
        }
        if (lane == 0) { wsum[warp][2 * j] = acc[j].c0; wsum[warp][2 * j + 1] = acc[j].c1; }
    }
    __syncthreads();
    // the points nobody evaluates stay zero
    const u32 w = threadIdx.x, pt = w >> 1, e = skip && pt ? pt - 1 : pt;
    const bool mine = pt < npe + skip && !(skip && pt == 1) && e >= e0 && e < e0 + NPT;
    u64 sum = 0;
    if (mine) {
        for (int v = 0; v < VMT / 32; v++) sum = gl_add(sum, wsum[v][2 * (e - e0) + (w & 1)]);
    }
    finish_round(step, sync, gridDim.x * gridDim.y * gridDim.z, mine, sum);
}

// points per thread and threads per pair for `npe` evaluated points
u32 vm_npt(u32 npe) { return npe <= (u32)vm::MAX_NPT ? npe : (npe + 1) / 2; }
size_t vm_fixed_bytes(const hlk::IrDev& p) { return (((size_t)p.n_code * 8 + 15) & ~(size_t)15) + (size_t)p.n_coefs * 16; }
// A thread per pair, at most four CTAs of them per SM (that many fit); where the pairs fill less than that, a pair's parts go to threads
// of their own.
struct VmGrid { u32 blocks, parts; };
VmGrid vm_grid(const hlk::IrDev& p, u32 half, int sm_count) {
    const u32 cap = (u32)sm_count * 4, b = (half + VMT - 1) / VMT;
    VmGrid g{b < 1 ? 1u : b > cap ? cap : b, 1u};
    g.parts = cap / g.blocks < p.parts ? cap / g.blocks : p.parts;
    return g;
}
constexpr size_t VM_SLOT_SMEM = 40 * 1024;  // above this the slots of a CTA go to global memory

template <int NPT>
cudaError_t launch_vm(const hlk::IrDev& p, const u64* tables, size_t stride, u32 half, int degree, u32 npe, bool skip, u64* slots, VmGrid g,
                      const ScStep& step, hlk::ScSync* sync, cudaStream_t s) {
    const size_t slot_bytes = (size_t)vm::slot_entries(p.p_slots, p.a_slots, NPT) * VMT * 16;
    const size_t smem = vm_fixed_bytes(p) + (slots ? 0 : slot_bytes);
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(k_sc_round_vm<NPT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    return chain_launch(k_sc_round_vm<NPT>, dim3(g.blocks + (step.between ? 1 : 0), (npe + NPT - 1) / NPT, g.parts), dim3(VMT), smem, s, tables, stride, half, p, degree, npe, skip,
                        reinterpret_cast<fp2*>(slots), step, sync);
}

template <int POLY, int K, int D>
cudaError_t launch_round(const u64* tables, size_t stride, u32 half, const u64* coefs, int eval_one, const ScStep& step, hlk::ScSync* sync, cudaStream_t s) {
    chain_launch(k_sc_round<POLY, K, D>, dim3(step.nblocks + (step.between ? 1 : 0)), dim3(RT), 0, s, tables, stride, half, coefs, eval_one, step, sync);
    return cudaGetLastError();
}

}  // namespace

namespace hlk {

u32 sc_round_blocks(u32 half, int sm_count) {
    u32 b = (half + RT - 1) / RT, cap = (u32)sm_count * 4;
    if (b < 1) b = 1;
    return b > cap ? cap : b;
}

// bytes of global memory for the slots of any round's grid, 0 where they fit shared memory
size_t sc_ir_slot_bytes(const IrDev& p, int sm_count) {
    size_t most = 0;
    for (u32 npe = p.eval_degree; npe <= p.eval_degree + 1; npe++) {
        if (npe == 0) continue;
        const u32 npt = vm_npt(npe);
        const size_t cta = (size_t)vm::slot_entries(p.p_slots, p.a_slots, (int)npt) * VMT * 16, all = cta * sm_count * 4 * ((npe + npt - 1) / npt);
        if (cta > VM_SLOT_SMEM && all > most) most = all;
    }
    return most;
}

cudaError_t sc_round_ir(const IrDev& p, const u64* tables, size_t stride, u32 half, int degree, int eval_one, u64* slots, int sm_count, const ScStep& step, ScSync* sync,
                        cudaStream_t s) {
    const bool skip = !eval_one && p.eval_degree >= 1;
    const u32 npe = p.eval_degree + (skip ? 0u : 1u), npt = vm_npt(npe);
    const size_t cta = (size_t)vm::slot_entries(p.p_slots, p.a_slots, (int)npt) * VMT * 16;
    u64* sl = cta > VM_SLOT_SMEM ? slots : nullptr;
    const VmGrid g = vm_grid(p, half, sm_count);
    switch (npt) {
        case 1: return launch_vm<1>(p, tables, stride, half, degree, npe, skip, sl, g, step, sync, s);
        case 2: return launch_vm<2>(p, tables, stride, half, degree, npe, skip, sl, g, step, sync, s);
        case 3: return launch_vm<3>(p, tables, stride, half, degree, npe, skip, sl, g, step, sync, s);
        case 4: return launch_vm<4>(p, tables, stride, half, degree, npe, skip, sl, g, step, sync, s);
        case 5: return launch_vm<5>(p, tables, stride, half, degree, npe, skip, sl, g, step, sync, s);
    }
    return cudaErrorInvalidValue;
}

bool sc_supported(int poly, int k, int degree) {
    if (poly == POLY_IR) return k >= 1 && k <= (int)ir::MAX_TABLES && degree >= 1 && degree < SC_MAX_POINTS;
    if (poly == POLY_PROD) return k >= 1 && k <= 6 && degree == k;
    if (poly == POLY_ZC || poly == POLY_LOGUP_T) return k == 4 && degree == 3;
    if (poly == POLY_LOGUP_Q) return k == 3 && degree == 3;
    return false;
}

cudaError_t sc_round(int poly, int k, const u64* tables, size_t stride, u32 half, const u64* coefs, int eval_one, const ScStep& step, ScSync* sync,
                     cudaStream_t s) {
#define R(P, K, D) return launch_round<P, K, D>(tables, stride, half, coefs, eval_one, step, sync, s)
    switch (poly) {
        case POLY_PROD:
            switch (k) {
                case 1: R(POLY_PROD, 1, 1);
                case 2: R(POLY_PROD, 2, 2);
                case 3: R(POLY_PROD, 3, 3);
                case 4: R(POLY_PROD, 4, 4);
                case 5: R(POLY_PROD, 5, 5);
                case 6: R(POLY_PROD, 6, 6);
            }
            break;
        case POLY_ZC: R(POLY_ZC, 4, 3);
        case POLY_LOGUP_Q: R(POLY_LOGUP_Q, 3, 3);
        case POLY_LOGUP_T: R(POLY_LOGUP_T, 4, 3);
    }
#undef R
    return cudaErrorInvalidValue;
}

cudaError_t sc_step(const ScStep& a, cudaStream_t s) {
    chain_launch(k_sc_step, dim3(1), dim3(STEP_T), 0, s, a);
    return cudaGetLastError();
}


cudaError_t sc_between(const ScStep& a, cudaStream_t s) { return chain_launch(k_sc_between, dim3(1), dim3(32), 0, s, a); }

cudaError_t sc_nonbase_mask(const u64* tables, size_t stride, size_t len, u32 k, u64* d_mask, int sm_count, cudaStream_t s) {
    size_t bx = (len + 255) / 256, cap = (size_t)sm_count * 8 / (k ? k : 1) + 1;
    if (bx > cap) bx = cap;
    k_sc_nonbase<<<dim3((unsigned)bx, k), 256, 0, s>>>(tables, stride, len, d_mask);
    return cudaGetLastError();
}

cudaError_t sc_finals(const u64* d_tables, size_t stride, u32 k, u64* d_out, cudaStream_t st) {  // k <= 64
    return chain_launch(k_sc_finals, dim3(1), dim3(64), 0, st, d_tables, stride, k, d_out);
}

cudaError_t sc_fold(u64* tables, size_t stride, u32 half, u32 k, const ScState* st, cudaStream_t s) {
    return chain_launch(k_sc_fold, dim3((half + 255) / 256, k), dim3(256), 0, s, tables, stride, half, st);
}

}  // namespace hlk
