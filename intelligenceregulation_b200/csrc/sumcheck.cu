// Sumcheck kernels: round polynomial, Fiat-Shamir step, table fold (sumcheck/rounds.rs:94-160).
//
// Tables are k arrays of `stride` Fp2 (16 bytes each); the live part of a table is its first
// `len` entries.  Variable 0 is the most significant index bit, so round j pairs entry i with
// entry i + len/2, and the fold writes the first half in place.
//
// k_sc_round   one grid pass over the pairs: each thread evaluates the slot polynomial at the
//              points 0..D by repeated addition of (T(i+half) - T(i)) and keeps D+1 running sums;
//              warp-shuffle tree, then a shared-memory tree across warps, one partial per CTA.
// k_sc_step    one warp: sums the CTA partials, recovers s(1) from the running claim, adds the
//              CFS mask c*g_j, absorbs "sc-round" into the transcript state, squeezes the
//              challenge, updates the claim and the mask's running terms (transcript.rs:67-148,
//              sumcheck.rs:260-299).  The host replays these rounds through its own transcript.
// k_sc_fold    T[i] += r (T[i+half] - T[i]) for every table, r read from device memory.
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

// Programmatic dependent launch: every kernel of a sumcheck is a link of one dependency chain in one stream.  A kernel opens with
// `chain_enter()`: it lets the next link be scheduled at once (its CTAs take the SM slots this grid leaves free and stop at their own
// wait) and then waits until the previous link has completed and its writes are visible.  Launched without the attribute the two
// instructions do nothing.  What the chain saves is the launch latency between dependent kernels, a few microseconds per link.
__device__ __forceinline__ void chain_enter() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
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

template <int POLY, int K, int D>
__global__ void __launch_bounds__(RT) k_sc_round(const u64* __restrict__ tables, size_t stride, u32 half, const u64* __restrict__ coefs,
                                                 int eval_one, u64* __restrict__ partials) {
    chain_enter();
    fp2 acc[D + 1];
#pragma unroll
    for (int d = 0; d <= D; d++) acc[d] = f2(0, 0);
    const fp2* cf = reinterpret_cast<const fp2*>(coefs);
    for (u32 i = blockIdx.x * RT + threadIdx.x; i < half; i += gridDim.x * RT) {
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
    if (threadIdx.x < 2 * (D + 1)) {
        u64 s = 0;
#pragma unroll
        for (int w = 0; w < RT / 32; w++) s = gl_add(s, wsum[w][threadIdx.x]);
        partials[(size_t)blockIdx.x * 2 * (D + 1) + threadIdx.x] = s;
    }
}

// The CTA partials of a round are summed by all STEP_T threads (independent loads, shared-memory tree);
// warp 0 then runs the Fiat-Shamir step.
constexpr int STEP_T = 512;
__global__ void __launch_bounds__(STEP_T) k_sc_step(ScStep a) {
    chain_enter();
    __shared__ StepSmem sm;
    __shared__ u64 red[STEP_T];
    // everything the serial step reads is fetched by the whole CTA while the partials are summed: the step itself then waits on
    // no global load (each one is most of a microsecond for a single warp)
    __shared__ hlk::ScState st_s;
    __shared__ __align__(16) u64 row_s[2 * hlk::SC_MAX_POINTS], tab_s[2 * hlk::SC_MAX_POINTS];
    __shared__ u64 invden_s[hlk::SC_MAX_POINTS], extrap_s[hlk::SC_MAX_POINTS * hlk::SC_MAX_POINTS];
    hlk::ScState* const st_global = a.state;
    {
        const u32* src = reinterpret_cast<const u32*>(a.state);
        u32* dst = reinterpret_cast<u32*>(&st_s);
        if (threadIdx.x < sizeof(hlk::ScState) / 4) dst[threadIdx.x] = src[threadIdx.x];
        const int t = (int)threadIdx.x - 64;
        if (a.mask && a.fs) {
            if (t >= 0 && t < 2 * a.degree) row_s[t] = a.mask[2 * (size_t)a.round * a.degree + t];
            if (t >= 16 && t < 16 + 2 * (a.degree + 1)) tab_s[t - 16] = a.mask_tab[2 * (size_t)a.round * (a.degree + 1) + (t - 16)];
        }
        if (t >= 40 && t < 40 + a.degree + 1) invden_s[t - 40] = a.inv_den[t - 40];
        const int ne = a.extrap ? (a.degree - a.eval_degree) * (a.eval_degree + 1) : 0;
        if (t >= 64 && t < 64 + ne) extrap_s[t - 64] = a.extrap[t - 64];
    }
    const int W = 2 * (a.degree + 1);              // <= 16 words per partial row
    const int w = threadIdx.x & 15, grp = threadIdx.x >> 4;  // STEP_T / 16 groups stride over the rows
    u64 s = 0;
    if (w < W) {
#pragma unroll 4
        for (u32 b = grp; b < a.nblocks; b += STEP_T / 16) s = gl_add(s, a.partials[(size_t)b * W + w]);
    }
    red[threadIdx.x] = s;
    __syncthreads();
    StepArgs x;
    x.degree = a.degree; x.recover = a.recover; x.fs = a.fs; x.mask_vars = a.mask_vars; x.eval_degree = a.eval_degree;
    x.rows = a.mask && a.fs ? reinterpret_cast<const fp2*>(row_s) : nullptr;
    x.tab = reinterpret_cast<const fp2*>(tab_s);
    x.row0 = a.round;  // this round's rows alone are staged
    x.inv_den = invden_s; x.extrap = a.extrap ? extrap_s : nullptr; x.state = &st_s; x.out = a.out;
    // warp 0 prepares the step, the others sum the groups' rows: 32 words per value
    fp2 g = f2(0, 0);
    const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp == 0) g = step_ahead(x, sm, a.round, (int)lane);
    for (u32 v = warp; warp > 0 && v - 1 < (u32)W; v += STEP_T / 32 - 1) {
        u64 z = red[lane * 16 + v - 1];
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) z = gl_add(z, shfl_down64(z, off));
        if (lane == 0) sm.sums[v - 1] = z;
    }
    __syncthreads();
    if (warp == 0) {
        const fp2 r = step_challenge(x, sm, a.round, a.use_claim != 0, g, (int)lane);
        step_after(x, sm, a.round, r, (int)lane);
        __syncwarp();
        const u32* src = reinterpret_cast<const u32*>(&st_s);
        u32* dst = reinterpret_cast<u32*>(st_global);
        for (u32 i = lane; i < sizeof(hlk::ScState) / 4; i += 32) dst[i] = src[i];
    }
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

// The fold with the previous challenge and the sums of the next round in ONE pass (the closed-form families): the tables are
// stored at length 2 n, unfolded; a thread reads T[i], T[i + n], T[i + half], T[i + half + n] (half = n / 2), writes the two
// folded entries T[i], T[i + half] - no other thread reads or writes those four places - and evaluates the round polynomial
// on them.  A table word is read once and written once per round, and a round is two launches (this one and the step).
template <int POLY, int K, int D>
__global__ void __launch_bounds__(RT) k_sc_fold_round(u64* __restrict__ tables, size_t stride, u32 n, const u64* __restrict__ coefs,
                                                      const hlk::ScState* __restrict__ st, int eval_one, u64* __restrict__ partials) {
    chain_enter();
    fp2 acc[D + 1];
#pragma unroll
    for (int d = 0; d <= D; d++) acc[d] = f2(0, 0);
    const fp2* cf = reinterpret_cast<const fp2*>(coefs);
    const fp2 r = st->r;
    const u32 half = n >> 1;
    for (u32 i = blockIdx.x * RT + threadIdx.x; i < half; i += gridDim.x * RT) {
        fp2 cur[K], dif[K];
#pragma unroll
        for (int t = 0; t < K; t++) {
            u64* tb = tables + 2 * (size_t)t * stride;
            const fp2 a0 = ld2(tb + 2 * (size_t)i), a1 = ld2(tb + 2 * ((size_t)i + n));
            const fp2 b0 = ld2(tb + 2 * ((size_t)i + half)), b1 = ld2(tb + 2 * ((size_t)i + half + n));
            const fp2 lo = f2_add(a0, f2_mul(r, f2_sub(a1, a0))), hi = f2_add(b0, f2_mul(r, f2_sub(b1, b0)));
            st2(tb + 2 * (size_t)i, lo);
            st2(tb + 2 * ((size_t)i + half), hi);
            cur[t] = lo;
            dif[t] = f2_sub(hi, lo);
        }
        acc[0] = f2_add(acc[0], hlk::poly_eval<POLY, K>(cur, cf));
#pragma unroll
        for (int d = 1; d <= D; d++) {
#pragma unroll
            for (int t = 0; t < K; t++) cur[t] = f2_add(cur[t], dif[t]);
            if (d != 1 || eval_one) acc[d] = f2_add(acc[d], hlk::poly_eval<POLY, K>(cur, cf));
        }
    }
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
    if (threadIdx.x < 2 * (D + 1)) {
        u64 s = 0;
#pragma unroll
        for (int w = 0; w < RT / 32; w++) s = gl_add(s, wsum[w][threadIdx.x]);
        partials[(size_t)blockIdx.x * 2 * (D + 1) + threadIdx.x] = s;
    }
}

__global__ void __launch_bounds__(256) k_sc_fold(u64* __restrict__ tables, size_t stride, u32 half, u32 k, const hlk::ScState* __restrict__ st) {
    chain_enter();
    const u32 i = blockIdx.x * blockDim.x + threadIdx.x, t = blockIdx.y;
    if (i >= half || t >= k) return;
    const fp2 r = st->r;
    u64* tb = tables + 2 * (size_t)t * stride;
    fp2 a = ld2(tb + 2 * (size_t)i), b = ld2(tb + 2 * ((size_t)i + half));
    st2(tb + 2 * (size_t)i, f2_add(a, f2_mul(r, f2_sub(b, a))));
}


// ---------------------------------------------------------------------------------------------
// Slot polynomials given as data: the long rounds, one pair per thread (or NPT of its points), the polynomial as a program (slot_vm.cuh)
// ---------------------------------------------------------------------------------------------
constexpr int VMT = 128;
template <int NPT>
__global__ void __launch_bounds__(VMT) k_sc_round_vm(const u64* __restrict__ tables, size_t stride, u32 half, hlk::IrDev p, int degree, u32 npe, bool skip,
                                                     fp2* __restrict__ slots_g, u64* __restrict__ partials) {
    chain_enter();
    extern __shared__ __align__(16) char vm_smem[];
    __shared__ u64 wsum[VMT / 32][2 * NPT];
    u64* code = reinterpret_cast<u64*>(vm_smem);
    fp2* cf = reinterpret_cast<fp2*>(vm_smem + (((size_t)p.n_code * 8 + 15) & ~(size_t)15));
    for (u32 x = threadIdx.x; x < p.n_code; x += VMT) code[x] = p.code[x];
    for (u32 x = threadIdx.x; x < p.n_coefs; x += VMT) cf[x] = ld2(p.coefs + 2 * (size_t)x);
    const u32 entries = vm::slot_entries(p.p_slots, p.a_slots, NPT), row = blockIdx.z * gridDim.x + blockIdx.x;
    fp2* slots = (slots_g ? slots_g + (size_t)(blockIdx.y * gridDim.x * gridDim.z + row) * entries * VMT : cf + p.n_coefs) + threadIdx.x;
    const u64* prog = gridDim.z > 1 ? code + p.start[blockIdx.z] : code;
    __syncthreads();
    const u32 e0 = blockIdx.y * NPT;  // this thread's first evaluated point, by its position among them
    const u32 first = skip && e0 ? e0 + 1 : e0;
    fp2 acc[NPT];
#pragma unroll
    for (int j = 0; j < NPT; j++) acc[j] = f2(0, 0);
    for (u32 i = blockIdx.x * VMT + threadIdx.x; i < half; i += gridDim.x * VMT) {
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
    // a partial row is every point of the declared degree: the points nobody evaluates are zero
    const u32 w = threadIdx.x, np = (u32)degree + 1;
    if (w < 2 * np) {
        const u32 pt = w >> 1, e = skip && pt ? pt - 1 : pt;
        u64* dst = partials + (size_t)row * 2 * np + w;
        if ((skip && pt == 1) || e >= npe) {
            if (blockIdx.y == 0) *dst = 0;
        } else if (e >= e0 && e < e0 + NPT) {
            u64 sum = 0;
            for (int v = 0; v < VMT / 32; v++) sum = gl_add(sum, wsum[v][2 * (e - e0) + (w & 1)]);
            *dst = sum;
        }
    }
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
    if (g.blocks * p.parts <= cap) g.parts = p.parts;
    return g;
}
constexpr size_t VM_SLOT_SMEM = 40 * 1024;  // above this the slots of a CTA go to global memory

template <int NPT>
cudaError_t launch_vm(const hlk::IrDev& p, const u64* tables, size_t stride, u32 half, int degree, u32 npe, bool skip, u64* slots, u64* partials, VmGrid g,
                      cudaStream_t s) {
    const size_t slot_bytes = (size_t)vm::slot_entries(p.p_slots, p.a_slots, NPT) * VMT * 16;
    const size_t smem = vm_fixed_bytes(p) + (slots ? 0 : slot_bytes);
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(k_sc_round_vm<NPT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    return chain_launch(k_sc_round_vm<NPT>, dim3(g.blocks, (npe + NPT - 1) / NPT, g.parts), dim3(VMT), smem, s, tables, stride, half, p, degree, npe, skip,
                        reinterpret_cast<fp2*>(slots), partials);
}

template <int POLY, int K, int D>
cudaError_t launch_round(const u64* tables, size_t stride, u32 half, const u64* coefs, int eval_one, u64* partials, u32 nblocks, cudaStream_t s) {
    chain_launch(k_sc_round<POLY, K, D>, dim3(nblocks), dim3(RT), 0, s, tables, stride, half, coefs, eval_one, partials);
    return cudaGetLastError();
}

}  // namespace

namespace hlk {

u32 sc_round_blocks(u32 half, int sm_count) {
    u32 b = (half + RT - 1) / RT, cap = (u32)sm_count * 4;
    if (b < 1) b = 1;
    return b > cap ? cap : b;
}

u32 sc_ir_rows(const IrDev& p, u32 half, int sm_count) {
    const VmGrid g = vm_grid(p, half, sm_count);
    return g.blocks * g.parts;
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

cudaError_t sc_round_ir(const IrDev& p, const u64* tables, size_t stride, u32 half, int degree, int eval_one, u64* slots, u64* partials, int sm_count,
                        cudaStream_t s) {
    const bool skip = !eval_one && p.eval_degree >= 1;
    const u32 npe = p.eval_degree + (skip ? 0u : 1u), npt = vm_npt(npe);
    const size_t cta = (size_t)vm::slot_entries(p.p_slots, p.a_slots, (int)npt) * VMT * 16;
    u64* sl = cta > VM_SLOT_SMEM ? slots : nullptr;
    const VmGrid g = vm_grid(p, half, sm_count);
    switch (npt) {
        case 1: return launch_vm<1>(p, tables, stride, half, degree, npe, skip, sl, partials, g, s);
        case 2: return launch_vm<2>(p, tables, stride, half, degree, npe, skip, sl, partials, g, s);
        case 3: return launch_vm<3>(p, tables, stride, half, degree, npe, skip, sl, partials, g, s);
        case 4: return launch_vm<4>(p, tables, stride, half, degree, npe, skip, sl, partials, g, s);
        case 5: return launch_vm<5>(p, tables, stride, half, degree, npe, skip, sl, partials, g, s);
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

cudaError_t sc_round(int poly, int k, const u64* tables, size_t stride, u32 half, const u64* coefs, int eval_one, u64* partials,
                     u32 nblocks, cudaStream_t s) {
#define R(P, K, D) return launch_round<P, K, D>(tables, stride, half, coefs, eval_one, partials, nblocks, s)
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

template <int POLY, int K, int D>
static cudaError_t launch_fold_round(u64* tables, size_t stride, u32 n, const u64* coefs, const ScState* st, int eval_one, u64* partials, u32 nblocks,
                                     cudaStream_t s) {
    chain_launch(k_sc_fold_round<POLY, K, D>, dim3(nblocks), dim3(RT), 0, s, tables, stride, n, coefs, st, eval_one, partials);
    return cudaGetLastError();
}

// fold with the challenge in `st` and the sums of the next round (table length n after the fold) in one pass
cudaError_t sc_fold_round(int poly, int k, u64* tables, size_t stride, u32 n, const u64* coefs, const ScState* st, int eval_one, u64* partials,
                          u32 nblocks, cudaStream_t s) {
#define R(P, K, D) return launch_fold_round<P, K, D>(tables, stride, n, coefs, st, eval_one, partials, nblocks, s)
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
    dim3 grid((half + 255) / 256, k);
    chain_launch(k_sc_fold, dim3(grid), dim3(256), 0, s, tables, stride, half, k, st);
    return cudaGetLastError();
}

}  // namespace hlk
