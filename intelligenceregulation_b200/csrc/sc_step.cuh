// The Fiat-Shamir step of a sumcheck round, by one warp (sumcheck/rounds.rs:94-160, transcript.rs:67-148, sumcheck.rs:194-299).
//
// A serial chain runs through every round: sums -> masked message -> two hashes -> challenge -> next round's tables.  So what does not
// lie on it is done beside it: the parts are called apart, and only `step_challenge` is waited for.
//
//   step_mask       before the sums are there: the mask's round polynomial, one evaluation point per lane (and step_head, the
//                   message's head).  The host scales the mask by its challenge c, so that no product is left for later:
//                   c g_j(x) = c 2^(N-1-j) (a0 + sum_{i>j} u_i(1)/2 + u_j(x))  [table]  + 2^(N-1-j) acc + x ap,
//                   acc = c sum_{i<j} u_i(r_i), ap = c a' prod_{i<j} r_i.
//   step_challenge  s(1) from the claim, the points above the attained degree, the message (one addition per point), absorb, squeeze.
//                   Every lane computes the hashes; lane 0 writes.
//   step_after      the next claim and the mask's running terms, which the NEXT round's message needs: it waits in the state (the round's
//                   sums, the challenge) and is taken by the next step, while the tables are folded and evaluated.
#pragma once
#include "b3.cuh"
#include "gl_field.cuh"
#include "sumcheck.h"

namespace {

__device__ __forceinline__ fp2 ld2(const u64* p) {
    ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
    return f2(v.x, v.y);
}
__device__ __forceinline__ void st2(u64* p, fp2 v) { *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(v.c0, v.c1); }

__device__ __forceinline__ u64 reduce_le16(const uint32_t* w) {  // 128-bit little-endian draw mod p (transcript.rs:133-148)
    return gl_reduce128(((u64)w[1] << 32) | w[0], ((u64)w[3] << 32) | w[2]);
}

// a CTA's sum of one word handed in, and the total taken out (ScSync::sums)
__device__ __forceinline__ void add_word(u64* lo_hi, u64 v) {
    atomicAdd(lo_hi, (u64)(u32)v);
    atomicAdd(lo_hi + 1, v >> 32);
}
__device__ __forceinline__ u64 take_word(u64* lo_hi) {
    const u64 lo = __ldcg(lo_hi), hi = __ldcg(lo_hi + 1);
    lo_hi[0] = 0;
    lo_hi[1] = 0;
    return gl_add(lo, gl_reduce128(hi << 32, hi >> 32));
}

struct StepSmem {
    __align__(16) u64 sums[2 * hlk::SC_MAX_POINTS];
    __align__(16) uint32_t msg[64];  // 256 bytes
};

// v 2^k mod p, 0 <= k <= 62
__device__ __forceinline__ u64 gl_mul_pow2(u64 v, int k) { return gl_reduce128(v << k, k ? v >> (64 - k) : 0ull); }

__device__ __forceinline__ fp2 shfl_down8_f2(fp2 v, int d) {  // within groups of eight lanes
    u32 a0 = __shfl_down_sync(0xffffffffu, (u32)v.c0, d, 8), a1 = __shfl_down_sync(0xffffffffu, (u32)(v.c0 >> 32), d, 8);
    u32 b0 = __shfl_down_sync(0xffffffffu, (u32)v.c1, d, 8), b1 = __shfl_down_sync(0xffffffffu, (u32)(v.c1 >> 32), d, 8);
    return f2(((u64)a1 << 32) | a0, ((u64)b1 << 32) | b0);
}

// What the steps of a batch read, resolved once: operands that sit in registers or shared memory.
struct StepArgs {
    int degree, recover, fs, mask_vars, eval_degree;
    const fp2* rows;    // c a_{j,e}: `degree` per round, from round `row0` on; NULL: no mask
    const fp2* tab;     // degree + 1 per round, likewise
    int row0;
    const u64* inv_den;
    const u64* extrap;  // or NULL
    hlk::ScState* state;
    u64* out;
};

// the message's head: state' = H(state || LE64(8) || "sc-round" || LE64(16 np) || bytes) (transcript.rs:67-74); the values go to word 14 on
__device__ __forceinline__ void step_head(const StepArgs& a, StepSmem& sm, int lane) {
    if (!a.fs) return;
    const int np = a.degree + 1, nw = 14 + 4 * np;
    for (int i = lane; i < 64; i += 32)
        if (i < 14 || i >= nw)
            sm.msg[i] = i < 8 ? a.state->state[i] : i == 8 ? 8u : i == 10 ? 0x722d6373u : i == 11 ? 0x646e756fu : i == 12 ? 16u * np : 0u;  // "sc-r" "ound"
    __syncwarp();
}

// c g_j(x) for the point x = lane of round j
__device__ __forceinline__ fp2 step_mask(const StepArgs& a, int j, int lane) {
    const int np = a.degree + 1;
    if (!a.fs || !a.rows || lane >= np || j >= a.mask_vars) return f2(0, 0);
    const int sh = a.mask_vars - 1 - j;  // mask_vars <= 63
    const fp2 g = f2_add(a.tab[(size_t)(j - a.row0) * np + lane], f2(gl_mul_pow2(a.state->acc.c0, sh), gl_mul_pow2(a.state->acc.c1, sh)));
    return f2_add(g, f2_mul_base(a.state->ap, (u64)lane));
}

// sm.sums holds the round's sums at the points 0 .. eval_degree (the point 1 left open when use_claim); returns the challenge in every lane
__device__ __forceinline__ fp2 step_challenge(const StepArgs& a, StepSmem& sm, int j, bool use_claim, fp2 g, int lane) {
    const int np = a.degree + 1;
    hlk::ScState* st = a.state;
    fp2* s = reinterpret_cast<fp2*>(sm.sums);
    if (lane == 0 && use_claim) s[1] = f2_sub(st->claim, s[0]);  // s(1) = claim - s(0) (rounds.rs:137-140)
    __syncwarp();
    if (a.extrap && a.eval_degree < a.degree) {
        // a polynomial of degree eval_degree is fixed by its values at 0..eval_degree: the points above, exactly
        fp2 v = f2(0, 0);
        if (lane > a.eval_degree && lane < np) {
            const u64* wrow = a.extrap + (size_t)(lane - a.eval_degree - 1) * (a.eval_degree + 1);
            for (int i = 0; i <= a.eval_degree; i++) v = f2_add(v, f2_mul_base(s[i], wrow[i]));
        }
        __syncwarp();
        if (lane > a.eval_degree && lane < np) s[lane] = v;
        __syncwarp();
    }
    u64* orow = a.out + (size_t)j * (2 * (size_t)np + 1) * 2;
    if (lane < np) st2(orow + 2 * lane, s[lane]);
    if (!a.fs) return f2(0, 0);  // plain round(): the host drives the transcript
    if (lane < np) {
        const fp2 m = f2_add(s[lane], g);
        st2(orow + 2 * (np + lane), m);
        uint2* mw = reinterpret_cast<uint2*>(sm.msg + 14 + 4 * lane);
        mw[0] = make_uint2((u32)m.c0, (u32)(m.c0 >> 32));
        mw[1] = make_uint2((u32)m.c1, (u32)(m.c1 >> 32));
    }
    __syncwarp();
    // The message's blocks and, behind them, squeeze: out = H(state' || "squeeze" || LE64(counter)); counter++; state = out
    // (transcript.rs:120-130), in one loop around one copy of the compression: it is twelve kilobytes of code.
    const uint32_t* key = st->keyed ? st->key : nullptr;
    const uint32_t mode = key ? b3::KEYED : 0u;
    const u32 bytes = 56 + 16 * np, nb = (bytes + 63) / 64;
    const u64 ctr = st->counter;
    uint32_t h[8];
    b3::init_cv(h, key);
#pragma unroll 1
    for (u32 b = 0; b <= nb; b++) {
        uint32_t m[16];
        u32 len, flags = mode;
        if (b < nb) {
            const uint4* w = reinterpret_cast<const uint4*>(sm.msg + 16 * b);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint4 v = w[i];
                m[4 * i] = v.x; m[4 * i + 1] = v.y; m[4 * i + 2] = v.z; m[4 * i + 3] = v.w;
            }
            len = b == nb - 1 ? bytes - 64 * b : 64;
            flags |= (b == 0 ? b3::CHUNK_START : 0u) | (b == nb - 1 ? (b3::CHUNK_END | b3::ROOT) : 0u);
        } else {
#pragma unroll
            for (int i = 0; i < 8; i++) m[i] = h[i];
            m[8] = 0x65757173u;                                   // "sque"
            m[9] = 0x00657a65u | ((uint32_t)(ctr & 0xff) << 24);  // "eze" then counter byte 0
            m[10] = (uint32_t)(ctr >> 8);
            m[11] = (uint32_t)(ctr >> 40);                        // counter bytes 5..7; the message ends there
            m[12] = m[13] = m[14] = m[15] = 0;
            len = 47;
            flags |= b3::CHUNK_START | b3::CHUNK_END | b3::ROOT;
            b3::init_cv(h, key);
        }
        b3::compress(h, m, 0, len, flags);
    }
    const fp2 r = f2(reduce_le16(h), reduce_le16(h + 4));
    __syncwarp();
    if (lane == 0) {
        st->counter = ctr + 1;
#pragma unroll
        for (int i = 0; i < 8; i++) st->state[i] = h[i];
        st->r = r;
        st->pending = j + 1;
        st2(orow + 4 * np, r);
    }
    if (lane < np) st->sums[lane] = s[lane];
    __syncwarp();
    return r;
}

// Every lane runs the SAME product tree over eight (or four) factors and one multiplier: lanes 0..7 a Lagrange numerator
// prod_{j != i} (r - j) times s_i / den_i, lanes 8..15 a power r^e times the mask coefficient, lane 16 the product r ap; sums over groups
// of eight lanes give the next claim (rounds.rs:145-147, mle.rs:338-351) and c u_j(r_j).
__device__ __forceinline__ void step_after(const StepArgs& a, int lane) {
    const int np = a.degree + 1;
    const bool masked = a.rows != nullptr;
    hlk::ScState* st = a.state;
    const int j = st->pending - 1;
    if (j < 0) return;
    const fp2 r = st->r;
    const int grp = lane >> 3, li = lane & 7;
    fp2 f[8], mult = f2(0, 0);
#pragma unroll
    for (int t = 0; t < 8; t++) f[t] = f2(1, 0);
    if (grp == 0) {
        if (a.recover && li < np) {
#pragma unroll
            for (int t = 0; t < 7; t++) {  // the points other than li, in order
                const int jj = t < li ? t : t + 1;
                if (jj < np) f[t] = f2(gl_sub(r.c0, (u64)jj), r.c1);
            }
            mult = f2_mul_base(st->sums[li], a.inv_den[li]);
        }
    } else if (grp == 1) {
        if (masked && li < a.degree) {  // r^(li + 1) c a_{j, li + 1}
#pragma unroll
            for (int t = 0; t < 7; t++)
                if (t <= li) f[t] = r;
            mult = a.rows[(size_t)(j - a.row0) * a.degree + li];
        }
    } else if (lane == 16 && masked) {
        f[0] = r;
        f[1] = st->ap;
        mult = f2(1, 0);
    }
    fp2 prod = f2_mul(f2_mul(f[0], f[1]), f2_mul(f[2], f[3]));
    if (a.degree > 4) prod = f2_mul(prod, f2_mul(f2_mul(f[4], f[5]), f2_mul(f[6], f[7])));
    fp2 term = f2_mul(prod, mult);
    const fp2 own = term;
#pragma unroll
    for (int off = 4; off >= 1; off >>= 1) term = f2_add(term, shfl_down8_f2(term, off));
    __syncwarp();
    if (lane == 0) {
        st->pending = 0;
        if (a.recover) st->claim = term;
    }
    if (lane == 8 && masked) st->acc = f2_add(st->acc, term);
    if (lane == 16 && masked) st->ap = own;
    __syncwarp();
}

}  // namespace
