// Row-encoder kernels: persistent CTAs, one row at a time per CTA (see encode_core.cuh).
#define GL_PLAIN_CANONICAL_FORMS 1  // see gl_field.cuh: this file is tuned around the 64-bit C forms
#include "encode_core.cuh"
#include "kernels.h"

namespace {

struct CtaSync {
    __device__ __forceinline__ void operator()() const { __syncthreads(); }
};

__global__ void k_encode_generic(enc::RowArgs a, u32 logn) {
    extern __shared__ u64 smem[];
    u64* S = smem;
    const u32 n = 1u << logn, tid = threadIdx.x, nt = blockDim.x;
    u64* X = a.scratch + (size_t)blockIdx.x * a.T * n;
    for (u32 row = blockIdx.x; row < a.rows; row += gridDim.x) {
        enc::Generic::load(a, row, logn, S, tid, nt);
        __syncthreads();
        for (u32 ln = logn; ln >= 1; ln--) {
            enc::Generic::dif_stage(a, logn, ln, S, tid, nt);
            __syncthreads();
        }
        enc::Generic::coeffs(a, row, logn, S, X, tid, nt);
        __syncthreads();
        for (u32 s = 0; s < (1u << a.logr); s++) {
            enc::Generic::twist(a, logn, s, X, S, tid, nt);
            __syncthreads();
            for (u32 ln = 1; ln <= logn; ln++) {
                enc::Generic::dit_stage(a, logn, ln, S, tid, nt);
                __syncthreads();
            }
            enc::Generic::store(a, row, logn, s, S, tid, nt);
            __syncthreads();
        }
    }
}

// CTA `cta` of `ctas`
template <int LOGN, int THREADS, int FORM, bool NARROW, bool LONG, bool SPLIT>
__device__ __forceinline__ void encode_fast(const enc::RowArgs& a, u32 cta, u32 ctas) {
    using F = enc::Fast<LOGN>;
    extern __shared__ u64 smem[];
    u64* S = smem;
    u64* TW = smem + F::N;
    const u32 tid = threadIdx.x;
    u64* X = a.scratch + (size_t)cta * a.T * F::N;
    F::load_twiddles(a, TW, tid, THREADS);
    __syncthreads();
    // a unit of work: a whole row, or (split) one output residue of a row with the row's inverse transform before it
    const u32 A = LONG ? 1u << a.loga : 1u, logR = LONG ? a.logr - a.loga : a.logr, R = 1u << logR;
    const u32 units = SPLIT ? a.rows << logR : a.rows;
    for (u32 unit = cta; unit < units; unit += ctas) {
        const u32 row = SPLIT ? unit >> logR : unit;
        if constexpr (FORM == enc::FORM_COEF) {
            F::row_given(a, row, X, tid, THREADS);
            __syncthreads();
        }
        const u32 first = SPLIT ? unit & (R - 1u) : 0u, end = A + A * (SPLIT ? 1u : R);
        for (u32 k = FORM == enc::FORM_COEF ? A : 0u; k < end; k++) {
            const u32 step = k < A ? k : k + A * first;
            F::template row_step<FORM, NARROW, LONG>(a, row, step, S, TW, X, tid, THREADS, CtaSync(), first);
            __syncthreads();  // the scratch slot is complete and shared memory is free again
        }
    }
}

template <int LOGN, int THREADS, int MINB, int FORM, bool NARROW, bool LONG, bool SPLIT>
__global__ void __launch_bounds__(THREADS, MINB) k_encode_fast(enc::RowArgs a) {
    encode_fast<LOGN, THREADS, FORM, NARROW, LONG, SPLIT>(a, blockIdx.x, gridDim.x);
}

// A masking commitment's two kinds of rows at once, a CTA for each (row, residue) of either: `a` messages by the first `ctas_a` CTAs, `b`
// coefficient rows by the others.  Neither kind fills the machine, and each takes as long as its longest row: 27 us and then 32 for 24
// masks in launches of their own.
template <int LOGN, int THREADS, int MINB>
__global__ void __launch_bounds__(THREADS, MINB) k_encode_mask(enc::RowArgs a, enc::RowArgs b, u32 ctas_a) {
    if (blockIdx.x < ctas_a) encode_fast<LOGN, THREADS, enc::FORM_COSET, false, false, true>(a, blockIdx.x, ctas_a);
    else encode_fast<LOGN, THREADS, enc::FORM_COEF, false, false, true>(b, blockIdx.x - ctas_a, gridDim.x - ctas_a);
}

// packed rows widened in a pass of their own: the shapes the fast path does not cover (rows below 2^8 or above 2^14 words)
__global__ void __launch_bounds__(256) k_widen_rows(const unsigned char* __restrict__ narrow, const u64* __restrict__ row_off,
                                                    const unsigned char* __restrict__ row_w, u64* __restrict__ out, u32 rows, u32 n) {
    const size_t total = (size_t)rows * n;
    for (size_t x = (size_t)blockIdx.x * blockDim.x + threadIdx.x; x < total; x += (size_t)gridDim.x * blockDim.x) {
        const u32 row = (u32)(x / n), i = (u32)(x - (size_t)row * n);
        out[x] = enc::widen_word(narrow + row_off[row], i, row_w[row]);
    }
}

template <int LOGN>
constexpr int fast_threads() {
    constexpr int g = (1 << LOGN) / 16;
    return g < 32 ? 32 : (g > 1024 ? 1024 : g);
}

// Registers for 1,024 threads an SM, which is also what the rows' shared memory allows (12 n bytes a CTA of n / 16 threads): 64 a
// thread.  With the 113 to 170 that the compiler takes otherwise only half as many fit, and rows wait on their passes' latencies:
// 1,480 rows of 2^13 574 -> 474 us, 2,600 of 2^11 261 -> 201, 300 of 2^12 79 -> 69 (38 rows of 2^12, a CTA for each residue:
// 32 -> 36, so split rows keep up to 128).
template <int LOGN>
constexpr int fast_min_ctas() {
    return 1024 / fast_threads<LOGN>();
}

template <int LOGN, int FORM, bool NARROW, bool LONG, bool SPLIT>
cudaError_t launch_fast_as(const enc::RowArgs& a, int sm_count, size_t scratch_words, cudaStream_t st, int* grid_out) {
    using F = enc::Fast<LOGN>;
    constexpr int T = fast_threads<LOGN>();
    auto kern = k_encode_fast<LOGN, T, SPLIT ? (T > 256 ? 1 : 512 / T) : fast_min_ctas<LOGN>(), FORM, NARROW, LONG, SPLIT>;
    size_t smem = (size_t)(F::N + F::TW_WORDS) * 8;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, T, smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) per_sm = 1;
    size_t grid = (size_t)sm_count * per_sm;
    const size_t units = SPLIT ? (size_t)a.rows << (a.logr - a.loga) : (size_t)a.rows;
    if (grid > units) grid = units;
    size_t max_by_scratch = scratch_words / ((size_t)a.T * F::N);
    if (grid > max_by_scratch) grid = max_by_scratch;
    if (grid < 1) return cudaErrorInvalidValue;
    *grid_out = (int)grid;
    kern<<<(unsigned)grid, T, smem, st>>>(a);
    return cudaGetLastError();
}

template <int LOGN>
cudaError_t launch_mask(const enc::RowArgs& a, const enc::RowArgs& b, cudaStream_t st) {
    using F = enc::Fast<LOGN>;
    constexpr int T = fast_threads<LOGN>();
    auto kern = k_encode_mask<LOGN, T, (T > 256 ? 1 : 512 / T)>;
    const size_t smem = (size_t)(F::N + F::TW_WORDS) * 8;
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const u32 ctas_a = a.rows << a.logr, ctas_b = b.rows << b.logr;
    kern<<<ctas_a + ctas_b, T, smem, st>>>(a, b, ctas_a);
    return cudaGetLastError();
}

// split rows are few: they get the registers that a row's latency wants
template <int LOGN, int FORM = enc::FORM_PCS, bool NARROW = false, bool LONG = false>
cudaError_t launch_fast(const enc::RowArgs& a, int sm_count, size_t scratch_words, cudaStream_t st, int* grid_out) {
    if (a.split) return launch_fast_as<LOGN, FORM, NARROW, LONG, true>(a, sm_count, scratch_words, st, grid_out);
    return launch_fast_as<LOGN, FORM, NARROW, LONG, false>(a, sm_count, scratch_words, st, grid_out);
}

}  // namespace

namespace hlk {

size_t encode_scratch_words(u32 logn, u32 T, int sm_count, u32 rows) {
    // enough for the largest grid any path launches: 32 CTAs per SM at most, one per row or, for a handful of rows, one per
    // (row, residue)
    size_t ctas = (size_t)sm_count * 32;
    const size_t units = encode_split_units(logn, sm_count);
    if (ctas > rows) ctas = rows > units ? rows : units;
    return ctas * T * ((size_t)1 << logn);
}

// How many (row, residue) CTAs a launch of split rows takes at once: one per SM, or half of those that an SM holds where a CTA is far from
// filling one
size_t encode_split_units(u32 logn, int sm_count) {
    const u32 t = logn > 9 ? 1u << (logn - 4) : 32u;
    return (size_t)sm_count * (t > 512 ? 1 : 512 / t);
}
// Splitting rows by residue repeats their inverse transform: 2 transforms a CTA instead of 1 + R, R times the CTAs.
// Where a CTA has an SM to itself (2^13 words and more) a turn of the machine takes as long as a lone CTA, and splitting pays when it takes
// fewer turns' transforms (38 rows of 2^14 103 -> 75 us, 74 of them 103 -> 74, 100 of them 103 -> 140; at rate 1/4 74
// rows 189 -> 152, 100 rows 189 -> 224).  Smaller CTAs share an SM, and a full turn takes twice a lone CTA's time, in proportion to the
// CTAs above that (measured for 2^8 .. 2^12 words at rates 1/2, 1/4, 1/8, and masks up to rate 1/64, as CTAs over the turn's CTAs where
// both ways take the same time: 0.75 - 1, 1.1 - 1.4, 2 - 2.5, 16; the line: 0.75, 1.25, 2.25, 16.25).  296 rows of 2^11 at rate 1/4 62 -> 87 us
// when split, 148 of them 58 -> 41.
bool encode_split_pays(u32 logn, u32 logR, u32 rows, int sm_count) {
    const u64 at_once = encode_split_units(logn, sm_count), units = (u64)rows << logR, whole = 1 + ((u64)1 << logR);
    if (logR < 1) return false;
    if (at_once > (u64)sm_count) return units * 4 < at_once * whole;
    return (units + at_once - 1) / at_once * 2 < (rows + at_once - 1) / at_once * whole;
}

cudaError_t encode_rows(const enc::RowArgs& a, u32 logn, bool allow_fast, int sm_count, size_t scratch_words,
                        cudaStream_t st, int* path_out) {
    int grid = 0;
    if (a.narrow) {  // packed rows: the widening first pass exists on the fast path only (the caller widens separately otherwise)
        if (!allow_fast || logn < 8 || logn > 14 || a.loga) return cudaErrorInvalidValue;
        if (path_out) *path_out = 2;
        switch (logn) {
            case 8: return launch_fast<8, enc::FORM_PCS, true>(a, sm_count, scratch_words, st, &grid);
            case 9: return launch_fast<9, enc::FORM_PCS, true>(a, sm_count, scratch_words, st, &grid);
            case 10: return launch_fast<10, enc::FORM_PCS, true>(a, sm_count, scratch_words, st, &grid);
            case 11: return launch_fast<11, enc::FORM_PCS, true>(a, sm_count, scratch_words, st, &grid);
            case 12: return launch_fast<12, enc::FORM_PCS, true>(a, sm_count, scratch_words, st, &grid);
            case 13: return launch_fast<13, enc::FORM_PCS, true>(a, sm_count, scratch_words, st, &grid);
            case 14: return launch_fast<14, enc::FORM_PCS, true>(a, sm_count, scratch_words, st, &grid);
        }
    }
    if (allow_fast && logn >= 8 && logn <= 14) {
        if (path_out) *path_out = 1;
        switch (logn) {
            case 8: return launch_fast<8>(a, sm_count, scratch_words, st, &grid);
            case 9: return launch_fast<9>(a, sm_count, scratch_words, st, &grid);
            case 10: return launch_fast<10>(a, sm_count, scratch_words, st, &grid);
            case 11: return launch_fast<11>(a, sm_count, scratch_words, st, &grid);
            case 12: return launch_fast<12>(a, sm_count, scratch_words, st, &grid);
            case 13: return launch_fast<13>(a, sm_count, scratch_words, st, &grid);
            case 14:
                if (a.loga) return launch_fast<14, enc::FORM_PCS, false, true>(a, sm_count, scratch_words, st, &grid);
                return launch_fast<14>(a, sm_count, scratch_words, st, &grid);
        }
    }
    if (logn < 1 || logn > 14) return cudaErrorInvalidValue;
    if (path_out) *path_out = 0;
    const u32 n = 1u << logn;
    int threads = (int)(n / 2 < 32 ? 32 : (n / 2 > 1024 ? 1024 : n / 2));
    size_t smem = (size_t)n * 8;
    cudaError_t e = cudaFuncSetAttribute(k_encode_generic, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(smem < 1024 ? 1024 : smem));
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_encode_generic, threads, smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) per_sm = 1;
    size_t g = (size_t)sm_count * per_sm;
    if (g > a.rows) g = a.rows;
    size_t max_by_scratch = scratch_words / ((size_t)a.T * n);
    if (g > max_by_scratch) g = max_by_scratch;
    if (g < 1) return cudaErrorInvalidValue;
    k_encode_generic<<<(unsigned)g, threads, smem, st>>>(a, logn);
    return cudaGetLastError();
}

cudaError_t widen_rows(const unsigned char* narrow, const u64* row_off, const unsigned char* row_w, u64* out, u32 rows, u32 n, int sm_count, cudaStream_t st) {
    const size_t total = (size_t)rows * n;
    size_t blocks = (total + 255) / 256, cap = (size_t)sm_count * 16;
    if (blocks > cap) blocks = cap;
    if (blocks < 1) blocks = 1;
    k_widen_rows<<<(unsigned)blocks, 256, 0, st>>>(narrow, row_off, row_w, out, rows, n);
    return cudaGetLastError();
}

// both kinds of rows of a masking commitment in one launch; a scratch slot of T x N words for each (row, residue) of either, a's first
cudaError_t encode_rows_mask(const enc::RowArgs& a, const enc::RowArgs& b, u32 logn, cudaStream_t st) {
    switch (logn) {
        case 8: return launch_mask<8>(a, b, st);
        case 9: return launch_mask<9>(a, b, st);
        case 10: return launch_mask<10>(a, b, st);
        case 11: return launch_mask<11>(a, b, st);
    }
    return cudaErrorInvalidValue;
}

// the rows of a masking commitment (messages of 2^8 .. 2^11 words): FORM_COSET or FORM_COEF, always the fast path
cudaError_t encode_rows_form(const enc::RowArgs& a, u32 logn, int form, int sm_count, size_t scratch_words, cudaStream_t st) {
    int grid = 0;
    const bool coef = form == enc::FORM_COEF;
    if (form != enc::FORM_COSET && !coef) return cudaErrorInvalidValue;
    switch (logn) {
        case 8: return coef ? launch_fast<8, enc::FORM_COEF>(a, sm_count, scratch_words, st, &grid) : launch_fast<8, enc::FORM_COSET>(a, sm_count, scratch_words, st, &grid);
        case 9: return coef ? launch_fast<9, enc::FORM_COEF>(a, sm_count, scratch_words, st, &grid) : launch_fast<9, enc::FORM_COSET>(a, sm_count, scratch_words, st, &grid);
        case 10: return coef ? launch_fast<10, enc::FORM_COEF>(a, sm_count, scratch_words, st, &grid) : launch_fast<10, enc::FORM_COSET>(a, sm_count, scratch_words, st, &grid);
        case 11: return coef ? launch_fast<11, enc::FORM_COEF>(a, sm_count, scratch_words, st, &grid) : launch_fast<11, enc::FORM_COSET>(a, sm_count, scratch_words, st, &grid);
    }
    return cudaErrorInvalidValue;
}

}  // namespace hlk
