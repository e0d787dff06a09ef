// Witness weight products (hashline/src/gpu/metal.rs:4646-4680 witness_product; private_block/witness.rs:979-991): the one
// dense contraction of the system, exact integers: int16 activations times int8 weights into int64.
//
//   k_wp_pack      x (int64, row stride xs) -> two byte planes per 128-token tile: hi = x >> 8 (signed), lo = x & 255
//                  (unsigned), K padded with zeros to a multiple of 128; an activation outside int16 raises the flag
//   k_wp_repack    weights the product kernel cannot read in place (in_out layout, or K not a multiple of 128) -> rows of Kp bytes
//                  in whole boxes, zeros included
//   k_wp_umma      out[128 x 256 tile] = 256 (A_hi B) + (A_lo B): tcgen05.mma kind::i8 (signed x signed for the high bytes,
//                  unsigned x signed for the low bytes), int32 accumulators in TMEM, int64 result written by the epilogue;
//                  split over K inside a cluster (partial sums through distributed shared memory), and beyond four CTAs of a
//                  cluster with integer atomics (integer addition: any order gives the same words)
// |sum lo w| <= K * 255 * 128 < 2^31 for K <= 65,536 (metal.rs:4234 states the same bound), so int32 never wraps.
#include <cuda.h>

#include <cstdlib>

#include "api_internal.h"
#include "umma.cuh"

using namespace hlapi;

namespace {

constexpr int WP_MT = 128;      // tokens per tile; the stacked tile has 2 * WP_MT rows (hi rows, then lo rows)
constexpr size_t WP_MAX_K = (size_t)1 << 16;

__global__ void __launch_bounds__(256) k_wp_pack(const long long* __restrict__ x, size_t xs, u32 t_rows, u32 K, u32 Kp,
                                                 uint8_t* __restrict__ A /* tiles x 2 x WP_MT x Kp */, int* __restrict__ flag,
                                                 long long* __restrict__ clear, size_t clear_words) {
    // the result plane's clear rides along (the product kernel runs after this one): one launch less on a launch-bound path
    for (size_t i = ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * blockDim.x + threadIdx.x; i < clear_words;
         i += (size_t)gridDim.x * gridDim.y * blockDim.x)
        clear[i] = 0;
    asm volatile("griddepcontrol.launch_dependents;\n" ::);  // the product kernel may set itself up and fetch weights meanwhile
    const u32 t = blockIdx.y;  // padded token index
    const u32 mt = t / WP_MT, r = t % WP_MT;
    uint8_t* hi = A + ((size_t)mt * 2 * WP_MT + r) * Kp;
    uint8_t* lo = hi + (size_t)WP_MT * Kp;
    // four activations (one 32-byte sector) per thread, one 4-byte word of each plane out
    for (u32 k = (blockIdx.x * blockDim.x + threadIdx.x) * 4; k < Kp; k += gridDim.x * blockDim.x * 4) {
        u32 h = 0, l = 0;
        bool bad = false;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            long long v = 0;
            if (t < t_rows && k + j < K) {
                v = x[(size_t)t * xs + k + j];
                if (v < -32768 || v > 32767) { bad = true; v = 0; }
            }
            h |= (u32)((v >> 8) & 255) << (8 * j);
            l |= (u32)(v & 255) << (8 * j);
        }
        if (bad) *reinterpret_cast<volatile int*>(flag) = 1;
        *reinterpret_cast<u32*>(hi + k) = h;
        *reinterpret_cast<u32*>(lo + k) = l;
    }
}

// four bytes from p on, of which the first `valid` belong to the row (the others read as zero); `lo` and `hi` bound the readable bytes
__device__ __forceinline__ u32 wp_load4(const int8_t* p, int valid, const int8_t* lo, const int8_t* hi) {
    const uintptr_t at = (uintptr_t)p & ~(uintptr_t)3;
    if (valid >= 4 && at >= (uintptr_t)lo && at + 8 <= (uintptr_t)hi) {
        const u32* w = reinterpret_cast<const u32*>(at);
        return __funnelshift_r(w[0], w[1], 8 * (u32)((uintptr_t)p & 3));
    }
    u32 v = 0;
    for (int j = 0; j < 4 && j < valid; j++) v |= (u32)(uint8_t)p[j] << (8 * j);
    return v;
}

// in_out: src[i * N + j] -> dst[j * Kp + i]; else src[j * K + i] -> dst[j * Kp + i]; zero beyond K and N.  A CTA fills 128 rows of 128
// bytes in 16-byte stores.  The transposing form turns 16 words (16 k, 4 n each) into 4 rows of 16 bytes per thread; the tile's words
// stand rotated by their row block, so that both its accesses take 32 banks.  Bound by memory: 16.8 MB transposed 26 us by single
// bytes, 12 now.  It reads nothing of the packing kernel's and may run beside it; it ends after it, so that whoever waits for this kernel has both.
__global__ void __launch_bounds__(256) k_wp_repack(const int8_t* __restrict__ src, size_t src_len, u32 K, u32 N, u32 Kp, int in_out, int8_t* __restrict__ dst) {
    __shared__ u32 tile[128][32];
    asm volatile("griddepcontrol.launch_dependents;\n" ::);
    const u32 k0 = blockIdx.x * 128, n0 = blockIdx.y * 128;
    const int8_t* end = src + src_len;
    const u32 seg = threadIdx.x & 7, grp = threadIdx.x >> 3;  // 16 bytes of a row; a group of four rows
    if (in_out) {
#pragma unroll 4
        for (u32 e = threadIdx.x; e < 128 * 32; e += 256) {
            const u32 kk = e >> 5, n4 = e & 31, n = n0 + 4 * n4;
            tile[kk][(n4 + 4 * (kk >> 4)) & 31] = k0 + kk < K && n < N ? wp_load4(src + (size_t)(k0 + kk) * N + n, (int)min(N - n, 4u), src, end) : 0u;
        }
        __syncthreads();
        u32 o[4][4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            u32 w[4];
#pragma unroll
            for (int j = 0; j < 4; j++) w[j] = tile[seg * 16 + 4 * q + j][(grp + 4 * seg) & 31];
            const u32 a = __byte_perm(w[0], w[1], 0x5140), b = __byte_perm(w[2], w[3], 0x5140), c = __byte_perm(w[0], w[1], 0x7362),
                      d = __byte_perm(w[2], w[3], 0x7362);
            o[0][q] = __byte_perm(a, b, 0x5410);
            o[1][q] = __byte_perm(a, b, 0x7632);
            o[2][q] = __byte_perm(c, d, 0x5410);
            o[3][q] = __byte_perm(c, d, 0x7632);
        }
#pragma unroll
        for (int r = 0; r < 4; r++)
            *reinterpret_cast<uint4*>(dst + (size_t)(n0 + 4 * grp + r) * Kp + k0 + 16 * seg) = make_uint4(o[r][0], o[r][1], o[r][2], o[r][3]);
    } else {
        const u32 k = k0 + 16 * seg;
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const u32 n = n0 + grp + 32 * r;
            u32 o[4] = {0, 0, 0, 0};
#pragma unroll
            for (u32 q = 0; q < 4; q++)
                if (n < N && k + 4 * q < K) o[q] = wp_load4(src + (size_t)n * K + k + 4 * q, (int)min(K - k - 4 * q, 4u), src, end);
            *reinterpret_cast<uint4*>(dst + (size_t)n * Kp + k) = make_uint4(o[0], o[1], o[2], o[3]);
        }
    }
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
}

// ---------------------------------------------------------------------------------------------------------------
// The product on the 5th-generation tensor cores: TMA tiles into shared memory, tcgen05.mma kind::i8, accumulators in TMEM.
// One CTA per SM owns a 128-token tile (two 128-row operands: the signed high bytes and the unsigned low bytes) and 256
// output columns.  Per K stage of 128 bytes one thread asks the TMA unit for two boxes (256 stacked activation rows and 256
// weight rows of 128 bytes, 128-byte swizzle) and, when they have landed, issues 4 x 2 instructions of shape 128 x 256 x 32
// (hi: s8 x s8 into TMEM columns 0..255, lo: u8 x s8 into columns 256..511); the epilogue reads both accumulators lane by
// lane and writes 256 hi + lo as int64 straight into the result plane (integer atomics when K is split).
// Shared-memory operands are K-major with the 128-byte swizzle the TMA unit writes: rows of 128 bytes, 8-row groups
// UM_SBO apart, a K step of 32 bytes is 32 bytes further along the row.
// Every wait is bounded: a wait that runs out sets the error word, every thread leaves together and TMEM is freed.
constexpr int UM_NT = 256, UM_KT = 128, UM_STAGES = 3, UM_THREADS = 256;
constexpr u32 UM_A_BYTES = WP_MT * UM_KT, UM_B_BYTES = UM_NT * UM_KT, UM_STAGE_BYTES = 2 * UM_A_BYTES + UM_B_BYTES;

// one box of the tensor map into shared memory; its bytes are counted on the mbarrier
__device__ __forceinline__ void um_tma_2d(u32 smem_dst, const CUtensorMap* map, u32 mbar, int x, int y) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n" ::"r"(smem_dst),
                 "l"((u64)map), "r"(mbar), "r"(x), "r"(y)
                 : "memory");
}
__device__ __forceinline__ void um_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
// 32 result words of one row; a lane's words are consecutive, so a vector store of 32 bytes fills a sector (8-byte stores alone took
// longer than the tile's arithmetic at 128 tokens)
__device__ __forceinline__ void um_store32(long long* o, const u32 (&hi)[32], const u32 (&lo)[32], u32 live, bool add, u32 align) {
    if (add || live < 32 || (align & 15)) {
#pragma unroll
        for (int j = 0; j < 32; j++) {
            if ((u32)j >= live) continue;
            const long long v = 256ll * (int)hi[j] + (int)lo[j];
            if (add) atomicAdd(reinterpret_cast<unsigned long long*>(o + j), (unsigned long long)v);
            else o[j] = v;
        }
    } else if (align & 31) {
#pragma unroll
        for (int j = 0; j < 32; j += 2)
            *reinterpret_cast<longlong2*>(o + j) = make_longlong2(256ll * (int)hi[j] + (int)lo[j], 256ll * (int)hi[j + 1] + (int)lo[j + 1]);
    } else {
#pragma unroll
        for (int j = 0; j < 32; j += 4)
            asm volatile("st.global.v4.b64 [%0], {%1, %2, %3, %4};\n" ::"l"(o + j), "l"(256ll * (int)hi[j] + (int)lo[j]),
                         "l"(256ll * (int)hi[j + 1] + (int)lo[j + 1]), "l"(256ll * (int)hi[j + 2] + (int)lo[j + 2]), "l"(256ll * (int)hi[j + 3] + (int)lo[j + 3])
                         : "memory");
    }
}

// grid (N tiles of 256, K splits, token tiles).  map_a: the packed activations, (tiles * 256) rows of Kp bytes; map_b: the weights,
// N rows of K bytes (rows past N read as zero).  Barriers: full[s] (the stage's two boxes have landed), empty[s] (the instructions
// that read the stage have completed), done.
// Clusters of S = 1, 2 or 4 CTAs along the K splits: CTA d of a cluster finishes the tile's columns [256 d / S, 256 (d + 1) / S).  The
// others hand it their partial sums (32-bit pairs: |sums| stay below 2^31 over all of K) into its stage memory, which is idle by then:
// (S - 1) x 128 x 256 / S pairs, at most the 192 KB there are.
// What bounds it: the operands' latency, two stages in flight a CTA (tensor pipe 31 % busy).  128 x 4096 x 14336, 56 tiles on 148
// SMs: 40 us unsplit, 27 in clusters of two, part of it beside the packing.  Tiles that start K at places of their own: the same.
__global__ void __launch_bounds__(UM_THREADS, 1) k_wp_umma(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, u32 N,
                                                          u32 Kp, u32 t_rows, size_t os, long long* __restrict__ out, int* __restrict__ err,
                                                          u32 S, u32 weights_first) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    __shared__ __align__(8) u64 bars[2 * UM_STAGES + 1];
    __shared__ u32 tmem_slot;
    __shared__ volatile u32 gave_up;  // set by the issuing thread when one of its waits ran out
    const u32 tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const u32 n0 = blockIdx.x * UM_NT, mt = blockIdx.z;
    const u32 kt_all = Kp / UM_KT, kt0 = (u32)((u64)kt_all * blockIdx.y / gridDim.y), kt1 = (u32)((u64)kt_all * (blockIdx.y + 1) / gridDim.y);
    const u32 nkt = kt1 - kt0;
    const u32 smem_base = ((u32)__cvta_generic_to_shared(smem_raw) + 1023u) & ~1023u;  // the swizzle pattern repeats every 1024 bytes
    const u32 bar_base = (u32)__cvta_generic_to_shared(bars);
    const u32 full0 = bar_base, empty0 = bar_base + 8 * UM_STAGES, done = bar_base + 16 * UM_STAGES;

    if (tid == 0) {
        gave_up = 0;
        for (int i = 0; i <= 2 * UM_STAGES; i++) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(bar_base + 8 * i));
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::);
    }
    if (warp == 0) {
        // all 512 columns: the allocation cannot wait on another CTA, because this kernel's shared memory (3 stages of 64 KB) lets
        // only one CTA live on an SM and no other kernel of the library holds TMEM
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"((u32)__cvta_generic_to_shared(&tmem_slot)), "r"(512u));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::);
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::);
    const u32 tmem = tmem_slot;

    bool ok = true;
    if (tid == 0) {
        auto load_a = [&](u32 kt, u32 st) {
            um_tma_2d(smem_base + st * UM_STAGE_BYTES, &map_a, full0 + 8 * st, (int)(kt * UM_KT), (int)(mt * 2 * WP_MT));
        };
        auto load_b = [&](u32 kt, u32 st) {
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(full0 + 8 * st), "r"(UM_STAGE_BYTES) : "memory");
            um_tma_2d(smem_base + st * UM_STAGE_BYTES + 2 * UM_A_BYTES, &map_b, full0 + 8 * st, (int)(kt * UM_KT), (int)n0);
        };
        auto load_stage = [&](u32 kt, u32 st) {
            load_b(kt, st);
            load_a(kt, st);
        };
        // the activations wait for the packing kernel, the caller's weights do not
        if (!weights_first) asm volatile("griddepcontrol.wait;\n" ::: "memory");
        for (u32 s = 0; s < UM_STAGES && s < nkt; s++) load_b(kt0 + s, s);
        if (weights_first) asm volatile("griddepcontrol.wait;\n" ::: "memory");
        for (u32 s = 0; s < UM_STAGES && s < nkt; s++) load_a(kt0 + s, s);
        for (u32 it = 0; it < nkt && ok; it++) {
            const u32 st = it % UM_STAGES;
            ok = um_wait(full0 + 8 * st, (it / UM_STAGES) & 1);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::);
            const u32 sa = smem_base + st * UM_STAGE_BYTES, sb = sa + 2 * UM_A_BYTES;
#pragma unroll
            for (u32 kk = 0; kk < UM_KT / 32; kk++) {
                const u64 bd = um_desc(sb + kk * 32);
                const u32 accumulate = (it | kk) ? 1u : 0u;
                um_mma(tmem, um_desc(sa + kk * 32), bd, um_idesc(true, true, WP_MT, UM_NT), accumulate);
                um_mma(tmem + 256, um_desc(sa + UM_A_BYTES + kk * 32), bd, um_idesc(false, true, WP_MT, UM_NT), accumulate);
            }
            um_commit(empty0 + 8 * st);  // arrives when the instructions above have read this stage
            // refill the stage read one iteration ago, once its instructions have completed
            if (it >= 1 && it - 1 + UM_STAGES < nkt) {
                ok = um_wait(empty0 + 8 * ((it - 1) % UM_STAGES), ((it - 1) / UM_STAGES) & 1);
                if (ok) load_stage(kt0 + it - 1 + UM_STAGES, (it - 1) % UM_STAGES);
            }
        }
        if (ok) um_commit(done);  // arrives when every instruction of this CTA has completed
        else gave_up = 1;
    }
    // everyone waits for the accumulators, in slices so that a wait the issuing thread gave up on ends the others' too
    bool ready = false;
    for (u32 round = 0; round < 1024 && !ready && !gave_up; round++) {
        for (u32 spin = 0; spin < (UM_SPIN_LIMIT >> 10) && !ready; spin++) {
            ready = um_try_wait(done, 0u);
            if (!ready) __nanosleep(128);  // the polling threads stay off the shared memory the tensor core is reading
        }
    }
    const bool failed = __syncthreads_or(!ready);
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::);
    asm volatile("griddepcontrol.wait;\n" ::: "memory");  // what the packing kernel cleared
    // warp w reads TMEM lanes 32 (w % 4) .. +31 (the rows of the token tile) and every other 32 columns
    const u32 q = warp & 3, half = warp >> 2, row = q * 32 + lane, t = mt * WP_MT + row;
    const u32 rank = S > 1 ? blockIdx.y % S : 0u, W = UM_NT / S;
    auto fetch = [&](u32 col, u32 (&hi)[32], u32 (&lo)[32]) {
        um_ld32(tmem + ((q * 32) << 16) + col, hi);
        um_ld32(tmem + ((q * 32) << 16) + 256 + col, lo);
        asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
    };
    if (S > 1) {
        um_cluster_sync();  // every CTA's instructions have read their stages (or it gave up: it comes here all the same)
        if (!failed) {
#pragma unroll 1
            for (u32 cc = half * 32; cc < UM_NT; cc += 64) {
                const u32 d = cc / W;
                if (d == rank) continue;
                u32 hi[32], lo[32], remote;
                fetch(cc, hi, lo);
                const u32 slot = rank < d ? rank : rank - 1;  // [slot][column][row], a pair each: lanes side by side
                const u32 at = smem_base + ((slot * W + cc % W) * WP_MT + row) * 8;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(remote) : "r"(at), "r"(d));
#pragma unroll
                for (int j = 0; j < 32; j++)
                    asm volatile("st.shared::cluster.v2.b32 [%0], {%1, %2};\n" ::"r"(remote + (u32)j * WP_MT * 8), "r"(hi[j]), "r"(lo[j]) : "memory");
            }
        }
        um_cluster_sync();
    }
    if (!failed) {
        const bool add = gridDim.y > S;
        const u32 align = (u32)((uintptr_t)out | (os * 8));
#pragma unroll 1
        for (u32 cc = rank * W + half * 32; cc < (rank + 1) * W; cc += 64) {
            u32 hi[32], lo[32];
            fetch(cc, hi, lo);
#pragma unroll 1
            for (u32 slot = 0; slot + 1 < S; slot++) {
                const u32 at = smem_base + ((slot * W + cc % W) * WP_MT + row) * 8;
#pragma unroll
                for (int j = 0; j < 32; j++) {
                    u32 h, l;
                    asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];\n" : "=r"(h), "=r"(l) : "r"(at + (u32)j * WP_MT * 8) : "memory");
                    hi[j] += h;
                    lo[j] += l;
                }
            }
            const u32 left = n0 + cc < N ? N - n0 - cc : 0;
            if (t < t_rows && left) um_store32(out + (size_t)t * os + n0 + cc, hi, lo, left, add, align);
        }
    }
    if (failed && tid == 0) *reinterpret_cast<volatile int*>(err) = 2;
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::);
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512u));
}

// everything on the context's stream; d_* are device pointers; *flag_out is read after one synchronisation
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// a byte matrix of `rows` rows of `inner` readable bytes, `pitch` bytes apart (a multiple of 16), read in boxes of 128 bytes x 256 rows
// with the 128-byte swizzle; rows and bytes outside the matrix read as zero
int byte_matrix_map(hl_ctx* c, const void* base, size_t inner, size_t rows, size_t pitch, CUtensorMap* map) {
    // looked up once per process (a function-local static is initialised under the language's own lock)
    static const EncodeTiledFn encode = [] {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) fn = nullptr;
        return (EncodeTiledFn)fn;
    }();
    if (!encode) return fail(c, HL_B200_ERR_DEVICE, "witness product: the driver has no tensor-map encoder");
    const cuuint64_t dims[2] = {(cuuint64_t)inner, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)pitch};
    const cuuint32_t box[2] = {(cuuint32_t)UM_KT, 256u}, elem[2] = {1u, 1u};
    const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? HL_B200_OK : fail(c, HL_B200_ERR_DEVICE, "witness product: tensor-map encoding refused");
}

int product_on_device(hl_ctx* c, size_t t_rows, const int64_t* d_x, size_t xs, const int8_t* d_w, size_t K, size_t N, size_t os, size_t out_len,
                      int in_out, int64_t* d_out, int* taken) {
    const u32 Kp = (u32)((K + UM_KT - 1) / UM_KT * UM_KT);
    const u32 tiles = (u32)((t_rows + WP_MT - 1) / WP_MT);
    // weights are read in place when their rows are whole K stages and there is at least one box of rows; else from a padded copy
    const bool in_place = !in_out && K % UM_KT == 0 && ((uintptr_t)d_w & 15) == 0 && N >= (size_t)UM_NT;
    const size_t n_pad = (N + UM_NT - 1) / UM_NT * UM_NT;
    const size_t a_bytes = (size_t)tiles * 2 * WP_MT * Kp, b_bytes = in_place ? 0 : n_pad * Kp;
    uint8_t* d_a = nullptr;
    int8_t* d_b = nullptr;
    int rc = dev_alloc(c, (void**)&d_a, a_bytes);
    if (!rc && !c->wp_flag) {  // the status word: page-locked host memory that the kernels write to when something is wrong, zero between calls
        if (cudaHostAlloc((void**)&c->wp_flag, 4, cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess) {
            c->wp_flag = nullptr;
            rc = fail(c, HL_B200_ERR_OOM, "witness product: status word");
        } else {
            *c->wp_flag = 0;
        }
    }
    int* d_flag = c->wp_flag;
    if (!rc && b_bytes) rc = dev_alloc(c, (void**)&d_b, b_bytes);
    CUtensorMap map_a, map_b;
    if (!rc) rc = byte_matrix_map(c, d_a, Kp, (size_t)tiles * 2 * WP_MT, Kp, &map_a);
    if (!rc) rc = byte_matrix_map(c, in_place ? (const void*)d_w : (const void*)d_b, Kp, in_place ? N : n_pad, Kp, &map_b);
    // The split over K, S CTAs of a cluster times sp clusters, by a cost model fitted to measurements on B200: a CTA streams one K stage
    // (64 KB of operands) in about 1.3 us, CTAs run in waves of one per SM (clusters of four leave some SMs out), handing partial sums
    // over inside a cluster takes about 3 us, and every cluster beyond the first adds a pass of 64-bit integer atomics over the result
    // plane at about 195 G atomics per second.
    const u32 n_tiles = (u32)((N + UM_NT - 1) / UM_NT), kt_all = Kp / UM_KT;
    const u32 base = n_tiles * tiles;
    u32 splits = 1, S = 1;
    double best = 1e30;
    for (u32 cl = 1; cl <= 4; cl *= 2) {
        const u32 slots = cl == 4 ? (u32)c->sm_count * 7 / 8 : (u32)c->sm_count;
        for (u32 sp = 1; sp * cl <= 64 && sp * cl <= kt_all; sp++) {
            const u64 ctas = (u64)base * sp * cl;
            const double waves = (double)((ctas + slots - 1) / slots), stages = (double)((kt_all + sp * cl - 1) / (sp * cl));
            const double cost = waves * (stages * 1.3e-6 + (cl > 1 ? 3e-6 : 0.0)) + (sp > 1 ? (double)sp * (double)t_rows * (double)N / 195e9 : 0.0);
            if (cost < best * 0.98) { best = cost; splits = sp * cl; S = cl; }
        }
    }
    int flag = 0;
    if (!rc) {
        Timed t(c, HL_T_WITNESS);
        // the plane is cleared unless the product kernel writes every word of it exactly once
        const bool dense = splits == S && os == N && out_len == t_rows * N;
        // the kernels after the packing may start beside the one before them and wait inside for what they read
        cudaLaunchAttribute at[2];
        at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[0].val.programmaticStreamSerializationAllowed = 1;
        at[1].id = cudaLaunchAttributeClusterDimension;
        at[1].val.clusterDim.x = 1; at[1].val.clusterDim.y = S; at[1].val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.stream = c->stream; cfg.attrs = at;
        k_wp_pack<<<dim3((Kp + 1023) / 1024, tiles * WP_MT), 256, 0, c->stream>>>((const long long*)d_x, xs, (u32)t_rows, (u32)K, Kp, d_a, d_flag,
                                                                                   (long long*)d_out, dense ? 0 : out_len);
        cudaError_t e = cudaGetLastError();
        c->stats.kernel_launches++;
        if (e == cudaSuccess && b_bytes) {
            cfg.gridDim = dim3(Kp / 128, (unsigned)(n_pad / 128)); cfg.blockDim = dim3(256); cfg.dynamicSmemBytes = 0; cfg.numAttrs = 1;
            e = cudaLaunchKernelEx(&cfg, k_wp_repack, d_w, K * N, (u32)K, (u32)N, Kp, in_out, d_b);
            c->stats.kernel_launches++;
        }
        const size_t smem = (size_t)UM_STAGES * UM_STAGE_BYTES + 1024;
        if (e == cudaSuccess && !c->wp_attr) {
            e = cudaFuncSetAttribute(k_wp_umma, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            c->wp_attr = e == cudaSuccess;
        }
        if (e == cudaSuccess) {
            cfg.gridDim = dim3(n_tiles, splits, tiles); cfg.blockDim = dim3(UM_THREADS); cfg.dynamicSmemBytes = smem; cfg.numAttrs = 2;
            e = cudaLaunchKernelEx(&cfg, k_wp_umma, map_a, map_b, (u32)N, Kp, (u32)t_rows, os, (long long*)d_out, d_flag, S, (u32)(in_place ? 1 : 0));
            c->stats.kernel_launches++;
        }
        if (e != cudaSuccess) rc = fail(c, HL_B200_ERR_DEVICE, "witness product launch", e);
    }
    if (!rc) rc = sync(c, "witness_product");
    if (d_flag) {
        flag = *reinterpret_cast<volatile int*>(d_flag);
        *d_flag = 0;  // for the next call
    }
    if (d_a) dev_free(c, d_a, a_bytes);
    if (d_b) dev_free(c, d_b, b_bytes);
    if (!rc && flag == 2) rc = fail(c, HL_B200_ERR_TIMEOUT, "witness product: a bounded wait on the tensor-core pipeline ran out");
    if (!rc) *taken = flag ? 0 : 1;
    return rc;
}

// witness_product_with's `fits` (metal.rs:4662-4674)
bool shape_fits(size_t t_rows, size_t x_len, size_t xs, size_t w_len, size_t inner, size_t outer, size_t os, size_t out_len) {
    // the reference's bounds are 2^30 rows and columns; the grids here take 2^15 rows and 2^21 columns
    if (t_rows < 1 || inner < 1 || outer < 1 || inner > WP_MAX_K || t_rows > ((size_t)1 << 15) || outer > ((size_t)1 << 21)) return false;
    if (xs < inner || os < outer || os > 0xFFFFFFFFull) return false;
    if (xs > ((size_t)1 << 40) || (t_rows - 1) * xs + inner > x_len) return false;
    if ((t_rows - 1) * os + outer > out_len) return false;
    return inner * outer <= w_len;
}

}  // namespace

extern "C" {

int hl_b200_witness_product_dev(hl_ctx* c, size_t t_rows, const int64_t* d_x, size_t x_len, size_t xs, const int8_t* d_w, size_t w_len, size_t inner,
                                size_t outer, size_t os, size_t out_len, int in_out, int64_t* d_out, int* taken) {
    if (!c || !taken) return fail(c, HL_B200_ERR_ARG, "witness_product: null argument");
    *taken = 0;
    if (!shape_fits(t_rows, x_len, xs, w_len, inner, outer, os, out_len)) return HL_B200_OK;
    if (!d_x || !d_w || !d_out) return fail(c, HL_B200_ERR_ARG, "witness_product: null argument");
    Call g(c);
    return product_on_device(c, t_rows, d_x, xs, d_w, inner, outer, os, out_len, in_out, d_out, taken);
}

int hl_b200_witness_product(hl_ctx* c, size_t t_rows, const int64_t* x, size_t x_len, size_t xs, const int8_t* w, size_t w_len, size_t inner,
                            size_t outer, size_t os, size_t out_len, int in_out, int64_t* out, int* taken) {
    if (!c || !taken) return fail(c, HL_B200_ERR_ARG, "witness_product: null argument");
    *taken = 0;
    if (!shape_fits(t_rows, x_len, xs, w_len, inner, outer, os, out_len)) return HL_B200_OK;
    if (!x || !w || !out) return fail(c, HL_B200_ERR_ARG, "witness_product: null argument");
    Call g(c);
    const size_t xb = ((t_rows - 1) * xs + inner) * 8, wb = inner * outer, ob = out_len * 8;
    int64_t *d_x = nullptr, *d_out = nullptr;
    int8_t* d_w = nullptr;
    int rc = dev_alloc(c, (void**)&d_x, xb);
    if (!rc) rc = dev_alloc(c, (void**)&d_w, wb);
    if (!rc) rc = dev_alloc(c, (void**)&d_out, ob);
    if (!rc) rc = h2d(c, d_x, x, xb);
    if (!rc) rc = h2d(c, d_w, w, wb);
    if (!rc) rc = product_on_device(c, t_rows, d_x, xs, d_w, inner, outer, os, out_len, in_out, d_out, taken);
    if (!rc && *taken) rc = d2h(c, out, d_out, ob);
    if (!rc) rc = sync(c, "witness_product");
    if (d_x) dev_free(c, d_x, xb);
    if (d_w) dev_free(c, d_w, wb);
    if (d_out) dev_free(c, d_out, ob);
    return rc;
}

}  // extern "C"
