// 5th-generation tensor cores, integer form: the few instructions that the library's kernels use (tcgen05.mma kind::i8 on operands in
// shared memory, accumulators in TMEM), and bounded waits.
#pragma once
#include "gl_field.cuh"

constexpr u32 UM_SBO = 1024;  // bytes between 8-row groups of an operand
constexpr u32 UM_SPIN_LIMIT = 1u << 22;  // some seconds

// K-major operand with the 128-byte swizzle: rows of 128 bytes, 8-row groups UM_SBO apart, a K step of 32 bytes is 32 bytes further
// along the row.  Start address and stride byte offset in 16-byte units (the leading offset is not used by a swizzled K-major operand
// and is set to 1 as the canonical form has it); descriptor version 1; layout type 2 = 128-byte swizzle
__device__ __forceinline__ u64 um_desc(u32 smem_addr) {
    return (u64)((smem_addr >> 4) & 0x3FFF) | (1ull << 16) | ((u64)(UM_SBO >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// instruction descriptor of kind::i8: D = s32, each operand signed or unsigned bytes, both K-major, M x N
__host__ __device__ constexpr u32 um_idesc(bool a_signed, bool b_signed, u32 m, u32 n) {
    return (2u << 4) | ((a_signed ? 1u : 0u) << 7) | ((b_signed ? 1u : 0u) << 10) | ((n >> 3) << 17) | ((m >> 4) << 24);
}

__device__ __forceinline__ void um_mma(u32 tmem_d, u64 a_desc, u64 b_desc, u32 idesc, u32 accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}\n" ::"r"(tmem_d),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(0u)
        : "memory");
}
__device__ __forceinline__ void um_commit(u32 mbar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(mbar) : "memory");
}
__device__ __forceinline__ bool um_try_wait(u32 mbar, u32 parity) {
    u32 ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
                 : "=r"(ok)
                 : "r"(mbar), "r"(parity)
                 : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool um_wait(u32 mbar, u32 parity) {
    for (u32 spin = 0; spin < UM_SPIN_LIMIT; spin++)
        if (um_try_wait(mbar, parity)) return true;
    return false;
}
__device__ __forceinline__ void um_ld32(u32 taddr, u32 (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, "
        "%23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
          "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
          "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
}
