// The closed-form slot polynomials of the sumcheck kernels, at one point (ids and meaning in sumcheck.h).
#pragma once
#include "gl_field.cuh"
#include "sumcheck.h"

namespace hlk {

template <int POLY, int K>
__device__ __forceinline__ fp2 poly_eval(const fp2 (&v)[K], const fp2* __restrict__ coefs) {
    if constexpr (POLY == POLY_PROD) {
        fp2 a = v[0];
#pragma unroll
        for (int t = 1; t < K; t++) a = f2_mul(a, v[t]);
        return a;
    } else if constexpr (POLY == POLY_ZC) {
        return f2_mul(v[0], f2_sub(f2_mul(v[1], v[2]), v[3]));
    } else if constexpr (POLY == POLY_LOGUP_Q) {
        return f2_mul(v[0], f2_sub(f2_mul(v[1], f2_sub(coefs[0], v[2])), f2(1, 0)));
    } else {
        return f2_mul(v[0], f2_sub(f2_mul(v[1], f2_sub(coefs[0], v[2])), v[3]));
    }
}

}  // namespace hlk
