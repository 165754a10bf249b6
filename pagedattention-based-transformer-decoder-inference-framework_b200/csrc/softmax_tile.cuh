// softmax_tile.cuh -- the exponentials of one query row over a tile of 64 scores held in registers (attention_tc.cu): one thread per row,
// two warps per scheduler.
//
// The special-function unit gives 16 exponentials a cycle and SM: 1024 cycles for the 256 rows of a CTA's two query tiles and 64 keys,
// about as much as the tensor pipe needs for them (1235).  Measured in a loop of their own, two warps a scheduler, with their maximum
// and sums: 1050 cycles; with one in four of them as a polynomial on the FMA pipe 980 there, but no faster in the kernels.
#pragma once
#include "f32x2.cuh"
#include "pa_common.cuh"

namespace pa {
namespace smx {

using namespace f32x2;

__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
// Largest of the 64 scores
__device__ __forceinline__ float row_max(const uint32_t (&s)[2][32]) {
    float m[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
    for (int k = 0; k < 32; ++k) m[k & 3] = max3(m[k & 3], __uint_as_float(s[k >> 4][(2 * k) & 31]), __uint_as_float(s[k >> 4][(2 * k + 1) & 31]));
    return fmaxf(fmaxf(m[0], m[1]), fmaxf(m[2], m[3]));
}

// Half of the row: w = pack(2^(s fe - ref)) of its 32 scores, two to a word; their sum is added to acc (two by two)
template <typename Pack>
__device__ __forceinline__ void exp_half(const uint32_t (&s)[32], float fe, float ref, uint32_t (&w)[16], uint64_t (&acc)[2], Pack pack) {
    const uint64_t f2 = pack2(fe, fe), r2 = pack2(-ref, -ref);
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        float e0, e1;
        unpack2(fma2(pack2(__uint_as_float(s[2 * k]), __uint_as_float(s[2 * k + 1])), f2, r2), e0, e1);
        e0 = fast_exp2(e0);
        e1 = fast_exp2(e1);
        acc[k & 1] = add2(acc[k & 1], pack2(e0, e1));
        w[k] = pack(e0, e1);
    }
}
__device__ __forceinline__ float sum_of(const uint64_t (&acc)[2]) {
    float lo, hi;
    unpack2(add2(acc[0], acc[1]), lo, hi);
    return lo + hi;
}

}  // namespace smx
}  // namespace pa
