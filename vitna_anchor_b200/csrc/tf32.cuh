// Products of float32 operands on the tensor cores with float32's precision, for the chunked recurrences.
//
// Products take float32 operands as two tf32 parts (x = high + low, 11 bits each and low's sign: 23 bits; high high + high low + low high, the eight terms of a k step
// summed by the tensor core and the steps in float32); the tensor cores do 159 such multiply-adds a cycle and multiprocessor where the float32 units do 124 and
// would need every operand from shared memory again for every 4 x 4 outputs.  Two bfloat16 parts would be twice as fast and lose a float32 state's last 7 bits.
#pragma once

#include <stdint.h>

namespace vk {

__device__ __forceinline__ void tf_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT> __device__ __forceinline__ void tf_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory"); }

__device__ __forceinline__ float tf_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// a float32 operand as two tf32 parts: its 11 leading bits rounded to the nearest, and the 11 leading bits (the tensor core does not read the others)
// of the at most 12 that this leaves.  A NaN or an infinity is a NaN in the low part, made by the subtraction: the sum on the bits may carry a NaN's
// high part over into the sign (0x7fffffff, which the arithmetic instructions make, becomes -0).  (cvt.rna.tf32 for the high part: 2 to 6 % of a mixer slower.)
struct Tf { uint32_t hi, lo; };
__device__ __forceinline__ Tf tf_split(float x) {
    const uint32_t hi = (__float_as_uint(x) + 0x1000u) & 0xffffe000u;
    return Tf{hi, __float_as_uint(x - __uint_as_float(hi))};
}
__device__ __forceinline__ bool tf_finite(float x) { return fabsf(x) <= 3.402823466e38f; }
__device__ __forceinline__ void tf_mma(float* d, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// d[m][n] += a[m] b[n] in three products a k step, the small ones first, on sums that begin at zero and are added to d in float32: the tensor core truncates what it
// adds, and sums that ran through a whole contraction there were 1.5 to 3 times as far from 64 bits as the float32 chains (mLSTM, 2,048 tokens, 8 heads of
// 128 x 256: outputs 5.7e-7 off, token after token 1.9e-7, this way 1.9e-7; gated linear attention 6.5e-7, 2.1e-7, 1.8e-7).  It costs 2 to 4 % of a mixer.
// Products of one sum stand M N instructions apart.
template <int M, int N>
__device__ __forceinline__ void tf_mma3(float* const (&d)[M][N], const Tf (&a)[M][4], const Tf (&b)[N][2]) {
    float t[M][N][4];
#pragma unroll
    for (int m = 0; m < M; m++)
#pragma unroll
        for (int n = 0; n < N; n++) {
            t[m][n][0] = t[m][n][1] = t[m][n][2] = t[m][n][3] = 0.0f;
            tf_mma(t[m][n], a[m][0].lo, a[m][1].lo, a[m][2].lo, a[m][3].lo, b[n][0].hi, b[n][1].hi);
        }
#pragma unroll
    for (int m = 0; m < M; m++)
#pragma unroll
        for (int n = 0; n < N; n++) tf_mma(t[m][n], a[m][0].hi, a[m][1].hi, a[m][2].hi, a[m][3].hi, b[n][0].lo, b[n][1].lo);
#pragma unroll
    for (int m = 0; m < M; m++)
#pragma unroll
        for (int n = 0; n < N; n++) tf_mma(t[m][n], a[m][0].hi, a[m][1].hi, a[m][2].hi, a[m][3].hi, b[n][0].hi, b[n][1].hi);
#pragma unroll
    for (int m = 0; m < M; m++)
#pragma unroll
        for (int n = 0; n < N; n++)
#pragma unroll
            for (int e = 0; e < 4; e++) d[m][n][e] += t[m][n][e];
}

}  // namespace vk
