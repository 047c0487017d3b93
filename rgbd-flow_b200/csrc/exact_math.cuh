// exact_math.cuh — correctly rounded FP32 quotients and square roots without the general routines' branches.
//
// The linearisation of a pixel takes 26 quotients and 7 inverse square roots.  IEEE division and square root
// of FP32 are each a dozen instructions around a branch to a routine for the operands that need care, which
// keeps neighbouring ones from overlapping.  Here the operands' range is looked at once for several results,
// and the results are computed in one straight line by Newton steps and a final correction by the exact
// remainder (P. Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor", IBM J.
// Res. Dev. 34 (1990): with y = 1/b rounded and q within an ulp of a / b, q + (a - b q) y rounds to the quotient
// rounded).  Outside the range the operators are used, so the inverse square roots and reciprocals are theirs bit for
// bit, and the quotients by whole numbers too but for a zero's sign and the last bit of some below 2^-126 (div_small).
// The quotients by the Laplacian's weights stay with the operator.  Instructions of a linearised pixel 1503 -> 1361, branches 97 ->
// 33; k_linearize on 640x480 (cold caches) 41.0 -> 35.6 us.
#pragma once
#include <cuda_runtime.h>

namespace rgbdflow {

__device__ __forceinline__ float approx_rcp(float x)
{
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float approx_rsqrt(float x)
{
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// x from 2^-62 to below 2^63 (|x| by the other): no step below over- or underflows.
__device__ __forceinline__ bool mid_range_pos(float x) { return __float_as_uint(x) - 0x20800000u < 0x3e800000u; }
__device__ __forceinline__ bool mid_range(float x) { return (__float_as_uint(x) & 0x7fffffffu) - 0x20800000u < 0x3e800000u; }

// x / D for a small whole D.  The remainder of the product with the rounded 1 / D is exact, so one step corrects it.
// -0 / D is +0 here, and a quotient below 2^-126 that lies halfway between two numbers may go to the other one.
template <int D>
__device__ __forceinline__ double div_small(double x) { return x / D; }
template <int D>
__device__ __forceinline__ float div_small(float x)
{
    constexpr float r = 1.0f / D;
    const float q = __fmul_rn(x, r);
    const float c = __fmaf_rn(__fmaf_rn(-(float)D, q, x), r, q);
    return fabsf(q) < __int_as_float(0x7f800000) ? c : q;  // an infinite or NaN one has no remainder
}

// y[i] = 1 / sqrt(x[i]), each operation rounded.
template <class T, int N>
__device__ __forceinline__ void inv_sqrt(const T* x, T* y)
{
    if constexpr (sizeof(T) == 8) {
        for (int i = 0; i < N; i++) y[i] = 1.0 / ::sqrt(x[i]);
    } else {
        float in[N];
        bool ok = true;
#pragma unroll
        for (int i = 0; i < N; i++) {
            in[i] = x[i];
            ok = ok && mid_range_pos(in[i]);
        }
        if (ok) {
#pragma unroll
            for (int i = 0; i < N; i++) {
                const float r0 = approx_rsqrt(in[i]);
                const float g0 = __fmul_rn(in[i], r0), h0 = __fmul_rn(0.5f, r0);
                const float d0 = __fmaf_rn(-g0, h0, 0.5f);
                const float g1 = __fmaf_rn(g0, d0, g0), h1 = __fmaf_rn(h0, d0, h0);
                const float s = __fmaf_rn(__fmaf_rn(-g1, g1, in[i]), h1, g1);  // sqrt(x)
                // not from 2 h1: where s is all ones, its error leaves 1 / s at a tie
                const float y0 = approx_rcp(s);
                const float y1 = __fmaf_rn(__fmaf_rn(-s, y0, 1.0f), y0, y0);
                y[i] = __fmaf_rn(__fmaf_rn(-s, y1, 1.0f), y1, y1);
            }
        } else {
#pragma unroll
            for (int i = 0; i < N; i++) y[i] = 1.0f / sqrtf(in[i]);
        }
    }
}

// x[i] = 1 / x[i].
template <class T, int N>
__device__ __forceinline__ void inverse(T* x)
{
    if constexpr (sizeof(T) == 8) {
        for (int i = 0; i < N; i++) x[i] = 1.0 / x[i];
    } else {
        bool ok = true;
#pragma unroll
        for (int i = 0; i < N; i++) ok = ok && mid_range(x[i]);
        if (ok) {
#pragma unroll
            for (int i = 0; i < N; i++) {
                const float y0 = approx_rcp(x[i]);
                const float y1 = __fmaf_rn(__fmaf_rn(-x[i], y0, 1.0f), y0, y0);
                x[i] = __fmaf_rn(__fmaf_rn(-x[i], y1, 1.0f), y1, y1);
            }
        } else {
#pragma unroll
            for (int i = 0; i < N; i++) x[i] = 1.0f / x[i];
        }
    }
}

}  // namespace rgbdflow
