// The epilogue activations shared by the GEMM store, the matrix-vector store and the stand-alone
// activation op (reference ops.jl:161-169,1665-1685): one definition, so a folded activation and the op it
// replaced give the same bits.
#pragma once
#include <cuda_fp16.h>

#include "../../include/b200dnn.h"
#include "ptx.cuh"

namespace b200 {

// geluexact on the fp16-rounded value (ops.jl:161-169,1665-1670): 0.5 x (1 + erf(x / sqrt 2)) with the reference's erf,
// Abramowitz & Stegun 7.1.26, as  relu(x) - |x| F(-|x|)  with  F(-q) = 2^P(q): F is 0.5 poly(t) exp(-q^2 / 2) of 7.1.26, P a
// polynomial of degree nine fitted (least squares on Chebyshev nodes, reweighted towards the smallest largest error) to its
// log2 on [0, 6].  Past 6 the second term is below half the smallest fp16 value; up to 9 P goes on falling with the function
// (|x| F off by 2.2e-11 at most, less than leaving the term out would be), and from there the smallest float stands for F, so
// that fp32 results go to zero (-1.3e-44) and fp16 ones to the packed form's.  Against 64 bits and the true erf, in
// brackets 7.1.26 step by step in fp32: over the fp16 grid 250 values round to another neighbour (458), fp32 results of
// N(0, 0.1), N(0, 1) and N(0, 3) are off by 1.0e-7, 8.1e-8 and 4.7e-8 in the 2-norm (1.5e-7, 8.5e-8, 4.9e-8).  One
// exponential an element and no sign to carry: a pair takes some 20 instructions where the steps take 32, two MUFU
// operations instead of four, and those bound the GEMM store of a short-K product (524288 x 448 x 112: 239 -> 222 us).
// Infinities and NaN give what the formula gives.
// Every multiply, add and fused multiply-add is spelled out, so that the packed form below, which the GEMM
// store uses, performs the same roundings and gives the same bits.
__device__ __forceinline__ constexpr float gelu_p(int i) {   // P's coefficients, of -q, ascending
    constexpr float c[10] = {-1.0f, 1.151112f, -0.45914048f, 0.052712347f, 0.0073685716f,
                             0.00034979929f, -0.00011288216f, -2.9053328e-05f, -2.9679443e-06f, -1.1896606e-07f};
    return c[i];
}

__device__ __forceinline__ float gelu_exact(float x) {
    const float nq = fmaxf(-fabsf(x), -9.0f);
    float p = gelu_p(9);
#pragma unroll
    for (int i = 8; i >= 0; --i) p = __fmaf_rn(p, nq, gelu_p(i));
    float g;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(g) : "f"(p));
    if (fabsf(x) > 9.0f) g = __uint_as_float(1u);
    const float hx = __fmul_rn(0.5f, x);
    return __fmaf_rn(nq, g, __fadd_rn(hx, fabsf(hx)));
}

// The same function on a pair, with the multiplies and FMAs as packed fp32-pair instructions (sm_100): half
// the instructions per element in the GEMM store, where the activation is what a short-K tile waits for.  For results that
// are rounded to fp16: past 9 it keeps P(-9), whose 2.0e-18 rounds to the same zero.
__device__ __forceinline__ uint64_t dup2(float c) { return pack2(c, c); }

__device__ __forceinline__ float2 gelu_exact2(float2 x) {
    const uint64_t nq = pack2(fmaxf(-fabsf(x.x), -9.0f), fmaxf(-fabsf(x.y), -9.0f));
    uint64_t p = dup2(gelu_p(9));
#pragma unroll
    for (int i = 8; i >= 0; --i) p = fma2(p, nq, dup2(gelu_p(i)));
    float p0, p1, g0, g1, h0, h1, r0, r1;
    unpack2(p, p0, p1);
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(g0) : "f"(p0));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(g1) : "f"(p1));
    unpack2(mul2(dup2(0.5f), pack2(x.x, x.y)), h0, h1);
    unpack2(fma2(nq, pack2(g0, g1), pack2(__fadd_rn(h0, fabsf(h0)), __fadd_rn(h1, fabsf(h1)))), r0, r1);
    return make_float2(r0, r1);
}
__device__ __forceinline__ float apply_act(int epi, float v) {
    switch (epi) {
        case B200_EPI_RELU: return fmaxf(v, 0.f);
        case B200_EPI_GELU: return gelu_exact(v);
        case B200_EPI_GELU_TANH: {
            float u = 0.7978845608028654f * (v + 0.044715f * v * v * v);
            return 0.5f * v * (1.0f + tanhf(u));
        }
        default: return v;
    }
}

} // namespace b200
