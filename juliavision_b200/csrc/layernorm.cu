// LayerNorm over the leading (contiguous) axis: one read of the input, one write of the
// output.  Bandwidth-bound: 16-byte vector loads, the whole group held in registers, fp32
// statistics reduced with warp shuffles, variance taken about the mean (two passes over
// registers, never E[x^2]-mean^2).
//
// Replaces layernorm_kernel! (reference kernels/layernorm.jl:44-114): 128 threads per
// group, shared-memory tree reductions and three strided passes over the group.
#include <cuda_fp16.h>

#include "internal.h"
#include "ptx.cuh"

namespace b200 {

template <typename T> struct Vec16;
template <> struct Vec16<__half> {
    static constexpr int N = 8;
    uint4 raw;
    __device__ __forceinline__ void to_f32(float* f) const {
        const __half2* h = reinterpret_cast<const __half2*>(&raw);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float2 t = __half22float2(h[i]);
            f[2 * i] = t.x;
            f[2 * i + 1] = t.y;
        }
    }
};
template <> struct Vec16<float> {
    static constexpr int N = 4;
    uint4 raw;
    __device__ __forceinline__ void to_f32(float* f) const {
        const float* p = reinterpret_cast<const float*>(&raw);
#pragma unroll
        for (int i = 0; i < 4; ++i) f[i] = p[i];
    }
};

template <int N> __device__ __forceinline__ void store_vec(__half* dst, const float* f) {
    static_assert(N == 8 || N == 4, "vector width");
    if constexpr (N == 8) {
        uint4 o;
        __half2* h = reinterpret_cast<__half2*>(&o);
#pragma unroll
        for (int i = 0; i < 4; ++i) h[i] = __floats2half2_rn(f[2 * i], f[2 * i + 1]);
        *reinterpret_cast<uint4*>(dst) = o;
    } else {
        uint2 o;
        __half2* h = reinterpret_cast<__half2*>(&o);
        h[0] = __floats2half2_rn(f[0], f[1]);
        h[1] = __floats2half2_rn(f[2], f[3]);
        *reinterpret_cast<uint2*>(dst) = o;
    }
}
template <int N> __device__ __forceinline__ void store_vec(float* dst, const float* f) {
#pragma unroll
    for (int i = 0; i < N; i += 4)
        *reinterpret_cast<float4*>(dst + i) = make_float4(f[i], f[i + 1], f[i + 2], f[i + 3]);
}

constexpr int LN_WIDE_THREADS = 256;   // block of a row too wide for one warp

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Sum over the LPG lanes of a group (LPG a power of two; the butterfly never leaves the aligned span).
template <int LPG>
__device__ __forceinline__ float group_sum(float v) {
#pragma unroll
    for (int o = LPG / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// The packed form (PACK): a row's moments and its output two elements per instruction, gamma and beta in one rounding.
// It is for launches whose rows come from and go to HBM (more than the L2 holds): 65536 x 1280 in fp16 63.1 -> 59.6 us
// (5.3 -> 5.6 TB/s, replayed over four operand sets), where the scalar form issues for about 25 us of the launch.  Rows that stay in the L2 are faster
// in the scalar form (14736 x 1176: 11.7 us, packed 12.9), so the row bytes decide, the same for the layer norm alone
// and the one behind a residual add, which therefore give the same bits.  The vectors of a lane are v = first,
// first + 32, ...; `x` is left holding x - mean.
__device__ __forceinline__ float pairs_sum(uint64_t s2) {
    float a, b;
    unpack2(s2, a, b);
    return a + b;
}
template <int VPL, int VN, int LPG>
__device__ __forceinline__ void ln_moments(uint64_t (&x)[VPL][VN / 2], int first, int nvec, int C, float eps, float& mu,
                                           float& r) {
    uint64_t s = pack2(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < VPL; ++i)
        if (first + 32 * i < nvec) {
#pragma unroll
            for (int j = 0; j < VN / 2; ++j) s = add2(s, x[i][j]);
        }
    const float n = (float)C;
    mu = group_sum<LPG>(pairs_sum(s)) / n;
    const uint64_t nmu = pack2(-mu, -mu);
    uint64_t s2 = pack2(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < VPL; ++i)
        if (first + 32 * i < nvec) {
#pragma unroll
            for (int j = 0; j < VN / 2; ++j) {
                x[i][j] = add2(x[i][j], nmu);
                s2 = fma2(x[i][j], x[i][j], s2);
            }
        }
    r = 1.0f / sqrtf(group_sum<LPG>(pairs_sum(s2)) / n + eps);
}
// One vector of the result: d = x - mean; y = d r, then gamma and beta in one rounding, or d r and beta in one.
template <typename InT, typename OutT>
__device__ __forceinline__ void ln_write(OutT* dst, const uint64_t* d, float r, bool has_g, const uint4& g, bool has_b,
                                         const uint4& b) {
    constexpr int VN = Vec16<InT>::N;
    Vec16<InT> tg, tb;
    float gf[VN], bf[VN], y[VN];
    tg.raw = g;
    tb.raw = b;
    if (has_g) tg.to_f32(gf);
    if (has_b) tb.to_f32(bf);
    const uint64_t rr = pack2(r, r);
#pragma unroll
    for (int j = 0; j < VN / 2; ++j) {
        uint64_t v;
        if (has_g && has_b) v = fma2(mul2(d[j], rr), pack2(gf[2 * j], gf[2 * j + 1]), pack2(bf[2 * j], bf[2 * j + 1]));
        else if (has_g) v = mul2(mul2(d[j], rr), pack2(gf[2 * j], gf[2 * j + 1]));
        else if (has_b) v = fma2(d[j], rr, pack2(bf[2 * j], bf[2 * j + 1]));
        else v = mul2(d[j], rr);
        unpack2(v, y[2 * j], y[2 * j + 1]);
    }
    store_vec<VN>(dst, y);
}

// One warp per group; lane l owns vectors l, l+32, ... (VPL of them at most).  Narrow groups (at most
// 16 or 8 vectors, VPL = 1) share a warp, LPG lanes each, so that no lane idles; the sums are the same
// butterflies with the empty upper steps left out, hence the same bits.
// LAT: the latency form, for launches small enough that every CTA is resident at once and what the kernel takes
// is a chain of round trips, not bytes (the encoder's 1500 rows): everything the row needs is asked for up front.
// It costs ~40 registers; launches of many waves, which want occupancy, take the lean form.
template <typename InT, typename OutT, int VPL, int LPG = 32, bool LAT = false, bool PACK = false>
__global__ void __launch_bounds__(128)
ln_warp_kernel(const InT* __restrict__ a, OutT* __restrict__ out, float* __restrict__ mean,
               float* __restrict__ rstd, const InT* __restrict__ gamma,
               const InT* __restrict__ beta, int64_t groups, int C, float eps) {
    constexpr int VN = Vec16<InT>::N;
    static_assert(LPG == 32 || VPL == 1, "only single-vector groups share a warp");
    static_assert(!(PACK && LAT), "the packed form is for launches of many waves");
    const int lane = threadIdx.x & (LPG - 1);
    const int64_t g = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / LPG;
    const int nvec = g < groups ? C / VN : 0;   // lanes past the last group idle through the shuffles
    const InT* src = a + g * (int64_t)C;
    // Narrow rows ask for gamma and beta together with the row, so that the normalised row does not wait for
    // them at the end (measured on the encoder pass with the add + layer-norm kernel below: 3.45 -> 3.37 ms).
    // Asking for them above the dependency wait would gain another 0.4 % when they are weights, and read stale
    // values when the previous kernel wrote them; nothing here knows which, so they are read below it.
    constexpr bool HOIST = LAT && VPL <= 6;
    grid_dep_wait();     // the input is the previous kernel's output
    grid_dep_launch();
    uint4 gw[HOIST ? VPL : 1], bw[HOIST ? VPL : 1];
    if constexpr (HOIST) {
#pragma unroll
        for (int i = 0; i < VPL; ++i) {
            const int v = lane + 32 * i;
            gw[i] = (gamma && v < nvec) ? __ldg(reinterpret_cast<const uint4*>(gamma) + v) : make_uint4(0u, 0u, 0u, 0u);
            bw[i] = (beta && v < nvec) ? __ldg(reinterpret_cast<const uint4*>(beta) + v) : make_uint4(0u, 0u, 0u, 0u);
        }
    }

    float mu, r;
    if constexpr (PACK) {
        uint64_t x[VPL][VN / 2];
#pragma unroll
        for (int i = 0; i < VPL; ++i) {
            const int v = lane + 32 * i;
            if (v < nvec) {
                Vec16<InT> t;
                float f[VN];
                t.raw = __ldg(reinterpret_cast<const uint4*>(src) + v);
                t.to_f32(f);
#pragma unroll
                for (int j = 0; j < VN / 2; ++j) x[i][j] = pack2(f[2 * j], f[2 * j + 1]);
            }
        }
        ln_moments<VPL, VN, LPG>(x, lane, nvec, C, eps, mu, r);
        OutT* dst = out + g * (int64_t)C;
#pragma unroll
        for (int i = 0; i < VPL; ++i) {
            const int v = lane + 32 * i;
            if (v < nvec) {
                uint4 gv = make_uint4(0u, 0u, 0u, 0u), bv = gv;
                if (gamma) gv = __ldg(reinterpret_cast<const uint4*>(gamma) + v);
                if (beta) bv = __ldg(reinterpret_cast<const uint4*>(beta) + v);
                ln_write<InT, OutT>(dst + (int64_t)v * VN, x[i], r, gamma != nullptr, gv, beta != nullptr, bv);
            }
        }
    } else {
        float x[VPL][VN];
        float s = 0.f;
#pragma unroll
        for (int i = 0; i < VPL; ++i) {
            int v = lane + 32 * i;
            if (v < nvec) {
                Vec16<InT> t;
                t.raw = __ldg(reinterpret_cast<const uint4*>(src) + v);
                t.to_f32(x[i]);
#pragma unroll
                for (int j = 0; j < VN; ++j) s += x[i][j];
            }
        }
        const float n = (float)C;
        mu = group_sum<LPG>(s) / n;
        float s2 = 0.f;
#pragma unroll
        for (int i = 0; i < VPL; ++i) {
            if (lane + 32 * i < nvec) {
#pragma unroll
                for (int j = 0; j < VN; ++j) {
                    float d = x[i][j] - mu;
                    s2 += d * d;
                }
            }
        }
        r = 1.0f / sqrtf(group_sum<LPG>(s2) / n + eps);

        OutT* dst = out + g * (int64_t)C;
#pragma unroll
        for (int i = 0; i < VPL; ++i) {
            int v = lane + 32 * i;
            if (v < nvec) {
                float y[VN];
#pragma unroll
                for (int j = 0; j < VN; ++j) y[j] = (x[i][j] - mu) * r;
                if (gamma) {
                    Vec16<InT> t;
                    float gf[VN];
                    if constexpr (HOIST) t.raw = gw[i];
                    else t.raw = __ldg(reinterpret_cast<const uint4*>(gamma) + v);
                    t.to_f32(gf);
#pragma unroll
                    for (int j = 0; j < VN; ++j) y[j] *= gf[j];
                }
                if (beta) {
                    Vec16<InT> t;
                    float bf[VN];
                    if constexpr (HOIST) t.raw = bw[i];
                    else t.raw = __ldg(reinterpret_cast<const uint4*>(beta) + v);
                    t.to_f32(bf);
#pragma unroll
                    for (int j = 0; j < VN; ++j) y[j] += bf[j];
                }
                store_vec<VN>(dst + (int64_t)v * VN, y);
            }
        }
    }
    if (lane == 0 && g < groups) {
        mean[g] = mu;
        rstd[g] = r;
    }
}

// Residual add (+ optional clamp) fused in front of the layer norm, fp16 only:
//     x <- clamp(fp16(x + h), lo, hi);   out <- LN(x)
// Bit-identical to running add.Tensor, clamp.default and native_layer_norm one after another
// (each rounds to fp16 where the separate ops would), but x and h are read once and the three
// launches become one.
// PAIRS: the order of the packed form, whose bits these are to be where the layer norm alone takes it, in scalar
// instructions: even and odd elements summed apart, gamma and beta (or the deviation and beta) in one rounding.  As packed
// instructions the row's two inputs and its pairs left a third fewer warps in flight (65536 x 1280: 136 us, 118.6 this way,
// 117.2 in the plain order; 43000 x 1480: 121, 104.0, 102.4); the bound on registers is the plain order's own count.
template <int VPL, int LPG = 32, bool LAT = false, bool PAIRS = false>
__global__ void __launch_bounds__(128, PAIRS ? (VPL <= 5 ? 8 : 7) : 0)
ln_add_warp_kernel(__half* __restrict__ x, const __half* __restrict__ h, __half* __restrict__ out,
                   float* __restrict__ mean, float* __restrict__ rstd, const __half* __restrict__ gamma,
                   const __half* __restrict__ beta, int64_t groups, int C, float eps, int use_clamp, float lo,
                   float hi) {
    constexpr int VN = 8;
    static_assert(LPG == 32 || VPL == 1, "only single-vector groups share a warp");
    static_assert(!(PAIRS && LAT), "the packed form is for launches of many waves");
    const int lane = threadIdx.x & (LPG - 1);
    const int64_t g = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / LPG;
    const int nvec = g < groups ? C / VN : 0;
    // gamma and beta are asked for together with the row (after the dependency wait: the previous kernel may have
    // written them), so that the normalised row does not wait for them at the end.
    // (Rows of up to 1536 elements; wider ones would spill, and read them where they are used.)
    constexpr bool HOIST = LAT && VPL <= 6;
    grid_dep_wait();     // x and h are the previous kernels' outputs
    grid_dep_launch();
    uint4 gw[HOIST ? VPL : 1], bw[HOIST ? VPL : 1];
    if constexpr (HOIST) {
#pragma unroll
        for (int i = 0; i < VPL; ++i) {
            const int vi = lane + 32 * i;
            gw[i] = (gamma && vi < nvec) ? __ldg(reinterpret_cast<const uint4*>(gamma) + vi) : make_uint4(0u, 0u, 0u, 0u);
            bw[i] = (beta && vi < nvec) ? __ldg(reinterpret_cast<const uint4*>(beta) + vi) : make_uint4(0u, 0u, 0u, 0u);
        }
    }
    __half* xr = x + g * (int64_t)C;
    const __half* hr = h + g * (int64_t)C;

    // every load of the row first, then the arithmetic: one round trip for the row whatever the compiler would
    // have made of loads and stores through the same pointer
    // (the latency form; the lean one reads each vector where it uses it)
    uint4 xraw[HOIST ? VPL : 1], hraw[HOIST ? VPL : 1];
    if constexpr (HOIST) {
#pragma unroll
        for (int i = 0; i < VPL; ++i) {
            const int vi = lane + 32 * i;
            if (vi < nvec) {
                xraw[i] = *(reinterpret_cast<const uint4*>(xr) + vi);
                hraw[i] = __ldg(reinterpret_cast<const uint4*>(hr) + vi);
            }
        }
    }
    float v[VPL][VN];
    float s = 0.f, so = 0.f;   // so: the odd elements' sum with PAIRS
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
        const int vi = lane + 32 * i;
        if (vi < nvec) {
            Vec16<__half> a, b;
            if constexpr (HOIST) {
                a.raw = xraw[i];
                b.raw = hraw[i];
            } else {
                a.raw = *(reinterpret_cast<const uint4*>(xr) + vi);
                b.raw = __ldg(reinterpret_cast<const uint4*>(hr) + vi);
            }
            float fa[VN], fb[VN];
            a.to_f32(fa);
            b.to_f32(fb);
#pragma unroll
            for (int j = 0; j < VN; ++j) {
                float t = __half2float(__float2half_rn(fa[j] + fb[j]));        // add.Tensor rounds here
                if (use_clamp) t = __half2float(__float2half_rn(fminf(fmaxf(t, lo), hi)));
                v[i][j] = t;
                if (PAIRS && (j & 1)) so += t;
                else s += t;
            }
            store_vec<VN>(xr + (int64_t)vi * VN, v[i]);                         // exact: already fp16 values
        }
    }
    const float n = (float)C;
    const float mu = group_sum<LPG>(PAIRS ? s + so : s) / n;
    float s2 = 0.f, s2o = 0.f;
#pragma unroll
    for (int i = 0; i < VPL; ++i)
        if (lane + 32 * i < nvec) {
#pragma unroll
            for (int j = 0; j < VN; ++j) {
                float d = v[i][j] - mu;
                if (PAIRS && (j & 1)) s2o = fmaf(d, d, s2o);
                else s2 = fmaf(d, d, s2);
            }
        }
    const float r = 1.0f / sqrtf(group_sum<LPG>(PAIRS ? s2 + s2o : s2) / n + eps);
    __half* dst = out + g * (int64_t)C;
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
        const int vi = lane + 32 * i;
        if (vi < nvec) {
            if constexpr (PAIRS) {   // two elements at a time: whole vectors of gamma and beta beside the row would spill
                uint4 gv = make_uint4(0u, 0u, 0u, 0u), bv = gv, ov;
                if (gamma) gv = __ldg(reinterpret_cast<const uint4*>(gamma) + vi);
                if (beta) bv = __ldg(reinterpret_cast<const uint4*>(beta) + vi);
                const __half2 *gh = reinterpret_cast<const __half2*>(&gv), *bh = reinterpret_cast<const __half2*>(&bv);
#pragma unroll
                for (int j = 0; j < VN / 2; ++j) {
                    const float2 g2 = __half22float2(gh[j]), b2 = __half22float2(bh[j]);
                    const float d0 = v[i][2 * j] - mu, d1 = v[i][2 * j + 1] - mu;
                    float y0 = __fmul_rn(d0, r), y1 = __fmul_rn(d1, r);
                    if (gamma && beta) {
                        y0 = fmaf(y0, g2.x, b2.x);
                        y1 = fmaf(y1, g2.y, b2.y);
                    } else if (gamma) {
                        y0 *= g2.x;
                        y1 *= g2.y;
                    } else if (beta) {
                        y0 = fmaf(d0, r, b2.x);
                        y1 = fmaf(d1, r, b2.y);
                    }
                    reinterpret_cast<__half2*>(&ov)[j] = __floats2half2_rn(y0, y1);
                }
                *(reinterpret_cast<uint4*>(dst) + vi) = ov;
                continue;
            }
            float y[VN];
#pragma unroll
            for (int j = 0; j < VN; ++j) y[j] = (v[i][j] - mu) * r;
            if (gamma) {
                Vec16<__half> t;
                float gf[VN];
                if constexpr (HOIST) t.raw = gw[i];
                else t.raw = __ldg(reinterpret_cast<const uint4*>(gamma) + vi);
                t.to_f32(gf);
#pragma unroll
                for (int j = 0; j < VN; ++j) y[j] *= gf[j];
            }
            if (beta) {
                Vec16<__half> t;
                float bf[VN];
                if constexpr (HOIST) t.raw = bw[i];
                else t.raw = __ldg(reinterpret_cast<const uint4*>(beta) + vi);
                t.to_f32(bf);
#pragma unroll
                for (int j = 0; j < VN; ++j) y[j] += bf[j];
            }
            store_vec<VN>(dst + (int64_t)vi * VN, y);
        }
    }
    if (lane == 0 && g < groups) {
        mean[g] = mu;
        rstd[g] = r;
    }
}

// Narrow rows (at most two vectors a lane) of launches of many waves: R rows per group of LPG lanes, so that a lane has R
// or more 16-byte loads in flight (2 R with the residual add in front, ADD) and gamma and beta are read once for all of them.
// Bound by HBM; with one row at a time the loads in flight were what bound it: 524288 x 112 fp16 69.0 -> 54.9 us (4.3 TB/s),
// 131072 x 224 35.6 -> 29.9, 200000 x 200 53.0 -> 43.3; behind the add 524288 x 112 86.2 -> 78.9 (6.0 TB/s), 32768 x 448
// 23.1 -> 20.6; smaller launches: ln_fills.  Eight rows lose (63.7: registers).  Alone, rows of two vectors a lane do not gain (32768 x 448 14.1 both
// ways, 16384 x 448 7.1 -> 7.4) and stay with ln_warp_kernel.  A row is kept as read (fp16 stays packed,
// also the sum x + h, which add.Tensor rounds to fp16), every operation and its order is that of the kernels
// above, hence the same bits.  The R rows' statistics leave in one store each.
template <typename InT, typename OutT, int VPL, int LPG, int R, bool ADD>
__global__ void __launch_bounds__(128)
ln_rows_kernel(const InT* a, InT* x, const InT* __restrict__ h, OutT* __restrict__ out, float* __restrict__ mean,
               float* __restrict__ rstd, const InT* __restrict__ gamma, const InT* __restrict__ beta, int64_t groups, int C,
               float eps, int use_clamp, float lo, float hi) {
    constexpr int VN = Vec16<InT>::N;
    constexpr int SIDE = 32 / LPG;   // rows side by side in a warp
    static_assert(LPG == 32 || VPL == 1, "only single-vector groups share a warp");
    static_assert(R <= LPG, "a lane per row writes the statistics");
    const int lane = threadIdx.x & (LPG - 1);
    const int64_t row0 = ((int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * (R * SIDE) + (threadIdx.x & 31) / LPG;
    const int nvec = C / VN;
    grid_dep_wait();     // the rows are the previous kernel's output
    grid_dep_launch();
    Vec16<InT> v[R][VPL], hv[ADD ? R : 1][ADD ? VPL : 1];
#pragma unroll
    for (int k = 0; k < R; ++k)
#pragma unroll
        for (int i = 0; i < VPL; ++i) {
            const int64_t g = row0 + k * SIDE;
            const int vi = lane + 32 * i;
            if (vi < nvec && g < groups) {
                v[k][i].raw = *(reinterpret_cast<const uint4*>((ADD ? x : a) + g * C) + vi);
                if constexpr (ADD) hv[k][i].raw = __ldg(reinterpret_cast<const uint4*>(h + g * C) + vi);
            } else {
                v[k][i].raw = make_uint4(0u, 0u, 0u, 0u);
            }
        }
    Vec16<InT> gw[VPL], bw[VPL];
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
        const int vi = lane + 32 * i;
        gw[i].raw = (gamma && vi < nvec) ? __ldg(reinterpret_cast<const uint4*>(gamma) + vi) : make_uint4(0u, 0u, 0u, 0u);
        bw[i].raw = (beta && vi < nvec) ? __ldg(reinterpret_cast<const uint4*>(beta) + vi) : make_uint4(0u, 0u, 0u, 0u);
    }
    float mu[R], r[R];
#pragma unroll
    for (int k = 0; k < R; ++k) {
        float s = 0.f;
#pragma unroll
        for (int i = 0; i < VPL; ++i) {
            const int vi = lane + 32 * i;
            if (vi < nvec) {
                float f[VN];
                v[k][i].to_f32(f);
                if constexpr (ADD) {
                    float fh[VN];
                    hv[k][i].to_f32(fh);
#pragma unroll
                    for (int j = 0; j < VN; ++j) {
                        f[j] = __half2float(__float2half_rn(f[j] + fh[j]));        // add.Tensor rounds here
                        if (use_clamp) f[j] = __half2float(__float2half_rn(fminf(fmaxf(f[j], lo), hi)));
                    }
                    store_vec<VN>(reinterpret_cast<InT*>(&v[k][i].raw), f);         // exact: already fp16 values
                    if (row0 + k * SIDE < groups)
                        *(reinterpret_cast<uint4*>(x + (row0 + k * SIDE) * C) + vi) = v[k][i].raw;
                }
#pragma unroll
                for (int j = 0; j < VN; ++j) s += f[j];
            }
        }
        mu[k] = s;
    }
#pragma unroll
    for (int o = LPG / 2; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < R; ++k) mu[k] += __shfl_xor_sync(0xffffffffu, mu[k], o);
    const float n = (float)C;
#pragma unroll
    for (int k = 0; k < R; ++k) {
        mu[k] /= n;
        float s2 = 0.f;
#pragma unroll
        for (int i = 0; i < VPL; ++i)
            if (lane + 32 * i < nvec) {
                float f[VN];
                v[k][i].to_f32(f);
#pragma unroll
                for (int j = 0; j < VN; ++j) {
                    const float d = f[j] - mu[k];
                    s2 = fmaf(d, d, s2);
                }
            }
        r[k] = s2;
    }
#pragma unroll
    for (int o = LPG / 2; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < R; ++k) r[k] += __shfl_xor_sync(0xffffffffu, r[k], o);
#pragma unroll
    for (int k = 0; k < R; ++k) r[k] = 1.0f / sqrtf(r[k] / n + eps);
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
        const int vi = lane + 32 * i;
        float gf[VN], bf[VN];
        gw[i].to_f32(gf);
        bw[i].to_f32(bf);
#pragma unroll
        for (int k = 0; k < R; ++k) {
            const int64_t g = row0 + k * SIDE;
            if (vi < nvec && g < groups) {
                float y[VN];
                v[k][i].to_f32(y);
#pragma unroll
                for (int j = 0; j < VN; ++j) y[j] = (y[j] - mu[k]) * r[k];
                if (gamma) {
#pragma unroll
                    for (int j = 0; j < VN; ++j) y[j] = __fmul_rn(y[j], gf[j]);
                }
                if (beta) {
#pragma unroll
                    for (int j = 0; j < VN; ++j) y[j] = __fadd_rn(y[j], bf[j]);
                }
                store_vec<VN>(out + g * C + (int64_t)vi * VN, y);
            }
        }
    }
    float m = mu[0], q = r[0];
#pragma unroll
    for (int k = 1; k < R; ++k)
        if (lane == k) {
            m = mu[k];
            q = r[k];
        }
    const int64_t g = row0 + lane * SIDE;
    if (lane < R && g < groups) {
        mean[g] = m;
        rstd[g] = q;
    }
}

__device__ __forceinline__ float ldf(const __half* p, int64_t i) { return __half2float(p[i]); }
__device__ __forceinline__ float ldf(const float* p, int64_t i) { return p[i]; }
__device__ __forceinline__ void stf(__half* p, int64_t i, float v) { p[i] = __float2half_rn(v); }
__device__ __forceinline__ void stf(float* p, int64_t i, float v) { p[i] = v; }

__device__ __forceinline__ float block_sum(float v, float* red) {
    v = warp_sum(v);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
    __syncthreads();
    if (l == 0) red[w] = v;
    __syncthreads();
    float t = l < nw ? red[l] : 0.f;
    return warp_sum(t);
}

// Rows of some 224 to 512 vectors: a block per row, a thread four to six vectors of it, kept as read (fp16 stays packed, 28 to
// 46 registers), moments and output two elements an instruction, the two sums through shared memory with one barrier each.
// Bound by HBM; a warp a row (ln_warp_kernel) holds 8 registers a vector and then has too few rows in flight.  Microseconds, a
// warp a row before -> now, 80 Mi elements of fp16: 1800 wide 70.5 -> 66.8, 2056
// 89.3 -> 68.8, 2560 84.6 -> 58.1 (5.5 TB/s), 3072 76.5 -> 60.8, 4096 112.3 -> 63.2; 40 Mi of fp32: 1280 53.8 -> 51.6,
// 2048 60.1 -> 52.3; in the L2, 1953 x 4096 16.8 -> 8.8; 64 x 4096 6.7 -> 3.2; behind the add 9765 x 4096 105 -> 51.7
// (6.2 TB/s), 600 x 4096 11.7 -> 6.1.  Narrower rows lose (52083 x 1536: 59.2 -> 64.8).  gamma and beta asked for with
// the row cost a fifth (registers), and so did rings of rows in shared memory that bulk copies fill, a warp a row (20480 x 4096: 98).
// With ADD the residual add (and clamp) of ln_add_warp_kernel comes first, for the same widths and the same bits.
template <typename InT, typename OutT, int VPT, bool ADD>
__global__ void __launch_bounds__(1024)
ln_split_kernel(const InT* a, InT* x, const InT* __restrict__ h, OutT* __restrict__ out, float* __restrict__ mean,
                float* __restrict__ rstd, const InT* __restrict__ gamma, const InT* __restrict__ beta, int C, float eps,
                int use_clamp, float lo, float hi) {
    constexpr int VN = Vec16<InT>::N;
    __shared__ float red[2][32];
    const int64_t g = blockIdx.x;
    const int nvec = C / VN, tid = threadIdx.x, T = blockDim.x, warp = tid >> 5, lane = tid & 31, warps = T >> 5;
    const uint4* src = reinterpret_cast<const uint4*>((ADD ? x : a) + g * (int64_t)C);
    grid_dep_wait();     // the input is the previous kernel's output
    grid_dep_launch();
    Vec16<InT> raw[VPT], hv[ADD ? VPT : 1];
#pragma unroll
    for (int i = 0; i < VPT; ++i)
        if (tid + T * i < nvec) {
            raw[i].raw = src[tid + T * i];
            if constexpr (ADD) hv[i].raw = __ldg(reinterpret_cast<const uint4*>(h + g * (int64_t)C) + tid + T * i);
        }
    uint64_t s = pack2(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < VPT; ++i)
        if (tid + T * i < nvec) {
            float f[VN];
            raw[i].to_f32(f);
            if constexpr (ADD) {
                float fh[VN];
                hv[i].to_f32(fh);
#pragma unroll
                for (int j = 0; j < VN; ++j) {
                    f[j] = __half2float(__float2half_rn(f[j] + fh[j]));        // add.Tensor rounds here
                    if (use_clamp) f[j] = __half2float(__float2half_rn(fminf(fmaxf(f[j], lo), hi)));
                }
                store_vec<VN>(reinterpret_cast<InT*>(&raw[i].raw), f);          // exact: already fp16 values
                *(reinterpret_cast<uint4*>(x + g * (int64_t)C) + tid + T * i) = raw[i].raw;
            }
#pragma unroll
            for (int j = 0; j < VN; j += 2) s = add2(s, pack2(f[j], f[j + 1]));
        }
    auto block_total = [&](float v, float* r) {
        v = warp_sum(v);
        if (lane == 0) r[warp] = v;
        __syncthreads();
        return warp_sum(lane < warps ? r[lane] : 0.f);
    };
    const float n = (float)C;
    const float mu = block_total(pairs_sum(s), red[0]) / n;
    const uint64_t nmu = pack2(-mu, -mu);
    s = pack2(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < VPT; ++i)
        if (tid + T * i < nvec) {
            float f[VN];
            raw[i].to_f32(f);
#pragma unroll
            for (int j = 0; j < VN; j += 2) {
                const uint64_t d = add2(pack2(f[j], f[j + 1]), nmu);
                s = fma2(d, d, s);
            }
        }
    const float r = 1.0f / sqrtf(block_total(pairs_sum(s), red[1]) / n + eps);
    OutT* dst = out + g * (int64_t)C;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
        const int v = tid + T * i;
        if (v < nvec) {
            float f[VN];
            uint64_t d[VN / 2];
            raw[i].to_f32(f);
#pragma unroll
            for (int j = 0; j < VN / 2; ++j) d[j] = add2(pack2(f[2 * j], f[2 * j + 1]), nmu);
            uint4 gv = make_uint4(0u, 0u, 0u, 0u), bv = gv;
            if (gamma) gv = __ldg(reinterpret_cast<const uint4*>(gamma) + v);
            if (beta) bv = __ldg(reinterpret_cast<const uint4*>(beta) + v);
            ln_write<InT, OutT>(dst + (int64_t)v * VN, d, r, gamma != nullptr, gv, beta != nullptr, bv);
        }
    }
    if (tid == 0) {
        mean[g] = mu;
        rstd[g] = r;
    }
}

// Rows of more than 512 vectors: 256 threads a row, the row in registers as it was read (fp16 stays packed: an SM holds twice the
// blocks that it does with the row in fp32), the two sums over the block through shared memory.  One order of sums whatever
// the number of rows, so that a row's bits do not depend on the rows beside it.  Bound by HBM; with scalar accesses and the row read
// three times 7112 x 4280 in fp32 took 71.6 us, now 44.5 (5.5 TB/s; replayed over four operand sets).  fp16, microseconds with the
// row in fp32 and now: 64 x 4104 3.3, 3.0; 592 x 5120 behind another kernel 5.3, 5.0; 1600 x 6144 13.8, 11.1; 10000 x 5120 56.0, 41.3;
// 4000 x 16384 75.9, 46.3.  The block a row above took 3.7, 5.6, 12.9, 39.4 and 64.6 there (700 x 5120: 6.0, here 4.6).
template <typename InT, typename OutT, int VPT>
__global__ void __launch_bounds__(LN_WIDE_THREADS)
ln_wide_kernel(const InT* __restrict__ a, OutT* __restrict__ out, float* __restrict__ mean, float* __restrict__ rstd,
               const InT* __restrict__ gamma, const InT* __restrict__ beta, int C, float eps) {
    constexpr int VN = Vec16<InT>::N;
    __shared__ float red[32];
    const int64_t g = blockIdx.x;
    const int nvec = C / VN, tid = threadIdx.x;
    const uint4* src = reinterpret_cast<const uint4*>(a + g * (int64_t)C);
    grid_dep_wait();     // the input is the previous kernel's output
    grid_dep_launch();
    Vec16<InT> raw[VPT];
#pragma unroll
    for (int i = 0; i < VPT; ++i)
        if (tid + LN_WIDE_THREADS * i < nvec) raw[i].raw = __ldg(src + tid + LN_WIDE_THREADS * i);
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i)
        if (tid + LN_WIDE_THREADS * i < nvec) {
            float x[VN];
            raw[i].to_f32(x);
#pragma unroll
            for (int j = 0; j < VN; ++j) s += x[j];
        }
    const float n = (float)C;
    const float mu = block_sum(s, red) / n;
    float s2 = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i)
        if (tid + LN_WIDE_THREADS * i < nvec) {
            float x[VN];
            raw[i].to_f32(x);
#pragma unroll
            for (int j = 0; j < VN; ++j) {
                const float d = x[j] - mu;
                s2 += d * d;
            }
        }
    const float r = 1.0f / sqrtf(block_sum(s2, red) / n + eps);
    OutT* dst = out + g * (int64_t)C;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
        const int v = tid + LN_WIDE_THREADS * i;
        if (v < nvec) {
            float x[VN], y[VN];
            raw[i].to_f32(x);
#pragma unroll
            for (int j = 0; j < VN; ++j) y[j] = (x[j] - mu) * r;
            if (sizeof(OutT) == 4 && gamma && beta) {
                // gamma and beta in one rounding, as in ln_block_kernel: with two, fp32 results were 7 % further from 64
                // bits (rounded to fp16 it does not show, and there both vectors at once cost registers and 17 % of the time)
                Vec16<InT> tg, tb;
                float gf[VN], bf[VN];
                tg.raw = __ldg(reinterpret_cast<const uint4*>(gamma) + v);
                tb.raw = __ldg(reinterpret_cast<const uint4*>(beta) + v);
                tg.to_f32(gf);
                tb.to_f32(bf);
#pragma unroll
                for (int j = 0; j < VN; ++j) y[j] = fmaf(y[j], gf[j], bf[j]);
                store_vec<VN>(dst + (int64_t)v * VN, y);
                continue;
            }
            if (gamma) {
                Vec16<InT> t;
                float gf[VN];
                t.raw = __ldg(reinterpret_cast<const uint4*>(gamma) + v);
                t.to_f32(gf);
#pragma unroll
                for (int j = 0; j < VN; ++j) y[j] *= gf[j];
            }
            if (beta) {
                Vec16<InT> t;
                float bf[VN];
                t.raw = __ldg(reinterpret_cast<const uint4*>(beta) + v);
                t.to_f32(bf);
#pragma unroll
                for (int j = 0; j < VN; ++j)   // fp32 without gamma: one rounding too (with two, 14 % further)
                    if constexpr (sizeof(OutT) == 4) y[j] = fmaf(x[j] - mu, r, bf[j]);
                    else y[j] += bf[j];
            }
            store_vec<VN>(dst + (int64_t)v * VN, y);
        }
    }
    if (tid == 0) {
        mean[g] = mu;
        rstd[g] = r;
    }
}

// Any C, any alignment: one block per group, scalar accesses, the group re-read from
// L1/L2 for the second and third pass.
template <typename InT, typename OutT>
__global__ void __launch_bounds__(256)
ln_block_kernel(const InT* __restrict__ a, OutT* __restrict__ out, float* __restrict__ mean,
                float* __restrict__ rstd, const InT* __restrict__ gamma,
                const InT* __restrict__ beta, int64_t C, float eps) {
    __shared__ float red[32];
    const int64_t g = blockIdx.x;
    const InT* src = a + g * C;
    float s = 0.f;
    for (int64_t i = threadIdx.x; i < C; i += blockDim.x) s += ldf(src, i);
    const float n = (float)C;
    const float mu = block_sum(s, red) / n;
    float s2 = 0.f;
    for (int64_t i = threadIdx.x; i < C; i += blockDim.x) {
        float d = ldf(src, i) - mu;
        s2 += d * d;
    }
    const float r = 1.0f / sqrtf(block_sum(s2, red) / n + eps);
    OutT* dst = out + g * C;
    for (int64_t i = threadIdx.x; i < C; i += blockDim.x) {
        float y = (ldf(src, i) - mu) * r;
        if (gamma) y *= ldf(gamma, i);
        if (beta) y += ldf(beta, i);
        stf(dst, i, y);
    }
    if (threadIdx.x == 0) {
        mean[g] = mu;
        rstd[g] = r;
    }
}

// fp16 rows of more than 96 MB, and as many bytes of results: they do not stay in the L2 (see the packed form).  A row's
// last bits therefore depend on the launch being this large, as they do on which kernel its width and alignment choose.
static bool ln_packs(int64_t groups, int64_t C) { return groups * C >= (int64_t)48 << 20; }
// The widths for which the packed form was measured to pay, as vectors per lane.  Four (60000 x 1000: 43.9 us scalar, 47.0
// packed) and eight (36000 x 1800: 60.0, 62.3; 32000 x 2048: 55.2, 57.2) lose: there its registers cost more warps than its
// instructions save; five and six gain (50000 x 1280: 51.8 -> 49.1, 43000 x 1480: 55.2 -> 52.1).
constexpr bool ln_pack_width(int vpl) { return vpl == 5 || vpl == 6; }

// Whether a launch of `rows` rows a group of `lpg` lanes fills every SM with `n` blocks of four warps: the rule for the kernel of
// several rows.  Its loads in flight pay where bytes bound the launch, its longer chain costs where latency does.  Microseconds,
// each launch behind another kernel, one row / two / four, 148 SMs: fp16 rows of 112 15000 4.1 / 4.7 / 5.2, 38000 (16 blocks of
// two) 7.3 / 6.9 / 7.3, 60000 (12 blocks of four) 10.3 / 9.7 / 9.4, of 64 24000 3.9 / 4.0 / 4.4, 150000 12.8 / 12.3 / 11.6; fp32 of
// 128 9500 (8 blocks of two) 4.5 / 4.5 / 4.9, 15000 5.7 / 5.2 / 5.9, 24000 8.1 / 6.6 / 6.7, 100000 28.7 / 21.4 / 20.4; behind the
// add, 112 24000 6.2 / 6.5 / 7.0, 70000 (30) 14.8 / 14.4 / 14.5, 150000 27.3 / 26.2 / 25.4; two vectors a lane, 448 9500 (8)
// 7.6 / 7.8, 14000 12.7 / 11.4.
static bool ln_fills(const b200_ctx* ctx, int64_t groups, int rows, int lpg, int64_t n) {
    return groups >= n * ctx->prop.multiProcessorCount * 4 * rows * (32 / lpg);
}

// Vectors a thread of ln_split_kernel, 0 for rows that stay with the other kernels.  Past 512 vectors 256 threads a row are as fast or
// faster: in fp32 2400 x 2600 12.6 us, 13.8, 11111 x 3600 50.5, 52.9; in fp16 see ln_wide_kernel.  fp32, six and four: 50000 x 1032 69, 77,
// 20000 x 1280 34.6, 36.3, 2400 x 1664 8.4, 7.8, 3200 x 2048 13.8, 12.6.  By the row's width alone, so that its bits do not depend on
// the rows beside it; what a launch of some 19 rows an SM of the narrowest loses, one round of warps and two of blocks (2800 x 2048 in
// fp16 5.0 us, 6.7; 3200 x 1032 in fp32 5.7, 7.6), it gives back at any other size (64 rows 4.0, 3.2; 20000 35.8, 32.4).
template <typename InT> static int ln_split(int nvec) {
    if (nvec > 512) return 0;
    if (sizeof(InT) == 4) return nvec <= 256 ? 0 : nvec <= 352 ? 6 : 4;
    return nvec <= 224 ? 0 : cdiv(cdiv(nvec, 5), 32) < cdiv(cdiv(nvec, 4), 32) ? 5 : 4;
}

template <typename InT, typename OutT>
static int launch_ln(b200_ctx* ctx, int64_t groups, int64_t C, const void* a, void* out, float* mean,
                     float* rstd, const void* gamma, const void* beta, float eps) {
    constexpr int VN = Vec16<InT>::N;
    const InT* ap = static_cast<const InT*>(a);
    OutT* op = static_cast<OutT*>(out);
    const InT* gp = static_cast<const InT*>(gamma);
    const InT* bp = static_cast<const InT*>(beta);
    auto al16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
    const size_t out_vec_bytes = VN * sizeof(OutT);
    const bool vec_ok = C % VN == 0 && C / VN <= 8 * LN_WIDE_THREADS && al16(a) && (!gamma || al16(gamma)) &&
                  (!beta || al16(beta)) &&
                  (reinterpret_cast<uintptr_t>(out) % (out_vec_bytes > 16 ? 16 : out_vec_bytes)) == 0;
    if (vec_ok) {
        const int nvec = (int)(C / VN);
        const int vpl = (nvec + 31) / 32;
        const int wpb = 4;
        dim3 grid((unsigned)cdiv(groups, wpb)), block(32 * wpb);
        constexpr bool PACKS = sizeof(InT) == 2 && sizeof(OutT) == 2;
        // few enough rows that every CTA is resident at once: the latency form (see the kernel)
        const bool lat = groups <= (int64_t)4 * wpb * ctx->prop.multiProcessorCount;
#define LN_GO(V)                                                                                            \
    do {                                                                                                    \
        if (lat)                                                                                            \
            B200_CUDA(launch_dep(ln_warp_kernel<InT, OutT, V, 32, true>, grid, block, 0, ctx->stream, 1, ap, op, mean, rstd, gp, \
                                 bp, groups, (int)C, eps));                                                 \
        else if (PACKS && ln_pack_width(V) && ln_packs(groups, C))                                          \
            B200_CUDA(launch_dep(ln_warp_kernel<InT, OutT, V, 32, false, PACKS && ln_pack_width(V)>, grid, block, 0, ctx->stream, 1, \
                                 ap, op, mean, rstd, gp, bp, groups, (int)C, eps));                         \
        else                                                                                                \
            B200_CUDA(launch_dep(ln_warp_kernel<InT, OutT, V>, grid, block, 0, ctx->stream, 1, ap, op, mean, rstd, gp, bp, \
                                 groups, (int)C, eps));                                                     \
    } while (0)
#define LN_GO_SHARED(L)                                                                                     \
    B200_CUDA(launch_dep(ln_warp_kernel<InT, OutT, 1, L>, dim3((unsigned)cdiv(groups, wpb * (32 / L))), block, 0,   \
                         ctx->stream, 1, ap, op, mean, rstd, gp, bp, groups, (int)C, eps))
#define LN_GO_ROWS(V, L, R)                                                                                 \
    B200_CUDA(launch_dep(ln_rows_kernel<InT, OutT, V, L, R, false>, dim3((unsigned)cdiv(groups, wpb * R * (32 / L))), block, 0, \
                         ctx->stream, 1, ap, (InT*)nullptr, (const InT*)nullptr, op, mean, rstd, gp, bp, groups, (int)C, eps, 0, \
                         0.f, 0.f))
#define LN_GO_NARROW(L, ONE)                                                                                \
    do {                                                                                                    \
        if (ln_fills(ctx, groups, 4, L, 12)) LN_GO_ROWS(1, L, 4);                                           \
        else if (ln_fills(ctx, groups, 2, L, sizeof(InT) == 4 ? 10 : 14)) LN_GO_ROWS(1, L, 2);              \
        else ONE;                                                                                           \
    } while (0)
#define LN_GO_WIDE(V)                                                                                       \
    B200_CUDA(launch_dep(ln_wide_kernel<InT, OutT, V>, dim3((unsigned)groups), dim3(LN_WIDE_THREADS), 0, ctx->stream, 1, ap, op, \
                         mean, rstd, gp, bp, (int)C, eps))
        // A block a row: the vectors a thread that leave fewer lanes idle (320 vectors: five of 64 threads, four would be of 96).
        const int split = ln_split<InT>(nvec);
        auto go_split = [&](auto kern) {
            return launch_dep(kern, dim3((unsigned)groups), dim3((unsigned)cdiv(cdiv(nvec, split), 32) * 32), 0, ctx->stream, 1, ap,
                              (InT*)nullptr, (const InT*)nullptr, op, mean, rstd, gp, bp, (int)C, eps, 0, 0.f, 0.f);
        };
        if (split == 4) B200_CUDA(go_split(ln_split_kernel<InT, OutT, 4, false>));
        else if (split == 5) B200_CUDA(go_split(ln_split_kernel<InT, OutT, 5, false>));
        else if (split == 6) B200_CUDA(go_split(ln_split_kernel<InT, OutT, 6, false>));
        else if (nvec <= 8) LN_GO_NARROW(8, LN_GO_SHARED(8));
        else if (nvec <= 16) LN_GO_NARROW(16, LN_GO_SHARED(16));
        else if (vpl <= 1) LN_GO_NARROW(32, LN_GO(1));
        else if (vpl <= 2) LN_GO(2);
        else if (vpl <= 3) LN_GO(3);
        else if (vpl <= 4) LN_GO(4);
        else if (vpl <= 5) LN_GO(5);
        else if (vpl <= 6) LN_GO(6);
        else if (vpl <= 8) LN_GO(8);
        else if (sizeof(InT) == 2 && nvec <= 3 * LN_WIDE_THREADS) LN_GO_WIDE(3);
        else if (nvec <= 4 * LN_WIDE_THREADS) LN_GO_WIDE(4);
        else if (sizeof(InT) == 2 && nvec <= 6 * LN_WIDE_THREADS) LN_GO_WIDE(6);
        else LN_GO_WIDE(8);
#undef LN_GO_WIDE
#undef LN_GO
#undef LN_GO_SHARED
#undef LN_GO_ROWS
#undef LN_GO_NARROW
    } else {
        ln_block_kernel<InT, OutT><<<(unsigned)groups, 256, 0, ctx->stream>>>(ap, op, mean, rstd, gp, bp,
                                                                             C, eps);
    }
    ctx->launches++;
    B200_CUDA(cudaGetLastError());
    return B200_OK;
}

} // namespace b200

using namespace b200;

extern "C" int b200_add_layernorm_f16(b200_ctx* ctx, int64_t groups, int64_t C, void* x, const void* h, int use_clamp,
                                      float lo, float hi, void* out, float* mean, float* rstd, const void* gamma,
                                      const void* beta, float eps) {
    B200_REQUIRE(ctx, B200_EINVAL, "add_layernorm: null ctx");
    B200_REQUIRE(groups >= 0 && C > 0, B200_EINVAL, "add_layernorm: groups=%lld C=%lld", (long long)groups,
                 (long long)C);
    if (groups == 0) return B200_OK;
    B200_REQUIRE(x && h && out && mean && rstd, B200_EINVAL, "add_layernorm: null array");
    B200_REQUIRE(groups < (1ll << 31), B200_DECLINE_EXTENT, "add_layernorm: %lld groups", (long long)groups);
    B200_CUDA(cudaSetDevice(ctx->device));
    auto al16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
    const bool vec = C % 8 == 0 && C / 8 <= 32 * 16 && al16(x) && al16(h) && al16(out) && (!gamma || al16(gamma)) &&
                     (!beta || al16(beta));
    if (!vec) {
        // Shapes the vector kernel does not take: the three ops one after another, same results.
        int rc = b200_add_f16(ctx, x, h, x, groups * C);
        if (rc == B200_OK && use_clamp) rc = b200_clamp_f16(ctx, x, x, groups * C, lo, hi);
        if (rc != B200_OK) return rc;
        return b200_layernorm(ctx, groups, C, x, B200_F16, out, B200_F16, mean, rstd, gamma, beta, eps);
    }
    const int nvec = (int)(C / 8), vpl = (nvec + 31) / 32, wpb = 4;
    dim3 grid((unsigned)cdiv(groups, wpb)), block(32 * wpb);
    const bool lat = groups <= (int64_t)4 * wpb * ctx->prop.multiProcessorCount;   // every CTA resident at once: the latency form
#define LNA_GO(V)                                                                                                 \
    do {                                                                                                          \
        if (lat)                                                                                                  \
            B200_CUDA(launch_dep(ln_add_warp_kernel<V, 32, true>, grid, block, 0, ctx->stream, 1, (__half*)x, (const __half*)h, \
                                 (__half*)out, mean, rstd, (const __half*)gamma, (const __half*)beta, groups, (int)C, eps, \
                                 use_clamp, lo, hi));                                                             \
        else if (ln_pack_width(V) && ln_packs(groups, C))                                                         \
            B200_CUDA(launch_dep(ln_add_warp_kernel<V, 32, false, ln_pack_width(V)>, grid, block, 0, ctx->stream, 1, (__half*)x, \
                                 (const __half*)h, (__half*)out, mean, rstd, (const __half*)gamma, (const __half*)beta, groups, (int)C, \
                                 eps, use_clamp, lo, hi));                                                        \
        else                                                                                                      \
            B200_CUDA(launch_dep(ln_add_warp_kernel<V>, grid, block, 0, ctx->stream, 1, (__half*)x, (const __half*)h,   \
                                 (__half*)out, mean, rstd, (const __half*)gamma, (const __half*)beta, groups, (int)C, eps, \
                                 use_clamp, lo, hi));                                                             \
    } while (0)
#define LNA_GO_SHARED(L)                                                                                          \
    B200_CUDA(launch_dep(ln_add_warp_kernel<1, L>, dim3((unsigned)cdiv(groups, wpb * (32 / L))), block, 0, ctx->stream, 1, \
                         (__half*)x, (const __half*)h, (__half*)out, mean, rstd, (const __half*)gamma,             \
                         (const __half*)beta, groups, (int)C, eps, use_clamp, lo, hi))
#define LNA_GO_ROWS(V, L, R)                                                                                      \
    B200_CUDA(launch_dep(ln_rows_kernel<__half, __half, V, L, R, true>, dim3((unsigned)cdiv(groups, wpb * R * (32 / L))), block, 0, \
                         ctx->stream, 1, (const __half*)nullptr, (__half*)x, (const __half*)h, (__half*)out, mean, rstd, \
                         (const __half*)gamma, (const __half*)beta, groups, (int)C, eps, use_clamp, lo, hi))
#define LNA_GO_NARROW(L, ONE)                                                                                     \
    do {                                                                                                          \
        if (ln_fills(ctx, groups, 4, L, 24)) LNA_GO_ROWS(1, L, 4);                                                \
        else if (ln_fills(ctx, groups, 2, L, 20)) LNA_GO_ROWS(1, L, 2);                                           \
        else ONE;                                                                                                 \
    } while (0)
    const int split = ln_split<__half>(nvec);
    auto go_split = [&](auto kern) {
        return launch_dep(kern, dim3((unsigned)groups), dim3((unsigned)cdiv(cdiv(nvec, split), 32) * 32), 0, ctx->stream, 1,
                          (const __half*)nullptr, (__half*)x, (const __half*)h, (__half*)out, mean, rstd, (const __half*)gamma,
                          (const __half*)beta, (int)C, eps, use_clamp, lo, hi);
    };
    if (split == 4) B200_CUDA(go_split(ln_split_kernel<__half, __half, 4, true>));
    else if (split == 5) B200_CUDA(go_split(ln_split_kernel<__half, __half, 5, true>));
    else if (nvec <= 8) LNA_GO_NARROW(8, LNA_GO_SHARED(8));
    else if (nvec <= 16) LNA_GO_NARROW(16, LNA_GO_SHARED(16));
    else if (vpl <= 1) LNA_GO_NARROW(32, LNA_GO(1));
    else if (vpl <= 2 && ln_fills(ctx, groups, 2, 32, 10)) LNA_GO_ROWS(2, 32, 2);
    else if (vpl <= 2) LNA_GO(2);
    else if (vpl <= 3) LNA_GO(3);
    else if (vpl <= 4) LNA_GO(4);
    else if (vpl <= 5) LNA_GO(5);
    else if (vpl <= 6) LNA_GO(6);
    else LNA_GO(8);
#undef LNA_GO
#undef LNA_GO_SHARED
#undef LNA_GO_ROWS
#undef LNA_GO_NARROW
    ctx->launches++;
    B200_CUDA(cudaGetLastError());
    return B200_OK;
}

extern "C" int b200_layernorm(b200_ctx* ctx, int64_t groups, int64_t C, const void* a, int in_dtype,
                              void* out, int out_dtype, float* mean, float* rstd, const void* gamma,
                              const void* beta, float eps) {
    B200_REQUIRE(ctx, B200_EINVAL, "layernorm: null ctx");
    B200_REQUIRE(groups >= 0 && C > 0, B200_EINVAL, "layernorm: groups=%lld C=%lld", (long long)groups,
                 (long long)C);
    if (groups == 0) return B200_OK;
    B200_REQUIRE(a && out && mean && rstd, B200_EINVAL, "layernorm: null array");
    B200_REQUIRE(groups < (1ll << 31), B200_DECLINE_EXTENT, "layernorm: %lld groups", (long long)groups);
    B200_REQUIRE((in_dtype == B200_F16 || in_dtype == B200_F32) &&
                     (out_dtype == B200_F16 || out_dtype == B200_F32),
                 B200_DECLINE_ELTYPE, "layernorm: dtype %d -> %d", in_dtype, out_dtype);
    B200_CUDA(cudaSetDevice(ctx->device));
    if (in_dtype == B200_F16 && out_dtype == B200_F16)
        return launch_ln<__half, __half>(ctx, groups, C, a, out, mean, rstd, gamma, beta, eps);
    if (in_dtype == B200_F16 && out_dtype == B200_F32)
        return launch_ln<__half, float>(ctx, groups, C, a, out, mean, rstd, gamma, beta, eps);
    if (in_dtype == B200_F32 && out_dtype == B200_F16)
        return launch_ln<float, __half>(ctx, groups, C, a, out, mean, rstd, gamma, beta, eps);
    return launch_ln<float, float>(ctx, groups, C, a, out, mean, rstd, gamma, beta, eps);
}
