// Bandwidth-bound glue ops the encoder graphs run between the dense kernels: residual add,
// clamp, standalone activation and the strided -> dense copy behind permute/contiguous.
// fp16 storage, fp32 arithmetic, one rounding at the store (reference ops.jl:186-197,
// 323-335, 1698-1702; execute.jl:257-277).
#include <cuda_fp16.h>

#include "act.cuh"
#include "internal.h"

namespace b200 {

enum { OP_ADD = 0, OP_CLAMP = 1, OP_ACT = 2 };

template <int OP>
__device__ __forceinline__ float ew(float a, float b, float lo, float hi, int epi) {
    if (OP == OP_ADD) return a + b;
    if (OP == OP_CLAMP) return fminf(fmaxf(a, lo), hi);
    return apply_act(epi, a);
}

// 8 halfs (16 B) per thread per step, grid-stride; the scalar tail is handled by the last
// few threads of the same launch.
template <int OP>
__global__ void __launch_bounds__(256)
ew_f16_kernel(const __half* __restrict__ a, const __half* __restrict__ b, __half* __restrict__ out,
              int64_t n, float lo, float hi, int epi, int vec) {
    const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
    int64_t done = 0;
    if (vec) {
        const int64_t nv = n / 8;
        for (int64_t i = tid; i < nv; i += nthreads) {
            uint4 ua = __ldg(reinterpret_cast<const uint4*>(a) + i);
            uint4 ub = OP == OP_ADD ? __ldg(reinterpret_cast<const uint4*>(b) + i) : ua;
            uint4 uo;
            const __half2* ha = reinterpret_cast<const __half2*>(&ua);
            const __half2* hb = reinterpret_cast<const __half2*>(&ub);
            __half2* ho = reinterpret_cast<__half2*>(&uo);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                float2 fa = __half22float2(ha[q]), fb = __half22float2(hb[q]);
                ho[q] = __floats2half2_rn(ew<OP>(fa.x, fb.x, lo, hi, epi), ew<OP>(fa.y, fb.y, lo, hi, epi));
            }
            reinterpret_cast<uint4*>(out)[i] = uo;
        }
        done = nv * 8;
    }
    for (int64_t i = done + tid; i < n; i += nthreads) {
        float fa = __half2float(a[i]);
        float fb = OP == OP_ADD ? __half2float(b[i]) : 0.f;
        out[i] = __float2half_rn(ew<OP>(fa, fb, lo, hi, epi));
    }
}

template <int OP>
static int launch_ew(b200_ctx* ctx, const void* a, const void* b, void* out, int64_t n, float lo, float hi,
                     int epi) {
    if (n == 0) return B200_OK;
    auto al = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
    const int vec = al(a) && al(out) && (OP != OP_ADD || al(b));
    int64_t work = vec ? cdiv(n, 8) : n;
    int64_t blocks = cdiv(work, 256);
    const int64_t cap = (int64_t)ctx->prop.multiProcessorCount * 16;
    if (blocks > cap) blocks = cap;
    ew_f16_kernel<OP><<<(unsigned)blocks, 256, 0, ctx->stream>>>((const __half*)a, (const __half*)b, (__half*)out,
                                                                  n, lo, hi, epi, vec);
    ctx->launches++;
    B200_CUDA(cudaGetLastError());
    return B200_OK;
}

// _to_copy between fp16 and fp32 (ops.jl:342-358): eight elements per thread when both ends are
// 16-byte aligned, a scalar loop for the tail.
template <typename SrcT, typename DstT>
__global__ void __launch_bounds__(256)
cast_kernel(const SrcT* __restrict__ src, DstT* __restrict__ dst, int64_t n, int vec) {
    const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
    auto tof = [](SrcT v) -> float {
        if constexpr (sizeof(SrcT) == 2) return __half2float(v);
        else return v;
    };
    auto fromf = [](float v) -> DstT {
        if constexpr (sizeof(DstT) == 2) return __float2half_rn(v);
        else return v;
    };
    int64_t done = 0;
    if (vec) {
        const int64_t nv = n / 8;
        for (int64_t i = tid; i < nv; i += nthreads) {
            SrcT in[8];
            DstT o[8];
            if constexpr (sizeof(SrcT) == 2) {
                *reinterpret_cast<uint4*>(in) = __ldg(reinterpret_cast<const uint4*>(src) + i);
            } else {
                *reinterpret_cast<uint4*>(in) = __ldg(reinterpret_cast<const uint4*>(src) + 2 * i);
                *reinterpret_cast<uint4*>(in + 4) = __ldg(reinterpret_cast<const uint4*>(src) + 2 * i + 1);
            }
#pragma unroll
            for (int q = 0; q < 8; ++q) o[q] = fromf(tof(in[q]));
            if constexpr (sizeof(DstT) == 2) {
                reinterpret_cast<uint4*>(dst)[i] = *reinterpret_cast<const uint4*>(o);
            } else {
                reinterpret_cast<uint4*>(dst)[2 * i] = *reinterpret_cast<const uint4*>(o);
                reinterpret_cast<uint4*>(dst)[2 * i + 1] = *reinterpret_cast<const uint4*>(o + 4);
            }
        }
        done = nv * 8;
    }
    for (int64_t i = done + tid; i < n; i += nthreads) dst[i] = fromf(tof(src[i]));
}

template <typename SrcT, typename DstT>
static int launch_cast(b200_ctx* ctx, const void* src, void* dst, int64_t n) {
    auto al = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
    const int vec = al(src) && al(dst);
    int64_t blocks = cdiv(vec ? cdiv(n, 8) : n, 256);
    const int64_t cap = (int64_t)ctx->prop.multiProcessorCount * 16;
    if (blocks > cap) blocks = cap;
    cast_kernel<SrcT, DstT><<<(unsigned)blocks, 256, 0, ctx->stream>>>((const SrcT*)src, (DstT*)dst, n, vec);
    ctx->launches++;
    B200_CUDA(cudaGetLastError());
    return B200_OK;
}

// Strided gather into a dense array: one thread per output element, output-coalesced.  I: 32-bit where the elements can be
// counted so (a step of the grid past them included); three 64-bit divisions an element are some 300 instructions.
template <typename T, typename I>
__global__ void __launch_bounds__(256)
permute4_kernel(const T* __restrict__ src, T* __restrict__ out, I n, I d0, I d1, I d2, int64_t s0, int64_t s1, int64_t s2, int64_t s3) {
    for (I i = blockIdx.x * (I)blockDim.x + threadIdx.x; i < n; i += (I)gridDim.x * blockDim.x) {
        I t = i / d0;
        const I i0 = i - t * d0, u = t / d1, i1 = t - u * d1, i3 = u / d2, i2 = u - i3 * d2;
        out[i] = src[(int64_t)i0 * s0 + (int64_t)i1 * s1 + (int64_t)i2 * s2 + (int64_t)i3 * s3];
    }
}
template <typename T>
static void permute4(b200_ctx* ctx, const T* src, T* out, int64_t n, int64_t d0, int64_t d1, int64_t d2, int64_t s0, int64_t s1, int64_t s2,
                     int64_t s3) {
    int64_t blocks = cdiv(n, 256);
    const int64_t cap = (int64_t)ctx->prop.multiProcessorCount * 32;
    if (blocks > cap) blocks = cap;
    if (n < (1ll << 31))   // no extent is larger than their product
        permute4_kernel<T, uint32_t><<<(unsigned)blocks, 256, 0, ctx->stream>>>(src, out, (uint32_t)n, (uint32_t)d0, (uint32_t)d1, (uint32_t)d2,
                                                                               s0, s1, s2, s3);
    else permute4_kernel<T, int64_t><<<(unsigned)blocks, 256, 0, ctx->stream>>>(src, out, n, d0, d1, d2, s0, s1, s2, s3);
}

// Same gather when the source is contiguous along output axis 1 (a transpose of the two
// fastest axes, the layout change behind permute(0,2,1,3)-style views): 32x32 tiles through
// shared memory so both the reads and the writes coalesce.
template <typename T>
__global__ void __launch_bounds__(256)
transpose01_kernel(const T* __restrict__ src, T* __restrict__ out, int d0, int d1, int64_t d2, int64_t s0,
                   int64_t s2, int64_t s3) {
    __shared__ T tile[32][33];
    const int64_t z = blockIdx.z;
    const int64_t i2 = z % d2, i3 = z / d2;
    const T* sp = src + i2 * s2 + i3 * s3;
    T* op = out + z * (int64_t)d0 * d1;
    const int b0 = blockIdx.x * 32, b1 = blockIdx.y * 32;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    for (int r = ty; r < 32; r += 8) {
        int i0 = b0 + r, i1 = b1 + tx; // read: i1 fastest in the source
        if (i0 < d0 && i1 < d1) tile[r][tx] = sp[(int64_t)i0 * s0 + i1];
    }
    __syncthreads();
    for (int r = ty; r < 32; r += 8) {
        int i1 = b1 + r, i0 = b0 + tx; // write: i0 fastest in the output
        if (i0 < d0 && i1 < d1) op[i0 + (int64_t)d0 * i1] = tile[tx][r];
    }
}

// The same for 2-byte elements whose rows lie on 16-byte boundaries on both sides: 64 x 64 tiles, read and written 16
// bytes at a time.  What bounds it is HBM; 2-byte accesses took three times as long: eight images of 65536 pixels x 112
// channels (117 MB each way) 158 -> 41 us.  A tile row is 33 words: a warp's stores hit every bank once, its loads twice.
__global__ void __launch_bounds__(256)
transpose01_vec_kernel(const uint16_t* __restrict__ src, uint16_t* __restrict__ out, int d0, int d1, int64_t d2, int64_t s0,
                       int64_t s2, int64_t s3) {
    __shared__ uint32_t tile[64][33];
    const int64_t z = blockIdx.z;
    const int64_t i2 = z % d2, i3 = z / d2;
    const uint16_t* sp = src + i2 * s2 + i3 * s3;
    uint16_t* op = out + z * (int64_t)d0 * d1;
    const int b0 = blockIdx.x * 64, b1 = blockIdx.y * 64;
    const int c = threadIdx.x & 7, r = threadIdx.x >> 3;
    uint4 v[2];
#pragma unroll
    for (int h = 0; h < 2; ++h)
        if (b0 + r + 32 * h < d0 && b1 + 8 * c < d1)
            v[h] = *reinterpret_cast<const uint4*>(sp + (int64_t)(b0 + r + 32 * h) * s0 + b1 + 8 * c);
        else v[h] = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        uint32_t* t = &tile[r + 32 * h][4 * c];
        t[0] = v[h].x;
        t[1] = v[h].y;
        t[2] = v[h].z;
        t[3] = v[h].w;
    }
    __syncthreads();
    // eight elements along axis 0 at positions 2 r and 2 r + 1 of axis 1
    uint32_t w[8], lo[4], hi[4];
#pragma unroll
    for (int u = 0; u < 8; ++u) w[u] = tile[8 * c + u][r];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        lo[u] = __byte_perm(w[2 * u], w[2 * u + 1], 0x5410);
        hi[u] = __byte_perm(w[2 * u], w[2 * u + 1], 0x7632);
    }
    const int i0 = b0 + 8 * c, i1 = b1 + 2 * r;
    if (i0 < d0) {
        if (i1 < d1) *reinterpret_cast<uint4*>(op + i0 + (int64_t)d0 * i1) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        if (i1 + 1 < d1) *reinterpret_cast<uint4*>(op + i0 + (int64_t)d0 * (i1 + 1)) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    }
}

template <typename T>
static int launch_permute(b200_ctx* ctx, const void* src, void* out, const int64_t* d, const int64_t* s) {
    const int64_t n = d[0] * d[1] * d[2] * d[3];
    if (n == 0) return B200_OK;
    // Axis 0 contiguous on both sides (a window partition moves whole runs of channels): the same gather
    // in 16-byte pieces.
    constexpr int64_t V = 16 / (int64_t)sizeof(T);
    auto al16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
    if (s[0] == 1 && d[0] % V == 0 && s[1] % V == 0 && s[2] % V == 0 && s[3] % V == 0 && al16(src) && al16(out)) {
        permute4<uint4>(ctx, (const uint4*)src, (uint4*)out, n / V, d[0] / V, d[1], d[2], 1, s[1] / V, s[2] / V, s[3] / V);
        ctx->launches++;
        B200_CUDA(cudaGetLastError());
        return B200_OK;
    }
    if (s[1] == 1 && s[0] != 1 && d[0] < (1ll << 30) && d[1] < (1ll << 30) && d[2] * d[3] < 65536 &&
        cdiv(d[1], 32) < 65536) {
        // an axis of one element is never stepped along
        const bool rows16 = sizeof(T) == 2 && d[0] % 8 == 0 && d[1] % 8 == 0 && s[0] % 8 == 0 && (d[2] == 1 || s[2] % 8 == 0) &&
                            (d[3] == 1 || s[3] % 8 == 0) && al16(src) && al16(out);
        dim3 grid((unsigned)cdiv(d[0], rows16 ? 64 : 32), (unsigned)cdiv(d[1], rows16 ? 64 : 32), (unsigned)(d[2] * d[3]));
        if (rows16)
            transpose01_vec_kernel<<<grid, 256, 0, ctx->stream>>>((const uint16_t*)src, (uint16_t*)out, (int)d[0], (int)d[1], d[2], s[0], s[2],
                                                                  s[3]);
        else transpose01_kernel<T><<<grid, 256, 0, ctx->stream>>>((const T*)src, (T*)out, (int)d[0], (int)d[1], d[2], s[0],
                                                            s[2], s[3]);
    } else {
        permute4<T>(ctx, (const T*)src, (T*)out, n, d[0], d[1], d[2], s[0], s[1], s[2], s[3]);
    }
    ctx->launches++;
    B200_CUDA(cudaGetLastError());
    return B200_OK;
}

// max_pool2d (reference kernels/resample.jl:121-141): out[ox,oy,c,n] = max over the window of
// x[ix,iy,c,n], positions outside the image skipped, the running maximum starting at the type's
// lowest value.  Both arrays are indexed (x, y, c, n) through element strides, so the planar layout
// of the reference's call and a channels-last token array go through the same kernel; VEC = 8 takes
// eight channels per thread when the channel axis is contiguous in both.
// I: as for the permuted copy.  TWO: a 2 x 2 window without padding, an image encoder's, is inside the image wherever it lies: its
// four loads go out together.  The six pools of an image encoder's pass over eight images (560 MB): 253 -> 167 us; its eight
// permuted copies 155 -> 108.
template <int VEC, bool TWO, typename I>
__global__ void __launch_bounds__(256)
maxpool2d_kernel(const __half* __restrict__ x, __half* __restrict__ out, int W, int H, int C, int OW, int OH, I total,
                 int64_t xs0, int64_t xs1, int64_t xs2, int64_t xs3, int64_t os0, int64_t os1, int64_t os2, int64_t os3,
                 int kx, int ky, int sx, int sy, int px, int py, int c_fast) {
    const I CV = C / VEC, ow = OW, oh = OH;
    for (I i = blockIdx.x * (I)blockDim.x + threadIdx.x; i < total; i += (I)gridDim.x * blockDim.x) {
        int ox, oy, c, n;
        I t = i;
        if (c_fast) {   // channel fastest: neighbouring threads touch neighbouring channels
            c = (int)(t % CV) * VEC; t /= CV;
            ox = (int)(t % ow); t /= ow;
            oy = (int)(t % oh); n = (int)(t / oh);
        } else {
            ox = (int)(t % ow); t /= ow;
            oy = (int)(t % oh); t /= oh;
            c = (int)(t % CV) * VEC; n = (int)(t / CV);
        }
        const int bx = ox * sx - px, by = oy * sy - py;
        const __half* xp = x + (int64_t)c * xs2 + (int64_t)n * xs3;
        if constexpr (VEC == 8) {
            __half2 acc[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) acc[u] = __half2half2(__ushort_as_half(0xFC00));   // -inf = typemin(Float16)
            auto take = [&](const uint4& w) {
                const __half2* hh = reinterpret_cast<const __half2*>(&w);
#pragma unroll
                for (int u = 0; u < 4; ++u) acc[u] = __hmax2_nan(acc[u], hh[u]);
            };
            if constexpr (TWO) {
                const __half* p0 = xp + (int64_t)bx * xs0 + (int64_t)by * xs1;
                uint4 w[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) w[e] = __ldg(reinterpret_cast<const uint4*>(p0 + (e & 1) * xs0 + (e >> 1) * xs1));
#pragma unroll
                for (int e = 0; e < 4; ++e) take(w[e]);
            } else {
                for (int dy = 0; dy < ky; ++dy) {
                    const int iy = by + dy;
                    if (iy < 0 || iy >= H) continue;
#pragma unroll 2   // two loads in flight: 5 x 5 / 2 over 4 of 14 x 14 x 64 6.5 -> 5.6 us
                    for (int dx = 0; dx < kx; ++dx) {
                        const int ix = bx + dx;
                        if (ix < 0 || ix >= W) continue;
                        // by value: a reference costs the loads their width (3 x 3 / 1 over 2 of 56 x 56 x 256: 6.4 -> 5.3 us)
                        const uint4 w = *reinterpret_cast<const uint4*>(xp + (int64_t)ix * xs0 + (int64_t)iy * xs1);
                        take(w);
                    }
                }
            }
            *reinterpret_cast<uint4*>(out + (int64_t)ox * os0 + (int64_t)oy * os1 + (int64_t)c * os2 + (int64_t)n * os3) =
                *reinterpret_cast<const uint4*>(acc);
        } else {
            __half acc = __ushort_as_half(0xFC00);
            for (int dy = 0; dy < ky; ++dy) {
                const int iy = by + dy;
                if (iy < 0 || iy >= H) continue;
                for (int dx = 0; dx < kx; ++dx) {
                    const int ix = bx + dx;
                    if (ix < 0 || ix >= W) continue;
                    acc = __hmax_nan(acc, xp[(int64_t)ix * xs0 + (int64_t)iy * xs1]);
                }
            }
            out[(int64_t)ox * os0 + (int64_t)oy * os1 + (int64_t)c * os2 + (int64_t)n * os3] = acc;
        }
    }
}

} // namespace b200

using namespace b200;

extern "C" {

int b200_maxpool2d_f16(b200_ctx* ctx, int64_t W, int64_t H, int64_t Cn, int64_t N, const void* x, const int64_t* xstride,
                       void* out, const int64_t* ostride, int64_t kx, int64_t ky, int64_t sx, int64_t sy, int64_t px,
                       int64_t py) {
    B200_REQUIRE(ctx && xstride && ostride, B200_EINVAL, "maxpool2d: null argument");
    B200_REQUIRE(W >= 0 && H >= 0 && Cn >= 0 && N >= 0, B200_EINVAL, "maxpool2d: negative extent");
    B200_REQUIRE(kx >= 1 && ky >= 1 && sx >= 1 && sy >= 1 && px >= 0 && py >= 0 && 2 * px <= kx && 2 * py <= ky,
                 B200_EINVAL, "maxpool2d: window %lldx%lld stride %lldx%lld pad %lldx%lld", (long long)kx, (long long)ky,
                 (long long)sx, (long long)sy, (long long)px, (long long)py);
    B200_REQUIRE(W < (1ll << 30) && H < (1ll << 30) && Cn < (1ll << 30) && N < (1ll << 30), B200_DECLINE_EXTENT,
                 "maxpool2d: extent");
    if (W + 2 * px < kx || H + 2 * py < ky) return B200_OK;   // no output position
    const int64_t OW = (W + 2 * px - kx) / sx + 1, OH = (H + 2 * py - ky) / sy + 1;
    if (OW * OH * Cn * N == 0) return B200_OK;
    B200_REQUIRE(x && out, B200_EINVAL, "maxpool2d: null array");
    B200_CUDA(cudaSetDevice(ctx->device));
    auto al16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
    bool vec = xstride[2] == 1 && ostride[2] == 1 && Cn % 8 == 0 && al16(x) && al16(out);
    for (int d = 0; d < 4; ++d)
        if (d != 2) vec = vec && xstride[d] % 8 == 0 && ostride[d] % 8 == 0;
    const int c_fast = ostride[2] == 1;
    const int64_t total = OW * OH * (vec ? Cn / 8 : Cn) * N;
    int64_t blocks = cdiv(total, 256);
    const int64_t cap = (int64_t)ctx->prop.multiProcessorCount * 32;
    if (blocks > cap) blocks = cap;
    auto go = [&](auto kern, auto count) {
        kern<<<(unsigned)blocks, 256, 0, ctx->stream>>>(
            (const __half*)x, (__half*)out, (int)W, (int)H, (int)Cn, (int)OW, (int)OH, count, xstride[0], xstride[1],
            xstride[2], xstride[3], ostride[0], ostride[1], ostride[2], ostride[3], (int)kx, (int)ky, (int)sx, (int)sy,
            (int)px, (int)py, c_fast);
    };
    const bool two = kx == 2 && ky == 2 && px == 0 && py == 0;
    if (total < (1ll << 31)) {
        if (vec && two) go(maxpool2d_kernel<8, true, uint32_t>, (uint32_t)total);
        else if (vec) go(maxpool2d_kernel<8, false, uint32_t>, (uint32_t)total);
        else go(maxpool2d_kernel<1, false, uint32_t>, (uint32_t)total);
    } else {
        if (vec && two) go(maxpool2d_kernel<8, true, int64_t>, total);
        else if (vec) go(maxpool2d_kernel<8, false, int64_t>, total);
        else go(maxpool2d_kernel<1, false, int64_t>, total);
    }
    ctx->launches++;
    B200_CUDA(cudaGetLastError());
    return B200_OK;
}

int b200_add_f16(b200_ctx* ctx, const void* a, const void* b, void* out, int64_t n) {
    B200_REQUIRE(ctx && n >= 0 && (n == 0 || (a && b && out)), B200_EINVAL, "add: bad argument");
    B200_CUDA(cudaSetDevice(ctx->device));
    return launch_ew<OP_ADD>(ctx, a, b, out, n, 0.f, 0.f, 0);
}
int b200_clamp_f16(b200_ctx* ctx, const void* a, void* out, int64_t n, float lo, float hi) {
    B200_REQUIRE(ctx && n >= 0 && (n == 0 || (a && out)), B200_EINVAL, "clamp: bad argument");
    B200_CUDA(cudaSetDevice(ctx->device));
    return launch_ew<OP_CLAMP>(ctx, a, nullptr, out, n, lo, hi, 0);
}
int b200_act_f16(b200_ctx* ctx, const void* a, void* out, int64_t n, int epilogue) {
    B200_REQUIRE(ctx && n >= 0 && (n == 0 || (a && out)), B200_EINVAL, "act: bad argument");
    B200_REQUIRE(epilogue >= B200_EPI_NONE && epilogue <= B200_EPI_GELU_TANH, B200_EINVAL, "act: epilogue %d",
                 epilogue);
    B200_CUDA(cudaSetDevice(ctx->device));
    return launch_ew<OP_ACT>(ctx, a, nullptr, out, n, 0.f, 0.f, epilogue);
}
int b200_cast(b200_ctx* ctx, const void* src, int src_dtype, void* dst, int dst_dtype, int64_t n) {
    B200_REQUIRE(ctx && n >= 0 && (n == 0 || (src && dst)), B200_EINVAL, "cast: bad argument");
    B200_REQUIRE((src_dtype == B200_F16 || src_dtype == B200_F32) && (dst_dtype == B200_F16 || dst_dtype == B200_F32),
                 B200_DECLINE_ELTYPE, "cast: dtypes %d -> %d", src_dtype, dst_dtype);
    if (n == 0) return B200_OK;
    B200_CUDA(cudaSetDevice(ctx->device));
    if (src_dtype == dst_dtype) {
        B200_CUDA(cudaMemcpyAsync(dst, src, (size_t)n * (src_dtype == B200_F16 ? 2 : 4), cudaMemcpyDeviceToDevice, ctx->stream));
        return B200_OK;
    }
    return src_dtype == B200_F16 ? launch_cast<__half, float>(ctx, src, dst, n) : launch_cast<float, __half>(ctx, src, dst, n);
}
int b200_permute4(b200_ctx* ctx, const void* src, void* out, const int64_t* shape, const int64_t* stride,
                  int elsize) {
    B200_REQUIRE(ctx && shape && stride, B200_EINVAL, "permute4: null argument");
    for (int i = 0; i < 4; ++i) B200_REQUIRE(shape[i] >= 0, B200_EINVAL, "permute4: negative extent");
    B200_REQUIRE(elsize == 2 || elsize == 4, B200_DECLINE_ELTYPE, "permute4: element size %d", elsize);
    if (shape[0] * shape[1] * shape[2] * shape[3] == 0) return B200_OK;
    B200_REQUIRE(src && out, B200_EINVAL, "permute4: null array");
    B200_CUDA(cudaSetDevice(ctx->device));
    return elsize == 2 ? launch_permute<uint16_t>(ctx, src, out, shape, stride)
                       : launch_permute<uint32_t>(ctx, src, out, shape, stride);
}

} // extern "C"
