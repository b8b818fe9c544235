// Matrix-vector product for the one-token case of matmul! (reference kernels/extern/matmul.jl:103-137,
// the MMGemvPlan / Lava.gemv! path): out[m] = epi(T(bias[m] + sum_k A[m,k] x[k])), A (M,K) with M
// contiguous (what hoistpermutes leaves), fp32 accumulation.  Bandwidth-bound when A is large, a chain of round trips
// when it is not: every byte of A is read once, as aligned 16-byte vectors whatever the leading dimension (a
// vocabulary of 51865 rows gives every column its own misalignment), a warp covering 512 contiguous bytes of a
// column, the K axis split over the warps of a block and, when M alone cannot fill the GPU, over the blocks of a
// cluster as well, whose sums meet in distributed shared memory and are added in one fixed order (so the result does not
// depend on timing).  1280 x 1280 in fp16 6.3 -> 5.0 us and 594 x 1685 in fp32 6.0 -> 4.1 against partial sums through
// the workspace and half as many columns in flight.
#include <cuda_fp16.h>

#include "act.cuh"
#include "internal.h"
#include "ptx.cuh"

namespace b200 {

template <typename T> __device__ __forceinline__ float gemv_tof(T v);
template <> __device__ __forceinline__ float gemv_tof<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float gemv_tof<float>(float v) { return v; }

// The activation sees the value rounded to the output type (ops.jl:161-169), as in the GEMM's store.
template <typename OutT>
__device__ __forceinline__ void gemv_store(OutT* out, int64_t m, float acc, int epi) {
    if constexpr (sizeof(OutT) == 2) out[m] = __float2half_rn(apply_act(epi, __half2float(__float2half_rn(acc))));
    else out[m] = apply_act(epi, acc);
}

constexpr int GEMV_WARPS = 16;          // a multiple of 8: a warp's columns share their offset from a 16-byte boundary
constexpr int GEMV_UNROLL = 8;          // columns in flight per lane: 128 bytes
constexpr int GEMV_BLOCKS_PER_SM = 2;   // resident blocks of 512 threads at 64 registers
constexpr int GEMV_SPLIT_MIN_K = 4096;  // (gemv_run)
constexpr int GEMV_MIN_COLS = 8;        // columns per warp below which a further K split only adds the join

// Pairwise sum of the warps, and of the parts.  With results kept in fp32 and K over fewer than eight parts (PAIRS) a warp's
// columns are added two at a time as well: as one chain over them and one over the warps, those results were up to 17 %
// further from 64 bits than with the fewer columns that a warp of gemv_split_kernel takes (10428 x 429: 1.24e-7 against
// 1.06e-7).  Eight parts leave a warp few enough (492 x 4415: 5.45 us, 5.68 in pairs), and rounded to fp16 none of this shows.
template <int N> __device__ __forceinline__ float gemv_pairs(float (&v)[N]) {
#pragma unroll
    for (int h = N / 2; h > 0; h /= 2)
#pragma unroll
        for (int i = 0; i < h; ++i) v[i] += v[i + h];
    return v[0];
}

// grid (m blocks, k parts); block (32, GEMV_WARPS); the k parts of an m block form a cluster.
//
// Warp w takes columns k0 + w, k0 + w + 16, ...  Their start addresses differ by multiples of
// 16 * lda * sizeof(T), a multiple of 16 bytes, so all of one warp's columns sit at the same offset s
// (in elements) from a 16-byte boundary.  The warp therefore keeps its accumulators aligned to memory,
// not to rows: lane l reads the aligned vector j = 31 * block + l of each column, whose VEC elements
// are rows VEC * j - s ... VEC * j - s + VEC - 1, with no shifting or masking in the loop.  A block owns
// 31 * VEC rows; the 32 vectors its lanes read cover them for every s (the neighbouring blocks read the
// first and last of them again, out of L2).  Elements a vector holds outside [0, M) (the end of the
// previous column, the start of the next, or the rest of an aligned 16-byte block at either end of the
// array) only reach accumulators that are thrown away; every vector read holds at least one element of
// A, so no read leaves the 16-byte blocks the array occupies.
template <typename T, typename OutT, bool PAIRS>
__global__ void __launch_bounds__(32 * GEMV_WARPS, GEMV_BLOCKS_PER_SM)
gemv_kernel(const T* __restrict__ A, int64_t lda, const T* __restrict__ x, const T* __restrict__ bias, OutT* __restrict__ out,
            int64_t M, int64_t K, int64_t kchunk, int epi) {
    constexpr int VEC = 16 / (int)sizeof(T);
    constexpr int ROWS = 31 * VEC;
    __shared__ float red[GEMV_WARPS][ROWS];
    __shared__ float sums[ROWS];
    const int lane = threadIdx.x, warp = threadIdx.y, tid = warp * 32 + lane;
    const int parts = gridDim.y;
    const int64_t k0 = (int64_t)blockIdx.y * kchunk;
    const int64_t k1 = k0 + kchunk < K ? k0 + kchunk : K;
    const int64_t j = (int64_t)blockIdx.x * 31 + lane;
    grid_dep_wait();
    grid_dep_launch();
    float acc[VEC];
#pragma unroll
    for (int v = 0; v < VEC; ++v) acc[v] = 0.f;
    int s = 0;
    int64_t k = k0 + warp;
    if (k < k1) {
        s = (int)((reinterpret_cast<uintptr_t>(A + k * lda) & 15u) / sizeof(T));
        if (VEC * j - s < M) {
            // first aligned vector of column k, then + j; columns are 16 * lda elements apart
            const uint4* vp = reinterpret_cast<const uint4*>(reinterpret_cast<const char*>(A + k * lda) - s * sizeof(T)) + j;
            const int64_t vstep = GEMV_WARPS * lda * (int64_t)sizeof(T) / 16;
            constexpr int UN = GEMV_UNROLL;
            for (; k < k1; k += UN * GEMV_WARPS, vp += UN * vstep) {
                uint4 a[UN];
                float xv[UN];
#pragma unroll
                for (int u = 0; u < UN; ++u) {
                    const bool in = k + u * GEMV_WARPS < k1;
                    a[u] = in ? __ldg(vp + u * vstep) : make_uint4(0u, 0u, 0u, 0u);
                    xv[u] = in ? gemv_tof<T>(x[k + u * GEMV_WARPS]) : 0.f;
                }
#pragma unroll
                for (int u = 0; u < UN; u += 2) {
                    const T* e = reinterpret_cast<const T*>(&a[u]);
                    const T* f = reinterpret_cast<const T*>(&a[u + 1]);
#pragma unroll
                    for (int v = 0; v < VEC; ++v) {
                        if constexpr (PAIRS) {   // two columns at a time: half the chain (see gemv_pairs)
                            acc[v] += fmaf(gemv_tof<T>(f[v]), xv[u + 1], gemv_tof<T>(e[v]) * xv[u]);
                        } else {
                            acc[v] = fmaf(gemv_tof<T>(e[v]), xv[u], acc[v]);
                            acc[v] = fmaf(gemv_tof<T>(f[v]), xv[u + 1], acc[v]);
                        }
                    }
                }
            }
        }
    }
    // accumulator v of lane l is row VEC * l + v - s of the block
#pragma unroll
    for (int v = 0; v < VEC; ++v) {
        const int r = VEC * lane + v - s;
        if (r >= 0 && r < ROWS) red[warp][r] = acc[v];
    }
    __syncthreads();
    auto finish = [&](int r, float t) {
        const int64_t m = (int64_t)blockIdx.x * ROWS + r;
        if (m >= M) return;
        if (bias != nullptr) t += gemv_tof<T>(bias[m]);
        gemv_store<OutT>(out, m, t, epi);
    };
    for (int r = tid; r < ROWS; r += 32 * GEMV_WARPS) {
        float v[GEMV_WARPS];
#pragma unroll
        for (int w = 0; w < GEMV_WARPS; ++w) v[w] = red[w][r];
        const float t = gemv_pairs(v);
        if (parts > 1) sums[r] = t;
        else finish(r, t);
    }
    if (parts == 1) return;
    cluster_sync_all();   // every part's sums are in its shared memory
    const int rank = (int)blockIdx.y;
    const uint32_t mine = smem_u32(sums);
    for (int r = tid * parts + rank; r < ROWS; r += 32 * GEMV_WARPS * parts) {
        float v[8];   // every part's load in flight together: a remote load takes a few hundred nanoseconds
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = q < parts ? ld_cluster_f32(mapa_u32(mine + r * 4, (uint32_t)q)) : 0.f;
        finish(r, gemv_pairs(v));
    }
    cluster_sync_all();   // nobody leaves while its sums may still be read
}

// The same in blocks of eight warps, four columns in flight, with the K axis over up to 64 blocks that are not a cluster
// (gemv_run says when).  Partial sums go through the workspace and are added in split order by
// whichever block of a row range finishes last, so the result does not depend on timing.
constexpr int GEMV_SPLIT_WARPS = 8;
template <typename T, typename OutT>
__global__ void __launch_bounds__(32 * GEMV_SPLIT_WARPS, 6)
gemv_split_kernel(const T* __restrict__ A, int64_t lda, const T* __restrict__ x, const T* __restrict__ bias, OutT* __restrict__ out,
            float* __restrict__ partial, int* __restrict__ arrived, int64_t M, int64_t K, int64_t kchunk, int epi) {
    constexpr int VEC = 16 / (int)sizeof(T);
    constexpr int ROWS = 31 * VEC;
    __shared__ float red[GEMV_SPLIT_WARPS][ROWS];
    __shared__ int last;
    const int lane = threadIdx.x, warp = threadIdx.y;
    const int64_t k0 = (int64_t)blockIdx.y * kchunk;
    const int64_t k1 = k0 + kchunk < K ? k0 + kchunk : K;
    const int64_t j = (int64_t)blockIdx.x * 31 + lane;
    float acc[VEC];
#pragma unroll
    for (int v = 0; v < VEC; ++v) acc[v] = 0.f;
    int s = 0;
    int64_t k = k0 + warp;
    if (k < k1) {
        s = (int)((reinterpret_cast<uintptr_t>(A + k * lda) & 15u) / sizeof(T));
        if (VEC * j - s < M) {
            // first aligned vector of column k, then + j; columns are 8 * lda elements apart
            const uint4* vp = reinterpret_cast<const uint4*>(reinterpret_cast<const char*>(A + k * lda) - s * sizeof(T)) + j;
            const int64_t vstep = GEMV_SPLIT_WARPS * lda * (int64_t)sizeof(T) / 16;
            constexpr int UN = 4;
            for (; k + (UN - 1) * GEMV_SPLIT_WARPS < k1; k += UN * GEMV_SPLIT_WARPS, vp += UN * vstep) {
                uint4 a[UN];
                float xv[UN];
#pragma unroll
                for (int u = 0; u < UN; ++u) {
                    a[u] = __ldg(vp + u * vstep);
                    xv[u] = gemv_tof<T>(x[k + u * GEMV_SPLIT_WARPS]);
                }
#pragma unroll
                for (int u = 0; u < UN; ++u) {
                    const T* e = reinterpret_cast<const T*>(&a[u]);
#pragma unroll
                    for (int v = 0; v < VEC; ++v) acc[v] = fmaf(gemv_tof<T>(e[v]), xv[u], acc[v]);
                }
            }
            for (; k < k1; k += GEMV_SPLIT_WARPS, vp += vstep) {
                const uint4 a = __ldg(vp);
                const float xv = gemv_tof<T>(x[k]);
                const T* e = reinterpret_cast<const T*>(&a);
#pragma unroll
                for (int v = 0; v < VEC; ++v) acc[v] = fmaf(gemv_tof<T>(e[v]), xv, acc[v]);
            }
        }
    }
    // accumulator v of lane l is row VEC * l + v - s of the block
#pragma unroll
    for (int v = 0; v < VEC; ++v) {
        const int r = VEC * lane + v - s;
        if (r >= 0 && r < ROWS) red[warp][r] = acc[v];
    }
    __syncthreads();
    for (int r = warp * 32 + lane; r < ROWS; r += 32 * GEMV_SPLIT_WARPS) {
        const int64_t m = (int64_t)blockIdx.x * ROWS + r;
        if (m >= M) continue;
        float t = 0.f;
#pragma unroll
        for (int w = 0; w < GEMV_SPLIT_WARPS; ++w) t += red[w][r];
        if (partial != nullptr) {
            partial[(int64_t)blockIdx.y * M + m] = t;
        } else {
            if (bias != nullptr) t += gemv_tof<T>(bias[m]);
            gemv_store<OutT>(out, m, t, epi);
        }
    }
    if (partial == nullptr) return;
    // K was split over gridDim.y blocks: the one that arrives last adds the partial sums of these rows in
    // split order (so the result does not depend on which block that is) and puts the counter back to zero
    // for the next launch.  Nobody waits on anybody.
    __threadfence();
    __syncthreads();
    if (warp == 0 && lane == 0) last = atomicAdd(arrived + blockIdx.x, 1) == (int)gridDim.y - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int r = warp * 32 + lane; r < ROWS; r += 32 * GEMV_SPLIT_WARPS) {
        const int64_t m = (int64_t)blockIdx.x * ROWS + r;
        if (m >= M) continue;
        float t = 0.f;
        for (unsigned y = 0; y < gridDim.y; ++y) t += __ldcg(partial + (int64_t)y * M + m);
        if (bias != nullptr) t += gemv_tof<T>(bias[m]);
        gemv_store<OutT>(out, m, t, epi);
    }
    if (warp == 0 && lane == 0) arrived[blockIdx.x] = 0;
}

template <typename T, typename OutT>
static int gemv_run(b200_ctx* ctx, int64_t M, int64_t K, const void* A, int64_t lda, const void* x, const void* bias, void* out,
                    int epi) {
    constexpr int ROWS = 31 * (16 / (int)sizeof(T));
    const int64_t mblocks = cdiv(M, ROWS);
    B200_REQUIRE(mblocks < (1ll << 31), B200_DECLINE_EXTENT, "gemv: M = %lld", (long long)M);
    // A cluster's parts: a power of two (clusters of 3 or 7 fill the GPCs badly: 7000 x 3000 in fp32 12 -> 15 us) that
    // leaves every block an SM of its own and every warp GEMV_MIN_COLS columns.
    const int64_t sms = ctx->prop.multiProcessorCount;
    int64_t parts = 1;
    while (parts < 8 && 2 * parts * mblocks <= sms && K >= 2 * parts * GEMV_WARPS * GEMV_MIN_COLS) parts *= 2;
    // Taken while a block has up to 290 KB to read, where round trips are what a call waits for (1280 x 1280 in fp16
    // 6.3 -> 5.0 us, 4390 x 721 in fp32 6.6 -> 5.5, 3000 x 5000 in fp16 10.0 -> 7.6).  With more to read, or more row
    // blocks than SMs, blocks of eight warps, six to an SM, stream with fewer gaps (9956 x 1817 in fp16 8.9 us against
    // 9.8, 51865 x 1280 25 against 31); and so few row blocks that eight parts would leave nine tenths of the SMs idle
    // over a long chain are split further that way (256 x 4096: 6.35 us, 6.44 as a cluster).
    const bool few = mblocks * 8 * 8 <= sms && K >= GEMV_SPLIT_MIN_K;
    const bool cluster = K == 0 || (!few && mblocks <= sms && M * K * (int64_t)sizeof(T) <= 290 * 1024 * mblocks * parts);
    if (!cluster && ctx->sk_flags != nullptr) {
        // K over blocks until the grid is one resident wave, sixteen columns a warp at least
        const int64_t slots = sms * 6;
        int64_t ksplit = mblocks >= slots || mblocks > GEMV_COUNTER_COUNT ? 1 : slots / mblocks;
        const int64_t most = K / (16 * GEMV_SPLIT_WARPS) > 0 ? K / (16 * GEMV_SPLIT_WARPS) : 1;
        if (ksplit > most) ksplit = most;
        if (ksplit > 64) ksplit = 64;
        const int64_t chunk = cdiv(K, ksplit);
        ksplit = cdiv(K, chunk);
        void* ws = nullptr;
        if (ksplit > 1) {
            int rc = ws_scratch(ctx, (size_t)ksplit * M * sizeof(float), &ws);
            if (rc) return rc;
        }
        gemv_split_kernel<T, OutT><<<dim3((unsigned)mblocks, (unsigned)ksplit), dim3(32, GEMV_SPLIT_WARPS), 0, ctx->stream>>>(
            (const T*)A, lda, (const T*)x, (const T*)bias, (OutT*)out, static_cast<float*>(ws), ctx->sk_flags + SK_FLAG_COUNT, M, K,
            chunk, epi);
        ctx->launches++;
        B200_CUDA(cudaGetLastError());
        return B200_OK;
    }
    const int64_t kchunk = K > 0 ? cdiv(K, parts) : 1;   // K = 0: one block per row range writes the bias
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)mblocks, (unsigned)parts, 1);
    cfg.blockDim = dim3(32, GEMV_WARPS, 1);
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = (unsigned)parts;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 2 : 1;
    const auto kern = sizeof(OutT) == 4 && parts < 8 ? gemv_kernel<T, OutT, sizeof(OutT) == 4> : gemv_kernel<T, OutT, false>;
    B200_CUDA(cudaLaunchKernelEx(&cfg, kern, (const T*)A, lda, (const T*)x, (const T*)bias, (OutT*)out, M, K, kchunk, epi));
    ctx->launches++;
    return B200_OK;
}

} // namespace b200

using namespace b200;

extern "C" {

int b200_gemv(b200_ctx* ctx, int64_t M, int64_t K, const void* A, int64_t lda, const void* x, const void* bias, int in_dtype,
              void* out, int out_dtype, int epilogue) {
    B200_REQUIRE(ctx, B200_EINVAL, "gemv: null context");
    B200_REQUIRE(M >= 0 && K >= 0 && lda >= (M > 0 ? M : 1), B200_EINVAL, "gemv: M=%lld K=%lld lda=%lld", (long long)M,
                 (long long)K, (long long)lda);
    B200_REQUIRE(in_dtype == B200_F16 || in_dtype == B200_F32, B200_DECLINE_ELTYPE, "gemv: operand dtype %d", in_dtype);
    B200_REQUIRE(out_dtype == B200_F32 || (out_dtype == B200_F16 && in_dtype == B200_F16), B200_DECLINE_ELTYPE,
                 "gemv: out dtype %d for operand dtype %d", out_dtype, in_dtype);
    B200_REQUIRE(epilogue >= B200_EPI_NONE && epilogue <= B200_EPI_GELU_TANH, B200_EINVAL, "gemv: epilogue %d", epilogue);
    if (M == 0) return B200_OK;
    B200_REQUIRE(out && (K == 0 || (A && x)), B200_EINVAL, "gemv: null array");
    B200_REQUIRE(reinterpret_cast<uintptr_t>(A) % (in_dtype == B200_F32 ? 4 : 2) == 0, B200_DECLINE_ALIGN,
                 "gemv: A is not aligned to its element size");
    B200_CUDA(cudaSetDevice(ctx->device));
    if (in_dtype == B200_F32) return gemv_run<float, float>(ctx, M, K, A, lda, x, bias, out, epilogue);
    if (out_dtype == B200_F16) return gemv_run<__half, __half>(ctx, M, K, A, lda, x, bias, out, epilogue);
    return gemv_run<__half, float>(ctx, M, K, A, lda, x, bias, out, epilogue);
}

} // extern "C"
