// Attention of at most 32 queries over any number of keys (a decoder's step over a long memory: 23 x 4096), E <= 128,
// with or without an additive mask: out = softmax(scale * Q K^T + mask) V, the arithmetic of attention_f16_tc_kernel
// (fp32 scores and softmax, P rounded to fp16 for the second product, fp32 accumulation; the key split and merge stand
// where attn_flash_cm_merge! stood, reference kernels/extern/flash.jl:1398-1421).
//
// What bounds it is the chain of round trips, not bytes or flops (23 x 4096 x 64 x 8 heads: 8 MB of keys and values,
// 1.3 us of HBM time): so the keys of a (head, batch) are spread over the CTAs of a cluster, each streams its share
// through a ring of 64-key blocks with cp.async, and the partial results meet in distributed shared memory inside the
// same launch.  The 128-row tensor-memory tiles of the large kernel would be mostly empty here, and its CTAs, one per
// SM, would pay tensor-memory and barrier set-up for two key blocks each and a second kernel for the merge; so the
// products are warp-level m16n8k16 tiles in registers, four warps sharing a block by queries and keys.  Measured against
// that: 23 x 4096, 8 heads 14.5 -> 9.2 us; masked, 3 x 477, 13 heads 29 -> 6, 2 x 7763, E = 128, 8 heads 419 -> 21.
#include <cuda_fp16.h>
#include <stdlib.h>

#include <mutex>
#include <type_traits>

#include "internal.h"
#include "ptx.cuh"

namespace b200 {

constexpr int AF_THREADS = 128;
constexpr int AF_BC = 64;    // keys per block of the ring
constexpr int AF_PARTS = 16; // CTAs of a cluster at most

// KS: key slots, i.e. how many of the four warps share a tile of 16 queries (4 / KS tiles per CTA, one or two).
template <int EP, int KS> struct AfCfg {
    static_assert(KS == 4 || (KS == 2 && EP == 64), "one query tile, or two of them at E <= 64");
    static constexpr int QT = 4 / KS, QR = 16 * QT;           // query tiles and rows of a CTA
    static constexpr int PITCH = EP + 8;                      // halves per shared row: an odd number of 16-byte units
    static constexpr int STAGES = EP == 64 ? 4 : 3;
    static constexpr int STAGE_HALVES = 2 * AF_BC * PITCH;    // K, then V
    static constexpr int RING_BYTES = STAGES * STAGE_HALVES * 2;
    // after the keys, over the ring: every warp's 16 x EP fp32 rows with (reference point, sum), then the CTA's rows
    static constexpr int ROW = EP + 4;                        // floats: the row, its reference point, its sum; 16-byte pitch
    static constexpr int PART_BYTES = 4 * 16 * ROW * 4;
    static_assert(PART_BYTES + QR * ROW * 4 <= RING_BYTES, "the partial results fit over the ring");
    static constexpr int SMEM_BYTES = RING_BYTES + QR * PITCH * 2;   // + Q
};

template <int V> struct AfInt {
    static constexpr int value = V;
};

struct FewParams {
    const __half *q, *k, *v, *bias;
    void* out;
    int64_t qsL, qsH, qsB, ksL, ksH, ksB, vsL, vsH, vsB, osL, osH, osB, bsK, bsQ, bsH, bsB;
    int E, Lq, Lk, out_f32;
    float scale_log2;
};

template <bool TRANS> __device__ __forceinline__ void af_ldmatrix(uint32_t (&r)[4], const __half* row) {
    const uint32_t addr = smem_u32(row);
    if constexpr (TRANS)
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
    else
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
// 16 bytes to shared memory, zeros when `live` is false (the address is then not read)
__device__ __forceinline__ void af_copy16(const __half* dst, const __half* src, bool live) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ uint32_t af_pack(float lo, float hi) {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}

// grid (key parts, heads, batch); the key parts form a cluster.
template <int EP, int KS, bool BIAS>
__global__ void __launch_bounds__(AF_THREADS, 2)
attention_few_kernel(const FewParams p) {
    using Cfg = AfCfg<EP, KS>;
    constexpr int PITCH = Cfg::PITCH, STAGES = Cfg::STAGES, QT = Cfg::QT, ROW = Cfg::ROW;
    constexpr int KW = AF_BC / KS, NT = KW / 8;     // keys of a block one warp takes, in tiles of 8
    extern __shared__ __align__(16) uint8_t af_smem[];
    __half* ring = reinterpret_cast<__half*>(af_smem);
    __half* Qs = reinterpret_cast<__half*>(af_smem + Cfg::RING_BYTES);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int qt = warp % QT, slot = warp / QT;
    const int parts = gridDim.x, rank = blockIdx.x, h = blockIdx.y, b = blockIdx.z;
    const int nblk_all = (p.Lk + AF_BC - 1) / AF_BC;
    const int jb0 = (int)((int64_t)rank * nblk_all / parts), nblk = (int)((int64_t)(rank + 1) * nblk_all / parts) - jb0;
    const __half* kbase = p.k + (int64_t)h * p.ksH + (int64_t)b * p.ksB;
    const __half* vbase = p.v + (int64_t)h * p.vsH + (int64_t)b * p.vsB;
    grid_dep_wait();
    grid_dep_launch();

    auto fetch = [&](int j) {   // block j of this part into its stage; a commit group even when there is none
        if (j < nblk) {
            __half* st = ring + (j % STAGES) * Cfg::STAGE_HALVES;
            const int key0 = (jb0 + j) * AF_BC;
#pragma unroll
            for (int i = 0; i < AF_BC * EP / 8 / AF_THREADS; ++i) {
                const int idx = tid + i * AF_THREADS, row = idx / (EP / 8), c = idx % (EP / 8) * 8;
                const bool live = key0 + row < p.Lk && c < p.E;
                const int64_t key = live ? key0 + row : 0;
                af_copy16(st + row * PITCH + c, kbase + key * p.ksL + (live ? c : 0), live);
                af_copy16(st + (AF_BC + row) * PITCH + c, vbase + key * p.vsL + (live ? c : 0), live);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    {
        const __half* qbase = p.q + (int64_t)h * p.qsH + (int64_t)b * p.qsB;
        for (int idx = tid; idx < Cfg::QR * EP / 8; idx += AF_THREADS) {   // with the first block's group
            const int row = idx / (EP / 8), c = idx % (EP / 8) * 8;
            const bool live = row < p.Lq && c < p.E;
            af_copy16(Qs + row * PITCH + c, qbase + (live ? row * p.qsL + c : 0), live);
        }
    }
#pragma unroll
    for (int j = 0; j < STAGES - 1; ++j) fetch(j);

    uint32_t qa[EP / 16][4];
    float o[EP / 8][4];
#pragma unroll
    for (int n = 0; n < EP / 8; ++n) o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f;
    float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;   // rows g and g + 8 of the tile
    const int r0 = qt * 16 + g;

    for (int j = 0; j < nblk; ++j) {
        const int kw0 = (jb0 + j) * AF_BC + slot * KW;           // the warp's first key of the block
        float bias[BIAS ? NT : 1][4];
        if constexpr (BIAS) {   // asked for before the wait for the block
            const __half* bp = p.bias + (int64_t)h * p.bsH + (int64_t)b * p.bsB;
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const int row = r0 + (c >> 1) * 8, key = kw0 + n * 8 + 2 * t + (c & 1);
                    bias[n][c] = row < p.Lq && key < p.Lk ? __half2float(__ldg(bp + row * p.bsQ + key * p.bsK)) : 0.f;
                }
        }
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncthreads();   // block j has landed for everyone, and block j - 1 has been read by everyone
        fetch(j + STAGES - 1);
        if (j == 0) {
#pragma unroll
            for (int ks = 0; ks < EP / 16; ++ks)
                af_ldmatrix<false>(qa[ks], Qs + (qt * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * PITCH + ks * 16 + (lane >> 4) * 8);
        }
        const __half* Ks = ring + (j % STAGES) * Cfg::STAGE_HALVES + slot * KW * PITCH;
        const __half* Vs = Ks + AF_BC * PITCH;
        float s[NT][4];
#pragma unroll
        for (int n = 0; n < NT; ++n) s[n][0] = s[n][1] = s[n][2] = s[n][3] = 0.f;
#pragma unroll
        for (int n = 0; n < NT; n += 2)
#pragma unroll
            for (int ks = 0; ks < EP / 16; ++ks) {
                uint32_t kb[4];
                af_ldmatrix<false>(kb, Ks + ((n + (lane >> 4)) * 8 + (lane & 7)) * PITCH + ks * 16 + ((lane >> 3) & 1) * 8);
                mma_16816(s[n], qa[ks], kb[0], kb[1]);
                mma_16816(s[n + 1], qa[ks], kb[2], kb[3]);
            }
        float x0 = -INFINITY, x1 = -INFINITY;
#pragma unroll
        for (int n = 0; n < NT; ++n) {
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                s[n][c] = BIAS ? fmaf(s[n][c], p.scale_log2, bias[BIAS ? n : 0][c] * 1.4426950408889634f) : s[n][c] * p.scale_log2;
                if (kw0 + n * 8 + 2 * t + (c & 1) >= p.Lk) s[n][c] = -INFINITY;
            }
            x0 = fmaxf(x0, fmaxf(s[n][0], s[n][1]));
            x1 = fmaxf(x1, fmaxf(s[n][2], s[n][3]));
        }
#pragma unroll
        for (int d = 1; d < 4; d *= 2) {   // a quad of lanes shares a row
            x0 = fmaxf(x0, __shfl_xor_sync(0xffffffffu, x0, d));
            x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, d));
        }
        x0 = fmaxf(m0, x0);
        x1 = fmaxf(m1, x1);
        // a row that has seen nothing but -inf keeps the reference point -inf and contributes zeros
        const float a0 = m0 == x0 ? 1.f : exp2f(m0 - x0), a1 = m1 == x1 ? 1.f : exp2f(m1 - x1);
        const float n0 = x0 == -INFINITY ? 0.f : x0, n1 = x1 == -INFINITY ? 0.f : x1;
        m0 = x0;
        m1 = x1;
        l0 *= a0;
        l1 *= a1;
#pragma unroll
        for (int n = 0; n < EP / 8; ++n) {
            o[n][0] *= a0;
            o[n][1] *= a0;
            o[n][2] *= a1;
            o[n][3] *= a1;
        }
        uint32_t pa[NT / 2][4];
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            const float e0 = exp2f(s[n][0] - n0), e1 = exp2f(s[n][1] - n0), e2 = exp2f(s[n][2] - n1), e3 = exp2f(s[n][3] - n1);
            l0 += e0 + e1;
            l1 += e2 + e3;
            pa[n >> 1][(n & 1) * 2] = af_pack(e0, e1);
            pa[n >> 1][(n & 1) * 2 + 1] = af_pack(e2, e3);
        }
#pragma unroll
        for (int kk = 0; kk < NT / 2; ++kk)
#pragma unroll
            for (int n = 0; n < EP / 8; n += 2) {
                uint32_t vb[4];
                af_ldmatrix<true>(vb, Vs + (kk * 16 + (lane & 15)) * PITCH + (n + (lane >> 4)) * 8);
                mma_16816(o[n], pa[kk], vb[0], vb[1]);
                mma_16816(o[n + 1], pa[kk], vb[2], vb[3]);
            }
    }
#pragma unroll
    for (int d = 1; d < 4; d *= 2) {
        l0 += __shfl_xor_sync(0xffffffffu, l0, d);
        l1 += __shfl_xor_sync(0xffffffffu, l1, d);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();   // the ring is free
    // This warp's rows: [row][EP values, reference point, sum]
    float* rows = reinterpret_cast<float*>(af_smem + Cfg::PART_BYTES);
    float* mine = reinterpret_cast<float*>(af_smem) + warp * 16 * ROW;
#pragma unroll
    for (int n = 0; n < EP / 8; ++n) {
        *reinterpret_cast<float2*>(mine + g * ROW + n * 8 + 2 * t) = make_float2(o[n][0], o[n][1]);
        *reinterpret_cast<float2*>(mine + (g + 8) * ROW + n * 8 + 2 * t) = make_float2(o[n][2], o[n][3]);
    }
    if (t == 0) {
        *reinterpret_cast<float2*>(mine + g * ROW + EP) = make_float2(m0, l0);
        *reinterpret_cast<float2*>(mine + (g + 8) * ROW + EP) = make_float2(m1, l1);
    }
    __syncthreads();
    // the key slots of a query tile
    for (int i = tid; i < Cfg::QR * (EP + 1); i += AF_THREADS) {
        const int row = i / (EP + 1), e = i % (EP + 1);
        const float* src = reinterpret_cast<const float*>(af_smem) + ((row >> 4) * 16 + (row & 15)) * ROW;   // slot 0; slot s: QT warps on
        float M = -INFINITY;
#pragma unroll
        for (int s = 0; s < KS; ++s) M = fmaxf(M, src[s * QT * 16 * ROW + EP]);
        float v = 0.f;
#pragma unroll
        for (int s = 0; s < KS; ++s) {
            const float m = src[s * QT * 16 * ROW + EP];
            const float w = m == -INFINITY ? 0.f : exp2f(m - M);
            v = fmaf(src[s * QT * 16 * ROW + (e < EP ? e : EP + 1)], w, v);
        }
        rows[row * ROW + (e < EP ? e : EP + 1)] = v;
        if (e == EP) rows[row * ROW + EP] = M;
    }
    if (parts > 1) cluster_sync_all();   // every part's rows are in its shared memory
    else __syncthreads();
    // A warp finishes rows, lane l its elements 4 l ... 4 l + 3.  Remote loads take a few hundred nanoseconds, so all
    // that a step needs are in flight together: (reference point, sum) of part l by lane l, then the row of PB parts at
    // a time; one row of all parts when there are no more rows than warps, else four rows of four parts.
    const uint32_t base = smem_u32(rows);
    auto finish = [&](auto rb, auto pb) {
        constexpr int RB = decltype(rb)::value, PB = decltype(pb)::value;
        for (int row0 = (rank * 4 + warp) * RB; row0 < p.Lq; row0 += parts * 4 * RB) {
            float w[RB], inv[RB];
            float4 acc[RB];
#pragma unroll
            for (int r = 0; r < RB; ++r) {
                const uint32_t at = base + (row0 + r < p.Lq ? row0 + r : row0) * (ROW * 4) + EP * 4;
                const float2 ml = lane < parts ? ld_cluster_f32x2(mapa_u32(at, (uint32_t)lane)) : make_float2(-INFINITY, 0.f);
                w[r] = ml.x;
                inv[r] = ml.y;
                acc[r] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int r = 0; r < RB; ++r) {
                float M = w[r];
#pragma unroll
                for (int d = 1; d < 32; d *= 2) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, d));
                w[r] = w[r] == -INFINITY ? 0.f : exp2f(w[r] - M);
                float den = inv[r] * w[r];
#pragma unroll
                for (int d = 1; d < 32; d *= 2) den += __shfl_xor_sync(0xffffffffu, den, d);
                inv[r] = 1.f / (den == 0.f ? 1.f : den);
            }
            for (int q0 = 0; q0 < parts; q0 += PB) {
                float4 v[RB][PB];
#pragma unroll
                for (int u = 0; u < PB; ++u) {
                    const bool in = q0 + u < parts && 4 * lane < EP;
                    const uint32_t src = mapa_u32(base + lane * 16, (uint32_t)(in ? q0 + u : 0));
#pragma unroll
                    for (int r = 0; r < RB; ++r)
                        v[r][u] = in ? ld_cluster_f32x4(src + (row0 + r < p.Lq ? row0 + r : row0) * (ROW * 4)) : make_float4(0.f, 0.f, 0.f, 0.f);
                }
#pragma unroll
                for (int u = 0; u < PB; ++u)
#pragma unroll
                    for (int r = 0; r < RB; ++r) {
                        const float f = __shfl_sync(0xffffffffu, w[r], q0 + u);   // zero past the last part
                        acc[r].x = fmaf(v[r][u].x, f, acc[r].x);
                        acc[r].y = fmaf(v[r][u].y, f, acc[r].y);
                        acc[r].z = fmaf(v[r][u].z, f, acc[r].z);
                        acc[r].w = fmaf(v[r][u].w, f, acc[r].w);
                    }
            }
#pragma unroll
            for (int r = 0; r < RB; ++r) {
                if (row0 + r >= p.Lq || 4 * lane >= p.E) continue;
                const float4 x = make_float4(acc[r].x * inv[r], acc[r].y * inv[r], acc[r].z * inv[r], acc[r].w * inv[r]);
                const int64_t dst = (row0 + r) * p.osL + (int64_t)h * p.osH + (int64_t)b * p.osB + 4 * lane;
                if (p.out_f32) *reinterpret_cast<float4*>(static_cast<float*>(p.out) + dst) = x;
                else *reinterpret_cast<uint2*>(static_cast<__half*>(p.out) + dst) = make_uint2(af_pack(x.x, x.y), af_pack(x.z, x.w));
            }
        }
    };
    if (p.Lq <= 4 * parts) finish(AfInt<1>{}, AfInt<AF_PARTS>{});
    else finish(AfInt<4>{}, AfInt<4>{});
    if (parts > 1) cluster_sync_all();   // nobody leaves while its rows may still be read
}

// How many CTAs of this kernel, and clusters of 2, 4, 8 and 16 of them, the device holds at once: [l] for 2^l, asked of the
// runtime once per device.  A GPC's SMs do not divide into large clusters without a rest, so that twice the SMs over the size is too many;
// sixteen is beyond the portable size besides, and a slice of a GPU may hold none.
struct AfRoom {
    int clusters[5];
};
template <typename Kern> static AfRoom af_ask(b200_ctx* ctx, Kern kern, size_t smem) {
    AfRoom room = {};
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, AF_THREADS, smem) != cudaSuccess) cudaGetLastError();
    room.clusters[0] = ctx->prop.multiProcessorCount * (per_sm > 0 ? per_sm : 1);
    const bool wide = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
    for (int l = 1; l <= (wide ? 4 : 3); ++l) {
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 1u << l;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(1u << l, 1, 1);
        cfg.blockDim = dim3(AF_THREADS, 1, 1);
        cfg.dynamicSmemBytes = smem;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int fit = 0;
        if (cudaOccupancyMaxActiveClusters(&fit, kern, &cfg) == cudaSuccess) room.clusters[l] = fit;
        else cudaGetLastError();
    }
    if (!wide) cudaGetLastError();
    return room;
}

template <int EP, int KS, bool BIAS> static cudaError_t af_rooms(b200_ctx* ctx, const AfRoom*& room) {
    static std::once_flag once[16];
    static AfRoom rooms[16];
    static cudaError_t set[16];
    auto kern = attention_few_kernel<EP, KS, BIAS>;
    const int d = ctx->device & 15;
    std::call_once(once[d], [&] {
        set[d] = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, AfCfg<EP, KS>::SMEM_BYTES);
        if (set[d] == cudaSuccess) rooms[d] = af_ask(ctx, kern, AfCfg<EP, KS>::SMEM_BYTES);
    });
    room = &rooms[d];
    return set[d];
}

static const char* af_forced() { return getenv("B200_ATTENTION_PARTS"); }   // debugging aid: this kernel, with clusters up to that size

// Key parts: as many, with two blocks or more each, as keep every cluster resident at once, two CTAs to an SM.  A second
// round of clusters costs more than the shorter walk saves (17 heads, 25 x 2405: 15.7 us with sixteen parts, of which
// sixteen clusters fit), and so does a third CTA on an SM (20 heads, 12 x 2003: 7.1 us with eight parts, 7.4 with sixteen).
static int af_parts(const AfRoom& room, int64_t sms, int64_t nblk, int64_t items) {
    const char* f = af_forced();
    const int most = f ? atoi(f) : AF_PARTS;
    int parts = 1;
    for (int l = 1; l <= 4 && (1 << l) <= most && nblk >= 2 << l; ++l)
        if (items <= room.clusters[l] && items << l <= 2 * sms) parts = 1 << l;
    return parts;
}

template <int EP, int KS, bool BIAS>
static int af_launch(b200_ctx* ctx, const FewParams& p, int64_t H, int64_t B) {
    const AfRoom* room;
    B200_CUDA((af_rooms<EP, KS, BIAS>(ctx, room)));
    const int parts = af_parts(*room, ctx->prop.multiProcessorCount, cdiv(p.Lk, AF_BC), H * B);
    B200_CUDA(launch_dep(attention_few_kernel<EP, KS, BIAS>, dim3((unsigned)parts, (unsigned)H, (unsigned)B), dim3(AF_THREADS, 1, 1),
                         AfCfg<EP, KS>::SMEM_BYTES, ctx->stream, parts, p));
    ctx->launches++;
    return B200_OK;
}

// f(head dim tier, key slots, mask) with the three as constants
template <typename F> static auto af_dispatch(int64_t E, int64_t Lq, bool masked, F f) {
    auto mask = [&](auto ep, auto ks) { return masked ? f(ep, ks, std::true_type{}) : f(ep, ks, std::false_type{}); };
    if (E > 64) return mask(AfInt<128>{}, AfInt<4>{});       // up to 16 queries
    return Lq <= 16 ? mask(AfInt<64>{}, AfInt<4>{}) : mask(AfInt<64>{}, AfInt<2>{});
}

// Whether a call of few queries is faster here than as tiles of 128 queries (attention_f16_tc_kernel, which cuts the keys
// too, and merges in a second launch).  Both times in us, fitted to 5060 shapes timed on both (4 to 290 heads in all, 1 to
// 32 queries, 16 to 8192 keys): the large kernel takes as long for 128 keys as this one for 64, but sets up tensor memory
// and merges.  16 to 32 queries over up to 384 keys are its (20 heads, 32 x 128: 4.4 us there, 7.2 here; 32 x 256 5.7, 6.7),
// and many heads over long keys with more than 16 queries (36 heads, 32 x 8192: 31, 36); up to 8 queries are nearly always
// this one's (8 heads, 1 x 1000: 9.5, 5.0).  The large kernel's constants, and that it cuts whatever leaves SMs idle into parts of two
// blocks or more, are of its form before whole warps issued and a cut was weighed; against the present one the choice is 0.4 % off the
// faster in the mean over 420 shapes (always here 5 %, always there 25 %), 26 of them more than 4 %, up to 1.3 times for a
// few queries' long masks (4 x 4, 3 x 6849 x 128: 35.3 us, 27.4 there).
bool attention_few_takes(b200_ctx* ctx, int64_t E, int64_t Lq, int64_t Lk, int64_t H, int64_t B, bool masked) {
    if (Lq > (E <= 64 ? 32 : 16)) return false;
    if (af_forced()) return true;
    struct Large { double wave, split, part, block; };
    struct Few { double start, join, finish, one, two; };   // per block: one CTA on an SM, or two
    static const Large large[2][2] = {{{3.16, 2.76, 0.34, 1.42}, {3.04, 2.72, 0.37, 2.22}}, {{3.05, 2.72, 0.40, 2.22}, {2.95, 2.73, 0.41, 3.09}}};
    static const Few few[3][2] = {{{3.41, 0.84, 0.83, 0.46, 0.78}, {3.47, 1.08, 1.07, 0.86, 1.21}},
                                  {{6.17, -0.51, 0.33, 0.50, 0.99}, {5.77, -0.66, 0.15, 1.77, 2.60}},
                                  {{4.58, 0.86, 0.79, 0.92, 1.52}, {4.27, 1.10, 1.25, 1.41, 2.35}}};
    const int64_t items = H * B, sms = ctx->prop.multiProcessorCount, blocks = cdiv(Lk, 128), nblk = cdiv(Lk, AF_BC);
    const Large& m = large[E > 64][masked];
    double there = m.wave * (double)cdiv(items, sms) + m.block * (double)(blocks * cdiv(items, sms));
    const int64_t rem = items % sms, cut = 2 * items <= sms ? items : (items > sms && rem > 0 && 2 * rem <= sms ? rem : 0);
    if (blocks >= 4 && cut > 0) {   // the keys of `cut` items over ns CTAs each
        int64_t ns = sms / cut;
        if (ns > blocks / 2) ns = blocks / 2;
        if (ns > 64) ns = 64;
        if (ns >= 2)
            there = m.wave * (double)(items / sms + 1) + m.split + m.part * (double)ns + m.block * (double)(blocks * (items / sms) + cdiv(blocks, ns));
    }
    const AfRoom* room = nullptr;
    const cudaError_t e = af_dispatch(E, Lq, masked, [&](auto ep, auto ks, auto bias) {
        return af_rooms<decltype(ep)::value, decltype(ks)::value, decltype(bias)::value>(ctx, room);
    });
    if (e != cudaSuccess) return true;   // the launch reports it
    const int parts = af_parts(*room, sms, nblk, items);
    const bool wide = E <= 64 && Lq > 16;   // two query tiles
    const Few& q = few[E > 64 ? 2 : wide][masked];
    const int64_t ctas = items * parts, waves = parts > 1 ? 1 : cdiv(items, room->clusters[0]);
    // (further rounds start under the ones before; a CTA's walk is its own up to an SM each, the heavier ones' up to seven
    // eighths of that: clusters do not spread evenly)
    const double each = ctas <= (wide || (masked && E > 64) ? sms * 7 / 8 : sms) ? q.one : q.two * (double)waves;
    const double here = q.start * 0.5 * (double)(waves + 1) + (parts > 1 ? q.join : 0.0) + (Lq > 4 * parts ? q.finish : 0.0) + each * (double)cdiv(nblk, parts);
    return here <= 1.03 * there;   // within the fits' own error the simpler launch
}

int attention_few_launch(b200_ctx* ctx, int64_t E, int64_t Lq, int64_t Lk, int64_t H, int64_t B, const b200_strided4* q,
                         const b200_strided4* k, const b200_strided4* v, const void* bias, const int64_t* bs,
                         const b200_strided4* o, int out_dtype, float scale) {
    FewParams p;
    p.q = static_cast<const __half*>(q->ptr);
    p.k = static_cast<const __half*>(k->ptr);
    p.v = static_cast<const __half*>(v->ptr);
    p.bias = static_cast<const __half*>(bias);
    p.out = const_cast<void*>(o->ptr);
    p.qsL = q->stride[1]; p.qsH = q->stride[2]; p.qsB = q->stride[3];
    p.ksL = k->stride[1]; p.ksH = k->stride[2]; p.ksB = k->stride[3];
    p.vsL = v->stride[1]; p.vsH = v->stride[2]; p.vsB = v->stride[3];
    p.osL = o->stride[1]; p.osH = o->stride[2]; p.osB = o->stride[3];
    p.bsK = bs[0]; p.bsQ = bs[1]; p.bsH = bs[2]; p.bsB = bs[3];
    p.E = (int)E; p.Lq = (int)Lq; p.Lk = (int)Lk;
    p.out_f32 = out_dtype == B200_F32;
    p.scale_log2 = scale * 1.4426950408889634f;
    return af_dispatch(E, Lq, bias != nullptr, [&](auto ep, auto ks, auto masked) {
        return af_launch<decltype(ep)::value, decltype(ks)::value, decltype(masked)::value>(ctx, p, H, B);
    });
}

} // namespace b200
