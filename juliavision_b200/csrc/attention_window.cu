// Attention over many short key sequences (windows of at most 64 keys, e.g. the 8x8-token windows of a
// hierarchical image encoder's first stages): out = softmax(scale * Q K^T) V per (window, head), the same
// arithmetic as attention_f16_tc_kernel (fp32 scores and softmax, P rounded to fp16 for the second
// product, fp32 accumulation, reference kernels/extern/flash.jl:459-1036 for the fused form).
//
// At this size the work per window is a megaflop and the operation is bound by HBM and by latency, not by
// the tensor pipe: the 128-row TMEM tiles of the large kernel are mostly empty and its per-CTA set-up
// (TMEM allocation, barriers, tensor maps) costs more than the window's arithmetic, with one CTA resident
// per SM.  So this kernel is small instead: CTAs of four warps, operands fetched with cp.async, and each warp's 16 x 64 scores
// and 16 x 64 output held in registers as warp-level m16n8k16 tiles.  A CTA takes one unit, 64 queries of one (window, head),
// six CTAs to an SM; or, where there are many more units of more than a few keys, four CTAs to an SM walk the units with the next
// one's operands on their way (two buffers of 27 KB) under this one's arithmetic.
// Microseconds, replayed (a unit a CTA with loads through registers / always walking / now): 8192 windows x 2 heads of 64 x 64 x
// 56 (470 MB) 118.6 / 107.1 / 106.3, 1024 x 2 in the L2 15.3 / 17.1 / 14.6, 2000 x 4 of 49 x 49 x 64 57.2 / 49.9 / 49.6, 600 x 4 of
// 16 x 16 x 56 9.9 / 9.6 / 8.5.
#include <cuda_fp16.h>

#include "internal.h"
#include "ptx.cuh"

namespace b200 {

constexpr int AW_THREADS = 128;
constexpr int AW_BQ = 64;      // queries per CTA (16 per warp)
constexpr int AW_LK = 64;      // keys per window at most
constexpr int AW_PITCH = 72;   // halves per shared row: 144 bytes, rows 4 banks apart, conflict-free fragments

struct WinParams {
    const __half *q, *k, *v;
    void* out;
    int64_t qsL, qsH, qsB, ksL, ksH, ksB, vsL, vsH, vsB, osL, osH, osB;
    int E, Lq, Lk, H, B, qtiles, out_f32;
    uint32_t units;
    float scale_log2;
};

__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], const __half* row) {
    const uint32_t addr = (uint32_t)__cvta_generic_to_shared(row);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}

__device__ __forceinline__ uint32_t pack_h2(float lo, float hi) {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}

__device__ __forceinline__ float win_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// rows [0, rows) x E halves of a strided (E, L) slice on their way into a [64][AW_PITCH] shared tile, zeros elsewhere already
__device__ __forceinline__ void win_fetch(__half* tile, const __half* base, int64_t sL, int rows, int E, int tid) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int idx = tid + i * AW_THREADS;          // 512 vectors: 64 rows x 8
        const int row = idx >> 3, vec = idx & 7;
        if (row < rows && vec * 8 < E)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(tile + row * AW_PITCH + vec * 8)),
                         "l"(base + (int64_t)row * sL + vec * 8)
                         : "memory");
    }
}

// One unit: 64 queries of one (window, head) out of its shared tiles.
__device__ __forceinline__ void window_unit(const WinParams& p, __half* Qs, const __half* Ks, const __half* Vs, int h, int b, int q0,
                                            int qrows, int warp, int lane, int g, int t) {
    const int r0 = warp * 16;
    if (r0 >= qrows) return;

    // S = Q K^T: 16 queries x 64 keys as eight n-tiles of 8 keys, four k-steps of 16 along E
    // Fragments come out of the row-major tiles with ldmatrix: four 8 x 8 blocks per instruction.
    uint32_t qa[4][4];
#pragma unroll
    for (int ks = 0; ks < 4; ++ks)      // blocks (rows 0-7 | 8-15) x (dims 16ks.. | 16ks+8..) of the warp's queries
        ldmatrix_x4(qa[ks], Qs + (r0 + (lane & 7) + ((lane >> 3) & 1) * 8) * AW_PITCH + ks * 16 + (lane >> 4) * 8);
    float s[8][4];
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) s[nt][0] = s[nt][1] = s[nt][2] = s[nt][3] = 0.f;
#pragma unroll
    for (int nt = 0; nt < 8; nt += 2) {
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
            uint32_t kb[4];             // blocks (keys 8nt.. | 8nt+8..) x (dims 16ks.. | 16ks+8..)
            ldmatrix_x4(kb, Ks + ((nt + (lane >> 4)) * 8 + (lane & 7)) * AW_PITCH + ks * 16 + ((lane >> 3) & 1) * 8);
            mma_16816(s[nt], qa[ks], kb[0], kb[1]);
            mma_16816(s[nt + 1], qa[ks], kb[2], kb[3]);
        }
    }
    // softmax over the keys of rows g (values 0,1) and g + 8 (values 2,3); a quad of lanes shares a row
    float m0 = -INFINITY, m1 = -INFINITY;
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int key = nt * 8 + 2 * t + (c & 1);
            s[nt][c] = key < p.Lk ? s[nt][c] * p.scale_log2 : -INFINITY;
        }
        m0 = fmaxf(m0, fmaxf(s[nt][0], s[nt][1]));
        m1 = fmaxf(m1, fmaxf(s[nt][2], s[nt][3]));
    }
    m0 = fmaxf(m0, __shfl_xor_sync(0xffffffffu, m0, 1));
    m0 = fmaxf(m0, __shfl_xor_sync(0xffffffffu, m0, 2));
    m1 = fmaxf(m1, __shfl_xor_sync(0xffffffffu, m1, 1));
    m1 = fmaxf(m1, __shfl_xor_sync(0xffffffffu, m1, 2));
    if (m0 == -INFINITY) m0 = 0.f;
    if (m1 == -INFINITY) m1 = 0.f;
    float l0 = 0.f, l1 = 0.f;
    uint32_t pa[4][4];
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
        // the row sum is taken over the fp16-rounded probabilities the second product uses
        const __half2 lo = __floats2half2_rn(win_ex2(s[nt][0] - m0), win_ex2(s[nt][1] - m0));
        const __half2 hi = __floats2half2_rn(win_ex2(s[nt][2] - m1), win_ex2(s[nt][3] - m1));
        const float2 flo = __half22float2(lo), fhi = __half22float2(hi);
        l0 += flo.x + flo.y;
        l1 += fhi.x + fhi.y;
        pa[nt >> 1][(nt & 1) * 2 + 0] = *reinterpret_cast<const uint32_t*>(&lo);
        pa[nt >> 1][(nt & 1) * 2 + 1] = *reinterpret_cast<const uint32_t*>(&hi);
    }
    l0 += __shfl_xor_sync(0xffffffffu, l0, 1);
    l0 += __shfl_xor_sync(0xffffffffu, l0, 2);
    l1 += __shfl_xor_sync(0xffffffffu, l1, 1);
    l1 += __shfl_xor_sync(0xffffffffu, l1, 2);

    // O = P V: 16 queries x 64 dims as eight n-tiles of 8 dims, four k-steps of 16 keys; V's fragments
    // come transposed out of its row-major tile
    float o[8][4];
#pragma unroll
    for (int ne = 0; ne < 8; ++ne) o[ne][0] = o[ne][1] = o[ne][2] = o[ne][3] = 0.f;
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
#pragma unroll
        for (int ne = 0; ne < 8; ne += 2) {
            uint32_t b0, b1, b2, b3;
            const __half* vrow = Vs + (kk * 16 + (lane & 15)) * AW_PITCH + (ne + (lane >> 4)) * 8;
            const uint32_t addr = (uint32_t)__cvta_generic_to_shared(vrow);
            asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                         : "=r"(b0), "=r"(b1), "=r"(b2), "=r"(b3)
                         : "r"(addr));
            mma_16816(o[ne], pa[kk], b0, b1);
            mma_16816(o[ne + 1], pa[kk], b2, b3);
        }
    }
    const float i0 = 1.f / l0, i1 = 1.f / l1;
    const int64_t obase = (int64_t)h * p.osH + (int64_t)b * p.osB;
    if (p.out_f32) {
        float* out = static_cast<float*>(p.out) + obase;
#pragma unroll
        for (int ne = 0; ne < 8; ++ne) {
            const int e = ne * 8 + 2 * t;
            if (e >= p.E) continue;
            if (r0 + g < qrows)
                *reinterpret_cast<float2*>(out + (int64_t)(q0 + r0 + g) * p.osL + e) = make_float2(o[ne][0] * i0, o[ne][1] * i0);
            if (r0 + g + 8 < qrows)
                *reinterpret_cast<float2*>(out + (int64_t)(q0 + r0 + g + 8) * p.osL + e) = make_float2(o[ne][2] * i1, o[ne][3] * i1);
        }
        return;
    }
    // fp16: through the warp's own 16 rows of the Q tile (its fragments are in registers by now), so that
    // a row leaves as whole 16-byte vectors
    __syncwarp();
#pragma unroll
    for (int ne = 0; ne < 8; ++ne) {
        if (ne * 8 >= p.E) continue;   // those columns stay zeros for the next unit, whatever this one's are
        __half* d = Qs + (r0 + g) * AW_PITCH + ne * 8 + 2 * t;
        *reinterpret_cast<uint32_t*>(d) = pack_h2(o[ne][0] * i0, o[ne][1] * i0);
        *reinterpret_cast<uint32_t*>(d + 8 * AW_PITCH) = pack_h2(o[ne][2] * i1, o[ne][3] * i1);
    }
    __syncwarp();
    __half* out = static_cast<__half*>(p.out) + obase;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int idx = lane + i * 32;                  // 128 vectors: 16 rows x 8
        const int row = idx >> 3, vec = idx & 7;
        if (r0 + row < qrows && vec * 8 < p.E)
            *reinterpret_cast<uint4*>(out + (int64_t)(q0 + r0 + row) * p.osL + vec * 8) =
                *reinterpret_cast<const uint4*>(Qs + (r0 + row) * AW_PITCH + vec * 8);
    }
}

constexpr int AW_TILE = 64 * AW_PITCH;                 // halves of one operand's tile
constexpr int AW_BUF_BYTES = 3 * AW_TILE * 2;          // one buffer of Q, K and V
constexpr int AW_CTAS_PER_SM = 4;                      // walking, two buffers
constexpr int AW_CTAS_PER_SM_ONE = 6;                  // a unit per CTA, one buffer
static_assert(AW_BQ == 64 && AW_LK == 64, "tiles of 64 rows");

// WALK: the grid's CTAs walk the units, two buffers each; else a CTA takes the one unit of its index.
template <bool WALK>
__global__ void __launch_bounds__(AW_THREADS, WALK ? AW_CTAS_PER_SM : AW_CTAS_PER_SM_ONE) attention_window_kernel(const WinParams p) {
    extern __shared__ __align__(16) __half win_smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    struct Unit { int h, b, q0, qrows; };
    auto unit = [&](uint32_t u) {
        Unit a;
        const int hb = (int)(u / (uint32_t)p.qtiles);
        a.b = hb / p.H;
        a.h = hb - a.b * p.H;
        a.q0 = (int)(u - (uint32_t)hb * (uint32_t)p.qtiles) * AW_BQ;
        a.qrows = min(AW_BQ, p.Lq - a.q0);
        return a;
    };
    auto fetch = [&](const Unit& a, int buf) {
        __half* tiles = win_smem + buf * 3 * AW_TILE;
        win_fetch(tiles, p.q + (int64_t)a.q0 * p.qsL + (int64_t)a.h * p.qsH + (int64_t)a.b * p.qsB, p.qsL, a.qrows, p.E, tid);
        win_fetch(tiles + AW_TILE, p.k + (int64_t)a.h * p.ksH + (int64_t)a.b * p.ksB, p.ksL, p.Lk, p.E, tid);
        win_fetch(tiles + 2 * AW_TILE, p.v + (int64_t)a.h * p.vsH + (int64_t)a.b * p.vsB, p.vsL, p.Lk, p.E, tid);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // Once: what no unit's copies cover (columns past E, keys past Lk) is read as zeros, and stays so.  Queries past a tile's
    // last give rows that are not stored.
#pragma unroll
    for (int tile = 0; tile < (WALK ? 6 : 3); ++tile)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int row = (tid >> 3) + 16 * i, vec = tid & 7;
            if (vec * 8 >= p.E || (tile % 3 != 0 && row >= p.Lk))
                *reinterpret_cast<uint4*>(win_smem + tile * AW_TILE + row * AW_PITCH + vec * 8) = make_uint4(0u, 0u, 0u, 0u);
        }
    grid_dep_wait();
    grid_dep_launch();
    Unit cur = unit(blockIdx.x);
    fetch(cur, 0);
    if constexpr (!WALK) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        window_unit(p, win_smem, win_smem + AW_TILE, win_smem + 2 * AW_TILE, cur.h, cur.b, cur.q0, cur.qrows, warp, lane, g, t);
        return;
    }
    int buf = 0;
    for (uint32_t u = blockIdx.x; u < p.units; u += gridDim.x, buf ^= 1) {
        Unit next = cur;
        if (u + gridDim.x < p.units) {
            next = unit(u + gridDim.x);
            fetch(next, buf ^ 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();   // every thread's copies of this unit have landed
        __half* Qs = win_smem + buf * 3 * AW_TILE;
        window_unit(p, Qs, Qs + AW_TILE, Qs + 2 * AW_TILE, cur.h, cur.b, cur.q0, cur.qrows, warp, lane, g, t);
        __syncthreads();   // the buffer is free for the unit after the next
        cur = next;
    }
}

int attention_window_launch(b200_ctx* ctx, int64_t E, int64_t Lq, int64_t Lk, int64_t H, int64_t B, const b200_strided4* q,
                            const b200_strided4* k, const b200_strided4* v, const b200_strided4* o, int out_dtype,
                            float scale) {
    WinParams p;
    p.q = static_cast<const __half*>(q->ptr);
    p.k = static_cast<const __half*>(k->ptr);
    p.v = static_cast<const __half*>(v->ptr);
    p.out = const_cast<void*>(o->ptr);
    p.qsL = q->stride[1]; p.qsH = q->stride[2]; p.qsB = q->stride[3];
    p.ksL = k->stride[1]; p.ksH = k->stride[2]; p.ksB = k->stride[3];
    p.vsL = v->stride[1]; p.vsH = v->stride[2]; p.vsB = v->stride[3];
    p.osL = o->stride[1]; p.osH = o->stride[2]; p.osB = o->stride[3];
    p.E = (int)E; p.Lq = (int)Lq; p.Lk = (int)Lk; p.H = (int)H; p.B = (int)B;
    p.qtiles = (int)cdiv(Lq, AW_BQ);
    p.out_f32 = out_dtype == B200_F32;
    p.scale_log2 = scale * 1.4426950408889634f;
    const int64_t units = (int64_t)p.qtiles * H * B, sms = ctx->prop.multiProcessorCount;
    B200_REQUIRE(units < (1ll << 31), B200_DECLINE_EXTENT, "attention: too many windows");
    p.units = (uint32_t)units;
    // A walking CTA of a single unit only pays for its second buffer, one of two or three takes longer than six CTAs side by side
    // with others behind them, and of few keys there is little to fetch ahead.  Between three and four units an SM both take the
    // same alone, and back to back walking CTAs, which leave no room for the next launch's, spread evenly.  Microseconds on 148
    // SMs, a unit a CTA / walking, each launch behind another kernel: 300 units of 64 x 64 x 56 6.2 / 6.2 (6.7 with every buffer
    // zeroed whole), 592 7.1 / 7.2 (back to back 7.0 / 5.8), 800 8.6 / 9.0, 888 8.7 / 9.8, 1600 in the L2 13.1 / 14.5, 2048
    // 16.1 / 17.3; of 49 x 49 x 64 2048 in the L2 14.0 / 14.7, 4096 27.5 / 26.5; of 36 x 36 x 48 2400 from memory 15.3 / 14.7; of
    // 16 x 16 x 56 300 4.5 / 4.6, 1800 8.2 / 9.4, 16000 51.1 / 51.2.
    if (Lk <= 32 || (units <= 14 * sms && (units <= 3 * sms || units > AW_CTAS_PER_SM * sms))) {
        B200_CUDA(launch_dep(attention_window_kernel<false>, dim3((unsigned)units, 1, 1), dim3(AW_THREADS, 1, 1), AW_BUF_BYTES, ctx->stream, 1, p));
        ctx->launches++;
        return B200_OK;
    }
    static bool attr_done[16] = {};
    if (!attr_done[ctx->device & 15]) {
        B200_CUDA(cudaFuncSetAttribute(attention_window_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 2 * AW_BUF_BYTES));
        attr_done[ctx->device & 15] = true;
    }
    const int64_t room = AW_CTAS_PER_SM * sms;
    B200_CUDA(launch_dep(attention_window_kernel<true>, dim3((unsigned)(units < room ? units : room), 1, 1), dim3(AW_THREADS, 1, 1),
                         2 * AW_BUF_BYTES, ctx->stream, 1, p));
    ctx->launches++;
    return B200_OK;
}

} // namespace b200
