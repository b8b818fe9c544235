// fp16 GEMM for operands a tensor map cannot express (leading dimensions that are not a multiple of 8 elements,
// pointers off a 16-byte boundary): out(M,N) = epi(T(bias + A(M,K) B(K,N))), fp32 accumulation, any alignment of A,
// B and out.  It is there for a decoder's vocabulary projection: A of 51865 x 1280 (132.8 MB, every column at its own
// misalignment) times a handful of tokens, where reading A once is all that should be paid.
//
// What bounds it: reading A, then the loads' latency (the accumulators leave room for fewer blocks per SM).  Measured
// against the one-thread-per-output kernel that ran these before (whole calls, B200): 17 x 1337 x 712 61 -> 8.6 us; 5 x 17579 x 4096
// takes 31.4 (4.6 TB/s of A).
//
// Columns k and k + 8 of A are 8 * lda * 2 bytes apart, a multiple of 16, so all columns k = w (mod 8) sit at the same
// offset s_w from a 16-byte boundary.  Warp w of a CTA takes exactly those columns and keeps its accumulators aligned
// to memory rather than to rows, as gemv_kernel does: the 16-byte vector at position j of a column holds rows
// 8 j - s_w ... 8 j - s_w + 7, and only the sum over the eight warps, through shared memory, shifts by s_w.  The order
// of a reduction axis and the names of a tile's rows are free, so the vectors become tensor-core fragments (m16n8k16,
// warp-level) with two byte permutes per register and
// no trip through shared memory: lane (g, t) holds four columns' vectors of rows 8 g ... 8 g + 7, and word p of them
// gives rows 2 p and 2 p + 1 of the group as the fragment's rows g and g + 8.
//
// Where A is long the product goes to gemm_rows_tc.cu, which finds tiles for tcgen05 in the same classes of columns.
//
// When row blocks alone do not fill the GPU the K axis is split over the CTAs of a cluster and the partial sums meet
// through distributed shared memory, added in rank order: no workspace, and the result does not depend on timing.
#include <cuda_fp16.h>

#include "act.cuh"
#include "gemm_rows.cuh"
#include "internal.h"
#include "ptx.cuh"

namespace b200 {

constexpr int GR_WARPS = 8;
constexpr int GR_STEP = 16 * GR_WARPS;   // columns of A one step of a CTA's warps covers

// NT: token tiles of 8.  MB: strips of 64 rows per warp.  CHUNK: steps of B staged in shared memory at a time.
template <int NT> struct GrCfg {
    static constexpr int MB = NT == 1 ? 2 : 1;
    static constexpr int CHUNK = NT <= 2 ? 11 : (NT == 4 ? 7 : 5);   // odd: rows of the staged B lie 4 (mod 8) 8-byte units apart
    static constexpr int ROWS = 64 * MB - 8;                          // rows a block owns: covered whatever the shift
    static constexpr int JP = 16 * CHUNK;                             // halves per staged (warp, token) row
    static constexpr int X_BYTES = GR_WARPS * NT * 8 * JP * 2;
    static constexpr int RP = 64 * MB + 1;                            // floats per row of a warp's partial tile: odd
    static constexpr int RED_BYTES = GR_WARPS * 8 * RP * 4;           // eight tokens at a time
    static constexpr int SUM_BYTES = NT * 8 * ROWS * 4;               // this CTA's sums, for the cluster
    static constexpr int SMEM_BYTES = (X_BYTES > RED_BYTES ? X_BYTES : RED_BYTES) + SUM_BYTES;
    static constexpr int MIN_BLOCKS = NT <= 4 ? 2 : 1;
};

// Out of line, and not called for nothing, in the two-tile form: inlined, its registers change the main loop's (115 for 96), 9 x
// 45001 x 2000, which gemm_rows_tc.cu takes now, 61.1 -> 62.8 us.  The other forms lose by it (4 x 20001 x 1280 18.8 -> 19.5).
__device__ __noinline__ float gr_act(int epi, float v) { return apply_act(epi, v); }

// grid (K parts, row blocks, token blocks), the K parts of a row block forming a cluster; 256 threads.  TWO: one of two
// launches that share the row blocks.
template <int NT, typename OutT, bool TWO>
__global__ void __launch_bounds__(32 * GR_WARPS, GrCfg<NT>::MIN_BLOCKS)
gemm_rows_kernel(const GrParams p) {
    using Cfg = GrCfg<NT>;
    constexpr int MB = Cfg::MB;
    extern __shared__ __align__(16) uint8_t gr_smem[];
    __half* xs = reinterpret_cast<__half*>(gr_smem);                       // [warp][token][j]: B(k = 8 j + warp, token)
    float* red = reinterpret_cast<float*>(gr_smem);                        // [warp][8 tokens][RP], after the main loop
    float* sums = reinterpret_cast<float*>(gr_smem + Cfg::SMEM_BYTES - Cfg::SUM_BYTES);   // [token][ROWS]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int64_t block = TWO ? p.block0 + blockIdx.y : blockIdx.y;
    // The tail, which reads what the first part reads, starts as the first part's blocks leave.  What follows the tail on the
    // stream and is launched to start early waits for it to end, hence for both.
    if constexpr (TWO) grid_dep_launch();
    const int64_t n0 = (int64_t)blockIdx.z * (NT * 8);
    const int ntok = (int)(p.N - n0 < NT * 8 ? p.N - n0 : NT * 8);
    const int64_t step0 = (int64_t)blockIdx.x * p.steps_per_cta;
    const int64_t nsteps_all = (p.K + GR_STEP - 1) / GR_STEP;
    const int nsteps = (int)(nsteps_all - step0 < p.steps_per_cta ? (nsteps_all > step0 ? nsteps_all - step0 : 0) : p.steps_per_cta);

    float acc[MB][4][NT][4];
#pragma unroll
    for (int mi = 0; mi < MB; ++mi)
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int v = 0; v < 4; ++v) acc[mi][q][nt][v] = 0.f;

    // Column k of this warp (k = warp mod 8): offset s from a 16-byte boundary, the same for all of them.
    const char* col0 = reinterpret_cast<const char*>(p.A + (int64_t)warp * p.lda);
    const int s = (int)(reinterpret_cast<uintptr_t>(col0) & 15u) >> 1;
    const int64_t cstep = 8 * p.lda * 2;                                   // bytes from one of the warp's columns to its next
    const int64_t jv = block * (Cfg::ROWS / 8);              // the block's first vector
    bool live[MB];
#pragma unroll
    for (int mi = 0; mi < MB; ++mi) live[mi] = 8 * (jv + 8 * mi + g) - s < p.M;   // the vector holds a row of A
    const char* vec0 = col0 - 2 * s + (jv + g) * 16;

    // the four columns lane t takes of a step: j = 16 step + 4 t + c
    auto fetch = [&](uint4 (&a)[MB][4], int64_t step) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int64_t j = 16 * step + 4 * t + c;
            const bool in = 8 * j + warp < p.K;
            const char* v = vec0 + j * cstep;
#pragma unroll
            for (int mi = 0; mi < MB; ++mi)
                a[mi][c] = in && live[mi] ? __ldg(reinterpret_cast<const uint4*>(v + mi * 128)) : make_uint4(0u, 0u, 0u, 0u);
        }
    };

    uint4 cur[MB][4], nxt[MB][4];
    if (nsteps > 0) fetch(cur, step0);
    for (int c0 = 0; c0 < nsteps; c0 += Cfg::CHUNK) {
        const int cn = nsteps - c0 < Cfg::CHUNK ? nsteps - c0 : Cfg::CHUNK;
        const int64_t kb = (step0 + c0) * GR_STEP;
        if (c0 > 0) __syncthreads();   // the previous chunk has been read
        // B(k, token), two groups of eight k per thread: element w of the groups goes to warp w's rows as one word.
        const int pairs = cn * 8;      // pairs of groups of eight columns in the chunk
        for (int i = tid; i < NT * 8 * pairs; i += 32 * GR_WARPS) {
            const int tok = i / pairs, pr = i - tok * pairs;
            const int64_t k = kb + 16 * (int64_t)pr;
            __align__(16) __half e[16];
            const __half* src = p.B + (n0 + tok) * p.ldb + k;
            if (tok < ntok && p.b_vec && k + 16 <= p.K) {
                *reinterpret_cast<uint4*>(e) = __ldg(reinterpret_cast<const uint4*>(src));
                *reinterpret_cast<uint4*>(e + 8) = __ldg(reinterpret_cast<const uint4*>(src) + 1);
            } else {
#pragma unroll
                for (int u = 0; u < 16; ++u) e[u] = tok < ntok && k + u < p.K ? src[u] : __ushort_as_half(0);
            }
#pragma unroll
            for (int w = 0; w < GR_WARPS; ++w)
                *reinterpret_cast<__half2*>(xs + (w * (NT * 8) + tok) * Cfg::JP + 2 * pr) = __halves2half2(e[w], e[w + 8]);
        }
        __syncthreads();
        const __half* xw = xs + (warp * (NT * 8) + g) * Cfg::JP + 4 * t;
        for (int st = 0; st < cn; ++st) {
            const int64_t step = step0 + c0 + st;
            if (c0 + st + 1 < nsteps) fetch(nxt, step + 1);
#pragma unroll
            for (int nt0 = 0; nt0 < NT; nt0 += 4) {
                uint2 b[NT < 4 ? NT : 4];
#pragma unroll
                for (int u = 0; u < (NT < 4 ? NT : 4); ++u)
                    b[u] = *reinterpret_cast<const uint2*>(xw + (nt0 + u) * 8 * Cfg::JP + 16 * st);
#pragma unroll
                for (int mi = 0; mi < MB; ++mi) {
                    const uint32_t* w0 = reinterpret_cast<const uint32_t*>(&cur[mi][0]);
                    const uint32_t* w1 = reinterpret_cast<const uint32_t*>(&cur[mi][1]);
                    const uint32_t* w2 = reinterpret_cast<const uint32_t*>(&cur[mi][2]);
                    const uint32_t* w3 = reinterpret_cast<const uint32_t*>(&cur[mi][3]);
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const uint32_t a0 = __byte_perm(w0[q], w1[q], 0x5410), a1 = __byte_perm(w0[q], w1[q], 0x7632);
                        const uint32_t a2 = __byte_perm(w2[q], w3[q], 0x5410), a3 = __byte_perm(w2[q], w3[q], 0x7632);
#pragma unroll
                        for (int u = 0; u < (NT < 4 ? NT : 4); ++u) mma_16816(acc[mi][q][nt0 + u], a0, a1, a2, a3, b[u].x, b[u].y);
                    }
                }
            }
#pragma unroll
            for (int mi = 0; mi < MB; ++mi)
#pragma unroll
                for (int c = 0; c < 4; ++c) cur[mi][c] = nxt[mi][c];
        }
    }

    // Sum over the warps, eight tokens at a time: row r of the block is accumulator row r + s of warp `warp`.
    const uint32_t nparts = cluster_nctarank();
    const int64_t m0 = block * Cfg::ROWS;
    auto store = [&](int tok, int r, float v) {
        const int64_t m = m0 + r, n = n0 + tok;
        if (p.bias != nullptr) v += __half2float(p.bias[p.bias_per_n ? n : m]);
        OutT* o = static_cast<OutT*>(p.out) + n * p.ldo + m;
        auto act = [&](float u) { return NT != 2 ? apply_act(p.epi, u) : p.epi == B200_EPI_NONE ? u : gr_act(p.epi, u); };
        if constexpr (sizeof(OutT) == 2) *o = __float2half_rn(act(__half2float(__float2half_rn(v))));
        else *o = act(v);
    };
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
        if (nt * 8 >= ntok) break;
        __syncthreads();
#pragma unroll
        for (int mi = 0; mi < MB; ++mi)
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    const int r = 64 * mi + 8 * g + 2 * q + (v >> 1) - s;
                    if (r >= 0 && r < Cfg::ROWS) red[(warp * 8 + 2 * t + (v & 1)) * Cfg::RP + r] = acc[mi][q][nt][v];
                }
        __syncthreads();
        for (int i = tid; i < 8 * Cfg::ROWS; i += 32 * GR_WARPS) {
            const int tk = i / Cfg::ROWS, r = i - tk * Cfg::ROWS;
            float v = 0.f;
#pragma unroll
            for (int w = 0; w < GR_WARPS; ++w) v += red[(w * 8 + tk) * Cfg::RP + r];
            if (nparts > 1) sums[(nt * 8 + tk) * Cfg::ROWS + r] = v;
            else if (nt * 8 + tk < ntok && m0 + r < p.M) store(nt * 8 + tk, r, v);
        }
    }
    if (nparts == 1) return;
    if (TWO && p.tail) grid_dep_wait();   // what follows on the stream runs after the first part as well
    cluster_sync_all();   // every part's sums are in its shared memory
    const uint32_t rank = cluster_ctarank();
    const uint32_t mine = smem_u32(sums);
    for (int i = tid + (int)rank * 32 * GR_WARPS; i < ntok * Cfg::ROWS; i += (int)nparts * 32 * GR_WARPS) {
        const int tok = i / Cfg::ROWS, r = i - tok * Cfg::ROWS;
        if (m0 + r >= p.M) continue;
        float a[8], v = 0.f;   // every part's load in flight together: a remote load takes a few hundred nanoseconds
#pragma unroll
        for (uint32_t q = 0; q < 8; ++q) a[q] = q < nparts ? ld_cluster_f32(mapa_u32(mine + i * 4, q)) : 0.f;
#pragma unroll
        for (uint32_t q = 0; q < 8; ++q) v += a[q];
        store(tok, r, v);
    }
    cluster_sync_all();   // nobody leaves while its sums may still be read
}

template <int NT, typename OutT>
static int gr_launch(b200_ctx* ctx, GrParams p) {
    using Cfg = GrCfg<NT>;
    static bool attr_done[16] = {};
    if (!attr_done[ctx->device & 15]) {
        B200_CUDA(cudaFuncSetAttribute(gemm_rows_kernel<NT, OutT, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES));
        B200_CUDA(cudaFuncSetAttribute(gemm_rows_kernel<NT, OutT, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES));
        attr_done[ctx->device & 15] = true;
    }
    const int64_t blocks = cdiv(p.M, Cfg::ROWS), tblocks = cdiv(p.N, NT * 8), steps = cdiv(p.K, GR_STEP);
    B200_REQUIRE(blocks < 65536 && tblocks < 65536, B200_DECLINE_EXTENT, "gemm: unaligned operands with M = %lld, N = %lld",
                 (long long)p.M, (long long)p.N);
    // K parts: until the resident blocks are used, each part keeping two steps or more
    const int64_t room = (int64_t)ctx->prop.multiProcessorCount * Cfg::MIN_BLOCKS;
    int64_t parts = 1;
    while (parts < 8 && 2 * parts * blocks * tblocks <= room && steps >= 4 * parts) parts *= 2;
    // Row blocks past the last full round of the resident ones, less than half a round of them, are a launch of their own,
    // split along K like few row blocks are: 433 blocks of 296 take a round and a half instead of two.  (A second launch may
    // start as the first one's blocks leave: see the kernel.)  17 x 20001 x 1024 31.5 -> 26.7 us.
    int64_t tail = 0, tail_parts = 1;
    if (parts == 1 && tblocks == 1 && blocks > room) {
        tail = blocks % room;
        while (tail_parts < 8 && 2 * tail_parts * tail <= room && steps >= 4 * tail_parts) tail_parts *= 2;
        if (tail_parts == 1) tail = 0;
    }
    auto kern = tail ? gemm_rows_kernel<NT, OutT, true> : gemm_rows_kernel<NT, OutT, false>;
    auto go = [&](int64_t first, int64_t n, int64_t k_parts, bool second) -> cudaError_t {
        p.block0 = first;
        p.tail = second;
        p.steps_per_cta = (int)cdiv(steps, k_parts);
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)k_parts, (unsigned)n, (unsigned)tblocks);
        cfg.blockDim = dim3(32 * GR_WARPS, 1, 1);
        cfg.dynamicSmemBytes = Cfg::SMEM_BYTES;
        cfg.stream = ctx->stream;
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)k_parts;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = second && pdl_enabled() ? 2 : 1;
        ctx->launches++;
        return cudaLaunchKernelEx(&cfg, kern, p);
    };
    if (blocks > tail) B200_CUDA(go(0, blocks - tail, parts, false));
    if (tail) B200_CUDA(go(blocks - tail, tail, tail_parts, true));
    return B200_OK;
}

// The rule: below about 32 k elements of A a launch takes the same few microseconds either way, and the scalar kernel's
// one thread per output is the reference's own arithmetic bit for bit.
bool gemm_rows_takes(int64_t M, int64_t N, int64_t K, int64_t nbatch) {
    return nbatch == 1 && N >= 2 && M >= 64 && M * K >= 32768 && M < (1ll << 21) && N < 65536 && K < (1ll << 31);
}

int gemm_rows_launch(b200_ctx* ctx, int64_t M, int64_t N, int64_t K, const void* A, int64_t lda, const void* B, int64_t ldb,
                     const void* bias, int bias_per_n, void* out, int64_t ldo, int out_dtype, int epilogue) {
    GrParams p;
    p.A = static_cast<const __half*>(A);
    p.B = static_cast<const __half*>(B);
    p.bias = static_cast<const __half*>(bias);
    p.out = out;
    p.lda = lda; p.ldb = ldb; p.ldo = ldo;
    p.M = M; p.N = N; p.K = K;
    p.bias_per_n = bias_per_n;
    p.epi = epilogue;
    p.b_vec = ldb % 8 == 0 && (reinterpret_cast<uintptr_t>(B) & 15u) == 0;
    p.steps_per_cta = 0;
    const bool h = out_dtype == B200_F16;
    if (const int nt = gemm_rows_tc_tokens(ctx, M, N, K)) return gemm_rows_tc_launch(ctx, p, nt, h);
    if (N <= 8) return h ? gr_launch<1, __half>(ctx, p) : gr_launch<1, float>(ctx, p);
    if (N <= 16) return h ? gr_launch<2, __half>(ctx, p) : gr_launch<2, float>(ctx, p);
    if (N <= 32) return h ? gr_launch<4, __half>(ctx, p) : gr_launch<4, float>(ctx, p);
    return h ? gr_launch<8, __half>(ctx, p) : gr_launch<8, float>(ctx, p);
}

} // namespace b200
