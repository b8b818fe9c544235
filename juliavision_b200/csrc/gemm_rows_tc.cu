// The product of gemm_rows.cu on tcgen05, where A is long.  The columns k = w (mod 8) of A, taken from the 16-byte boundary below the first of
// them, are a matrix whose columns are whole multiples of 16 bytes apart: a tensor map can express it, and TMA brings its tiles as
// they are, rows s_w ... of the matrix for rows 0 ... of A.  So a tile of 128 such rows is multiplied class by class, each class into
// its own columns of tensor memory, and the sum over the eight classes, through shared memory, shifts class w's rows by s_w.
// A CTA turns B into the classes once and walks row blocks, A's ring running on from one block into the next; a class's columns are
// given back as soon as they have been read, and the sum of one class hides behind the copies of the next ones.
// The row blocks are cut equal, so that every CTA has the same number of them.  A class has two accumulators, a half of its columns
// each, and classes are added in pairs: against 64 bits the error is 0.55 to 0.7 of gemm_rows.cu's and of this form's with one
// (1.40e-7 of the norm for 2.08e-7 and 2.32e-7, 5 x 51865 x 1280), at the same speed.
//
// What bounds it: the copies.  A row of 128 bytes that starts off a 128-byte line takes two requests, and a copy costs about 0.1 us of
// the copy engine however few rows it has: the fewer and larger the stages the better (5 x 71039 x 1280, ring of 96 KB: stages of 16
// columns 80, of 32 46.4, of 64 36.1, of 80 37.5, of 112 36.1 us), down to three of them (two: 50.6).  51865 x 1280: 26.7 us for 5
// tokens (5.0 TB/s of A), 33.4 for 48, 46.0 for 64, where B leaves a ring of three stages; by gemm_rows.cu 32.4, 129, 139.
#include "act.cuh"
#include "gemm_rows.cuh"
#include "internal.h"
#include "ptx.cuh"

namespace b200 {

__device__ __noinline__ float gt_act(int epi, float v) { return apply_act(epi, v); }   // out of line: the loop over tokens is unrolled

struct GrMaps { CUtensorMap m[8]; };   // class w: {M + s_w, its columns}, boxes of 64 x j

constexpr int GT_ROWS = 128, GT_COL_BYTES = GT_ROWS * 2, GT_RING = 112 * 1024, GT_MAX_STAGES = GT_RING / (16 * GT_COL_BYTES);
template <int NT> struct GtCfg {
    static constexpr int GROUPS = NT == 48 ? 3 : NT > 16 ? 2 : 1, THREADS = 128 + 128 * GROUPS;   // groups of four warps that sum, each its share of the tokens
    static constexpr int SHARE = NT / GROUPS, CW = 16;               // tokens of a group, and those that cross shared memory at a time
    static constexpr int RED_BYTES = GROUPS * CW * GT_ROWS * 4;      // and their room: twice for one barrier an exchange instead of two
    static_assert(2 * RED_BYTES >= 8 * 2048 && (GROUPS == 1 || RED_BYTES >= 8 * 2048), "the warps' rooms for turning B");
    static constexpr int B_BLOCK_BYTES = NT * 32;                    // sixteen j of a class of B: a row of 32 bytes a token, 32-byte swizzle
    static constexpr int SLOTS = NT <= 32 ? 8 : 512 / (2 * NT), TMEM = NT <= 16 ? 256 : 512;   // of tensor memory: two accumulators of a class
    static constexpr int TAIL_BYTES = (2 * GT_MAX_STAGES + 16) * 8 + 16;
    static int64_t fixed(int64_t K, int rooms) { return cdiv(K, 128) * 8 * B_BLOCK_BYTES + rooms * RED_BYTES + TAIL_BYTES; }
    static int64_t ring(int64_t K, int rooms) { return 232448 - fixed(K, rooms); }
    static int rooms(int64_t K) { return GROUPS == 1 || ring(K, 2) >= 8 * 8192 ? 2 : 1; }
    static bool fits(int64_t K) { return ring(K, rooms(K)) >= 4 * 8192; }
};
struct GtParams {
    GrParams g;
    int* d_status;
    int rows, j, steps, stages, rooms;   // rows a block owns (a multiple of 8); columns of a class a stage holds, sixteens of them in all; ring; RED_BYTES
};

template <int NT, typename OutT>
__global__ void __launch_bounds__(GtCfg<NT>::THREADS, 1) gemm_rows_tc_kernel(const __grid_constant__ GrMaps maps, const GtParams p) {
    using Cfg = GtCfg<NT>;
    extern __shared__ __align__(1024) uint8_t gr_smem[];
    if ((smem_u32(gr_smem) & 1023u) != 0) {
        if (threadIdx.x == 0) atomicCAS(p.d_status, 0, KST_SMEM_LAYOUT);
        return;
    }
    uint8_t* sb = gr_smem + p.stages * p.j * GT_COL_BYTES;                                   // [class][chunk] blocks of B
    float* red = reinterpret_cast<float*>(sb + 8 * p.steps * Cfg::B_BLOCK_BYTES);       // [buffer][token][row]
    uint64_t* full = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(red) + p.rooms * Cfg::RED_BYTES);
    uint64_t* empty = full + p.stages;
    uint64_t* tfull = empty + p.stages;
    uint64_t* tempty = tfull + 8;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 8);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const GrParams& g = p.g;
    const int nblocks = (int)((g.M + p.rows - 1) / p.rows);
    const int64_t n0 = (int64_t)blockIdx.y * NT;
    const int ntok = (int)(g.N - n0 < NT ? g.N - n0 : NT);

    if (tid == 0) {
        for (int s = 0; s < p.stages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int w = 0; w < Cfg::SLOTS; ++w) {
            mbar_init(&tfull[w], 1);
            mbar_init(&tempty[w], 4 * Cfg::GROUPS);
        }
        *abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, Cfg::TMEM);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    grid_dep_wait();
    grid_dep_launch();

    const bool both = p.rows > 56;   // whether a block's rows, wherever they start, reach past the first 64
    const int half = p.j * (GT_COL_BYTES / 2);
    int block = blockIdx.x, cls = 0, y = 0, stage = 0, phase = 0;   // the producer's place
    uint8_t* place = gr_smem;
    auto load = [&]() {
        mbar_arrive_expect_tx(&full[stage], both ? 2 * half : half);
        tma_load_2d(place, &maps.m[cls], &full[stage], block * p.rows, y);
        if (both) tma_load_2d(place + half, &maps.m[cls], &full[stage], block * p.rows + 64, y);
        place += 2 * half;
        if (++stage == p.stages) {
            stage = 0;
            phase ^= 1;
            place = gr_smem;
        }
        y += p.j;
        if (y >= 16 * p.steps) {
            y = 0;
            if (++cls == 8) {
                cls = 0;
                block += gridDim.x;
            }
        }
    };
    if (warp == 0 && lane == 0)
        for (int s = 0; s < p.stages && block < nblocks; ++s) load();
    // B(8 j + w, token): 64 k of a token are eight j of every class.  A warp reads sixteen such items whole, through shared memory
    // (rows of 128 bytes, 16-byte pieces permuted), and a lane then takes four classes of one.
    {
        const int sets = NT / 16 * 2 * p.steps, c = lane & 15, hi = lane >> 4;
        uint8_t* raw = reinterpret_cast<uint8_t*>(red) + warp * 2048;
        auto read = [&](uint4 (&e)[4], int set) {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int tok = set % (NT / 16) * 16 + 4 * u + (lane >> 3);
                const int64_t k = 64 * (int64_t)(set / (NT / 16)) + 8 * (lane & 7);
                const __half* src = g.B + (n0 + tok) * g.ldb + k;
                if (set < sets && tok < ntok && g.b_vec && k + 8 <= g.K) e[u] = __ldg(reinterpret_cast<const uint4*>(src));
                else {
                    __align__(16) __half h[8];
#pragma unroll
                    for (int v = 0; v < 8; ++v) h[v] = set < sets && tok < ntok && k + v < g.K ? src[v] : __ushort_as_half(0);
                    e[u] = *reinterpret_cast<const uint4*>(h);
                }
            }
        };
        uint4 e[4], f[4];
        if (warp < 8) read(e, warp);
        for (int set = warp; warp < 8 && set < sets; set += 8) {
            read(f, set + 8);
            __syncwarp();
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int item = 4 * u + (lane >> 3);
                *reinterpret_cast<uint4*>(raw + item * 128 + (((lane & 7) ^ (item & 7)) << 4)) = e[u];
                e[u] = f[u];
            }
            __syncwarp();
            const int tok = set % (NT / 16) * 16 + c, jg = set / (NT / 16);
            uint2 d[8];   // four classes of the item's group u
#pragma unroll
            for (int u = 0; u < 8; ++u) d[u] = *reinterpret_cast<const uint2*>(raw + c * 128 + ((u ^ (c & 7)) << 4) + hi * 8);
            uint8_t* dst = sb + (jg >> 1) * Cfg::B_BLOCK_BYTES + tok * 32 + (((jg ^ (tok >> 2)) & 1) << 4);
#pragma unroll
            for (int w = 0; w < 4; ++w) {
                uint32_t o[4];
#pragma unroll
                for (int v = 0; v < 4; ++v)
                    o[v] = __byte_perm(w < 2 ? d[2 * v].x : d[2 * v].y, w < 2 ? d[2 * v + 1].x : d[2 * v + 1].y, w & 1 ? 0x7632 : 0x5410);
                *reinterpret_cast<uint4*>(dst + (4 * hi + w) * p.steps * Cfg::B_BLOCK_BYTES) = make_uint4(o[0], o[1], o[2], o[3]);
            }
        }
    }
    fence_proxy_async_smem();
    __syncthreads();

    if (warp == 0) {
        if (lane == 0)
            while (block < nblocks) {
                if (!mbar_wait_spin(&empty[stage], (uint32_t)phase ^ 1, p.d_status, KST_WAIT_EMPTY, abort_flag)) break;
                load();
            }
    } else if (warp == 1) {
        constexpr uint32_t idesc = make_idesc_f16(GT_ROWS, NT, /*a MN-major*/ 1, /*b K-major*/ 0);
        // one thread's chain of instructions a stage is what sets the pace of small stages: addresses only advance
        const uint64_t adesc = smem_desc_at(make_smem_desc(half, 1024), smem_u32(gr_smem));
        const uint64_t bdesc = smem_desc_at((uint64_t(1) << 16) | (uint64_t(256 >> 4) << 32) | (uint64_t(1) << 46) | (uint64_t(6) << 61), smem_u32(sb));
        const uint32_t a_hi = (uint32_t)(adesc >> 32), b_hi = (uint32_t)(bdesc >> 32), a_first = (uint32_t)adesc;
        auto desc = [](uint32_t hi, uint32_t lo) { return uint64_t(hi) << 32 | lo; };
        uint32_t a_lo = a_first;
        const int first = (p.steps + 1) / 2;   // steps into the first of a class's two accumulators
        bool ok = true;
        uint32_t round = 0;
        int slot = 0;
        for (int b = blockIdx.x; ok && b < nblocks; b += gridDim.x) {
            uint32_t b_lo = (uint32_t)bdesc;
            for (int w = 0; ok && w < 8; ++w) {
                ok = __all_sync(0xffffffffu, mbar_wait_spin(&tempty[slot], round ^ 1, p.d_status, KST_WAIT_TMEM_EMPTY, abort_flag));
                const uint32_t d = tmem_base + slot * (2 * NT);
                for (int i = 0; ok && i < p.steps; i += p.j / 16) {
                    const int kn = min(p.j / 16, p.steps - i);
                    ok = __all_sync(0xffffffffu, mbar_wait_spin(&full[stage], (uint32_t)phase, p.d_status, KST_WAIT_FULL, abort_flag));
                    if (!ok) break;
                    tc_fence_after();
                    if (elect_one()) {
#pragma unroll 2
                        for (int k = 0; k < kn; ++k)
                            umma_ss(i + k < first ? d : d + NT, desc(a_hi, a_lo + k * (2048 >> 4)), desc(b_hi, b_lo + k * (Cfg::B_BLOCK_BYTES >> 4)), idesc,
                                    i + k != 0 && i + k != first);
                        umma_commit(&empty[stage]);
                        if (i + kn == p.steps) umma_commit(&tfull[slot]);
                    }
                    __syncwarp();
                    b_lo += kn * (Cfg::B_BLOCK_BYTES >> 4);
                    a_lo += half >> 3;
                    if (++stage == p.stages) {
                        stage = 0;
                        phase ^= 1;
                        a_lo = a_first;
                    }
                }
                if (++slot == Cfg::SLOTS) {
                    slot = 0;
                    round ^= 1;
                }
            }
        }
    } else if (warp >= 4) {
        const int quad = warp & 3, row = quad * 32 + lane, part = (warp >> 2) - 1, t0 = part * Cfg::SHARE;
        const uint32_t tacc = tmem_base + (uint32_t(quad * 32) << 16) + t0;
        float* const mine = red + part * (Cfg::CW * GT_ROWS);
        const int ng = ntok - t0;   // tokens from the group's first on
        bool ok = true;
        uint32_t round = 0, buf = 0;
        int slot = 0;
        for (int b = blockIdx.x; ok && b < nblocks; b += gridDim.x) {
            float acc[Cfg::SHARE], even[Cfg::SHARE];
#pragma unroll
            for (int n = 0; n < Cfg::SHARE; ++n) acc[n] = 0.f;
#pragma unroll 2
            for (int w = 0; w < 8; ++w) {
                ok = mbar_wait(&tfull[slot], round, p.d_status, KST_WAIT_TMEM_FULL, abort_flag);
                if (named_bar_or(4 + part, 128, !ok)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const int s = (int)(reinterpret_cast<uintptr_t>(g.A + (int64_t)w * g.lda) & 15u) >> 1;
                const int from = row + s < GT_ROWS ? row + s : GT_ROWS - 1;   // past the last: a row no block owns
#pragma unroll
                for (int h = 0; h < Cfg::SHARE; h += Cfg::CW) {
                    float* rb = mine + buf * (Cfg::RED_BYTES / 4);
                    if (p.rooms == 2) buf ^= 1;
                    else named_bar_sync(7 + part, 128);   // what was there has been read
                    uint32_t r[16], r2[16];
                    tmem_ld16(tacc + slot * (2 * NT) + h, r);
                    tmem_ld16(tacc + slot * (2 * NT) + (p.steps > 1 ? NT : 0) + h, r2);
                    tmem_wait_ld();
                    if (h + Cfg::CW >= Cfg::SHARE) {
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&tempty[slot]);
                    }
#pragma unroll
                    for (int n = 0; n < Cfg::CW; ++n)
                        if (h + n < ng) rb[n * GT_ROWS + row] = __uint_as_float(r[n]) + (p.steps > 1 ? __uint_as_float(r2[n]) : 0.f);
                    named_bar_sync(1 + part, 128);
#pragma unroll
                    for (int n = 0; n < Cfg::CW; ++n)
                        if (h + n < ng) {
                            const float v = rb[n * GT_ROWS + from];
                            if (w & 1) acc[h + n] += even[h + n] + v;
                            else even[h + n] = v;
                        }
                }
                if (++slot == Cfg::SLOTS) {
                    slot = 0;
                    round ^= 1;
                }
            }
            const int64_t m = (int64_t)b * p.rows + row;
            if (ok && row < p.rows && m < g.M) {
                const float bm = g.bias != nullptr && !g.bias_per_n ? __half2float(g.bias[m]) : 0.f;
                OutT* o = static_cast<OutT*>(g.out) + (n0 + t0) * g.ldo + m;
#pragma unroll
                for (int n = 0; n < Cfg::SHARE; ++n) {
                    if (n >= ng) break;
                    const float v = acc[n] + (g.bias != nullptr && g.bias_per_n ? __half2float(g.bias[n0 + t0 + n]) : bm);
                    if constexpr (sizeof(OutT) == 2) {
                        const __half r = __float2half_rn(v);
                        o[n * g.ldo] = g.epi == B200_EPI_NONE ? r : __float2half_rn(gt_act(g.epi, __half2float(r)));
                    } else o[n * g.ldo] = g.epi == B200_EPI_NONE ? v : gt_act(g.epi, v);
                }
            }
        }
    }
    if (*abort_flag) {   // let any TMA copy still in flight into this CTA's shared memory land before exit
        for (int i = 0; i < 4; ++i) __nanosleep(1000000);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, Cfg::TMEM);
    }
}

template <int NT, typename OutT>
static int gt_launch(b200_ctx* ctx, const GrParams& g) {
    using Cfg = GtCfg<NT>;
    auto kern = gemm_rows_tc_kernel<NT, OutT>;
    static bool attr_done[16] = {};
    if (!attr_done[ctx->device & 15]) {
        B200_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448));
        attr_done[ctx->device & 15] = true;
    }
    const int64_t sms = ctx->prop.multiProcessorCount;
    const int64_t turns = cdiv(cdiv(g.M, GT_ROWS - 8), sms);
    GtParams p;
    p.g = g;
    p.d_status = ctx->d_status;
    p.rows = (int)(cdiv(cdiv(g.M, turns * sms), (int64_t)8) * 8);
    p.steps = (int)cdiv(g.K, 128);
    p.rooms = Cfg::rooms(g.K);
    const int ring = (int)Cfg::ring(g.K, p.rooms);
    int parts = (int)cdiv(p.steps, 7);   // of a class's columns: as few as leave three stages
    while (3 * cdiv(p.steps, parts) * 16 * GT_COL_BYTES > ring) ++parts;
    p.j = (int)cdiv(p.steps, parts) * 16;
    p.stages = (ring < GT_RING ? ring : GT_RING) / (p.j * GT_COL_BYTES);
    GrMaps maps;
    for (int w = 0; w < 8; ++w) {
        const char* col = reinterpret_cast<const char*>(g.A + w * g.lda);
        const int off = (int)(reinterpret_cast<uintptr_t>(col) & 15u);
        const uint64_t dims[2] = {(uint64_t)(g.M + off / 2), (uint64_t)cdiv(g.K - w, 8)}, str[1] = {(uint64_t)g.lda * 16};
        const uint32_t box[2] = {64, (uint32_t)p.j};
        const int rc = make_tmap(ctx, &maps.m[w], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, col - off, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B);
        if (rc != B200_OK) return rc;
    }
    const int64_t blocks = cdiv(g.M, p.rows);
    const dim3 grid((unsigned)(blocks < sms ? blocks : sms), (unsigned)cdiv(g.N, NT));
    B200_CUDA(launch_dep(kern, grid, dim3(Cfg::THREADS), (size_t)(p.stages * p.j * GT_COL_BYTES + Cfg::fixed(g.K, p.rooms)), ctx->stream, 1, maps, p));
    ctx->launches++;
    return B200_OK;
}

// This form turns all of B in every CTA and ends with a sum that nothing hides, some 4 us of a call; A has to be long enough to pay for
// it, more so for few tokens, whose row blocks cost gemm_rows.cu little.  B stays in shared memory, so a long reduction takes the ring's
// room, and then the copies stand.  By gemm_rows.cu and by this form, us:
// 5 tokens: x 51865 x 1280 32.4, 26.7; x 54687 x 768 25.2, 23.6; x 42001 x 1000 23.2, 23.5; x 51865 x 384 15.6, 16.8; x 300001 x 136 45, 69.  Where
//   the ring is not whole: x 13125 x 3200 24.8, 25.8; x 17579 x 4096 31.4, 34.7; x 8301 x 5120 20.9, 41.6.  And many rows, which the other
//   form reads at 4.8 TB/s and this one at 4.0: x 171875 x 1280 92.5, 95.9; x 300001 x 1000 135, 153;
// 16: x 51865 x 1280 47.7, 27.4; x 24001 x 1200 25.6, 19.2; x 147657 x 256 42.5, 45.6; x 112251 x 259 41.3, 37.0; x 10921 x 4150 50.6, 46.5;
//   x 11825 x 4879 59.8, 60.9; x 14407 x 5162 63.6, 72.1;
// 32: x 51865 x 1280 62.9, 29.5; x 14765 x 2560 34.8, 29.1;  18: x 11641 x 2764 49.9, 53.9;
// 48: x 51865 x 1280 129, 33.4; x 9001 x 1280 27.2, 15.5;  64: x 51865 x 1280 139, 46.0; x 9001 x 1280 28.7, 19.9, and where B leaves the
//   least ring x 9001 x 1350 41.4, 42.8 (49 tokens 36.4, 42.0), x 15121 x 1321 59.6, 44.0;
// A read twice, by blocks of 32: 64 x 17001 x 2000 73.9, 40.4; 40 x 17007 x 2315 91.2, 71.6; 34 x 12241 x 2406 64.0, 67.5; 48 x 9951 x 2199 57.9, 68.9;
//   60 x 18749 x 2759 136, 151.
// Over 1700 products of 2 to 150 tokens drawn beside those that the lines were laid by, no call is more than 1.05 times as slow as by
// gemm_rows.cu; of the others 2 x 36001 x 2000 (34.0, 36.9: little more there than one round of row blocks).
// The lines of 9 and 21 million elements do not lie where the forms meet but above: 33 x 16577 x 520 (8.6 million) takes 27 us and would
// take 13, 32 x 12001 x 1000 16.7 and 12.9.  Under them the other form's two launches are what runs and is tested.
// And a CTA has to have rows: 16 x 2001 x 4800, 16 rows a CTA, 15.0, 34.4.
int gemm_rows_tc_tokens(const b200_ctx* ctx, int64_t M, int64_t N, int64_t K) {
    const int64_t per = cdiv(N, cdiv(N, 64)), steps = cdiv(K, 128), size = M * K;   // tokens of a token block
    if (M < 56 * (int64_t)ctx->prop.multiProcessorCount) return 0;
    if (N <= 8) return K >= 768 && size >= 45000000 && M < 170000 && GtCfg<16>::ring(K, 2) >= GT_RING ? 16 : 0;
    if (N <= 16) return K > 256 && steps <= 36 && size >= 21000000 ? 16 : 0;
    if (K < 64 || size < (N <= 32 ? 21000000 : 9000000)) return 0;
    if (N <= 32) return steps <= 21 ? 32 : 0;
    if (per <= 48 && GtCfg<48>::fits(K)) return 48;
    if (GtCfg<64>::fits(K) && (steps <= 10 || size >= 16000000)) return 64;
    return steps <= 20 && size >= (steps > 16 && N <= 64 ? 30000000 : 21000000) ? 32 : 0;
}

int gemm_rows_tc_launch(b200_ctx* ctx, const GrParams& p, int tokens, bool half_out) {
    switch (tokens) {
        case 16: return half_out ? gt_launch<16, __half>(ctx, p) : gt_launch<16, float>(ctx, p);
        case 32: return half_out ? gt_launch<32, __half>(ctx, p) : gt_launch<32, float>(ctx, p);
        case 48: return half_out ? gt_launch<48, __half>(ctx, p) : gt_launch<48, float>(ctx, p);
        default: return half_out ? gt_launch<64, __half>(ctx, p) : gt_launch<64, float>(ctx, p);
    }
}

} // namespace b200
