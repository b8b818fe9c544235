// Fused non-causal attention for sm_100a: one pass over the keys with an online softmax,
// the query tile resident in shared memory, K/V streamed by TMA straight from the strided
// (E,L,H,B) operands, S = Q K' and O += P V on the tcgen05 tensor cores with S and O in TMEM.
//
// Replaces attn_flash_cm! / attn_flash_cm_merge! / attn_flash! (reference
// kernels/extern/flash.jl:160-271,459-1036,1398-1421) and the layout passes that fed them
// (toLE_tiled_*, densify, padE: kernels/extern/attention.jl:342-396,448-463): the tensor maps
// read the operands through their strides, pad E to the MMA granule with zero fill and
// zero-fill the ragged key/query tails, so no operand is copied, padded or clamped.
//
// Rounding points kept from the reference: the scale multiplies the fp32 scores
// (flash.jl:672-675), the softmax runs in fp32, P is rounded to fp16 before P V
// (flash.jl:725,765), O accumulates in fp32, and a row whose sum is zero divides by one
// (flash.jl:1015).
//
// One CTA owns 256 queries (two tiles of 128) of one (head, batch) and walks the keys in blocks of 128, or, for many
// windows of up to 256 keys, one tile in blocks of 64; the kernel comment below gives the roles and the pipeline.
#include <cuda_fp16.h>

#include <mutex>
#include <type_traits>

#include "internal.h"
#include "ptx.cuh"

namespace b200 {

constexpr int ATT_BR = 128;  // queries per tile (TMEM lanes)
constexpr int ATT_TILE_BYTES = 128 * 128; // one swizzle atom of an operand tile: 128 rows x 128 B (64 fp16 of E)
// Four forms of CTA, by the head dimension, the mask and, the first, by short keys:
//   EP = 64, NT = 1:           one query tile, key blocks of 64, P over S, 128 tensor-memory columns and 48 KB, so that
//                              four CTAs share an SM
//   EP = 64  (E <= 64):        two query tiles of 128 per CTA, K/V rings of 4 stages x 16 KB
//   EP = 80  (64 < E <= 80):   as EP = 128, but O has 80 columns per tile, which leaves P 48 columns of its own: 96 of a
//                              block's 128 keys, the other 32 go through shared memory (A operand of the last two steps
//                              of P V).  8 heads x 4096 x 72 replayed: 70.9 us with P over S, 58.5 so (70.6 and 61.7 by
//                              calls); no mask (no room for it)
//   EP = 128 (80 < E <= 128, with a mask 64 < E):  two query tiles of 128 per CTA as well; every operand tile is two swizzle atoms along
//                              E (columns 0-63, 64-127, the second zero-filled past E by the tensor map), S = Q K'
//                              runs over both, O has 128 columns per tile — S 2 x 128 + O 2 x 128 fill the tensor
//                              memory, so P is written over the first 64 columns of its tile's S once the softmax
//                              has pulled S into registers, and a tile's Q K'(j+1) is issued after its P V(j)
//                              (the two tiles' chains interleave on the tensor core); K/V rings of 2 stages x 32 KB
// The reference's own fused tiling is E = 72 padded to 80 (flash.jl:1149-1157, flashepad kernelplans.jl).
// With an additive mask each tile also stages a block's 128 x 128 mask entries (BIAS_ROW_WORDS words per row, see
// the softmax); at EP = 128 the room for it comes from the V ring, which keeps one stage: V(j+1) is asked for when
// both tiles' P V(j) are done and needed a softmax later, more than a fetch takes.
// Through a tensor map the entries come as two boxes of 64 keys, swizzled, asked for by a warp of their own as soon as the
// block before is read.  Copied by the softmax's own warps, they cost a block 1800 clocks of standing in front of a full queue
// (4 heads x 4000 x 56: 69.3 -> 51.0 us, 8 x 2048 x 72 49.8 -> 37.6); copies of 8 bytes by warps of their own were no faster.
// A row staged by the softmax's warps: 128 entries.  Rows on 8-byte boundaries are copied and read 8 bytes at a time, 66 words apart
// (an odd number of 8-byte units, so that a warp's 32 rows lie in all banks); others word by word, from the 4-byte
// boundary at or one entry before the first, 65 words apart (odd, for the same reason).
constexpr int BIAS_ROW_WORDS = 66;
template <int EP, bool BIAS = false, int NT_ = 2> struct AttCfg {
    static_assert(EP == 64 || EP == 80 || EP == 128, "head dim is padded to one or two swizzle atoms, O to EP columns");
    static constexpr int ATOMS = EP == 64 ? 1 : 2;     // 16 KB atoms per operand tile
    static constexpr int NT = NT_;                     // query tiles per CTA
    static_assert(NT == 2 || (NT == 1 && EP == 64 && !BIAS), "one tile per CTA is built for E <= 64 without a mask");
    static_assert(EP != 80 || !BIAS, "a mask leaves no room for the tail of P");
    static constexpr int BC = NT == 2 ? 128 : 64;      // keys per block
    static constexpr int CTAS_PER_SM = NT == 2 ? 1 : 4;
    static constexpr int THREADS = 128 * NT + 128;     // NT softmax warpgroups, then TMA and UMMA warps and one that fetches the mask or idles
    static constexpr int TMA_WARP = 4 * NT, ISSUE_WARP = 4 * NT + 1;
    // registers of a softmax thread and of the others: (NT x 128 x one + 128 x the other) is what the launch holds
    static constexpr int SOFTMAX_REGS = NT == 2 ? 232 : 96, OTHER_REGS = NT == 2 ? 40 : 32;
    static constexpr int TMEM_COLS = NT == 2 ? 512 : 128;
    // S of tile t at BC t, O at O_COL + EP t, P of its own at P_COL + P_COLS t
    static constexpr int O_COL = NT * BC, P_COL = O_COL + NT * EP;
    static constexpr bool P_TAIL = EP == 80;               // the last 32 keys of a block's P lie in shared memory
    static constexpr int P_COLS = P_TAIL ? 48 : 64;
    static constexpr int K_STAGES = NT == 2 && EP == 64 ? 4 : 2;
    static constexpr int V_STAGES = NT == 2 && EP == 64 ? 4 : (BIAS ? 1 : 2);
    static constexpr bool P_IN_S = EP == 128 || NT == 1;   // P shares its tile's S columns (tensor memory is full otherwise)
    static constexpr int Q_BYTES = ATOMS * ATT_TILE_BYTES;    // one Q tile
    static constexpr int KV_ATOM = BC * 128, KV_BYTES = ATOMS * KV_ATOM;   // one K or V tile
    // shared-memory map
    static constexpr int S_Q = 0;                              // NT tiles
    static constexpr int S_K = NT * Q_BYTES;                   // K_STAGES tiles
    static constexpr int S_V = S_K + K_STAGES * KV_BYTES;      // V_STAGES tiles
    static constexpr int S_P = S_V + V_STAGES * KV_BYTES;      // P_TAIL: NT tiles of 128 rows x 128 B, the first 64 used
    static constexpr int S_END = S_P + (P_TAIL ? NT * ATT_TILE_BYTES : 0);
    static constexpr int BIAS_TILE_BYTES = BIAS ? ATT_BR * BIAS_ROW_WORDS * 4 : 0;
    static constexpr int S_BARS = S_END + NT * BIAS_TILE_BYTES;   // the barriers, then the tensor-memory address and the abort flag
    static constexpr int BARRIERS = 2 + 2 * K_STAGES + 2 * V_STAGES + 10 + (EP == 128 ? 2 : 0) + (BIAS ? 4 : 0);
    static constexpr int SMEM_BYTES = S_BARS + (BARRIERS + 1) * 8;
    static_assert(CTAS_PER_SM * (SMEM_BYTES + 1024) <= 233472, "shared memory over budget");
    // Joining: a CTA's share of an item's rows from all of them, over the operand tiles, [part][four columns][row] of 16 bytes (16 more
    // between columns, so that neighbouring fours of a row lie in other banks); behind them [part][row] (reference point, sum).
    static constexpr int join_bytes(int parts) {
        const int share = (NT * ATT_BR + parts - 1) / parts;
        return parts * (EP / 4 * (share * 16 + 16) + share * 8);
    }
    static_assert(NT == 1 || (join_bytes(2) <= S_V + V_STAGES * KV_BYTES && join_bytes(8) <= S_V + V_STAGES * KV_BYTES),
                  "the rows to join fit over the operand tiles");
};
constexpr int JOIN_MOST = 8;   // CTAs of a portable cluster
// tensor-memory map of two tiles (512 columns): S of tile t, fp32, at [128 t, 128 t + 128); O of tile t, fp32, at
// [256 + EP t, ... + EP); P of tile t, fp16 packed two keys per column, at [384 + 64 t, ... + 64) for EP = 64, at
// [416 + 48 t, ... + 48) for EP = 80 and over the first 64 columns of S_t for EP = 128

struct AttnParams {
    int E, Lq, Lk, H, B;
    float scale, scale_log2;   // scale_log2 = scale * log2(e)
    void* out;
    int64_t osL, osH, osB;  // element strides of out along L, H, B (E is contiguous)
    int out_f32;
    int qpairs;         // work items per (head, batch): groups of NT query tiles ("pairs" when NT = 2)
    int pair_ctas;      // CTAs [0, pair_ctas) own a whole item; the rest own one tile of a pair, or a key range of an item
    int* d_status;
    unsigned long long* trace;  // optional timeline of CTA (0,0,0) (globaltimer ns), null in normal use
    // Additive mask of the mem-efficient variant (attention.jl:55-59), (Lk,Lq,H,B) fp16 with element
    // strides (0 on a broadcast axis); null when absent.
    const __half* bias;
    int64_t bsK, bsQ, bsH, bsB;
    int mask;           // how the mask's blocks reach the softmax: one of MASK_*
    // Keys split over nsplit CTAs per query pair (few queries, many keys): each writes its unnormalised
    // fp32 O rows to part_o[split][tail pair][256 rows][E] and (reference point, row sum) to part_ml[...][2];
    // attention_merge_kernel combines them (the reference's attn_flash_cm_merge!, flash.jl:1398-1421).
    int nsplit;
    int ntail;          // pairs that are split (the last ntail of them)
    float* part_o;
    float* part_ml;
};

// Entry by entry from global memory (keys not contiguous); copied to shared memory ahead of use by words, or 8 bytes at
// a time where every row starts on an 8-byte boundary; through a tensor map.
enum { MASK_DIRECT = 0, MASK_WORDS = 1, MASK_EIGHTS = 2, MASK_TMA = 3 };

#define ATT_TRACE(slot)                                                                              \
    do {                                                                                             \
        if (p.trace != nullptr && blockIdx.x == 0 && (slot) < 128) \
            p.trace[(slot)] = globaltimer_ns();                                                      \
    } while (0)

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async8(uint32_t dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void st_shared16(uint32_t at, const uint32_t* v) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
}
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[32]) { tmem_ld32(taddr, r); }
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[16]) { tmem_ld16(taddr, r); }
__device__ __forceinline__ float fmax3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ void tmem_st16_raw(uint32_t taddr, const uint32_t* r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}

// Two tiles (NT = 2): 256 queries of one (head, batch), one CTA per SM:
//   warps 0-3  softmax of tile 0, warps 4-7 softmax of tile 1: one thread per query row, the whole
//              128-score row in registers (these two warpgroups take registers from the third)
//   warp 8     TMA producer: both Q tiles once, then K and V blocks through the rings of AttCfg
//   warps 9,10 UMMA issuers, one warp per tile, which waits together and has one thread issue: S_t = Q_t K' and O_t += P_t V per key block;
//              the two chains are independent, so the tensor core works on one tile while the
//              other tile's softmax runs
//   warp 11    asks for the mask's entries where a tensor map is over them
// One tile (NT = 1): warps 0-3 its softmax, 64 scores a thread, warp 4 the producer, warp 5 the issuer; four CTAs per SM.
// P stays out of shared memory, but for a quarter of it at EP = 80: the softmax threads write it as packed fp16 into tensor memory
// and the P V product takes its A operand from there, so the shared-memory port feeds K and V.
// BIAS: the scaled score gets an additive fp16 mask before the softmax; a row whose keys are all
// blocked (-inf everywhere) comes out as zeros, as in attn_softmax (attention.jl:73-100).
// JOIN: the CTAs an item's keys are cut over are a cluster, which joins their rows through distributed shared memory: an instance of
// its own (in one with the others its code cost their loop 13 %).
template <int EP, bool BIAS, int NT_, bool JOIN>
__global__ void __launch_bounds__(AttCfg<EP, BIAS, NT_>::THREADS, AttCfg<EP, BIAS, NT_>::CTAS_PER_SM)
attention_f16_tc_kernel(const __grid_constant__ CUtensorMap tmapQ,
                        const __grid_constant__ CUtensorMap tmapK,
                        const __grid_constant__ CUtensorMap tmapV,
                        const __grid_constant__ CUtensorMap tmapM, const AttnParams p) {
    using Cfg = AttCfg<EP, BIAS, NT_>;
    constexpr int K_STAGES = Cfg::K_STAGES, V_STAGES = Cfg::V_STAGES;
    constexpr int BC = Cfg::BC, NC = BC / 32;   // keys per block, and per-thread pieces of 32 of them
    constexpr int NT = Cfg::NT;
    // Where P lies over S, everything after P waits for P V: it is issued in two halves of the block, the first under the second
    // half's exponentials.  12 x 1500 x 96 32.2 -> 31.7 us, masked 8 x 2048 x 72 50.6 -> 49.9 (before the whole warp issued);
    // with columns of its own the turns hide as much and the extra hand-over costs (12 x 4096 x 64: 85.9 -> 88.1).
    constexpr bool HALVES = EP == 128;
    constexpr bool OWN_P = !Cfg::P_IN_S;     // P in columns (and shared memory) of its own
    constexpr bool FREE = OWN_P && !BIAS;    // its tiles go their own ways after the start, see the softmax
    constexpr int ITEM_ROWS = NT * ATT_BR;   // queries one whole work item covers
    extern __shared__ __align__(1024) uint8_t smem[];
    // Uniform across the grid: a base that is not 1024-aligned makes every thread leave before
    // any barrier or TMEM allocation exists.
    if ((smem_u32(smem) & 1023u) != 0) {
        if (threadIdx.x == 0) atomicCAS(p.d_status, 0, KST_SMEM_LAYOUT);
        return;
    }
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::S_BARS);
    uint64_t* q_full = bars + 0;                           // [2]
    uint64_t* k_full = bars + 2;                           // [K_STAGES]
    uint64_t* k_empty = k_full + K_STAGES;                 // [K_STAGES]
    uint64_t* v_full = k_empty + K_STAGES;                 // [V_STAGES]
    uint64_t* v_empty = v_full + V_STAGES;                 // [V_STAGES]
    uint64_t* s_full = v_empty + V_STAGES;                 // [2]
    uint64_t* s_empty = s_full + 2;                        // [2]
    uint64_t* p_full = s_empty + 2;                        // [2]
    uint64_t* pv_done = p_full + 2;                        // [2]
    uint64_t* exp_turn = pv_done + 2;                      // [2]: whose turn it is to run its exponentials
    uint64_t* p_half = exp_turn + 2;                       // [2]: HALVES, the first half of a block's P is written
    uint64_t* mask_full = p_half + (HALVES ? 2 : 0);       // [2]: BIAS, a block's mask entries have landed (MASK_TMA)
    uint64_t* mask_empty = mask_full + 2;                  // [2]: and have been read
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(mask_full + (BIAS ? 4 : 0));
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    static_assert(Cfg::BARRIERS == 2 + 2 * K_STAGES + 2 * V_STAGES + 10 + (HALVES ? 2 : 0) + (BIAS ? 4 : 0), "barriers counted by the layout");

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    // Work item of this CTA.  Most CTAs own a pair of query tiles; when the pairs do not fill the
    // last wave of SMs, the pairs of that wave are handed out as single tiles instead (twice as
    // many, half as long), which shortens the tail.
    // CTAs [0, pair_ctas) own a whole pair.  The pairs after those are the tail: either each is cut along
    // the keys into nsplit CTAs whose partial results are merged afterwards (nsplit > 1), or each is
    // handed out as two single tiles.
    // A join's CTAs all belong to the tail; the whole pairs before it, if any, are a launch of their own.
    int item = blockIdx.x + (JOIN ? p.pair_ctas : 0), half = -1, split = 0, nsp = 1;
    if (item >= p.pair_ctas) {
        const int t = item - p.pair_ctas;
        if (p.nsplit > 1) {
            nsp = p.nsplit;
            split = t % nsp;
            item = p.pair_ctas + t / nsp;
        } else {
            half = t & 1;
            item = p.pair_ctas + (t >> 1);
        }
    }
    const int tailpair = item - p.pair_ctas;   // index among the split pairs (when nsp > 1)
    const int qp = item % p.qpairs;
    const int h = (item / p.qpairs) % p.H;
    const int b = item / (p.qpairs * p.H);
    const int q0 = qp * ITEM_ROWS + (half > 0 ? ATT_BR : 0);
    const int nblk_all = (p.Lk + BC - 1) / BC;
    const int jb0 = (int)((int64_t)split * nblk_all / nsp);           // first key block of this CTA
    const int nblk = (int)((int64_t)(split + 1) * nblk_all / nsp) - jb0;
    const int ntiles = (NT == 2 && half < 0 && q0 + ATT_BR < p.Lq) ? 2 : 1;   // the second tile may lie wholly past Lq

    if (threadIdx.x == 0) {
        ATT_TRACE(0);
        for (int t = 0; t < 2; ++t) {
            mbar_init(&q_full[t], 1);
            mbar_init(&s_full[t], 1);
            mbar_init(&s_empty[t], 4);   // one arrival per softmax warp
            mbar_init(&p_full[t], 4);
            if (HALVES) mbar_init(&p_half[t], 4);
            mbar_init(&pv_done[t], 1);
            mbar_init(&exp_turn[t], 4);
            if (BIAS) {
                mbar_init(&mask_full[t], 1);
                mbar_init(&mask_empty[t], 4);
            }
        }
        for (int s = 0; s < K_STAGES; ++s) {
            mbar_init(&k_full[s], 1);
            mbar_init(&k_empty[s], ntiles);   // freed when every tile's issuer is done with it
        }
        for (int s = 0; s < V_STAGES; ++s) {
            mbar_init(&v_full[s], 1);
            mbar_init(&v_empty[s], ntiles);
        }
        *abort_flag = 0;
        fence_barrier_init();
        prefetch_tmap(&tmapQ);
        prefetch_tmap(&tmapK);
        prefetch_tmap(&tmapV);
    }
    if (warp == Cfg::TMA_WARP) {
        tmem_alloc(tmem_slot, Cfg::TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // Everything above overlapped the previous kernel's tail; from here on its results are needed.
    // (A joined tail reads only what its whole pairs' launch has waited for, and by TMA alone, which reads the L2, so it starts as that
    // one's CTAs leave; what follows the tail on the stream waits for it to end, hence, by the wait at its end, for both.)
    if (!JOIN || p.pair_ctas == 0) grid_dep_wait();
    grid_dep_launch();

    bool met = false;   // joining: this warp has passed the barrier behind which the rows are there

    // Register budget: the two softmax warpgroups hold a full score row per thread; the third
    // warpgroup (a TMA lane, the warps that issue and the mask's lane) needs almost nothing and hands its
    // share over (setmaxnreg at the head of each role's branch).
    if (warp == 4 * NT + 3 || (NT == 1 && warp == 6)) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Cfg::OTHER_REGS));
        if (BIAS && p.mask == MASK_TMA && lane == 0) {   // a block's 128 x 128 entries per tile, as soon as the block before is read
            bool ok = true;
            for (int j = 0; ok && j < nblk; ++j)
                for (int t = 0; ok && t < ntiles; ++t) {
                    if (j > 0 && !mbar_wait(&mask_empty[t], (uint32_t)((j - 1) & 1), p.d_status, KST_WAIT_EMPTY, abort_flag)) {
                        ok = false;
                        break;
                    }
                    mbar_arrive_expect_tx(&mask_full[t], 2 * ATT_TILE_BYTES);
#pragma unroll
                    for (int a = 0; a < 2; ++a)
                        tma_load_4d(smem + Cfg::S_END + t * Cfg::BIAS_TILE_BYTES + a * ATT_TILE_BYTES, &tmapM, &mask_full[t],
                                    (jb0 + j) * BC + 64 * a, q0 + t * ATT_BR, p.bsH ? h : 0, p.bsB ? b : 0);
                }
        }
    } else if (warp == Cfg::TMA_WARP) {
        // ------------------------------------------------------------- TMA producer
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Cfg::OTHER_REGS));
        if (lane == 0) {
            for (int t = 0; t < ntiles; ++t) {
                mbar_arrive_expect_tx(&q_full[t], Cfg::Q_BYTES);
#pragma unroll
                for (int a = 0; a < Cfg::ATOMS; ++a)
                    tma_load_4d(smem + Cfg::S_Q + t * Cfg::Q_BYTES + a * ATT_TILE_BYTES, &tmapQ, &q_full[t], a * 64, q0 + t * ATT_BR, h, b);
            }
            for (int j = 0; j < nblk; ++j) {
                const int s = j % K_STAGES, sv = j % V_STAGES;
                const uint32_t ph = (uint32_t)((j / K_STAGES) & 1), phv = (uint32_t)((j / V_STAGES) & 1);
                if (!mbar_wait(&k_empty[s], ph ^ 1, p.d_status, KST_WAIT_EMPTY, abort_flag)) break;
                mbar_arrive_expect_tx(&k_full[s], Cfg::KV_BYTES);
#pragma unroll
                for (int a = 0; a < Cfg::ATOMS; ++a)
                    tma_load_4d(smem + Cfg::S_K + s * Cfg::KV_BYTES + a * Cfg::KV_ATOM, &tmapK, &k_full[s], a * 64, (jb0 + j) * BC, h, b);
                if (!mbar_wait(&v_empty[sv], phv ^ 1, p.d_status, KST_WAIT_EMPTY, abort_flag)) break;
                mbar_arrive_expect_tx(&v_full[sv], Cfg::KV_BYTES);
#pragma unroll
                for (int a = 0; a < Cfg::ATOMS; ++a)
                    tma_load_4d(smem + Cfg::S_V + sv * Cfg::KV_BYTES + a * Cfg::KV_ATOM, &tmapV, &v_full[sv], a * 64, (jb0 + j) * BC, h, b);
            }
        }
    } else if (warp == Cfg::ISSUE_WARP || (NT == 2 && warp == Cfg::ISSUE_WARP + 1)) {
        // ------------------------------------------------------------- UMMA issuers
        // One issuing warp per query tile (warp 9: tile 0, warp 10: tile 1).  Each walks its own
        // chain  S_t(j+1) = Q_t K(j+1)'  as soon as the softmax has pulled S_t(j) into registers,
        // then  O_t += P_t(j) V(j)  once P_t(j) is written.  The two chains share only the
        // K/V rings.  (Issuing a UMMA blocks while the tensor pipe is busy, so the issuing warps
        // are not softmax warps.)
        // The whole warp walks the chain and waits; the thread elect.sync picks (the same one every time) issues, every
        // operand being the same for the warp.  With one lane running it under `if (lane == 0)`, P written -> P V
        // issued took 1000 clocks and S taken -> Q K' issued 1300, with nothing else on the tensor core; now 290 and
        // 430.  16 heads x 2048 x 128 35.4 -> 33.7 us, masked 8 x 2048 x 72 49.9 -> 45.1, 1024 x 8 windows of 256 x 56 374 -> 359.
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Cfg::OTHER_REGS));
        const int t = warp - Cfg::ISSUE_WARP;
        if (t < ntiles) {
            // S = Q K': both operands K-major (E contiguous), from shared memory.  O += P V: P from
            // tensor memory (P_TAIL: its last 32 keys K-major from shared memory), V MN-major (E contiguous per key) from
            // shared memory.
            constexpr uint32_t idesc_s = make_idesc_f16(ATT_BR, BC, 0, 0);
            constexpr uint32_t idesc_o = make_idesc_f16(ATT_BR, EP, 0, 1);
            constexpr uint64_t kdesc0 = make_smem_desc(16, 1024);
            constexpr uint64_t vdesc0 = make_smem_desc(Cfg::KV_ATOM, 1024);
            const uint32_t q_addr = smem_u32(smem + Cfg::S_Q + t * Cfg::Q_BYTES);
            const uint32_t tail_addr = smem_u32(smem + Cfg::S_P + t * ATT_TILE_BYTES);
            const uint32_t s_tmem = tmem_base + t * BC;
            const uint32_t o_tmem = tmem_base + Cfg::O_COL + t * EP;
            const uint32_t p_tmem = OWN_P ? tmem_base + Cfg::P_COL + t * Cfg::P_COLS : s_tmem;

            auto wait = [&](uint64_t* bar, uint32_t parity, int code) -> bool {   // one answer per warp
                return __all_sync(0xffffffffu, mbar_wait(bar, parity, p.d_status, code, abort_flag));
            };
            auto issue_qk = [&](int j) -> bool {
                const int sk = j % K_STAGES;
                if (!wait(&k_full[sk], (uint32_t)((j / K_STAGES) & 1), KST_WAIT_FULL)) return false;
                // With P in S's columns this product is issued after P V(j-1), which read P after the softmax had taken
                // S(j-1), and UMMAs of one thread run in issue order: nothing else to wait for.
                if (OWN_P && j > 0 && !wait(&s_empty[t], (uint32_t)((j - 1) & 1), KST_WAIT_SOFTMAX)) return false;
                tc_fence_after();
                if (elect_one()) {
                    const uint32_t k_addr = smem_u32(smem + Cfg::S_K + sk * Cfg::KV_BYTES);
#pragma unroll
                    for (int k = 0; k < EP / 16; ++k) {
                        // past the head dim both operands are zeros
                        if (EP == 128 && k >= 5 && k * 16 >= p.E) break;
                        // 16 elements of E = 32 B inside the swizzle row; every fourth step moves to the next atom
                        const uint32_t in = (uint32_t)(k & 3) * 32;
                        umma_ss(s_tmem, smem_desc_at(kdesc0, q_addr + (uint32_t)(k >> 2) * ATT_TILE_BYTES + in),
                                smem_desc_at(kdesc0, k_addr + (uint32_t)(k >> 2) * Cfg::KV_ATOM + in), idesc_s, k != 0);
                    }
                    umma_commit(&s_full[t]);
                    umma_commit(&k_empty[sk]);   // one of `ntiles` arrivals that free this K stage
                    if (j >= 1 && j < 7) ATT_TRACE(64 * t + 8 + 8 * (j - 1) + 0);   // Q K'(j) issued, filed under block j-1
                }
                __syncwarp();
                return true;
            };
            // P V of block j, steps [k0, k1) of 16 keys.
            auto issue_pv = [&](int j, int sv, int k0, int k1) {
                const uint32_t v_addr = smem_u32(smem + Cfg::S_V + sv * Cfg::KV_BYTES);
#pragma unroll
                for (int k = k0; k < k1; ++k) {
                    // P comes from tensor memory: 16 keys = 8 packed columns per step.
                    // V: 16 key rows = two 8-row groups = 2048 B.
                    const uint64_t vdesc = smem_desc_at(vdesc0, v_addr + k * 2048);
                    if (Cfg::P_TAIL && k >= BC / 16 - 2) umma_ss(o_tmem, smem_desc_at(kdesc0, tail_addr + (k - (BC / 16 - 2)) * 32), vdesc, idesc_o, 1);
                    else umma_ts(o_tmem, p_tmem + k * 8, vdesc, idesc_o, (j | k) != 0);
                }
            };

            bool ok = wait(&q_full[t], 0, KST_WAIT_FULL);
            if (ok && nblk > 0) ok = issue_qk(0);
            for (int j = 0; ok && j < nblk; ++j) {
                if (OWN_P && j + 1 < nblk && !issue_qk(j + 1)) break;
                const int sv = j % V_STAGES;
                if (!wait(&v_full[sv], (uint32_t)((j / V_STAGES) & 1), KST_WAIT_FULL)) break;
                if (j < 6 && lane == 0) ATT_TRACE(64 * t + 8 + 8 * j + 7);   // issuer reaches its wait for P(j)
                constexpr int FIRST = HALVES ? BC / 32 : 0;   // steps that do not wait for the whole of P
                if constexpr (HALVES) {
                    if (!wait(&p_half[t], (uint32_t)(j & 1), KST_WAIT_SOFTMAX)) break;
                    tc_fence_after();
                    if (elect_one()) issue_pv(j, sv, 0, FIRST);
                    __syncwarp();
                }
                if (!wait(&p_full[t], (uint32_t)(j & 1), KST_WAIT_SOFTMAX)) break;
                tc_fence_after();
                if (elect_one()) {
                    issue_pv(j, sv, FIRST, BC / 16);
                    umma_commit(&pv_done[t]);
                    umma_commit(&v_empty[sv]);   // one of `ntiles` arrivals that free this V stage
                    if (j < 6) ATT_TRACE(64 * t + 8 + 8 * j + 1);   // P V(j) issued
                }
                __syncwarp();
                if (!OWN_P && j + 1 < nblk && !issue_qk(j + 1)) break;   // overwrites P(j): after the product that reads it
            }
        }
    } else {
        // ------------------------------------------------------- softmax + epilogue
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(Cfg::SOFTMAX_REGS));
        const int t = warp >> 2;               // which query tile this warpgroup owns
        const int quad = warp & 3;             // TMEM lane quadrant
        const int row = quad * 32 + lane;
        if (t < ntiles) {
            const uint32_t lane_base = uint32_t(quad * 32) << 16;
            const uint32_t s_tmem = tmem_base + lane_base + t * BC;
            const uint32_t o_tmem = tmem_base + lane_base + Cfg::O_COL + t * EP;
            const uint32_t p_tmem = OWN_P ? tmem_base + lane_base + Cfg::P_COL + t * Cfg::P_COLS : s_tmem;
            const float sc = BIAS ? p.scale : p.scale_log2;
            const float sce = BIAS ? 1.4426950408889634f : sc;   // with a bias the scores are scaled when it is added
            float m_run = -INFINITY, l_run = 0.f;
            bool ok = true;
            // Both tiles take the same time per block, and in step both would want the MUFU pipe in the same half of
            // every period and leave it idle in the other.  Where P has a place of its own and there is no mask it is enough that tile 1
            // starts behind: nothing brings the two together again (12 heads x 4096 x 64, its tail not joined: 79.6 us, 84.5 in step, 86.3
            // with a turn handed over every block).
            // With P over S, or a mask, a tile's block is one long chain and the exponential phases take turns (tile 0 block j, tile 1
            // block j, tile 0 block j+1, ...): while one tile owns the MUFU pipe the other does its max / rescale / waits
            // and its tensor-core work runs (16 heads x 2048 x 128: 33.7 us, 38.5 without).
            const bool pingpong = ntiles == 2;
            // After which quarter of its exponentials a tile passes the turn.  The mean over 12 shapes of 2 to 40 heads and 800 to 16384
            // keys, after the first, second, third and last: 64 wide 1, 1.05, 0.99, 0.98, and the 32-layer encoder 3189 us, 3234, 3148, 3150;
            // 72 wide 1, 0.99, 1.03, 1.04 (8 heads x 4096: 58.5, 58.2, 62.7, 63.5); 128 wide 1, 0.99, 0.96, 0.96; masked 64 wide alike within 1 %,
            // 80 wide 1, 0.99, 0.95, 0.97.
            constexpr int TURN_AT = !FREE ? 3 : EP == 64 ? 2 : 0;
            // A mask no tensor map is over, its keys contiguous: each warp copies the next block's entries of its own 32 rows to
            // shared memory (cp.async, a row's entries across the lanes) while it works on this block, and every thread
            // then reads its row back.  Nothing but the warp itself is involved, so no barrier is.  Rows may start at
            // any element: when not all of them lie on 8-byte boundaries (an odd number of keys puts every other row in
            // the middle of a word) words are copied from the 4-byte boundary at or below a row's first entry and
            // shifted when read.  Every piece copied holds an entry of the mask.  Read straight from global memory, one
            // row per thread, 20 heads x 1500 x 1500 took 152 us, with words copied 56, with 8 bytes at a time 45 (24
            // without a mask: adding it is 64 more packed FMAs, 128 conversions and the reads per thread and block).
            uint32_t* bias_rows = reinterpret_cast<uint32_t*>(smem + Cfg::S_END) + (t * ATT_BR + quad * 32) * BIAS_ROW_WORDS;
            const bool bias_async = BIAS && (p.mask == MASK_WORDS || p.mask == MASK_EIGHTS);
            const bool bias8 = BIAS && p.mask == MASK_EIGHTS;
            auto bias_fetch = [&](int j) {
                const int keys = min(BC, p.Lk - (jb0 + j) * BC);
                const int rows = min(32, p.Lq - (q0 + t * ATT_BR + quad * 32));   // rows of this warp that exist
                const char* src = reinterpret_cast<const char*>(p.bias + (int64_t)(q0 + t * ATT_BR + quad * 32) * p.bsQ +
                                                                (int64_t)h * p.bsH + (int64_t)b * p.bsB + (int64_t)(jb0 + j) * BC);
                const uint32_t dst = smem_u32(bias_rows);
                if (bias8) {
                    if (4 * lane < keys) {
                        src += lane * 8;
#pragma unroll 8
                        for (int r = 0; r < rows; ++r, src += p.bsQ * 2) cp_async8(dst + lane * 8 + r * 264, src);
                    }
                } else {
                    const char* s = src;
#pragma unroll 4
                    for (int r = 0; r < rows; ++r, s += p.bsQ * 2) {
                        const int words = (keys + 1 + (int)((reinterpret_cast<uintptr_t>(s) >> 1) & 1)) >> 1;
                        const char* a = reinterpret_cast<const char*>(reinterpret_cast<uintptr_t>(s) & ~(uintptr_t)3) + lane * 4;
                        if (lane < words) cp_async4(dst + lane * 4 + r * 260, a);
                        if (lane + 32 < words) cp_async4(dst + lane * 4 + r * 260 + 128, a + 128);
                    }
                    if (lane < rows) {   // a row's 65th word, when its 128 entries start in the middle of a word
                        const uintptr_t a = reinterpret_cast<uintptr_t>(src) + (int64_t)lane * p.bsQ * 2;
                        if ((a & 2) && keys == BC)
                            cp_async4(dst + lane * 260 + 256, reinterpret_cast<const char*>((a & ~(uintptr_t)3) + 256));
                    }
                }
                cp_async_commit();
            };
            if (bias_async) bias_fetch(0);

            uint32_t r[NC][32];
            // The whole row of S (128 fp32) comes into registers in one round trip.
            auto scores = [&](int j) -> bool {
                if (!mbar_wait(&s_full[t], (uint32_t)(j & 1), p.d_status, KST_WAIT_TMEM_FULL, abort_flag)) return false;
                __syncwarp();
                tc_fence_after();
#pragma unroll
                for (int c = 0; c < NC; ++c) tmem_ld32(s_tmem + c * 32, r[c]);
                return true;
            };
            for (int j = 0; ok && j < nblk; ++j) {
                if (BIAS && p.mask == MASK_TMA && !mbar_wait(&mask_full[t], (uint32_t)(j & 1), p.d_status, KST_WAIT_SOFTMAX, abort_flag)) { ok = false; break; }
                if (!scores(j)) { ok = false; break; }
                const int nvalid = p.Lk - (jb0 + j) * BC; // keys of this block that exist (>= BC when full)
                if (lane == 0 && quad == 0 && j < 6) ATT_TRACE(64 * t + 8 + 8 * j + 2);  // S(0, j) ready
                tmem_wait_ld();
#pragma unroll
                for (int c = 0; c < NC; ++c)
#pragma unroll
                    for (int i = 0; i < 32; ++i) asm volatile("" : "+r"(r[c][i]));   // in registers from here on
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&s_empty[t]);   // free for the next Q K' of this tile
                if (lane == 0 && quad == 0 && j < 6) ATT_TRACE(64 * t + 8 + 8 * j + 3);  // S in registers

                if constexpr (BIAS) {
                    // r <- s * scale + bias: from here on the scores are in the mask's units and the scale below is log2(e).
                    // (A reference point beyond 2^12, where every key of a row carries the type's lowest value, is itself
                    // rounded by more than fp16 tells from one: there the heaviest key's P is rounded like the others'.)
                    const int lq = q0 + t * ATT_BR + row;
                    {
                        const __half* brow = p.bias + (int64_t)(lq < p.Lq ? lq : 0) * p.bsQ + (int64_t)h * p.bsH +
                                             (int64_t)b * p.bsB + (int64_t)(jb0 + j) * BC * p.bsK;
                        const uint64_t sc2b = pack2(sc, sc);
                        // score * scale + mask for two keys: the mask's units, the exponent's factor follows later
                        auto add = [&](int c, int i, uint32_t two) {
                            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&two));
                            float x0, x1;
                            unpack2(fma2(pack2(__uint_as_float(r[c][2 * i]), __uint_as_float(r[c][2 * i + 1])), sc2b, pack2(f.x, f.y)),
                                    x0, x1);
                            r[c][2 * i] = __float_as_uint(x0);
                            r[c][2 * i + 1] = __float_as_uint(x1);
                        };
                        if (p.mask == MASK_TMA) {
                            const uint8_t* w = smem + Cfg::S_END + t * Cfg::BIAS_TILE_BYTES + row * 128;   // rows of 64 entries, 128-byte swizzle
#pragma unroll
                            for (int c = 0; c < BC / 8; ++c) {
                                const uint4 eight = *reinterpret_cast<const uint4*>(w + (c >> 3) * ATT_TILE_BYTES + (((c & 7) ^ (row & 7)) << 4));
                                add(c >> 2, (c & 3) * 4, eight.x);
                                add(c >> 2, (c & 3) * 4 + 1, eight.y);
                                add(c >> 2, (c & 3) * 4 + 2, eight.z);
                                add(c >> 2, (c & 3) * 4 + 3, eight.w);
                            }
                            __syncwarp();   // every lane has read its row
                            if (lane == 0) mbar_arrive(&mask_empty[t]);
                        } else if (bias_async) {
                            cp_async_wait_all();
                            __syncwarp();
                            if (bias8) {
                                const uint2* w = reinterpret_cast<const uint2*>(bias_rows + lane * 66);
#pragma unroll
                                for (int c = 0; c < NC; ++c)
#pragma unroll
                                    for (int i = 0; i < 16; i += 2) {
                                        const uint2 four = w[c * 8 + i / 2];
                                        add(c, i, four.x);
                                        add(c, i + 1, four.y);
                                    }
                            } else {
                                const uint32_t* w = bias_rows + lane * 65;
                                const uint32_t shift = (uint32_t)(reinterpret_cast<uintptr_t>(brow) & 2) * 8;   // 16: the row starts mid-word
                                uint32_t lo = w[0];
#pragma unroll
                                for (int c = 0; c < NC; ++c)
#pragma unroll
                                    for (int i = 0; i < 16; ++i) {
                                        const uint32_t hi = w[c * 16 + i + 1];
                                        add(c, i, __funnelshift_r(lo, hi, shift));
                                        lo = hi;
                                    }
                            }
                            __syncwarp();   // every lane has read its row
                            if (j + 1 < nblk) bias_fetch(j + 1);
                        } else {
#pragma unroll
                            for (int c = 0; c < NC; ++c)
#pragma unroll
                                for (int i = 0; i < 32; ++i) {
                                    const float bv = (c * 32 + i < nvalid) ? __half2float(brow[(int64_t)(c * 32 + i) * p.bsK]) : 0.f;
                                    r[c][i] = __float_as_uint(fmaf(__uint_as_float(r[c][i]), sc, bv));
                                }
                        }
                    }
                }
                // Row maximum of the raw scores (the scale is positive, so it commutes with max);
                // eight independent chains instead of one 128-long dependent one.
                if (nvalid < BC) {
#pragma unroll
                    for (int c = 0; c < NC; ++c)
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            if (c * 32 + i >= nvalid) r[c][i] = 0xff800000u; // -inf: a key that does not exist gives 2^-inf = 0
                }
                float mxa = -INFINITY, mxb = -INFINITY, mxc = -INFINITY, mxd = -INFINITY;
#pragma unroll
                for (int c = 0; c < NC; ++c) {
#pragma unroll
                    for (int i = 0; i < 32; i += 8) {   // three-input max: two scores per instruction
                        mxa = fmax3(mxa, __uint_as_float(r[c][i]), __uint_as_float(r[c][i + 1]));
                        mxb = fmax3(mxb, __uint_as_float(r[c][i + 2]), __uint_as_float(r[c][i + 3]));
                        mxc = fmax3(mxc, __uint_as_float(r[c][i + 4]), __uint_as_float(r[c][i + 5]));
                        mxd = fmax3(mxd, __uint_as_float(r[c][i + 6]), __uint_as_float(r[c][i + 7]));
                    }
                }
                const float mx = fmaxf(fmaxf(mxa, mxb), fmaxf(mxc, mxd));
                // The reference point of the exponentials only has to keep 2^(x - m) inside fp16:
                // it follows the true maximum lazily, moving (and rescaling O and the running sum)
                // only when the maximum has grown by more than 2^8.  Any reference point gives the
                // same quotient O / l; the lazy one makes rescales rare after the first blocks.
                // The key at the reference point has P = 1, which fp16 holds exactly, and it is the key with the largest
                // weight: so the first 128 keys give their maximum in every form, also where they are two blocks (left
                // lazy there, the result of 256-key windows was 1.6 to 2 % further from 64 bits, for 2 % of their time).
                const float m_blk = mx * sce;
                const float slack = (BC < 128 && j == 1) ? 0.0f : 8.0f;
                const float m_new = (m_blk > m_run + slack) ? m_blk : m_run;
                // With a mask a row may have seen nothing but -inf so far: then the reference point stays -inf.
                const float m_sub = (BIAS && m_new == -INFINITY) ? 0.f : m_new;
                float alpha = 1.0f;
                bool pv_known = false;
                // O is in use by the previous block's P V; so are P's columns where nothing else says that it is done.
                auto pv_wait = [&]() -> bool {
                    if (j > 0 && !pv_known && !mbar_wait(&pv_done[t], (uint32_t)((j - 1) & 1), p.d_status, KST_WAIT_SOFTMAX, abort_flag)) return false;
                    pv_known = true;
                    tc_fence_after();
                    return true;
                };
                if (!FREE && !pv_wait()) { ok = false; break; }
                auto rescale = [&]() -> bool {
                    alpha = (BIAS && m_run == m_new) ? 1.0f : ex2(m_run - m_new);   // 0 on the first block (m_run = -inf), else 1 or < 2^-8
                    if (j == 0) return true;
                    if (!pv_wait()) return false;
#pragma unroll 1
                    for (int c = 0; c < EP / 16; ++c) {   // 16 columns at a time: S is live in registers
                        uint32_t o16[16];
                        tmem_ld16(o_tmem + c * 16, o16);
                        tmem_wait_ld();
#pragma unroll
                        for (int i = 0; i < 16; ++i) o16[i] = __float_as_uint(__uint_as_float(o16[i]) * alpha);
                        tmem_st16_raw(o_tmem + c * 16, o16);
                    }
                    tmem_wait_st();
                    return true;
                };
                if (!FREE && __any_sync(0xffffffffu, m_new != m_run) && !rescale()) { ok = false; break; }
                if (lane == 0 && quad == 0 && j < 6) ATT_TRACE(64 * t + 8 + 8 * j + 4);  // max done
                if (pingpong && (FREE ? t == 1 && j == 0 : t == 1 || j > 0)) {
                    // tile 0 waits for tile 1's block j-1, tile 1 for tile 0's block j
                    const uint32_t par = (uint32_t)((t == 1 ? j : j - 1) & 1);
                    if (!mbar_wait(&exp_turn[t], par, p.d_status, KST_WAIT_SOFTMAX, abort_flag)) { ok = false; break; }
                }
                if (lane == 0 && quad == 0 && j < 6) ATT_TRACE(64 * t + 8 + 8 * j + 5);  // rescale done, my turn
                // P = 2^(s*scale - m): fp32 exponentials, their fp32 row sum, and P rounded to fp16
                // (two keys per 32-bit column) straight into tensor memory for the P V product.
                const uint64_t sc2 = pack2(sce, sce), nm2 = pack2(-m_sub, -m_sub);
                uint64_t lsa = pack2(0.f, 0.f), lsb = pack2(0.f, 0.f);
                uint32_t pk[NC][16];
                bool pv_seen = false;   // asked half way, so that the answer is there when it is needed
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    if (FREE && c == NC / 2) pv_seen = j == 0 || mbar_test_wait(&pv_done[t], (uint32_t)((j - 1) & 1));
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        // two scores per FMA and per add (packed fp32 pairs), one ex2 each, one convert for the pair
                        const uint64_t x2 = fma2(pack2(__uint_as_float(r[c][2 * i]), __uint_as_float(r[c][2 * i + 1])), sc2, nm2);
                        float x0, x1;
                        unpack2(x2, x0, x1);
                        const float e0 = ex2(x0), e1 = ex2(x1);
                        if (i & 1) lsb = add2(lsb, pack2(e0, e1));
                        else lsa = add2(lsa, pack2(e0, e1));
                        const __half2 h2 = __floats2half2_rn(e0, e1);
                        pk[c][i] = *reinterpret_cast<const uint32_t*>(&h2);
                    }
                    if (!FREE) tmem_st16_raw(p_tmem + c * 16, pk[c]);
                    if (c == TURN_AT && NC == 4 && pingpong && (!FREE || j == 0)) {
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&exp_turn[1 - t]);
                    }
                    if (HALVES && c == NC / 2 - 1) {
                        tmem_wait_st();
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&p_half[t]);
                    }
                }
                if constexpr (FREE) {
                    pv_known = __all_sync(0xffffffffu, pv_seen);   // one answer per warp
                    if (__any_sync(0xffffffffu, m_new != m_run) && !rescale()) { ok = false; break; }
                    if (!pv_wait()) { ok = false; break; }
#pragma unroll
                    for (int c = 0; c < (Cfg::P_TAIL ? NC - 1 : NC); ++c) tmem_st16_raw(p_tmem + c * 16, pk[c]);
                    if (Cfg::P_TAIL) {
                        const uint32_t at = smem_u32(smem + Cfg::S_P + t * ATT_TILE_BYTES) + row * 128;
#pragma unroll
                        for (int c = 0; c < 4; ++c) st_shared16(at + ((c ^ (row & 7)) << 4), &pk[NC - 1][4 * c]);
                        fence_proxy_async_smem();
                    }
                }
                tmem_wait_st();
                float ls0, ls1;
                unpack2(add2(lsa, lsb), ls0, ls1);
                l_run = l_run * alpha + (ls0 + ls1);
                m_run = m_new;
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&p_full[t]);
                if (lane == 0 && quad == 0 && j < 6) ATT_TRACE(64 * t + 8 + 8 * j + 6);  // P written
                if (lane == 0 && j == 3) ATT_TRACE(56 + 64 * t + quad);                  // per-warp P written, block 3
            }

            // Epilogue: O / l to global through the caller's output strides.
            if (ok && nblk > 0)
                ok = mbar_wait(&pv_done[t], (uint32_t)((nblk - 1) & 1), p.d_status, KST_WAIT_SOFTMAX, abort_flag);
            constexpr int W = EP % 32 ? 16 : 32;   // columns a step
            if (JOIN) {
                cluster_sync_all();       // nobody in the cluster reads its K, V or Q any more
                met = true;
                const int share = (ITEM_ROWS + nsp - 1) / nsp, nch = p.E >> 2;   // rows a CTA finishes, fours of a row
                const int r = t * ATT_BR + row, owner = r / share, col = share * 16 + 16;
                const uint32_t to = mapa_u32(smem_u32(smem), owner);
                if (ok) {
                    tc_fence_after();
                    const uint32_t at = to + split * nch * col + (r - owner * share) * 16;
#pragma unroll 1
                    for (int c = 0; c < EP / W; ++c) {
                        uint32_t v[W];
                        tmem_ld(o_tmem + c * W, v);
                        tmem_wait_ld();
#pragma unroll
                        for (int i = 0; i < W; i += 4)
                            if (c * W + i < p.E) st_cluster_v4(at + (c * W + i) / 4 * col, v[i], v[i + 1], v[i + 2], v[i + 3]);
                    }
                    st_cluster_f32x2(to + nsp * nch * col + (split * share + r - owner * share) * 8, m_run, l_run);
                }
            } else if (ok) {
                tc_fence_after();
                const int lq = q0 + t * ATT_BR + row;
                if (nsp > 1) {
                    // Unnormalised rows and their (reference point, sum) for the merge.  tcgen05.ld is a
                    // warp-wide (.sync.aligned) instruction: every lane executes it, whether or not its
                    // row exists; only the stores are predicated.
                    const int64_t prow = ((int64_t)split * p.ntail + tailpair) * ITEM_ROWS + t * ATT_BR + row;
                    float* po = p.part_o + prow * p.E;
#pragma unroll 1
                    for (int c = 0; c < EP / W; ++c) {
                        uint32_t r[W];
                        tmem_ld(o_tmem + c * W, r);
                        tmem_wait_ld();
                        if (lq < p.Lq) {
#pragma unroll
                            for (int i = 0; i < W; i += 4)
                                if (c * W + i < p.E)
                                    *reinterpret_cast<float4*>(po + c * W + i) =
                                        make_float4(__uint_as_float(r[i]), __uint_as_float(r[i + 1]), __uint_as_float(r[i + 2]),
                                                    __uint_as_float(r[i + 3]));
                        }
                    }
                    if (lq < p.Lq) {
                        p.part_ml[prow * 2] = m_run;
                        p.part_ml[prow * 2 + 1] = l_run;
                    }
                } else {
                const float inv = 1.0f / (l_run == 0.f ? 1.0f : l_run);
                const int64_t obase = lq * p.osL + h * p.osH + b * p.osB;
#pragma unroll 1
                for (int c = 0; c < EP / W; ++c) {
                    uint32_t r[W];
                    tmem_ld(o_tmem + c * W, r);
                    tmem_wait_ld();
                    if (lq < p.Lq) {
                        if (p.out_f32) {
                            float* o = static_cast<float*>(p.out) + obase + c * W;
#pragma unroll
                            for (int i = 0; i < W; i += 4) {
                                if (c * W + i < p.E)
                                    *reinterpret_cast<float4*>(o + i) =
                                        make_float4(__uint_as_float(r[i]) * inv, __uint_as_float(r[i + 1]) * inv,
                                                    __uint_as_float(r[i + 2]) * inv, __uint_as_float(r[i + 3]) * inv);
                            }
                        } else {
                            __half* o = static_cast<__half*>(p.out) + obase + c * W;
#pragma unroll
                            for (int i = 0; i < W; i += 8) {
                                if (c * W + i < p.E) {
                                    uint4 w;
                                    __half2* hh = reinterpret_cast<__half2*>(&w);
#pragma unroll
                                    for (int u = 0; u < 4; ++u)
                                        hh[u] = __floats2half2_rn(__uint_as_float(r[i + 2 * u]) * inv,
                                                                  __uint_as_float(r[i + 2 * u + 1]) * inv);
                                    *reinterpret_cast<uint4*>(o + i) = w;
                                }
                            }
                        }
                    }
                }
                }   // nsplit == 1
            }
        }
        if constexpr (JOIN) {
            // Each CTA of the cluster finishes its share of the rows, in split order, as attention_merge_kernel does:
            // out = sum_s O_s 2^(m_s - M) / sum_s l_s 2^(m_s - M), M the largest reference point.
            if (!met) cluster_sync_all();
            met = true;
            cluster_sync_all();   // every part's rows are there
            // share <= 128 rows, so at least two threads a row, each every per-th four of it
            const int share = (ITEM_ROWS + nsp - 1) / nsp, nch = p.E >> 2;
            const int r0 = split * share, n = min(min(share, ITEM_ROWS - r0), p.Lq - q0 - r0), col = share * 16 + 16;
            const int per = 128 * NT / share, r = threadIdx.x / per;
            if (r < n) {
                const float2* ml = reinterpret_cast<const float2*>(smem + nsp * nch * col + r * 8);
                float w[JOIN_MOST], M = -INFINITY, den = 0.f;
                float2 f[JOIN_MOST];
#pragma unroll
                for (int s = 0; s < JOIN_MOST; ++s) f[s] = s < nsp ? ml[s * share] : make_float2(-INFINITY, 0.f);
#pragma unroll
                for (int s = 0; s < JOIN_MOST; ++s) M = fmaxf(M, f[s].x);
#pragma unroll
                for (int s = 0; s < JOIN_MOST; ++s) {
                    w[s] = (f[s].x == -INFINITY) ? 0.f : exp2f(f[s].x - M);
                    den = fmaf(f[s].y, w[s], den);
                }
                const float inv = 1.0f / (den == 0.f ? 1.0f : den);
                const int64_t at0 = (q0 + r0 + r) * p.osL + h * p.osH + b * p.osB;
#pragma unroll 2
                for (int c = threadIdx.x - r * per; c < nch; c += per) {
                    const uint8_t* o = smem + c * col + r * 16;
                    float4 v[JOIN_MOST], num = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                    for (int s = 0; s < JOIN_MOST; ++s)
                        if (s < nsp) v[s] = *reinterpret_cast<const float4*>(o + s * nch * col);
#pragma unroll
                    for (int s = 0; s < JOIN_MOST; ++s)
                        if (s < nsp) {
                            num.x = fmaf(v[s].x, w[s], num.x);
                            num.y = fmaf(v[s].y, w[s], num.y);
                            num.z = fmaf(v[s].z, w[s], num.z);
                            num.w = fmaf(v[s].w, w[s], num.w);
                        }
                    const int64_t at = at0 + 4 * c;
                    if (p.out_f32) {
                        *reinterpret_cast<float4*>(static_cast<float*>(p.out) + at) = make_float4(num.x * inv, num.y * inv, num.z * inv, num.w * inv);
                    } else {
                        uint2 h2;
                        *reinterpret_cast<__half2*>(&h2.x) = __floats2half2_rn(num.x * inv, num.y * inv);
                        *reinterpret_cast<__half2*>(&h2.y) = __floats2half2_rn(num.z * inv, num.w * inv);
                        *reinterpret_cast<uint2*>(static_cast<__half*>(p.out) + at) = h2;
                    }
                }
            }
        }
    }

    if (JOIN && !met) {   // the roles without rows: the two barriers of a join
        cluster_sync_all();
        cluster_sync_all();
    }
    if (JOIN && p.pair_ctas > 0) grid_dep_wait();
    if (*abort_flag) {
        for (int i = 0; i < 4; ++i) __nanosleep(1000000);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == Cfg::TMA_WARP) {
        tc_fence_after();
        tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
    }
}

// Combine the partial results of a key split (attn_flash_cm_merge!, flash.jl:1398-1421): one warp per
// query row; out = sum_s O_s 2^(m_s - M) / sum_s l_s 2^(m_s - M), M the largest reference point.
__global__ void __launch_bounds__(128)
attention_merge_kernel(const float* __restrict__ part_o, const float* __restrict__ part_ml, int nsplit, int ntail,
                       int first_pair, int qpairs, int item_rows, int E, int Lq, int H, void* out, int64_t osL, int64_t osH,
                       int64_t osB, int out_f32) {
    grid_dep_wait();
    const int lane = threadIdx.x & 31;
    const int64_t rows = (int64_t)ntail * item_rows;
    const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= rows) return;
    const int pair = first_pair + (int)(row / item_rows);
    const int lq = (pair % qpairs) * item_rows + (int)(row % item_rows);
    if (lq >= Lq) return;
    const int h = (pair / qpairs) % H, b = pair / (qpairs * H);
    float M = -INFINITY;
    for (int s = 0; s < nsplit; ++s) M = fmaxf(M, part_ml[(s * rows + row) * 2]);
    float den = 0.f, num[4] = {0.f, 0.f, 0.f, 0.f};   // E <= 128: up to four elements per lane
    for (int s = 0; s < nsplit; ++s) {
        const float m = part_ml[(s * rows + row) * 2], l = part_ml[(s * rows + row) * 2 + 1];
        const float w = (m == -INFINITY) ? 0.f : exp2f(m - M);
        den = fmaf(l, w, den);
        const float* po = part_o + (s * rows + row) * E;
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (lane + 32 * u < E) num[u] = fmaf(po[lane + 32 * u], w, num[u]);
    }
    const float inv = 1.0f / (den == 0.f ? 1.0f : den);
    const int64_t obase = lq * osL + h * osH + b * osB;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        if (lane + 32 * u >= E) continue;
        if (out_f32) static_cast<float*>(out)[obase + lane + 32 * u] = num[u] * inv;
        else static_cast<__half*>(out)[obase + lane + 32 * u] = __float2half_rn(num[u] * inv);
    }
}

// Scalar path for operands a tensor map cannot express (E > 128, E not a multiple of 8,
// unaligned strides): one warp per query row, two passes over the keys.
__global__ void attention_f16_scalar_kernel(int E, int Lq, int Lk, int H, int B, const __half* q, int64_t qsE, int64_t qsL, int64_t qsH, int64_t qsB,
                                            const __half* k, int64_t ksE, int64_t ksL, int64_t ksH, int64_t ksB,
                                            const __half* v, int64_t vsE, int64_t vsL, int64_t vsH, int64_t vsB,
                                            void* out, int64_t osL, int64_t osH, int64_t osB, int out_f32, float scale,
                                            const __half* bias, int64_t bsK, int64_t bsQ, int64_t bsH, int64_t bsB) {
    const int lane = threadIdx.x & 31;
    const int64_t rowid = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (rowid >= (int64_t)Lq * H * B) return;
    const int lq = (int)(rowid % Lq);
    const int h = (int)((rowid / Lq) % H);
    const int b = (int)(rowid / ((int64_t)Lq * H));
    const __half* qp = q + qsL * lq + qsH * h + qsB * b;
    const __half* kp = k + ksH * h + ksB * b;
    const __half* vp = v + vsH * h + vsB * b;
    const __half* bp = bias ? bias + bsQ * lq + bsH * h + bsB * b : nullptr;
    float m = -INFINITY;
    for (int lk = lane; lk < Lk; lk += 32) {
        float a = 0.f;
        for (int e = 0; e < E; ++e) a = fmaf(__half2float(qp[qsE * e]), __half2float(kp[ksL * lk + ksE * e]), a);
        a *= scale;
        if (bp) a += __half2float(bp[bsK * lk]);
        m = fmaxf(m, a);
    }
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (m == -INFINITY) m = 0.f;   // every key blocked: all exponentials are zero and the row divides by one
    // Each lane accumulates its own keys into E partial outputs held two per lane-pass.
    float l = 0.f;
    extern __shared__ float acc_sm[]; // [warps][E]
    float* acc = acc_sm + (threadIdx.x >> 5) * E;
    for (int e = lane; e < E; e += 32) acc[e] = 0.f;
    __syncwarp();
    for (int lk0 = 0; lk0 < Lk; lk0 += 32) {
        const int lk = lk0 + lane;
        float pexp = 0.f;
        if (lk < Lk) {
            float a = 0.f;
            for (int e = 0; e < E; ++e) a = fmaf(__half2float(qp[qsE * e]), __half2float(kp[ksL * lk + ksE * e]), a);
            a *= scale;
            if (bp) a += __half2float(bp[bsK * lk]);
            pexp = __expf(a - m);
            l += pexp;
            pexp = __half2float(__float2half_rn(pexp));
        }
        for (int t = 0; t < 32 && lk0 + t < Lk; ++t) {
            const float pt = __shfl_sync(0xffffffffu, pexp, t);
            for (int e = lane; e < E; e += 32) acc[e] = fmaf(pt, __half2float(vp[vsL * (lk0 + t) + vsE * e]), acc[e]);
        }
    }
    for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    const float inv = 1.0f / (l == 0.f ? 1.0f : l);
    const int64_t obase = lq * osL + h * osH + b * osB;
    for (int e = lane; e < E; e += 32) {
        if (out_f32) static_cast<float*>(out)[obase + e] = acc[e] * inv;
        else static_cast<__half*>(out)[obase + e] = __float2half_rn(acc[e] * inv);
    }
}

// ----------------------------------------------------------------------- the two-GEMM route
// Attention as two batched tensor-core GEMMs with a softmax between them, for head dims the fused kernel's
// tensor memory cannot hold (E > 128): S(Lk, Lq) = Kt(Lk, E) . Q(E, Lq) in fp32, P = softmax over the keys
// (fp16, already divided by the row sum), O(E, Lq) = V(E, Lk) . P(Lk, Lq) written straight into out.  The
// reference's second tier, sdpa_coopmat! + attn_softmax_rows! (attention.jl:528-705), restated for this
// GEMM's orientation: only K is transposed (one permuted copy), Q and V are read through their strides, and
// the scores keep the keys contiguous so that the softmax reads and writes whole rows.
//
// One warp per (query, head*batch) column of S: scale (+ additive mask), maximum, exponentials, sum, P.  A
// column whose keys are all blocked comes out as zeros (attn_softmax, attention.jl:73-100).
__global__ void __launch_bounds__(256)
attn_softmax_cols_kernel(const float* __restrict__ S, __half* __restrict__ P, int Lk, int64_t ldS, int CH, int64_t ncols,
                         float scale, const __half* __restrict__ bias, int64_t bsK, int64_t bsQ, int64_t bsH, int64_t bsB,
                         int q0, int Lq, int H) {
    const int lane = threadIdx.x & 31;
    const int64_t col = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);   // lq_local + CH * hb
    if (col >= ncols) return;
    const int lq = q0 + (int)(col % CH);
    if (lq >= Lq) return;   // a short last chunk: the columns past it hold an earlier chunk's scores and are not used
    const int hb = (int)(col / CH);
    const float* s = S + col * ldS;
    __half* p = P + col * ldS;
    const __half* bp = bias ? bias + (int64_t)lq * bsQ + (int64_t)(hb % H) * bsH + (int64_t)(hb / H) * bsB : nullptr;
    float m = -INFINITY;
    for (int k = lane; k < Lk; k += 32) {
        float a = s[k] * scale;
        if (bp) a += __half2float(bp[(int64_t)k * bsK]);
        m = fmaxf(m, a);
    }
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (m == -INFINITY) m = 0.f;
    float l = 0.f;
    for (int k = lane; k < Lk; k += 32) {
        float a = s[k] * scale;
        if (bp) a += __half2float(bp[(int64_t)k * bsK]);
        l += __expf(a - m);
    }
    for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    const float inv = 1.0f / (l == 0.f ? 1.0f : l);
    for (int k = lane; k < Lk; k += 32) {
        float a = s[k] * scale;
        if (bp) a += __half2float(bp[(int64_t)k * bsK]);
        p[k] = __float2half_rn(__expf(a - m) * inv);
    }
}

static int attention_two_gemm(b200_ctx* ctx, int64_t E, int64_t Lq, int64_t Lk, int64_t H, int64_t B,
                              const b200_strided4* q, const b200_strided4* k, const b200_strided4* v,
                              const __half* bias, const int64_t* bs, const b200_strided4* o, int out_dtype, float scale) {
    const int64_t HB = H * B;
    const size_t osz = out_dtype == B200_F16 ? 2 : 4;
    int rc;
    // Kt(Lk, E, H, B), dense: the one layout pass of this route (the reference transposes Q and V as well)
    void* kT = nullptr;
    if ((rc = ws_scratch(ctx, (size_t)(Lk * E * HB) * 2, &kT))) return rc;
    {
        const int64_t shape[4] = {Lk, E, H, B};
        const int64_t stride[4] = {k->stride[1], 1, k->stride[2], k->stride[3]};
        if ((rc = b200_permute4(ctx, k->ptr, kT, shape, stride, 2))) return rc;
    }
    // Queries are taken in chunks so that the fp32 scores and the fp16 probabilities stay within ~256 MB.
    int64_t CH = (int64_t)(256ll << 20) / (Lk * HB * 6);
    if (CH > Lq) CH = Lq;
    CH = CH / 8 * 8;
    if (CH < 8) CH = Lq < 8 ? Lq : 8;
    void *S = nullptr, *P = nullptr;
    if ((rc = ws_scratch(ctx, (size_t)(Lk * CH * HB) * 4, &S))) return rc;
    if ((rc = ws_scratch(ctx, (size_t)(Lk * CH * HB) * 2, &P))) return rc;
    // One batched launch over (h, b) when the operands' head and batch strides fold into one, else one per image.
    auto folds = [&](const b200_strided4* t) { return B == 1 || t->stride[3] == H * t->stride[2]; };
    const bool one = folds(q) && folds(v) && folds(o);
    const int64_t nb = one ? HB : H, reps = one ? 1 : B;
    for (int64_t q0 = 0; q0 < Lq; q0 += CH) {
        const int64_t n = Lq - q0 < CH ? Lq - q0 : CH;
        for (int64_t r = 0; r < reps; ++r) {
            const __half* qp = (const __half*)q->ptr + q0 * q->stride[1] + r * q->stride[3];
            if ((rc = gemm_f16_run(ctx, Lk, n, E, (const __half*)kT + r * H * Lk * E, Lk, qp, q->stride[1], nullptr, 0,
                                   (float*)S + r * H * Lk * CH, Lk, B200_F32, B200_EPI_NONE, nb, Lk * E, q->stride[2],
                                   Lk * CH)))
                return rc;
        }
        const int64_t ncols = CH * HB;
        attn_softmax_cols_kernel<<<(unsigned)cdiv(ncols, 8), 256, 0, ctx->stream>>>(
            (const float*)S, (__half*)P, (int)Lk, Lk, (int)CH, ncols, scale, bias, bs[0], bs[1], bs[2], bs[3], (int)q0, (int)Lq,
            (int)H);
        ctx->launches++;
        B200_CUDA(cudaGetLastError());
        for (int64_t r = 0; r < reps; ++r) {
            const __half* vp = (const __half*)v->ptr + r * v->stride[3];
            char* op = (char*)const_cast<void*>(o->ptr) + (size_t)(q0 * o->stride[1] + r * o->stride[3]) * osz;
            if ((rc = gemm_f16_run(ctx, E, n, Lk, vp, v->stride[1], (const __half*)P + r * H * Lk * CH, Lk, nullptr, 0, op,
                                   o->stride[1], out_dtype, B200_EPI_NONE, nb, v->stride[2], Lk * CH, o->stride[2])))
                return rc;
        }
    }
    return B200_OK;
}

static int tc_reason(int64_t E, int64_t Lq, int64_t Lk, int64_t H, int64_t B, const int64_t* qs,
                     const int64_t* ks, const int64_t* vs) {
    if (E < 1 || Lq < 1 || Lk < 1 || H < 1 || B < 1) return B200_DECLINE_EXTENT;
    if (E > 128 || E % 8 != 0) return B200_DECLINE_TILING;
    if (H > 65535 || B > 65535 || Lq >= (1ll << 31) || Lk >= (1ll << 31)) return B200_DECLINE_EXTENT;
    const int64_t* ss[3] = {qs, ks, vs};
    for (int i = 0; i < 3; ++i) {
        const int64_t ext[4] = {E, i == 0 ? Lq : Lk, H, B};
        if (ss[i][0] != 1) return B200_DECLINE_ALIGN;
        // A tensor map wants every stride a multiple of 16 bytes; an axis of extent one is
        // never stepped along, so its stride is free.
        for (int d = 1; d < 4; ++d)
            if (ext[d] > 1 && (ss[i][d] % 8 != 0 || ss[i][d] <= 0)) return B200_DECLINE_ALIGN;
    }
    return B200_OK;
}

static int make_qkv_map(b200_ctx* ctx, CUtensorMap* m, const b200_strided4* t, int64_t E, int64_t L,
                        int64_t H, int64_t B, uint32_t rows) {
    uint64_t dims[4] = {(uint64_t)E, (uint64_t)L, (uint64_t)H, (uint64_t)B};
    // A unit-extent axis may carry any stride; give the encoder a legal one.
    auto st = [&](int d, uint64_t fallback) {
        uint64_t s = (uint64_t)t->stride[d] * 2;
        return (dims[d] == 1 || s == 0) ? fallback : s;
    };
    uint64_t s1 = st(1, (uint64_t)E * 2 < 16 ? 16 : (uint64_t)((E * 2 + 15) / 16 * 16));
    uint64_t s2 = st(2, s1 * (uint64_t)L);
    uint64_t s3 = st(3, s2 * (uint64_t)H);
    uint64_t str[3] = {s1, s2, s3};
    uint32_t box[4] = {64, rows, 1, 1};   // one swizzle atom; a head dim above 64 takes two boxes per tile
    return make_tmap(ctx, m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, t->ptr, dims, str, box,
                     CU_TENSOR_MAP_SWIZZLE_128B);
}

// How many clusters of 2 to JOIN_MOST CTAs of an SM each the GPU holds at once (a GPC's SMs do not divide without a rest: 45 of
// three, not 49): asked once per device.
struct AttRooms { int clusters[JOIN_MOST + 1]; };
static const AttRooms& att_rooms(b200_ctx* ctx) {
    static std::once_flag once[16];
    static AttRooms rooms[16];
    const int d = ctx->device & 15;
    std::call_once(once[d], [&] {
        using Cfg = AttCfg<64>;
        auto kern = attention_f16_tc_kernel<64, false, 2, false>;
        AttRooms& got = rooms[d];
        got = {};
        if (cudaSetDevice(ctx->device) != cudaSuccess ||
            cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES) != cudaSuccess) {
            cudaGetLastError();
            return;
        }
        for (int n = 2; n <= JOIN_MOST; ++n) {
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = (unsigned)n;
            attr[0].val.clusterDim.y = 1;
            attr[0].val.clusterDim.z = 1;
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3((unsigned)(ctx->prop.multiProcessorCount / n * n), 1, 1);
            cfg.blockDim = dim3(Cfg::THREADS, 1, 1);
            cfg.dynamicSmemBytes = Cfg::SMEM_BYTES;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            int fit = 0;
            if (cudaOccupancyMaxActiveClusters(&fit, kern, &cfg) == cudaSuccess) got.clusters[n] = fit;
            else cudaGetLastError();
        }
    });
    return rooms[d];
}

// Over how many CTAs the keys of each of `pairs` items are cut, and whether those are a cluster that joins its rows in the launch.
// The estimate beside a call's start, in us, fitted to 250 shapes of 2 to 18 heads and 400 to 2040 keys (2 to 7 % off): `block` and
// `load` x the SMs used per key block, a cluster's `join`, or a second launch that merges (`merge` and `rows` x the parts' rows / 256).
// Items of one tile have few rows to merge and do not join (16 heads, 40 x 8192 x 128: 24.9 us merged, 29.0); clusters that would
// fill their room exactly may take two rounds (45 of three: 14.9 us and 23).
// A join is the cheapest cut wherever its clusters are resident at once: 1.05 to 1.65 times as fast as merging, 1.29 in the mean
// (9 heads x 2040 x 64 28.0 -> 21.5 us, 18 x 1020 22.2 -> 15.0, 12 x 900 x 128 23.2 -> 18.9); two and three key blocks, and many
// pairs of four, stay whole (12 heads x 400: 9.9 us, 13.0 merged).  More than eight parts are worth a merge where pairs are few.
// The tail of `waves` full rounds of items is cut the same way.  Its clusters wait for SMs of one group that fall free one by one, up
// to 7 % of the rounds apart: joined rather than merged, 12 heads x 4096 x 4096 x 64 80.3 -> 76.9 us, x 1200 39.3 -> 34.1, 10 heads x
// 4096 x 4096 x 72 80.0 -> 71.9, but x 8000 138.6 -> 140.7.  Wider heads take three-CTA clusters up to one short of their room
// (44 of 45, 12 heads x 4096 x 4096 x 72: 89.5 -> 103.5, two rounds of them).  Masked tails go on merging, their CTAs' ends lie
// further apart (12 heads x 4096 x 4096 111.6 -> 117.3, 14 x 2900 86.1 -> 89.8; short ones would gain, 38 x 1024 x 640 31.1 -> 29.4).
struct AttSplit { int parts; bool join; };
static AttSplit att_split(b200_ctx* ctx, int64_t pairs, int64_t nblk, int64_t Lq, int64_t E, bool masked, int64_t waves, double staged) {
    struct Cost { double block, load, join, merge, rows; };
    static const Cost costs[5] = {{1.35, 0.37, 3.65, 4.15, 0.035}, {1.44, 0.57, 4.4, 4.75, 0.038}, {1.83, 0.46, 4.7, 5.4, 0.038},
                                  {2.07, 0.56, 3.9, 5.15, 0.035}, {2.44, 0.77, 4.7, 5.6, 0.042}};
    const Cost& c = costs[masked ? 3 + (E > 64) : (E > 64) + (E > 80)];
    const int64_t sms = ctx->prop.multiProcessorCount;
    auto walk = [&](int64_t n) { return (double)cdiv(nblk, n) * (c.block + staged + c.load * (double)(pairs * n) / (double)sms); };
    const AttRooms& rooms = att_rooms(ctx);
    AttSplit best = {1, false};
    double least = walk(1);
    const double apart = 0.07 * ((double)(waves * nblk) * (c.block + c.load) - 20.0);
    const double join = c.join + (apart > 0.0 ? apart : 0.0);
    for (int n = 2; n <= JOIN_MOST && n <= nblk && Lq > ATT_BR && !(waves && masked); ++n)
        if (pairs + (waves && E > 64) < rooms.clusters[n] + (n == 2) && walk(n) + join < least) {
            least = walk(n) + join;
            best = {n, true};
        }
    int64_t n = sms / pairs;
    if (n > nblk / 2) n = nblk / 2;
    if (n > 64) n = 64;
    if (n >= 2 && walk(n) + c.merge + c.rows * (double)(pairs * n) * (Lq < 2 * ATT_BR ? (double)Lq / (2 * ATT_BR) : 1.0) < least) best = {(int)n, false};
    return best;
}

// A mask whose rows lie on 16-byte boundaries: one warp a row.  Any strides; rows of contiguous keys are read by words from the 4-byte
// boundary at or below each eight's first entry, every word holding one.  What is behind a row's last key in its last eight is what
// the last word had there or zero; the tensor map's extent ends before it.
__global__ void __launch_bounds__(256)
mask_rows_kernel(const __half* __restrict__ mask, uint4* __restrict__ out, int Lq, int Lk, int64_t rows, int planesH, int64_t bsK,
                 int64_t bsQ, int64_t bsH, int64_t bsB) {
    grid_dep_wait();
    grid_dep_launch();
    const int lane = threadIdx.x & 31;
    const int64_t row = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (row >= rows) return;
    const int64_t plane = row / Lq;
    const __half* src = mask + (row - plane * Lq) * bsQ + (plane % planesH) * bsH + (plane / planesH) * bsB;
    const int n8 = (Lk + 7) / 8;
    uint4* dst = out + row * n8;
    for (int c = lane; c < n8; c += 32) {
        const int n = min(8, Lk - c * 8);
        uint32_t v[4] = {0, 0, 0, 0};
        if (bsK == 1) {
            const uintptr_t a = reinterpret_cast<uintptr_t>(src + c * 8);
            const uint32_t* w = reinterpret_cast<const uint32_t*>(a & ~(uintptr_t)3);
            const int odd = (int)(a >> 1) & 1, words = (n + odd + 1) >> 1;
            uint32_t x[5];
#pragma unroll
            for (int i = 0; i < 5; ++i) x[i] = i < words ? __ldg(w + i) : 0;
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] = __funnelshift_r(x[i], x[i + 1], 16 * odd);
        } else {
#pragma unroll
            for (int i = 0; i < 8; ++i)
                if (i < n) v[i >> 1] |= (uint32_t)__half_as_ushort(src[(int64_t)(c * 8 + i) * bsK]) << (16 * (i & 1));
        }
        dst[c] = make_uint4(v[0], v[1], v[2], v[3]);
    }
}

// What a mask's way to the softmax costs, in us.
// The softmax warps' own staging: `block` for every key block of a CTA, 0.2 of it for the first, whose entries are waited for either way.
// 1.1 by copies of 8 bytes, 1.2 so beside wider heads, 2.5 by words, less for the warps of a tile that have no rows (0.4 of it for 32
// queries); entry by entry, keys apart, 6 and for the first as well.
// `copy`: a launch that lays the rows on 16-byte boundaries for the tensor map, 1.4, 0.9 per million entries and 0.3 for every trip of a
// row's warp, 256 keys (keys apart 2 and 8 per million).
// Fitted to 930 masks of 9 to 3900 queries and 50 to 9000 keys, either way taken: the cheaper one by this is 0.4 % off in the mean and 1.13
// at worst (always the copy 5 %, never 7 %).  20 heads x 1500 x 1500 42.1 -> 36.9 us, 2 x 8 x 1001 x 1001 31.1 -> 26.7, 4 x 20 x 1001 x 1001 x 32 88.8 -> 62.6; 2 x 2001 x
// 2001 x 128 would go 24.6 -> 26.8, 8 x 100 x 3001 16.2 -> 17.9, 16 x 35 x 4391 x 128 26.5 -> 32.2 and one block, 2 x 32 x 575 x 50, 14.4 -> 16.3.
// Keys apart, 20 x 1500 x 1500 193 -> 92, 4 x 300 x 300 44.6 -> 14.5.  The workspace keeps what a copy took and half as much again, so
// there is a most to it: 256 MiB are 11584 x 11584 entries, and a larger mask is read in place, as every one that is not copied.
constexpr int64_t MASK_COPY_MOST = (int64_t)256 << 20;
struct MaskWay {
    bool lies;      // rows on 16-byte boundaries: the map is over the mask itself
    bool apart;
    double block, copy;
    int64_t rows, bytes;   // of a copy
    bool copied(int64_t blocks, int64_t walks) const {
        return block * ((double)blocks - (apart ? 0.0 : 0.8 * (double)walks)) >= copy && bytes <= MASK_COPY_MOST;
    }
};
static MaskWay mask_way(const __half* bptr, const int64_t* bs, int64_t E, int64_t Lq, int64_t Lk, int64_t H, int64_t B, int mask) {
    const int64_t ext[4] = {Lk, Lq, bs[2] != 0 ? H : 1, bs[3] != 0 ? B : 1};
    MaskWay w;
    w.lies = (bs[0] == 1 || Lk == 1) && reinterpret_cast<uintptr_t>(bptr) % 16 == 0;
    for (int d = 1; d < 4; ++d) w.lies = w.lies && (ext[d] == 1 || (bs[d] > 0 && bs[d] % 8 == 0 && bs[d] < (1ll << 38)));
    w.apart = mask == MASK_DIRECT;
    w.rows = Lq * ext[2] * ext[3];
    w.bytes = w.rows * cdiv(Lk, 8) * 16;
    const double entries = (double)(w.rows * Lk);
    if (w.apart) {
        w.block = Lq < 2 * ATT_BR ? 6.0 * (double)Lq / (2 * ATT_BR) : 6.0;
        w.copy = 2.0 + 8e-6 * entries;
    } else {
        w.block = (mask == MASK_WORDS ? 2.5 : E <= 64 ? 1.1 : 1.2) * (Lq < ATT_BR ? 0.2 + 0.8 * (double)Lq / ATT_BR : 1.0);
        w.copy = 1.4 + 0.9e-6 * entries + 0.3 * (double)cdiv(Lk, 256);
    }
    return w;
}

// The mask's tensor map, over the mask itself where its rows lie on 16-byte boundaries, else over a copy of it whose rows do
// where that is worth a launch.  Leaves p->mask as it is where neither is to be had.
// Nor where many CTAs fetch boxes of few keys, rows of parts of a line, the same ones at the same time, and each waits for its first: 80
// items of 144 queries x 8 keys 7.2 us staged, 10.7; x 24 7.3, 9.0; of 29 queries x 72 5.8, 6.7; x 64 and x 128 gain (0.95, 0.94 of
// the staged time), and so do launches of up to some 48 items (16 x 99 x 96: 5.5, 5.0).
// `blocks`: key blocks a CTA walks, `walks`: from how many first ones; `items`: of two tiles.
static int mask_map(b200_ctx* ctx, const __half* bptr, const int64_t* bs, const MaskWay& way, int64_t Lq, int64_t Lk, int64_t H, int64_t B,
                    int64_t blocks, int64_t walks, int64_t items, AttnParams* p, CUtensorMap* tm) {
    const int64_t ext[4] = {Lk, Lq, bs[2] != 0 ? H : 1, bs[3] != 0 ? B : 1};
    uint64_t dims[4], str[3], dense = (uint64_t)cdiv(Lk, 8) * 16;   // a legal stride for an axis of extent one
    for (int d = 0; d < 4; ++d) {
        dims[d] = (uint64_t)ext[d];
        if (d == 0) continue;
        str[d - 1] = way.lies && ext[d] != 1 ? (uint64_t)bs[d] * 2 : dense;
        dense *= (uint64_t)ext[d];
    }
    if (way.lies && items > 48 && Lk < 128 && Lk != 64 && (Lk < 64 || Lq < ATT_BR)) return B200_OK;
    const void* base = bptr;
    if (!way.lies) {
        const size_t mark = ctx->ws_used;
        void* ws = nullptr;
        if (!way.copied(blocks, walks)) {
            // A context's first masked call leaves it a workspace, if only the smallest: one recorded later finds room for a small copy.
            if (ctx->ws_buf == nullptr && ws_scratch(ctx, 0, &ws) == B200_OK) ctx->ws_used = mark;
            return B200_OK;
        }
        const int rc = ws_scratch(ctx, (size_t)way.bytes, &ws);
        if (rc == B200_ENOMEM) return B200_OK;
        if (rc) return rc;
        B200_CUDA(launch_dep(mask_rows_kernel, dim3((unsigned)cdiv(way.rows, 8), 1, 1), dim3(256, 1, 1), 0, ctx->stream, 1, bptr, (uint4*)ws,
                             (int)Lq, (int)Lk, way.rows, (int)ext[2], bs[0], bs[1], bs[2], bs[3]));
        ctx->launches++;
        base = ws;
    }
    uint32_t box[4] = {64, ATT_BR, 1, 1};
    const int rc = make_tmap(ctx, tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, base, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
    p->mask = MASK_TMA;
    return B200_OK;
}

} // namespace b200

using namespace b200;

extern "C" {

int b200_attention_f16_supported(int64_t E, int64_t Lq, int64_t Lk, int64_t H, int64_t B,
                                 const int64_t* qstride, const int64_t* kstride, const int64_t* vstride,
                                 int has_bias) {
    (void)has_bias;   // an additive mask no longer declines: b200_attention_f16_bias takes it
    if (!qstride || !kstride || !vstride) return B200_EINVAL;
    return tc_reason(E, Lq, Lk, H, B, qstride, kstride, vstride);
}

int b200_attention_f16_route(int64_t E, int64_t Lq, int64_t Lk, int64_t H, int64_t B, const int64_t* qstride,
                             const int64_t* kstride, const int64_t* vstride) {
    if (!qstride || !kstride || !vstride) return -1;
    if (tc_reason(E, Lq, Lk, H, B, qstride, kstride, vstride) == B200_OK) return 0;
    // Two batched GEMMs and a softmax: head dims past the fused kernel's, when the GEMM's tensor maps can take the
    // operands as they lie (E contiguous and a multiple of 8) and the problem is worth three launches.
    if (E > 128 && E % 8 == 0 && E <= 4096 && Lq >= 1 && Lk >= 1 && H >= 1 && B >= 1 && Lk < (1ll << 31) && Lq < (1ll << 31) &&
        qstride[0] == 1 && kstride[0] == 1 && vstride[0] == 1 && Lq * Lk >= 64 * 64)
        return 1;
    return 2;
}

int b200_attention_f16(b200_ctx* ctx, int64_t E, int64_t Lq, int64_t Lk, int64_t H, int64_t B,
                       const b200_strided4* q, const b200_strided4* k, const b200_strided4* v, void* out,
                       int out_dtype, float scale) {
    b200_strided4 o;
    o.ptr = out;
    o.stride[0] = 1;
    o.stride[1] = E;
    o.stride[2] = E * Lq;
    o.stride[3] = E * Lq * H;
    return b200_attention_f16_strided(ctx, E, Lq, Lk, H, B, q, k, v, &o, out_dtype, scale);
}

int b200_attention_f16_strided(b200_ctx* ctx, int64_t E, int64_t Lq, int64_t Lk, int64_t H, int64_t B,
                               const b200_strided4* q, const b200_strided4* k, const b200_strided4* v,
                               const b200_strided4* o, int out_dtype, float scale) {
    return b200_attention_f16_bias(ctx, E, Lq, Lk, H, B, q, k, v, nullptr, o, out_dtype, scale);
}

int b200_attention_f16_bias(b200_ctx* ctx, int64_t E, int64_t Lq, int64_t Lk, int64_t H, int64_t B,
                            const b200_strided4* q, const b200_strided4* k, const b200_strided4* v,
                            const b200_strided4* bias, const b200_strided4* o, int out_dtype, float scale) {
    B200_REQUIRE(ctx && q && k && v && o, B200_EINVAL, "attention: null argument");
    const __half* bptr = (bias != nullptr) ? static_cast<const __half*>(bias->ptr) : nullptr;
    const int64_t bs[4] = {bptr ? bias->stride[0] : 0, bptr ? bias->stride[1] : 0, bptr ? bias->stride[2] : 0,
                           bptr ? bias->stride[3] : 0};
    void* out = const_cast<void*>(o->ptr);
    B200_REQUIRE(E >= 0 && Lq >= 0 && Lk >= 0 && H >= 0 && B >= 0, B200_EINVAL, "attention: negative extent");
    B200_REQUIRE(out_dtype == B200_F16 || out_dtype == B200_F32, B200_DECLINE_ELTYPE, "attention: out dtype %d",
                 out_dtype);
    if (E == 0 || Lq == 0 || H == 0 || B == 0) return B200_OK;
    B200_REQUIRE(out && q->ptr, B200_EINVAL, "attention: null array");
    B200_CUDA(cudaSetDevice(ctx->device));
    const size_t osz = out_dtype == B200_F16 ? 2 : 4;
    const int64_t oal = out_dtype == B200_F16 ? 8 : 4; // elements per 16-byte vector store
    B200_REQUIRE(o->stride[0] == 1, B200_DECLINE_ALIGN, "attention: out must be contiguous along E");
    const bool odense = o->stride[1] == E && (H == 1 || o->stride[2] == E * Lq) && (B == 1 || o->stride[3] == E * Lq * H);
    const bool oaligned = (Lq == 1 || o->stride[1] % oal == 0) && (H == 1 || o->stride[2] % oal == 0) &&
                          (B == 1 || o->stride[3] % oal == 0);
    if (Lk == 0) {
        // Softmax over no keys: every row is the all-blocked case, a zero row divided by one.
        B200_REQUIRE(odense, B200_DECLINE_ALIGN, "attention: Lk = 0 with a strided out");
        B200_CUDA(cudaMemsetAsync(out, 0, (size_t)(E * Lq * H * B) * osz, ctx->stream));
        return B200_OK;
    }
    B200_REQUIRE(k->ptr && v->ptr, B200_EINVAL, "attention: null array");
    auto al16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
    const bool tc = tc_reason(E, Lq, Lk, H, B, q->stride, k->stride, v->stride) == B200_OK && al16(q->ptr) &&
                    al16(k->ptr) && al16(v->ptr) && al16(out) && oaligned && scale > 0.f;
    if (!tc && b200_attention_f16_route(E, Lq, Lk, H, B, q->stride, k->stride, v->stride) == 1 && scale > 0.f &&
        o->stride[1] > 0 && o->stride[2] > 0 && o->stride[3] > 0)
        return attention_two_gemm(ctx, E, Lq, Lk, H, B, q, k, v, bptr, bs, o, out_dtype, scale);
    if (!tc) {
        B200_REQUIRE(E <= 1024, B200_DECLINE_EXTENT, "attention: E = %lld", (long long)E);
        const int wpb = 4;
        const int64_t rows = Lq * H * B;
        attention_f16_scalar_kernel<<<(unsigned)cdiv(rows, wpb), 32 * wpb, wpb * E * sizeof(float), ctx->stream>>>(
            (int)E, (int)Lq, (int)Lk, (int)H, (int)B, (const __half*)q->ptr, q->stride[0], q->stride[1],
            q->stride[2], q->stride[3], (const __half*)k->ptr, k->stride[0], k->stride[1], k->stride[2],
            k->stride[3], (const __half*)v->ptr, v->stride[0], v->stride[1], v->stride[2], v->stride[3], out,
            o->stride[1], o->stride[2], o->stride[3], out_dtype == B200_F32, scale, bptr, bs[0], bs[1], bs[2], bs[3]);
        ctx->launches++;
        B200_CUDA(cudaGetLastError());
        return B200_OK;
    }
    static bool attr_done[16] = {};
    if (!attr_done[ctx->device & 15]) {
        auto allow = [](auto kern, int bytes) { return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes); };
        B200_CUDA(allow(attention_f16_tc_kernel<64, false, 1, false>, AttCfg<64, false, 1>::SMEM_BYTES));
        B200_CUDA(allow(attention_f16_tc_kernel<64, false, 2, false>, AttCfg<64>::SMEM_BYTES));
        B200_CUDA(allow(attention_f16_tc_kernel<64, false, 2, true>, AttCfg<64>::SMEM_BYTES));
        B200_CUDA(allow(attention_f16_tc_kernel<64, true, 2, false>, AttCfg<64, true>::SMEM_BYTES));
        B200_CUDA(allow(attention_f16_tc_kernel<64, true, 2, true>, AttCfg<64, true>::SMEM_BYTES));
        B200_CUDA(allow(attention_f16_tc_kernel<80, false, 2, false>, AttCfg<80>::SMEM_BYTES));
        B200_CUDA(allow(attention_f16_tc_kernel<80, false, 2, true>, AttCfg<80>::SMEM_BYTES));
        B200_CUDA(allow(attention_f16_tc_kernel<128, false, 2, false>, AttCfg<128>::SMEM_BYTES));
        B200_CUDA(allow(attention_f16_tc_kernel<128, false, 2, true>, AttCfg<128>::SMEM_BYTES));
        B200_CUDA(allow(attention_f16_tc_kernel<128, true, 2, false>, AttCfg<128, true>::SMEM_BYTES));
        B200_CUDA(allow(attention_f16_tc_kernel<128, true, 2, true>, AttCfg<128, true>::SMEM_BYTES));
        attr_done[ctx->device & 15] = true;
    }
    // Many windows of at most 64 keys: bound by HBM and latency, not by the tensor pipe; the small-tile
    // kernel keeps four or six CTAs per SM in flight where this one's set-up would cost more than the arithmetic.
    if (bptr == nullptr && E <= 64 && Lk <= 64 && B * H * cdiv(Lq, 64) > 2 * ctx->prop.multiProcessorCount)
        return attention_window_launch(ctx, E, Lq, Lk, H, B, q, k, v, o, out_dtype, scale);
    // A few queries: their tile would be mostly empty (see attention_few.cu).
    if (attention_few_takes(ctx, E, Lq, Lk, H, B, bptr != nullptr))
        return attention_few_launch(ctx, E, Lq, Lk, H, B, q, k, v, bptr, bs, o, out_dtype, scale);
    const bool wide = E > 64;                              // two swizzle atoms along E
    const int64_t sms = ctx->prop.multiProcessorCount;
    // Up to 256 keys and more than two tiles per SM (16 x 16 windows): one tile per CTA, four CTAs per SM, so that one's
    // set-up, loads and hand-offs run under the others' arithmetic: 1024 x 2 heads of 256 x 256, E = 56: 118 -> 91 us,
    // 287 x 2 heads of 196 x 196, E = 64: 30.5 -> 26.9.  With long keys its blocks of 64 hold the tensor pipe as long as blocks of 128 (64 cycles a UMMA
    // whatever N), and it loses: 12 heads x 4096 x 4096 85.7 -> 126.7.
    const bool single = !wide && bptr == nullptr && Lk <= 256 && cdiv(Lq, ATT_BR) * H * B > 2 * sms;
    const int block = single ? AttCfg<64, false, 1>::BC : AttCfg<64>::BC;
    CUtensorMap tq, tk, tv;
    int rc;
    if ((rc = make_qkv_map(ctx, &tq, q, E, Lq, H, B, ATT_BR))) return rc;
    if ((rc = make_qkv_map(ctx, &tk, k, E, Lk, H, B, block))) return rc;
    if ((rc = make_qkv_map(ctx, &tv, v, E, Lk, H, B, block))) return rc;
    AttnParams p;
    p.E = (int)E; p.Lq = (int)Lq; p.Lk = (int)Lk; p.H = (int)H; p.B = (int)B;
    p.scale = scale;
    p.scale_log2 = scale * 1.4426950408889634f;
    p.out = out;
    p.osL = o->stride[1]; p.osH = o->stride[2]; p.osB = o->stride[3];
    p.out_f32 = out_dtype == B200_F32;
    p.d_status = ctx->d_status;
    p.trace = ctx->gemm_trace;
    p.bias = bptr;
    p.bsK = bs[0]; p.bsQ = bs[1]; p.bsH = bs[2]; p.bsB = bs[3];
    p.mask = !(bs[0] == 1 || Lk == 1) ? MASK_DIRECT
             : reinterpret_cast<uintptr_t>(bptr) % 8 == 0 && bs[1] % 4 == 0 && bs[2] % 4 == 0 && bs[3] % 4 == 0 ? MASK_EIGHTS : MASK_WORDS;
    CUtensorMap tm = tq;   // not read unless there is a mask
    MaskWay way = {};
    if (bptr) way = mask_way(bptr, bs, E, Lq, Lk, H, B, p.mask);
    const int64_t nblk_all = cdiv(Lk, block);
    const int64_t item_rows = single ? ATT_BR : 2 * ATT_BR;
    auto launch = [&](dim3 grid, int cluster = 1) -> cudaError_t {
        auto go = [&](auto kern, int threads, size_t smem) {
            return launch_dep(kern, grid, dim3(threads, 1, 1), smem, ctx->stream, cluster, tq, tk, tv, tm, p);
        };
        if (single) return go(attention_f16_tc_kernel<64, false, 1, false>, AttCfg<64, false, 1>::THREADS, AttCfg<64, false, 1>::SMEM_BYTES);
        auto either = [&](auto ep, auto bias) {
            using Cfg = AttCfg<decltype(ep)::value, decltype(bias)::value>;
            return cluster > 1 ? go(attention_f16_tc_kernel<decltype(ep)::value, decltype(bias)::value, 2, true>, Cfg::THREADS, Cfg::SMEM_BYTES)
                               : go(attention_f16_tc_kernel<decltype(ep)::value, decltype(bias)::value, 2, false>, Cfg::THREADS, Cfg::SMEM_BYTES);
        };
        using Int64 = std::integral_constant<int, 64>;
        using Int80 = std::integral_constant<int, 80>;
        using Int128 = std::integral_constant<int, 128>;
        if (bptr) return wide ? either(Int128(), std::true_type()) : either(Int64(), std::true_type());
        return !wide ? either(Int64(), std::false_type()) : E <= 80 ? either(Int80(), std::false_type()) : either(Int128(), std::false_type());
    };
    p.qpairs = (int)cdiv(Lq, item_rows);
    const int64_t pairs = (int64_t)p.qpairs * H * B;      // work items: pairs of query tiles, or single tiles of short keys
    B200_REQUIRE(pairs < (1ll << 30), B200_DECLINE_EXTENT, "attention: too many query tiles");
    // Pairs that do not fill the SMs are cut along the keys (att_split): over a cluster's CTAs, which join their rows in the same
    // launch, or over more of them with a merge behind.  A last wave that would leave most SMs idle has its pairs cut the same way,
    // so that the wave is as short as that allows instead of a whole pair long.
    p.nsplit = 1;
    p.ntail = 0;
    p.part_o = p.part_ml = nullptr;
    int join = 1;   // CTAs of a cluster an item's keys are cut over
    const int64_t rem = pairs % sms;
    const bool tail = nblk_all >= 4 && pairs > sms && rem > 0 && 2 * rem <= sms;
    const size_t ws_mark = ctx->ws_used;
    const bool frugal = bptr != nullptr || Lq <= (E <= 64 ? 32 : 16);
    if (!single) {
        int64_t ntail = 0, ns = 1;
        if (2 * pairs <= sms || tail) {
            const double staged = bptr && !way.lies && !way.apart && !way.copied(cdiv(pairs, sms) * nblk_all, cdiv(pairs, sms)) ? way.block : 0.0;
            const AttSplit cut = att_split(ctx, tail ? rem : pairs, nblk_all, Lq, E, bptr != nullptr, tail ? pairs / sms : 0, staged);
            if (cut.join) {
                join = cut.parts;
            } else {
                ntail = tail ? rem : pairs;
                ns = cut.parts;
            }
        }
        if (ntail > 0 && ns >= 2) {
            const int64_t rows = ntail * item_rows;
            void* ws = nullptr;
            rc = ws_scratch(ctx, (size_t)(ns * rows * (E + 2)) * sizeof(float), &ws);
            // A masked call, and one of as few queries as attention_few.cu takes, does not depend on the workspace: it runs
            // unsplit when that is refused (a graph recorded without an eager call before), and gives its share back below.
            if (rc && !(frugal && rc == B200_ENOMEM)) return rc;
            if (!rc) {
                p.nsplit = (int)ns;
                p.ntail = (int)ntail;
                p.part_o = static_cast<float*>(ws);
                p.part_ml = p.part_o + ns * rows * E;
            }
        }
    }
    if (bptr) {
        const int64_t waves = join > 1 ? (tail ? pairs / sms : 0) : p.nsplit > 1 ? (pairs - p.ntail) / sms : cdiv(pairs, sms);
        const int64_t serial = waves * nblk_all + (join > 1 ? cdiv(nblk_all, join) : p.nsplit > 1 ? cdiv(nblk_all, p.nsplit) : 0);
        if ((rc = mask_map(ctx, bptr, bs, way, Lq, Lk, H, B, serial, waves + (join > 1 || p.nsplit > 1), pairs, &p, &tm))) return rc;
    }
    if (join > 1) {
        p.ntail = (int)(tail ? rem : pairs);
        p.pair_ctas = (int)(pairs - p.ntail);
        if (tail) {
            B200_CUDA(launch(dim3((unsigned)p.pair_ctas, 1, 1)));
            ctx->launches++;
        }
        p.nsplit = join;
        B200_CUDA(launch(dim3((unsigned)(p.ntail * join), 1, 1), join));
        ctx->launches++;
        if (frugal) ctx->ws_used = ws_mark;
        return B200_OK;
    }
    if (p.nsplit > 1) {
        p.pair_ctas = (int)(pairs - p.ntail);
        const int64_t ctas = p.pair_ctas + (int64_t)p.ntail * p.nsplit;
        B200_CUDA(launch(dim3((unsigned)ctas, 1, 1)));
        const int64_t rows = (int64_t)p.ntail * item_rows;
        B200_CUDA(launch_dep(attention_merge_kernel, dim3((unsigned)cdiv(rows, 4), 1, 1), dim3(128, 1, 1), 0, ctx->stream, 1,
                             (const float*)p.part_o, (const float*)p.part_ml, p.nsplit, p.ntail, p.pair_ctas, p.qpairs, (int)item_rows, (int)E,
                             (int)Lq, (int)H, out, o->stride[1], o->stride[2], o->stride[3], (int)(out_dtype == B200_F32)));
        ctx->launches += 2;
        if (frugal) ctx->ws_used = ws_mark;   // what comes next on the stream runs after the merge has read the partial rows
        return B200_OK;
    }
    // Split the pairs of a last wave that would leave more than half of the SMs idle — but not a
    // pair whose second tile does not exist.
    int64_t nsplit = (!single && pairs > sms && rem > 0 && 2 * rem <= sms && Lq % (2 * ATT_BR) == 0) ? rem : 0;
    p.pair_ctas = (int)(pairs - nsplit);
    B200_CUDA(launch(dim3((unsigned)(pairs + nsplit), 1, 1)));
    ctx->launches++;
    if (frugal) ctx->ws_used = ws_mark;   // a repacked mask, as above
    return B200_OK;
}

} // extern "C"
