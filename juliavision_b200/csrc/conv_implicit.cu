// Convolution as an implicit GEMM on the sm_100a tensor cores: the im2col matrix exists only as the shared-memory
// tiles the UMMAs read.  out(OW,OH,Cout,N) = act(bias + w * x); x (W,H,Cin,N), w (KW,KH,Cin,Cout), the general form of
// the reference's im2col + GEMM route (kernels/extern/conv_coopmat.jl:246-392).
//
// What bounds it: the gather, element by element, because a tap moves the image by one element and a TMA copy or a
// vector load by multiples of eight; and, with few input channels, the output's way to HBM.  Against the materialised
// matrix it saves that matrix's write and read and a launch; and because the pixels sit on the tensor-memory lanes,
// the store of one channel is 32 consecutive elements per warp whatever the alignment, so an image of any size runs
// on the tensor cores.
//
// One CTA takes 128 pixels of one image and up to 256 output channels, two CTAs per SM so that one's gather runs under
// the other's waits and store:
//   warps 0-7  gather: D's A operand, 64 rows (cin, kh, kw) x 128 pixels per k-block, pixels contiguous (MN-major),
//              written with the 128-byte swizzle.  A warp takes eight rows, whose tap is then uniform, and a lane two
//              pairs of neighbouring pixels of each, so that a load instruction touches one or two lines and a store
//              every bank once; four rows are loaded while the four before them are stored.
//              Afterwards the epilogue, TMEM -> +bias, round, act -> global
//   warp 8     TMA producer of the weight tile (K-major, straight from w)
//   warp 9     UMMA issuer
// In words and in runs, launches of more CTAs than that take four smaller ones per SM (CiCfg).
// Measured (us, B200) against the im2col + GEMM route: 1024 x 1024 x 3 -> 112, 7 x 7 / 4: 35 -> 23.6; 300 x 296 x 16 -> 64,
// 3 x 3: 42.5 -> 24.6; against the scalar GEMM odd pixel counts had: 43 x 42 x 256 -> 256, 3 x 3 / 2: 229 -> 14.2, two of
// 230 x 225 x 32 -> 80, 3 x 3: 890 -> 43.  What is left is the gather's load latency.
// An even stride takes the image in whole words instead (G): the pixels' first taps are then 8 (stride 4, 8, ...) or 4
// bytes apart, so one pixel's taps of a kernel row, with the element or two before or after them that fill the words, are
// two aligned loads, masked to the taps.  The reduction is laid out (cin, kh, G columns), G = 8 or 4, the weight the same
// with zeros between, the tile K-major: a thread's pixel and eight columns are one 16-byte store.  A seventh and a third more
// columns than taps (7 x 7 / 4, 3 x 3 / 2) and a tenth of the instructions: us, before and
// now: 1024 x 1024 x 3 -> 112, 7 x 7 / 4 24.8 -> 17.0, eight of them 166 -> 93, 512 x 512 x 3 -> 64 18.4 -> 6.4, 3 x 3 / 2
// 256 x 256 x 32 -> 128 19.4 -> 9.2, 128 x 128 x 128 -> 256 22.5 -> 18.1.  What is left is a CTA's chain of latencies.
// A convolution of stride one whose rows of results are as long as the image's (3 x 3 padded by 1) is read in runs: the taps of eight
// neighbouring pixels are eight elements in a row in memory, over the ends of image rows as well, so a thread reads the two aligned
// vectors they lie in, shifts them into place, blanks what is outside the image by bits it has worked out once, and stores a whole
// 16-byte piece of the tile; the reduction's order and bits are the taps'.  500 x 495 x 16 -> 40: 837 warp instructions a k-block and
// warp by taps; us, by taps and in runs: 64.6, 42.1, 1000 x 991 x 16 -> 32 267, 165, two of 106 x 97 x 136 -> 80 47.7, 35.4, two of 185 x
// 181 x 16 -> 56 19.4, 12.8, 300 x 296 x 16 -> 64 24.1, 17.5 (with the four smaller CTAs an SM; 57.3, -, 40.2, 18.9, 22.5 with two and
// dearer masks).
// A small image (fewer CTAs than the GPU holds) splits the reduction over the CTAs of a cluster, whose fp32 tiles
// meet in distributed shared memory, added in rank order.
#include <cuda_fp16.h>

#include <type_traits>

#include "act.cuh"
#include "internal.h"
#include "ptx.cuh"

namespace b200 {

constexpr int CI_PIX = 128;              // pixels per CTA (TMEM lanes)
constexpr int CI_BK = 64;                // one 128-byte swizzle row of the weight tile
constexpr int CI_A_BYTES = CI_PIX * CI_BK * 2;

// SMALL: half the gather warps and a third to half of the ring, four CTAs to an SM, for launches of more than two an SM read in
// words: a CTA's chain of waits is what takes the time, and four run beside each other (us on the device, two and four:
// 1024 x 1024 x 3 -> 112, 7 x 7 / 4 15.7, 14.2, eight of them 92.8, 72.6; 512 x 512 x 16 -> 64, 3 x 3 / 2 12.9, 12.0; launches that
// two an SM hold lose, 256 x 256 x 3 -> 96, 7 x 7 / 4 5.8, 6.9).  Issue slots are 45 % used then, the longest wait is for loads.
template <int BN, bool SMALL = false> struct CiCfg {
    static constexpr int GATHER = SMALL ? 128 : 256;   // gather / epilogue threads
    static constexpr int THREADS = GATHER + 64;
    static constexpr int CTAS = SMALL ? 4 : 2;
    static constexpr int STAGES = SMALL ? (BN == 64 ? 2 : 1) : BN == 256 ? 2 : (BN == 128 ? 3 : 4);
    static constexpr int B_BYTES = BN * CI_BK * 2;
    static constexpr int STAGE_BYTES = CI_A_BYTES + B_BYTES;
    static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + BN * 4 + 128;
    static constexpr bool SPLITS = !SMALL && BN * CI_PIX * 4 <= STAGES * STAGE_BYTES;   // the fp32 tile fits over the drained ring
    static_assert(CTAS * (SMEM_BYTES + 1024) <= 233472 && CTAS * BN <= 512, "shared or tensor memory over budget");
};

struct ConvParams {
    const __half* x;
    const __half* bias;
    void* out;
    int64_t x_img, out_img;   // elements from one image to the next
    int W, H, CRS, Cout, OW, P, tiles;   // tiles of CI_PIX pixels per image
    int sx, sy, px, py, dx, dy;
    int KW, KH;
    int rows;                 // G: kernel rows of all channels, Cin * KH
    uint32_t mask[4];         // G: the words of a kernel row that are taps
    uint32_t mKW, mKH;        // ceil(2^32 / KW), ceil(2^32 / KH): exact quotients below 2^16
    int epi;
    int* d_status;
};

__device__ __forceinline__ uint32_t div_magic(uint32_t v, uint32_t d, uint32_t magic) {
    return d == 1 ? v : __umulhi(v, magic);
}

// The element at p, or zero: a predicated load, no branch.
__device__ __forceinline__ uint32_t ldg_u16_if(const uint16_t* p, bool in) {
    uint32_t v;
    asm volatile(
        "{\n\t"
        ".reg .pred P;\n\t"
        ".reg .b16 h;\n\t"
        "setp.ne.u32 P, %2, 0;\n\t"
        "mov.b16 h, 0;\n\t"
        "@P ld.global.nc.b16 h, [%1];\n\t"
        "cvt.u32.u16 %0, h;\n\t"
        "}\n"
        : "=r"(v)
        : "l"(p), "r"((uint32_t)in));
    return v;
}

// The words of a piece of a kernel row, or zeros: predicated loads, no branch.
__device__ __forceinline__ void ldg_words_if(uint32_t (&v)[2], const uint16_t* p, bool in) {
    asm volatile(
        "{\n\t"
        ".reg .pred P;\n\t"
        "setp.ne.u32 P, %3, 0;\n\t"
        "mov.b32 %0, 0;\n\t"
        "mov.b32 %1, 0;\n\t"
        "@P ld.global.nc.v2.b32 {%0, %1}, [%2];\n\t"
        "}\n"
        : "=&r"(v[0]), "=&r"(v[1])
        : "l"(p), "r"((uint32_t)in));
}
__device__ __forceinline__ void ldg_words_if(uint32_t (&v)[1], const uint16_t* p, bool in) {
    asm volatile(
        "{\n\t"
        ".reg .pred P;\n\t"
        "setp.ne.u32 P, %2, 0;\n\t"
        "mov.b32 %0, 0;\n\t"
        "@P ld.global.nc.b32 %0, [%1];\n\t"
        "}\n"
        : "=&r"(v[0])
        : "l"(p), "r"((uint32_t)in));
}

// Bits 0 ... 7 of m as halves of ones or zeros.  (Bit i of four goes to the top of byte i, whose sign prmt repeats.)
__device__ __forceinline__ void halves_of_bits(uint32_t (&w)[4], uint32_t m) {
    const uint32_t lo = ((m & 15u) * 0x10204080u) & 0x80808080u, hi = ((m >> 4) * 0x10204080u) & 0x80808080u;
    asm("prmt.b32 %0, %1, %1, 0x9988;" : "=r"(w[0]) : "r"(lo));
    asm("prmt.b32 %0, %1, %1, 0xBBAA;" : "=r"(w[1]) : "r"(lo));
    asm("prmt.b32 %0, %1, %1, 0x9988;" : "=r"(w[2]) : "r"(hi));
    asm("prmt.b32 %0, %1, %1, 0xBBAA;" : "=r"(w[3]) : "r"(hi));
}

// grid (K parts, pixel tiles of all images, channel tiles); the K parts of a tile form a cluster.  G: columns of the
// reduction per kernel row where the image is read in words, 0: tap by tap, -1: tap by tap in runs of eight pixels.
template <int BN, typename OutT, int G, bool SMALL>
__global__ void __launch_bounds__((CiCfg<BN, SMALL>::THREADS), (CiCfg<BN, SMALL>::CTAS))
conv_implicit_kernel(const __grid_constant__ CUtensorMap tmapW,   // w: {CRS, Cout}, boxes of 64 x BN
                     const ConvParams p) {
    using Cfg = CiCfg<BN, SMALL>;
    constexpr int CI_GATHER = Cfg::GATHER, TMA_WARP = CI_GATHER / 32, ISSUE_WARP = TMA_WARP + 1;
    static_assert(!SMALL || G != 0, "the small CTA reads the image in words or runs");
    extern __shared__ __align__(1024) uint8_t smem[];
    if ((smem_u32(smem) & 1023u) != 0) {
        if (threadIdx.x == 0) atomicCAS(p.d_status, 0, KST_SMEM_LAYOUT);
        return;
    }
    float* sbias = reinterpret_cast<float*>(smem + Cfg::STAGES * Cfg::STAGE_BYTES);
    uint64_t* bars = reinterpret_cast<uint64_t*>(sbias + BN);
    uint64_t* full = bars;
    uint64_t* empty = bars + Cfg::STAGES;
    uint64_t* tfull = bars + 2 * Cfg::STAGES;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tfull + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int img = blockIdx.y / p.tiles, m0 = (blockIdx.y - img * p.tiles) * CI_PIX, c0 = blockIdx.z * BN;
    const int parts = gridDim.x, rank = blockIdx.x;
    const int nkb_all = (p.CRS + CI_BK - 1) / CI_BK;
    const int kb0 = rank * nkb_all / parts, nkb = (rank + 1) * nkb_all / parts - kb0;

    if (tid == 0) {
        for (int s = 0; s < Cfg::STAGES; ++s) {
            mbar_init(&full[s], CI_GATHER / 32 + 1);   // the gather warps and the weight tile's bytes
            mbar_init(&empty[s], 1);
        }
        mbar_init(tfull, 1);
        *abort_flag = 0;
        fence_barrier_init();
        prefetch_tmap(&tmapW);
    }
    if (warp == TMA_WARP) {
        tmem_alloc(tmem_slot, BN);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // Every warp, in words too: the launch before lays out the weight and has itself waited for the image, but a kernel's writes are
    // visible to the grid that waits, and the gather reads past the L1's coherence (ld.global.nc).
    grid_dep_wait();
    grid_dep_launch();

    // Channel c of the tile at pixel pix, rounded before the activation sees it.  The activation is a template
    // argument: a switch in the unrolled store cost more than the gather.
    OutT* const out0 = static_cast<OutT*>(p.out) + (int64_t)img * p.out_img + (int64_t)c0 * p.P;
    auto store = [&](OutT* dst, float o, auto act) {
        if constexpr (sizeof(OutT) == 2) *dst = __float2half_rn(act(__half2float(__float2half_rn(o))));
        else *dst = act(o);
    };
    auto by_act = [&](auto body) {
        switch (p.epi) {
            case B200_EPI_NONE: body([](float v) { return v; }); break;
            case B200_EPI_RELU: body([](float v) { return fmaxf(v, 0.f); }); break;
            case B200_EPI_GELU: body([](float v) { return gelu_exact(v); }); break;
            default: body([](float v) { return apply_act(B200_EPI_GELU_TANH, v); }); break;
        }
    };
    if (warp == TMA_WARP) {
        if (lane == 0) {
            for (int kb = 0; kb < nkb; ++kb) {
                const int s = kb % Cfg::STAGES;
                if (!mbar_wait(&empty[s], (uint32_t)((kb / Cfg::STAGES) & 1) ^ 1, p.d_status, KST_WAIT_EMPTY, abort_flag)) break;
                mbar_arrive_expect_tx(&full[s], Cfg::B_BYTES);
                tma_load_2d(smem + s * Cfg::STAGE_BYTES + CI_A_BYTES, &tmapW, &full[s], (kb0 + kb) * CI_BK, c0);
            }
        }
    } else if (warp == ISSUE_WARP) {
        // the warp waits together and the thread elect.sync picks issues, as in the GEMM
        constexpr uint32_t idesc = make_idesc_f16(CI_PIX, BN, /*a MN-major, in words K-major*/ G <= 0, /*b K-major*/ 0);
        constexpr uint64_t adesc0 = G <= 0 ? make_smem_desc(64 * CI_BK * 2, 1024) : make_smem_desc(16, 1024);
        constexpr uint64_t bdesc0 = make_smem_desc(16, 1024);
        bool ok = true;
        for (int kb = 0; kb < nkb; ++kb) {
            const int s = kb % Cfg::STAGES;
            ok = mbar_wait(&full[s], (uint32_t)((kb / Cfg::STAGES) & 1), p.d_status, KST_WAIT_FULL, abort_flag);
            if (__any_sync(0xffffffffu, !ok)) { ok = false; break; }
            tc_fence_after();
            if (elect_one()) {
                const uint32_t a = smem_u32(smem + s * Cfg::STAGE_BYTES), b = a + CI_A_BYTES;
#pragma unroll
                for (int k = 0; k < CI_BK / 16; ++k) {   // 16 k: two 8-row groups of an MN-major A, 32 bytes inside a K-major swizzle row
                    if (G < 0 && (kb0 + kb) * CI_BK + k * 16 >= p.CRS) break;   // not gathered
                    umma_ss(tmem_base, smem_desc_at(adesc0, a + k * (G <= 0 ? 2048 : 32)), smem_desc_at(bdesc0, b + k * 32), idesc, (kb | k) != 0);
                }
                umma_commit(&empty[s]);
                if (kb + 1 == nkb) umma_commit(tfull);
            }
            __syncwarp();
        }
    } else {
        for (int j = tid; j < BN; j += CI_GATHER)   // read in the epilogue, a barrier among these warps later
            sbias[j] = p.bias != nullptr && c0 + j < p.Cout ? __half2float(p.bias[c0 + j]) : 0.f;
        bool ok = true;
        if constexpr (G > 0) {
            const uint16_t* xi = reinterpret_cast<const uint16_t*>(p.x) + (int64_t)img * p.x_img;
            // Pixel tid % 128; of a k-block's eight 16-byte pieces those of one parity, in SMALL all, the even ones first.
            constexpr int VL = G / 2, RPC = 8 / G;   // elements a load, kernel rows a piece
            constexpr int HALVES = SMALL ? 2 : 1;   // SMALL: a thread takes all eight pieces of its pixel, four at a time
            const int pix = tid & 127, par = tid >> 7, m = m0 + pix;
            const int oh = m / p.OW, ow = m - oh * p.OW;
            const int bx = ow * p.sx - p.px, by = m < p.P ? oh * p.sy - p.py : -(1 << 30);   // never inside the image
            const bool in0 = (uint32_t)bx < (uint32_t)p.W, in1 = (uint32_t)(bx + VL) < (uint32_t)p.W;   // whole words: W is a multiple
            const int base = by * p.W + bx;
            uint32_t v[2][4][RPC][2][VL / 2];
            auto load = [&](int st, int b) {
                const int kb = st / HALVES, par1 = SMALL ? st & 1 : par;
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int u = 0; u < RPC; ++u) {
                        const int r = ((kb0 + kb) * 8 + 2 * i + par1) * RPC + u;   // the same for the warp
                        const int cin = (int)div_magic((uint32_t)r, p.KH, p.mKH), ky = (r - cin * p.KH) * p.dy;
                        const bool row = r < p.rows && (uint32_t)(by + ky) < (uint32_t)p.H;
                        const uint16_t* src = xi + (base + (cin * p.H + ky) * p.W);
                        ldg_words_if(v[b][i][u][0], src, row && in0);
                        ldg_words_if(v[b][i][u][1], src + VL, row && in1);
                    }
            };
            load(0, 0);
            const int nsteps = nkb * HALVES;
            auto step = [&](int st, int b) -> bool {
                const int kb = st / HALVES, s = kb % Cfg::STAGES, par1 = SMALL ? b : par;
                if (st + 1 < nsteps) load(st + 1, b ^ 1);
                if ((!SMALL || b == 0) && ok && !mbar_wait(&empty[s], (uint32_t)((kb / Cfg::STAGES) & 1) ^ 1, p.d_status, KST_WAIT_EMPTY, abort_flag)) ok = false;
                if (__any_sync(0xffffffffu, !ok)) return ok = false;
                const uint32_t a = smem_u32(smem + s * Cfg::STAGE_BYTES) + pix * 128;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    uint32_t w[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) w[e] = v[b][i][e / (4 / RPC)][(e / (VL / 2)) & 1][e % (VL / 2)] & p.mask[e];
                    st_shared_v4(a + (((2 * i + par1) ^ (pix & 7)) << 4), w);
                }
                if (SMALL && b == 0) return true;
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(&full[s]);
                return true;
            };
            for (int st = 0; st < nsteps; st += 2) {   // by twos: the registers of a step are named at compile time
                if (!step(st, 0)) break;
                if (st + 1 < nsteps && !step(st + 1, 1)) break;
            }
        } else if constexpr (G < 0) {
            // Pixels 8 (lane % 16) ... of the tile, a run of memory for every tap.  What of it lies outside the image is masked: byte
            // kx of `xm` are the eight pixels' columns that are inside with that tap, byte ky of `ym` the rows.
            const uint16_t* xi = reinterpret_cast<const uint16_t*>(p.x) + (int64_t)img * p.x_img;
            const int c = lane & 15, up = lane >> 4, m = m0 + 8 * c, y0 = m / p.W, x0 = m - y0 * p.W;
            uint32_t xm = 0, ym = 0;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int wrap = x0 + j >= p.W, x = x0 + j - (wrap ? p.W : 0) - p.px;   // W is eight at the least
                const int y = m + j < p.P ? y0 + wrap - p.py : -(1 << 30);
#pragma unroll
                for (int t = 0; t < 4; ++t) {   // bits of taps that are not there are not looked at
                    xm |= (uint32_t)((uint32_t)(x + t * p.dx) < (uint32_t)p.W) << (8 * t + j);
                    ym |= (uint32_t)((uint32_t)(y + t * p.dy) < (uint32_t)p.H) << (8 * t + j);
                }
            }
            const int base = m - p.py * p.W - p.px, total = p.CRS / (p.KW * p.KH) * p.H * p.W;
            // A warp takes rows warp + WARPS r of a k-block, four at a time, a half of it each of two.
            constexpr int WARPS = CI_GATHER / 32, STEPS = 16 / WARPS;
            const int row = WARPS == 8 ? warp : warp + 4 * up;   // in its eight rows
            uint8_t* const to = smem + (c >> 3) * (64 * CI_BK * 2) + (WARPS == 8 ? up * 1024 : 0) + row * 128 + (((c & 7) ^ row) << 4);
            int koff, kxy;   // of row r by lane r: offset in the image, and 8 kx, 8 ky; past the reduction negative
            auto taps = [&](int kb) {
                const uint32_t k = (uint32_t)((kb0 + kb) * CI_BK + warp + WARPS * (lane & (64 / WARPS - 1)));
                const uint32_t t = div_magic(k, p.KW, p.mKW), cin = div_magic(t, p.KH, p.mKH);
                const int kx = (int)(k - t * p.KW), ky = (int)(t - cin * p.KH);
                koff = ((int)cin * p.H + ky * p.dy) * p.W + kx * p.dx;
                kxy = k < (uint32_t)p.CRS ? 8 * kx | 8 * ky << 8 : -1;
            };
            struct Run { uint4 v[2]; uint32_t how; };   // the vectors the run lies in; its first element there, and the mask << 8
            auto load = [&](Run (&run)[2], int step) {   // r = 4 step + 2 i + up of the k-block whose taps are held
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const int o = __shfl_sync(0xffffffffu, koff, 4 * step + 2 * i + up), t = __shfl_sync(0xffffffffu, kxy, 4 * step + 2 * i + up);
                    const uint32_t mask = t < 0 ? 0u : xm >> (t & 255) & ym >> (t >> 8) & 255u;
                    const int e = base + o;
                    const uint16_t* a = xi + e;
                    const int s = (int)(reinterpret_cast<uintptr_t>(a) >> 1) & 7, ev = e - s;
                    const uint4* v = reinterpret_cast<const uint4*>(a - s);
                    run[i].how = (uint32_t)s | mask << 8;
                    // a vector is read if it holds an element of the image
                    run[i].v[0] = mask != 0 && ev > -8 && ev < total ? __ldg(v) : make_uint4(0u, 0u, 0u, 0u);
                    run[i].v[1] = mask != 0 && s != 0 && ev > -16 && ev + 8 < total ? __ldg(v + 1) : make_uint4(0u, 0u, 0u, 0u);
                }
            };
            auto put = [&](const Run (&run)[2], int stage, int step) {
                uint8_t* a = to + stage * Cfg::STAGE_BYTES + step * (512 * WARPS);
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const uint32_t s = run[i].how & 7u, mask = run[i].how >> 8;
                    const uint4 v0 = run[i].v[0], v1 = run[i].v[1];
                    // by two words, one word, one element
                    const bool b2 = s & 4, b1 = s & 2;
                    const uint32_t t0 = b2 ? v0.z : v0.x, t1 = b2 ? v0.w : v0.y, t2 = b2 ? v1.x : v0.z, t3 = b2 ? v1.y : v0.w, t4 = b2 ? v1.z : v1.x,
                                   t5 = b2 ? v1.w : v1.y;
                    const uint32_t u[5] = {b1 ? t1 : t0, b1 ? t2 : t1, b1 ? t3 : t2, b1 ? t4 : t3, b1 ? t5 : t4};
                    uint32_t w[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) w[q] = __funnelshift_r(u[q], u[q + 1], (s & 1u) << 4);
                    uint32_t in[4];
                    halves_of_bits(in, mask);
#pragma unroll
                    for (int q = 0; q < 4; ++q) w[q] &= in[q];
                    *reinterpret_cast<uint4*>(a + i * (256 * WARPS)) = make_uint4(w[0], w[1], w[2], w[3]);
                }
            };
            Run ra[2], rb[2];
            taps(0);
            load(ra, 0);
            for (int kb = 0; kb < nkb; ++kb) {
                const int s = kb % Cfg::STAGES;
                const int n = (p.CRS - (kb0 + kb) * CI_BK + CI_BK / STEPS - 1) / (CI_BK / STEPS);   // steps with a row of the reduction
                if (n > 1) load(rb, 1);
                if (ok && !mbar_wait(&empty[s], (uint32_t)((kb / Cfg::STAGES) & 1) ^ 1, p.d_status, KST_WAIT_EMPTY, abort_flag)) ok = false;
                if (__any_sync(0xffffffffu, !ok)) { ok = false; break; }
                put(ra, s, 0);
                if constexpr (STEPS == 4) {
                    if (n > 2) load(ra, 2);
                    if (n > 1) put(rb, s, 1);
                    if (n > 3) load(rb, 3);
                    if (n > 2) put(ra, s, 2);
                }
                if (kb + 1 < nkb) {
                    taps(kb + 1);
                    load(ra, 0);
                }
                if (n >= STEPS) put(rb, s, STEPS - 1);
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(&full[s]);
            }
        } else {
        // Pixels 2 lane, 2 lane + 1 of either half of the tile.
        int bx[4], by[4], base[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int m = m0 + 64 * (q >> 1) + 2 * lane + (q & 1);
            const int oh = m / p.OW, ow = m - oh * p.OW;
            bx[q] = ow * p.sx - p.px;
            by[q] = m < p.P ? oh * p.sy - p.py : -(1 << 30);   // never inside the image
            base[q] = by[q] * p.W + bx[q];
        }
        const uint16_t* xi = reinterpret_cast<const uint16_t*>(p.x) + (int64_t)img * p.x_img;
        const int row_off = warp * 128 + (((lane >> 2) ^ warp) << 4) + (lane & 3) * 4;   // row warp + 8 r: r * 1024 further
        // The taps of the warp's eight rows of a k-block, row r by lane r: offset in the image and (x, y) shift.  A row
        // past the reduction gets a shift that is never inside.
        int koff, kx, ky;
        auto taps = [&](int kb) {
            const uint32_t k = (uint32_t)((kb0 + kb) * CI_BK + warp + 8 * (lane & 7));
            const uint32_t t = div_magic(k, p.KW, p.mKW), cin = div_magic(t, p.KH, p.mKH);
            kx = k < (uint32_t)p.CRS ? (int)(k - t * p.KW) * p.dx : -(1 << 30);
            ky = (int)(t - cin * p.KH) * p.dy;
            koff = ((int)cin * p.H + ky) * p.W + kx;
        };
        auto load = [&](uint32_t (&v)[4][4], int half) {   // rows 4 half ... of the k-block whose taps are held
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int o = __shfl_sync(0xffffffffu, koff, 4 * half + i), x = __shfl_sync(0xffffffffu, kx, 4 * half + i),
                          y = __shfl_sync(0xffffffffu, ky, 4 * half + i);
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    v[i][q] = ldg_u16_if(xi + (base[q] + o), (uint32_t)(bx[q] + x) < (uint32_t)p.W && (uint32_t)(by[q] + y) < (uint32_t)p.H);
            }
        };
        auto put = [&](const uint32_t (&v)[4][4], int step) {
            uint8_t* a = smem + ((step >> 1) % Cfg::STAGES) * Cfg::STAGE_BYTES + (step & 1) * 4096 + row_off;
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    *reinterpret_cast<uint32_t*>(a + h * (64 * CI_BK * 2) + i * 1024) = v[i][2 * h] | (v[i][2 * h + 1] << 16);
        };
        uint32_t va[4][4], vb[4][4];
        taps(0);
        load(va, 0);
        for (int kb = 0; kb < nkb; ++kb) {
            const int s = kb % Cfg::STAGES;
            load(vb, 1);
            if (ok && !mbar_wait(&empty[s], (uint32_t)((kb / Cfg::STAGES) & 1) ^ 1, p.d_status, KST_WAIT_EMPTY, abort_flag)) ok = false;
            if (__any_sync(0xffffffffu, !ok)) { ok = false; break; }
            put(va, 2 * kb);
            if (kb + 1 < nkb) {
                taps(kb + 1);
                load(va, 0);
            }
            put(vb, 2 * kb + 1);
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[s]);
        }
        }
        // ------------------------------------------------------------------ epilogue
        named_bar_sync(1, CI_GATHER);   // sbias
        if (ok && !mbar_wait(tfull, 0, p.d_status, KST_WAIT_TMEM_FULL, abort_flag)) ok = false;
        if (!__any_sync(0xffffffffu, !ok)) {
            tc_fence_after();
            constexpr int SHARES = CI_GATHER / 128;
            const int quad = warp & 3, part = warp >> 2;   // tensor-memory lane quadrant, share of the channels
            const int pix = m0 + quad * 32 + lane;
            const uint32_t tacc = tmem_base + (uint32_t(quad * 32) << 16);
            const int cend = min((part + 1) * (BN / SHARES), p.Cout - c0);
            if (Cfg::SPLITS && parts > 1) {
                float* acc = reinterpret_cast<float*>(smem) + quad * 32 + lane;   // [channel][pixel], over the drained ring
#pragma unroll 1
                for (int c = part * (BN / SHARES); c < cend; c += 16) {
                    uint32_t r[16];
                    tmem_ld16(tacc + c, r);
                    tmem_wait_ld();
#pragma unroll
                    for (int t = 0; t < 16; ++t) acc[(c + t) * CI_PIX] = __uint_as_float(r[t]);
                }
            } else {
                by_act([&](auto act) {
#pragma unroll 1
                    for (int c = part * (BN / SHARES); c < cend; c += 16) {
                        uint32_t r[16];
                        tmem_ld16(tacc + c, r);
                        tmem_wait_ld();
                        OutT* dst = out0 + (int64_t)c * p.P + pix;
                        if (pix < p.P) {
                            if (c + 16 <= cend) {
#pragma unroll
                                for (int t = 0; t < 16; ++t, dst += p.P) store(dst, __uint_as_float(r[t]) + sbias[c + t], act);
                            } else {
#pragma unroll
                                for (int t = 0; t < 16; ++t, dst += p.P)
                                    if (c + t < cend) store(dst, __uint_as_float(r[t]) + sbias[c + t], act);
                            }
                        }
                        __syncwarp();
                    }
                });
            }
        }
    }
    if (Cfg::SPLITS && parts > 1) {
        cluster_sync_all();   // every part's tile is in its shared memory
        if (warp < TMA_WARP) {
            const uint32_t mine = smem_u32(smem) + (tid & 127) * 4;
            const int pix = m0 + (tid & 127);
            // four channels' loads from every part in flight together: a remote load takes a few hundred nanoseconds
            by_act([&](auto act) {
                for (int c = rank * (BN / parts) + (tid >> 7); c < (rank + 1) * (BN / parts); c += 8) {
                    float v[4][8];
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        const uint32_t src = mapa_u32(mine + c * (CI_PIX * 4), q < parts ? q : 0);
#pragma unroll
                        for (int u = 0; u < 4; ++u) v[u][q] = q < parts ? ld_cluster_f32(src + u * (2 * CI_PIX * 4)) : 0.f;
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        float o = 0.f;
#pragma unroll
                        for (int q = 0; q < 8; ++q) o += v[u][q];
                        if (pix < p.P && c0 + c + 2 * u < p.Cout)
                            store(out0 + (int64_t)(c + 2 * u) * p.P + pix, o + sbias[c + 2 * u], act);
                    }
                }
            });
        }
        cluster_sync_all();   // nobody leaves while its tile may still be read
    }
    if (*abort_flag) {   // let any TMA copy still in flight into this CTA's shared memory land before exit
        for (int i = 0; i < 4; ++i) __nanosleep(1000000);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == TMA_WARP) {
        tc_fence_after();
        tmem_dealloc(tmem_base, BN);
    }
}

template <int BN, typename OutT, int G, bool SMALL = false>
static int ci_launch(b200_ctx* ctx, const CUtensorMap& tw, const ConvParams& p, int64_t N, int parts) {
    using Cfg = CiCfg<BN, SMALL>;
    static bool attr_done[16] = {};
    auto kern = conv_implicit_kernel<BN, OutT, G, SMALL>;
    if (!attr_done[ctx->device & 15]) {
        B200_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES));
        attr_done[ctx->device & 15] = true;
    }
    dim3 grid((unsigned)parts, (unsigned)(p.tiles * N), (unsigned)cdiv(p.Cout, BN));
    B200_CUDA(launch_dep(kern, grid, dim3(Cfg::THREADS, 1, 1), Cfg::SMEM_BYTES, ctx->stream, parts, tw, p));
    ctx->launches++;
    return B200_OK;
}

bool conv_implicit_takes(int64_t W, int64_t H, int64_t Cin, int64_t N, int64_t KW, int64_t KH, int64_t Cout, int64_t P) {
    return cdiv(P, CI_PIX) * N < 65536 && P < (1ll << 30) && W * H * Cin < (1ll << 31) && KW * KH * Cin < 65536 && KW < 65536 && KH < 65536 &&
           Cout < (1 << 20) && W < (1 << 28) && H < (1 << 28);
}

// Whether the image can be read in words, and the columns of the reduction a kernel row then takes (0: no).  The pixels'
// first taps have to lie `word` elements apart with every row of the image starting on one, and a row's taps in two words.
// One word would do for narrow kernels and half of the reduction would be zeros; they stay with the taps.
int conv_words(int64_t W, int64_t KW, int64_t sx, int64_t px, int64_t dx, const void* x, int64_t x_img) {
    for (const int64_t word : {4, 2}) {
        const int64_t lead = (word - px % word) % word;
        if (sx % word == 0 && W % word == 0 && x_img % word == 0 && dx == 1 && reinterpret_cast<uintptr_t>(x) % (2 * word) == 0 &&
            KW + lead > word && KW + lead <= 2 * word)
            return (int)(2 * word);
    }
    return 0;
}

// The weight for it: (Cout, CRS) -> (Cout, Cin KH, g), each kernel row's taps behind `lead` zeros; rows in whole 16 bytes.
int64_t conv_words_ldw(int64_t rows, int g) { return cdiv(rows * g, 8) * 8; }

__global__ void conv_words_weight_kernel(__half* __restrict__ dst, const __half* __restrict__ src, int KW, int g, int lead, int rows,
                                         int ldw, int64_t n) {
    grid_dep_wait();     // the weight may be the previous kernel's output
    grid_dep_launch();
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t co = i / ldw;
        const int k = (int)(i - co * ldw), row = k / g, t = k - row * g - lead;
        dst[i] = row < rows && t >= 0 && t < KW ? src[(co * rows + row) * KW + t] : __float2half_rn(0.f);
    }
}

int conv_words_weight(b200_ctx* ctx, void* dst, const void* w, int64_t KW, int64_t px, int64_t rows, int64_t Cout, int g) {
    const int64_t ldw = conv_words_ldw(rows, g), n = Cout * ldw, word = g / 2, cap = (int64_t)ctx->prop.multiProcessorCount * 8;
    const int64_t blocks = cdiv(n, 256);
    B200_CUDA(launch_dep(conv_words_weight_kernel, dim3((unsigned)(blocks < cap ? blocks : cap), 1, 1), dim3(256, 1, 1), 0, ctx->stream, 1,
                         (__half*)dst, (const __half*)w, (int)KW, g, (int)((word - px % word) % word), (int)rows, (int)ldw, n));
    ctx->launches++;
    return B200_OK;
}

// Channels per CTA: all of them up to 256, since every channel tile gathers the pixels again; but a launch that
// leaves half of the GPU's CTAs unused splits the reduction, two k-blocks a part at least, which the 256-wide
// tile has no shared memory for; four a part where they are read in words and take less than a cluster's barriers
// (256 x 256 x 32 -> 128, 3 x 3 / 2: 15.8 us with two, 9.2).  Eight parts up to the clusters a GPC's SMs hold at once (48 x 44 x
// 256 -> 256, 3 x 3, 34 clusters: 25.5 us, with four parts 21.1).  tiles: pixel tiles of all images; cols: of the reduction.
struct CiTiles { int bn, parts; int64_t nkb; };
static CiTiles ci_tiles(const b200_ctx* ctx, int64_t tiles, int64_t cols, int64_t Cout, int g) {
    const int64_t room = 2 * (int64_t)ctx->prop.multiProcessorCount, nkb = cdiv(cols, CI_BK);
    CiTiles t = {Cout <= 64 ? 64 : (Cout <= 128 || (2 * tiles * cdiv(Cout, 128) <= room && nkb >= 4) ? 128 : 256), 1, nkb};
    if (t.bn < 256)
        while (t.parts < 8 && (2 * t.parts + (t.parts == 4)) * tiles * cdiv(Cout, t.bn) <= room && nkb >= (g ? 8 : 4) * t.parts) t.parts *= 2;
    return t;
}

// What a convolution takes through the im2col matrix of a small image, one after the other, in microseconds (fitted as below).
static double ci_matrix(int64_t N, int64_t P, int64_t crs, int64_t Cout) {
    return (double)N * (6.9 + 2.36e-6 * (double)P * (double)crs + 1.3e-9 * (double)P * (double)crs * (double)Cout + 0.0012 * (double)crs) +
           (crs % 8 != 0 ? 1.2 : 0.0);
}

// Which of the convolutions that can be read in words gain by it.  Not where laying out the weight is more than reading the
// image (34 x 34 x 256 -> 256, 3 x 3 / 2: 14.3 us, 15.1 in words), nor a kernel no wider than a word, half of whose columns are
// zeros, on a short reduction (72 x 66 x 16 -> 8, 2 x 2 / 2 padded by 1: 4.5 us by taps, 5.2).  The implicit kernel by taps loses to
// it otherwise (`taps`; 560 x 556 x 3 -> 32, 7 x 7 / 4: 12.2 us, 6.8); against the im2col matrix of a small image the cheaper one
// is taken, in microseconds as fitted to 280 convolutions of 16 to 512 pixels a side, 1 to 384 -> 8 to 512 channels: the first
// moves and multiplies more, the second has a long chain a CTA (64 x 60 x 64 -> 256, 3 x 3 / 2: 9.0 us, 12.6 in words; 128 x 128 x
// 128 -> 128: 20.1, 15.2).  That is 0.3% off the faster of the two in the mean, always words was 1.7%, and 1.15 times it at worst (1.66).
bool conv_words_gains(const b200_ctx* ctx, int64_t W, int64_t H, int64_t Cin, int64_t N, int64_t KW, int64_t KH, int64_t Cout, int64_t P,
                      int g, bool taps) {
    const int64_t cols = Cin * KH * g, tiles = cdiv(P, CI_PIX) * N;
    if (conv_words_ldw(Cin * KH, g) * Cout > N * Cin * W * H || (2 * KW <= g && cols <= 4 * CI_BK)) return false;
    if (taps) return true;
    const CiTiles t = ci_tiles(ctx, tiles, cols, Cout, g);
    const double load = (double)(tiles * cdiv(Cout, t.bn) * t.parts) / (2.0 * ctx->prop.multiProcessorCount);   // of the resident CTAs
    const double words = 3.1 + 4.8e-6 * (double)(cols * Cout) + (double)cdiv(t.nkb, t.parts) * (0.41 + 0.84 * load) +
                         0.0129 * t.bn * (load > 1.0 ? load : 1.0) + (t.parts > 1 ? 2.5 + 1.8 * load : 0.0);
    return 1.04 * words < ci_matrix(N, P, KW * KH * Cin, Cout);
}

// Whether the pixels' taps are runs of memory as the pixels are: a row of results as long as the image's, pixel by pixel.
bool conv_runs(int64_t W, int64_t KW, int64_t KH, int64_t sx, int64_t sy, int64_t OW) {
    return sx == 1 && sy == 1 && OW == W && W >= 8 && KW <= 4 && KH <= 4;
}

// Whether a small image read in runs beats its im2col matrix, by an estimate fitted to 190 of 3 x 3, 16 to 512 pixels a side and 1 to
// 384 -> 8 to 512 channels, in microseconds: the route it picks is 0.3 % off the faster one in the mean and 8 % at worst (always runs
// 2.5 and 46 %, always the matrix 73 % in the mean).  64 x 60 x 64 -> 64: 12.8 -> 8.2 us, two images 25.2 -> 11.2, 128 x 124 x 128 ->
// 128 50.8 -> 24.2, 128 x 124 x 64 -> 64 29.2 -> 15.1; a reduction off eights, whose weight either route copies, stays with the matrix
// more often (48 x 47 x 133 -> 488: 20.1, 29.3).
bool conv_runs_gain(const b200_ctx* ctx, int64_t Cin, int64_t N, int64_t KW, int64_t KH, int64_t Cout, int64_t P) {
    const int64_t crs = KW * KH * Cin, tiles = cdiv(P, CI_PIX) * N;
    const CiTiles t = ci_tiles(ctx, tiles, crs, Cout, 0);
    const double load = (double)(tiles * cdiv(Cout, t.bn) * t.parts) / (2.0 * ctx->prop.multiProcessorCount), rounds = load > 1.0 ? load : 1.0;
    const double blocks = t.parts > 1 ? (double)cdiv(t.nkb, t.parts) : (double)crs / CI_BK;
    const double runs = 0.81 + blocks * (0.55 + 1.65 * load) + (0.012 * t.bn + 2.47) * rounds + (t.parts > 1 ? 2.44 + 0.7 * load : 0.0) +
                        (crs % 8 != 0 ? 1.75 + 4.3e-6 * (double)(crs * Cout) : 0.0);
    return 0.95 * runs < ci_matrix(N, P, crs, Cout);
}

int conv_implicit_launch(b200_ctx* ctx, int64_t W, int64_t H, int64_t Cin, int64_t N, int64_t KW, int64_t KH, int64_t Cout,
                         int64_t sx, int64_t sy, int64_t px, int64_t py, int64_t dx, int64_t dy, int64_t OW, int64_t P,
                         const void* x, int64_t x_img, const void* w, int64_t ldw, const void* bias, void* out,
                         int64_t out_img, int out_dtype, int epilogue, int g) {
    ConvParams p;
    p.x = static_cast<const __half*>(x);
    p.bias = static_cast<const __half*>(bias);
    p.out = out;
    p.x_img = x_img; p.out_img = out_img;
    p.W = (int)W; p.H = (int)H; p.CRS = (int)(KW * KH * Cin); p.Cout = (int)Cout; p.OW = (int)OW; p.P = (int)P;
    p.sx = (int)sx; p.sy = (int)sy; p.px = (int)px; p.py = (int)py; p.dx = (int)dx; p.dy = (int)dy;
    p.KW = (int)KW; p.KH = (int)KH;
    p.mKW = KW > 1 ? (uint32_t)(((1ull << 32) + KW - 1) / KW) : 0;
    p.mKH = KH > 1 ? (uint32_t)(((1ull << 32) + KH - 1) / KH) : 0;
    p.epi = epilogue;
    p.d_status = ctx->d_status;
    p.tiles = (int)cdiv(P, CI_PIX);
    p.rows = (int)(Cin * KH);
    if (g) {
        const int64_t word = g / 2, lead = (word - px % word) % word;
        p.CRS = (int)(Cin * KH * g);
        p.px = (int)(px + lead);
        for (int e = 0; e < 4; ++e) {
            p.mask[e] = 0;
            for (int h = 0; h < 2; ++h) {
                const int64_t t = (2 * e + h) % g - lead;
                if (t >= 0 && t < KW) p.mask[e] |= 0xFFFFu << (16 * h);
            }
        }
    }
    const CiTiles t = ci_tiles(ctx, p.tiles * N, p.CRS, Cout, g);
    const int bn = t.bn, parts = t.parts;
    const bool small = parts == 1 && p.tiles * N * cdiv(Cout, bn) > 2 * ctx->prop.multiProcessorCount;
    CUtensorMap tw;
    uint64_t dims[2] = {(uint64_t)p.CRS, (uint64_t)Cout};
    uint64_t str[1] = {(uint64_t)ldw * 2};
    uint32_t box[2] = {CI_BK, (uint32_t)bn};
    int rc = make_tmap(ctx, &tw, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, w, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
    auto go = [&](auto zero, auto G) -> int {
        using T = decltype(zero);
        constexpr int g = decltype(G)::value;
        if constexpr (g != 0) {
            if (small && bn == 128) return ci_launch<128, T, g, true>(ctx, tw, p, N, 1);
            if (small && bn == 64) return ci_launch<64, T, g, true>(ctx, tw, p, N, 1);
        }
        if (bn == 256) return ci_launch<256, T, g>(ctx, tw, p, N, 1);
        if (bn == 128) return ci_launch<128, T, g>(ctx, tw, p, N, parts);
        return ci_launch<64, T, g>(ctx, tw, p, N, parts);
    };
    auto typed = [&](auto G) { return out_dtype == B200_F16 ? go(__half(), G) : go(float(), G); };
    if (g == 8) return typed(std::integral_constant<int, 8>());
    if (g == 4) return typed(std::integral_constant<int, 4>());
    if (conv_runs(W, KW, KH, sx, sy, OW)) return typed(std::integral_constant<int, -1>());
    return typed(std::integral_constant<int, 0>());
}

} // namespace b200
