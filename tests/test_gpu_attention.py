import math
import os

import numpy as np
import pytest

import juliavision_b200 as jv

from .conftest import relerr
from .gpu_helpers import attention_gpu, describe, qkv_views

pytestmark = pytest.mark.gpu
G = os.path.join(os.path.dirname(__file__), "golden")
TOL = 5e-3  # the reference's fused-attention gate: max|d|/max|ref| (test_flash.jl:142,204)


def test_golden(ctx):
    g = np.load(os.path.join(G, "attention.npz"))
    got, plan = attention_gpu(ctx, g["q"], g["k"], g["v"], float(g["scale"]), out_dtype=np.float32)
    assert isinstance(plan, jv.FlashTCPlan)
    assert relerr(got, g["out"]) < TOL, describe(got, g["out"], TOL)


# torch (B,H,Lq,Lk,E); covers the reference's test shapes that fit E <= 64 (test_flash.jl:36,189-190),
# the Whisper shape's ragged 1500 and the Hiera head dim 56
SHAPES = [(1, 4, 128, 128, 64), (1, 1, 64, 64, 64), (2, 2, 256, 256, 64), (1, 8, 23, 4096, 16),
          (1, 8, 23, 23, 32), (1, 8, 4096, 23, 16), (1, 4, 23, 17, 16), (1, 3, 1500, 1500, 64),
          (3, 2, 300, 200, 56), (1, 2, 129, 257, 8), (1, 1, 1, 1, 64)]


@pytest.mark.parametrize("B,H,Lq,Lk,E", SHAPES)
@pytest.mark.parametrize("out_dtype", [np.float16, np.float32])
def test_vs_oracle(ctx, ora, B, H, Lq, Lk, E, out_dtype):
    rng = np.random.default_rng(B * 1000 + H * 100 + Lq + Lk + E)
    q = np.float16(rng.standard_normal((B, H, Lq, E)))
    k = np.float16(rng.standard_normal((B, H, Lk, E)))
    v = np.float16(rng.standard_normal((B, H, Lk, E)))
    scale = 1 / np.sqrt(E)
    got, plan = attention_gpu(ctx, q, k, v, scale, out_dtype)
    assert isinstance(plan, jv.FlashTCPlan), plan
    assert got.shape == (B, H, Lq, E) and got.dtype == out_dtype
    ref = ora.attention_ref(q, k, v, scale)
    assert np.max(np.abs(got)) > 1e-3
    assert relerr(got, ref) < TOL, describe(got, ref, TOL)
    # and within the stated tolerance of the runtime's own unfused decomposition
    tp = ora.attention_threepass(q, k, v, scale)
    assert relerr(got, tp) < 1e-2, describe(got, tp, 1e-2)


def test_interleaved_heads(ctx, ora):
    """Operands as the projections leave them: (E,H,L,B) memory viewed as (E,L,H,B); fused qkv."""
    rng = np.random.default_rng(11)
    B, L, H, E = 2, 200, 5, 64
    buf = np.float16(rng.standard_normal((B, L, 3, H, E)))
    q, k, v = (buf[:, :, i].transpose(0, 2, 1, 3) for i in range(3))
    got, plan = attention_gpu(ctx, q, k, v, 0.125)
    assert isinstance(plan, jv.FlashTCPlan)
    ref = ora.attention_ref(q, k, v, 0.125)
    assert relerr(got, ref) < TOL, describe(got, ref, TOL)


def test_token_major_output_view(ctx, ora):
    """out given as an (E,L,H,B) view of a token-major buffer: the permute copy after sdpa is folded
    into the store; values are those of the dense call."""
    from .gpu_helpers import qkv_views
    rng = np.random.default_rng(13)
    B, H, L, E = 2, 5, 200, 64
    q, k, v = (np.float16(rng.standard_normal((B, H, L, E))) for _ in range(3))
    dq, dk, dv = qkv_views(ctx, q, k, v)
    dense, _ = attention_gpu(ctx, q, k, v, 0.125)
    buf = ctx.allocate(np.float16, E * H, L, B)                     # torch (B, L, H*E)
    ctx.fill_bytes(buf, 0xFF)
    view = jv.DeviceArray(ctx, buf.ptr, np.float16, (E, L, H, B), (1, E * H, E, E * H * L), owner=buf)
    jv.sdpa(ctx, dq, dk, dv, None, 0.125, out=view)
    ctx.synchronize()
    got = buf.to_host().reshape(B, L, H, E).transpose(0, 2, 1, 3)
    assert np.array_equal(got, dense)


# (E, Lq, Lk, H, B): the reference's own fused tiling and its tests are at head dim 72 (test_flash.jl:36,
# 189-190, 221; FLASHCM_TILINGS flash.jl:1149-1157), SAM 2's windowed shape is (72,256,256,8,16)
# (tools/attn_lab.jl:11-14); 80/96/104/128 cover the rest of the two-atom range
WIDE = [(72, 64, 64, 1, 1), (72, 128, 128, 2, 1), (72, 256, 256, 2, 1), (72, 128, 256, 2, 2), (72, 64, 4096, 2, 1),
        (72, 256, 256, 8, 16), (72, 1000, 700, 3, 2), (80, 300, 300, 2, 1), (96, 257, 129, 1, 2), (104, 130, 513, 2, 1),
        (128, 384, 384, 2, 1), (128, 23, 4096, 4, 1)]


@pytest.mark.parametrize("E,Lq,Lk,H,B", WIDE)
def test_head_dims_above_one_swizzle_row_run_on_the_tensor_cores(ctx, ora, E, Lq, Lk, H, B):
    """Head dims 72..128: two swizzle atoms along E, one query tile per CTA; same contract and tolerance
    as the narrow kernel, ragged query/key tails and the few-queries key split included."""
    rng = np.random.default_rng(E * 7 + Lq + Lk)
    q = np.float16(rng.standard_normal((B, H, Lq, E)) * 0.2)
    k = np.float16(rng.standard_normal((B, H, Lk, E)) * 0.2)
    v = np.float16(rng.standard_normal((B, H, Lk, E)) * 0.2)
    scale = 1 / np.sqrt(E)
    for out_dtype in (np.float32, np.float16):
        got, plan = attention_gpu(ctx, q, k, v, scale, out_dtype)
        assert isinstance(plan, jv.FlashTCPlan), plan
        assert np.all(np.isfinite(got))
        ref = ora.attention_ref(q, k, v, scale)
        assert np.max(np.abs(got)) > 1e-3
        assert relerr(got, ref) < TOL, describe(got, ref, TOL)


def test_sam2_global_shape_head_dim_72_sampled_rows(ctx, ora):
    """(E72, L4096, H8, B1), the global-attention shape of the reference's flagship encoder
    (tools/attn_lab.jl:11-14), checked on sampled query rows against the fp32 reference."""
    rng = np.random.default_rng(72)
    B, H, L, E = 1, 8, 4096, 72
    q, k, v = (np.float16(rng.standard_normal((B, H, L, E)) * 0.5) for _ in range(3))
    scale = 1 / np.sqrt(E)
    got, plan = attention_gpu(ctx, q, k, v, scale)
    assert isinstance(plan, jv.FlashTCPlan)
    rows = np.unique(np.concatenate([np.arange(0, L, 97), [127, 128, 255, 256, L - 1]]))
    ref = ora.attention_ref(q[:, :, rows], k, v, scale)
    assert relerr(got[:, :, rows], ref) < TOL, describe(got[:, :, rows], ref, TOL)


# (B, H, Lq, Lk, E), mask shape or None: head dims past the fused kernel's run as two batched GEMMs and a softmax
TWO_GEMM = [((1, 2, 300, 264, 256), None), ((2, 3, 128, 512, 136), None), ((1, 2, 100, 77, 160), None),   # Lk = 77: unaligned scores
            ((2, 2, 200, 200, 192), (2, 1, 200, 200)), ((1, 4, 1030, 520, 256), None)]


@pytest.mark.parametrize("shape,bshape", TWO_GEMM)
def test_head_dims_above_128_run_as_two_gemms_and_a_softmax(ctx, ora, shape, bshape):
    """sdpa_coopmat! + attn_softmax_rows! (attention.jl:528-705): S = Kt Q in fp32, P = softmax over the keys in fp16,
    O = V P; against the fp32 reference at the fused kernel's tolerance and the three-pass form at 1e-2; with and
    without the additive mask (whose all-blocked rows come out as zeros)."""
    B, H, Lq, Lk, E = shape
    rng = np.random.default_rng(sum(shape))
    q = np.float16(rng.standard_normal((B, H, Lq, E)) * 0.3)
    k = np.float16(rng.standard_normal((B, H, Lk, E)) * 0.3)
    v = np.float16(rng.standard_normal((B, H, Lk, E)) * 0.3)
    bias = None
    if bshape is not None:
        bias = np.float16(rng.standard_normal(bshape))
        bias[rng.random(bshape) < 0.3] = -np.inf
        bias[:, :, 5, :] = -np.inf
    scale = 1 / np.sqrt(E)
    for out_dtype in (np.float16, np.float32):
        got, plan = attention_gpu(ctx, q, k, v, scale, out_dtype, bias=bias)
        assert isinstance(plan, jv.TwoGemmPlan), plan
        assert np.all(np.isfinite(got))
        ref = ora.attention_ref(q, k, v, scale, bias=bias)
        assert relerr(got, ref) < TOL, describe(got, ref, TOL)
        if bias is not None:
            assert np.all(got[:, :, 5] == 0)


def test_two_gemm_route_with_heads_interleaved_in_the_token_row(ctx, ora):
    """q, k, v as views of one (tokens, 3 d) projection and the result token-major: the head and batch strides do not
    fold into one, so the route runs one batched launch per image; values are those of the dense call."""
    from .gpu_helpers import qkv_views
    rng = np.random.default_rng(77)
    B, H, L, E = 2, 2, 160, 136
    d = H * E
    qkv = np.float16(rng.standard_normal((B, L, 3, H, E)) * 0.3)
    q, k, v = (qkv[:, :, i].transpose(0, 2, 1, 3) for i in range(3))     # (B, H, L, E) strided views
    dq, dk, dv = qkv_views(ctx, q, k, v)
    assert isinstance(jv.sdpaplan(ctx, dq, dk, dv), jv.TwoGemmPlan)
    buf = ctx.allocate(np.float16, d, L, B)
    ctx.fill_bytes(buf, 0xFF)
    view = jv.DeviceArray(ctx, buf.ptr, np.float16, (E, L, H, B), (1, d, E, d * L), owner=buf)
    jv.sdpa(ctx, dq, dk, dv, None, 1 / np.sqrt(E), out=view)
    ctx.synchronize()
    got = buf.to_host().reshape(B, L, H, E).transpose(0, 2, 1, 3)
    ref = ora.attention_ref(np.ascontiguousarray(q), np.ascontiguousarray(k), np.ascontiguousarray(v), 1 / np.sqrt(E))
    assert relerr(got, ref) < TOL, describe(got, ref, TOL)


def test_head_dim_not_a_multiple_of_eight_takes_the_scalar_kernel(ctx, ora):
    rng = np.random.default_rng(12)
    q, k, v = (np.float16(rng.standard_normal((1, 2, 64, 132)) * 0.2) for _ in range(3))
    got, plan = attention_gpu(ctx, q, k, v, 1 / np.sqrt(132), np.float32)
    assert isinstance(plan, jv.AttnScalarPlan)
    assert relerr(got, ora.attention_ref(q, k, v, 1 / np.sqrt(132))) < TOL


# torch (B,H,Lq,Lk,E) and the bias shape as torch (B|1, H|1, Lq|1, Lk|1)
BIAS_CASES = [((2, 3, 256, 384, 64), (2, 3, 256, 384)),    # full mask, rows read 8 keys at a time
              ((2, 3, 300, 200, 56), (2, 3, 300, 200)),    # ragged keys: the guarded scalar reads
              ((2, 4, 256, 256, 64), (2, 1, 1, 256)),      # key-padding mask broadcast over heads and queries
              ((1, 2, 130, 257, 32), (1, 1, 130, 257)),    # broadcast over heads, odd row stride
              ((1, 2, 64, 64, 72), (1, 2, 64, 64)),        # head dim past one swizzle row: two atoms along E
              ((2, 2, 300, 260, 96), (2, 1, 300, 260)),
              ((1, 1, 40, 40, 132), (1, 1, 40, 40))]       # not a multiple of 8: scalar kernel


@pytest.mark.parametrize("shape,bshape", BIAS_CASES)
def test_additive_bias_vs_oracle(ctx, ora, shape, bshape):
    """The additive mask of the mem-efficient variant (attention.jl:55-59), which the reference runs
    unfused: random finite values, -inf on a share of the keys, and some rows blocked entirely."""
    B, H, Lq, Lk, E = shape
    rng = np.random.default_rng(sum(shape) + sum(bshape))
    q = np.float16(rng.standard_normal((B, H, Lq, E)))
    k = np.float16(rng.standard_normal((B, H, Lk, E)))
    v = np.float16(rng.standard_normal((B, H, Lk, E)))
    bias = np.float16(rng.standard_normal(bshape))
    bias[rng.random(bshape) < 0.3] = -np.inf
    if bshape[2] > 1:
        bias[:, :, 5, :] = -np.inf            # a query every key is hidden from
        bias[:, :, bshape[2] - 1, : Lk // 2] = -np.inf
    scale = 1 / np.sqrt(E)
    for out_dtype in (np.float16, np.float32):
        got, plan = attention_gpu(ctx, q, k, v, scale, out_dtype, bias=bias)
        assert isinstance(plan, jv.FlashTCPlan if E <= 128 else jv.AttnScalarPlan), plan
        assert np.all(np.isfinite(got))
        ref = ora.attention_ref(q, k, v, scale, bias=bias)
        assert relerr(got, ref) < TOL, describe(got, ref, TOL)
        if bshape[2] > 1:
            assert np.all(got[:, :, 5] == 0)   # all keys blocked: a zero row (attention.jl:73-100)
        tp = ora.attention_threepass(q, k, v, scale, bias=bias)
        assert relerr(got, tp) < 1e-2, describe(got, tp, 1e-2)


def test_zero_bias_changes_nothing(ctx):
    rng = np.random.default_rng(5)
    q, k, v = (np.float16(rng.standard_normal((1, 2, 256, 64))) for _ in range(3))
    plain, _ = attention_gpu(ctx, q, k, v, 0.125)
    masked, _ = attention_gpu(ctx, q, k, v, 0.125, bias=np.zeros((1, 1, 256, 256), np.float16))
    assert relerr(masked, plain) < 1e-3


def test_declines(ctx):
    q = ctx.allocate(np.float16, 64, 128, 2, 1)
    assert jv.sdpaplan(ctx, q, q, q, bias=q) == jv.Decline("bias")          # a mask that does not broadcast
    q32 = ctx.allocate(np.float32, 64, 128, 2, 1)
    assert jv.sdpaplan(ctx, q32, q32, q32) == jv.Decline("eltype")
    k = ctx.allocate(np.float16, 32, 128, 2, 1)
    assert jv.sdpaplan(ctx, q, k, k) == jv.Decline("extent")
    with pytest.raises(jv.B200Error):
        jv.sdpa(ctx, q, q, q, bias=q)


def test_config2_properties_at_full_size(ctx):
    """BASELINE config 2 (B1 H12 L4096 E64). Size-independent checks: V = 1 gives exactly-normalised
    rows, attention is linear in V, and permuting the keys (with their values) changes nothing
    beyond rounding."""
    rng = np.random.default_rng(20260102)
    B, H, L, E = 1, 12, 4096, 64
    q = np.float16(rng.standard_normal((B, H, L, E)))
    k = np.float16(rng.standard_normal((B, H, L, E)))
    v = np.float16(rng.standard_normal((B, H, L, E)))
    ones = np.ones_like(v)
    o1, _ = attention_gpu(ctx, q, k, ones, 0.125, np.float32)
    assert np.max(np.abs(o1 - 1)) < 2e-3
    ov, _ = attention_gpu(ctx, q, k, v, 0.125, np.float32)
    o2v, _ = attention_gpu(ctx, q, k, np.float16(2) * v, 0.125, np.float32)
    assert np.max(np.abs(o2v - 2 * ov)) < 1e-5 * max(1.0, float(np.max(np.abs(ov))))
    perm = rng.permutation(L)
    op, _ = attention_gpu(ctx, q, k[:, :, perm], v[:, :, perm], 0.125, np.float32)
    assert relerr(op, ov) < TOL


def test_config2_sample_rows_vs_oracle(ctx, ora):
    """Config 2 at full key length, checked against the oracle on a sample of query rows."""
    rng = np.random.default_rng(20260103)
    B, H, L, E = 1, 12, 4096, 64
    q, k, v = (np.float16(rng.standard_normal((B, H, L, E))) for _ in range(3))
    got, _ = attention_gpu(ctx, q, k, v, 0.125)
    rows = np.sort(rng.choice(L, 64, replace=False))
    ref = ora.attention_ref(np.ascontiguousarray(q[:, :, rows]), k, v, 0.125)
    assert relerr(got[:, :, rows], ref) < TOL, describe(got[:, :, rows], ref, TOL)


@pytest.mark.parametrize("B,H,Lq,Lk,E", [(512, 2, 64, 64, 56), (1024, 4, 16, 64, 56), (300, 2, 64, 64, 64), (256, 2, 49, 49, 32),
                                         (200, 3, 100, 40, 8), (400, 1, 1, 64, 16), (310, 1, 23, 1, 24), (150, 2, 129, 64, 48),
                                         (16, 8, 256, 256, 56), (40, 2, 64, 256, 56), (64, 3, 130, 200, 64), (90, 2, 17, 65, 16)])
def test_many_small_windows(ctx, ora, B, H, Lq, Lk, E):
    """Attention windows of a few dozen tokens, token-major with the windows back to back (what the image
    encoder hands over): many of them take the small-tile kernel (64 queries of one window and head per
    CTA).  Values must be those of independent windows: checked against the oracle window by window, and
    a window's result must not change when its neighbours do."""
    from .gpu_helpers import qkv_views
    rng = np.random.default_rng(B + Lq + Lk)
    qb = np.float16(rng.standard_normal((B, Lq, H, E)))
    kb = np.float16(rng.standard_normal((B, Lk, H, E)))
    vb = np.float16(rng.standard_normal((B, Lk, H, E)))
    q, k, v = (t.transpose(0, 2, 1, 3) for t in (qb, kb, vb))            # torch (B,H,L,E) views
    scale = 1 / np.sqrt(E)

    def run(q, k, v):
        dq, dk, dv = qkv_views(ctx, q, k, v)
        buf = ctx.allocate(np.float16, E * H, Lq, B)                      # torch (B, Lq, H*E)
        ctx.fill_bytes(buf, 0xFF)
        view = jv.DeviceArray(ctx, buf.ptr, np.float16, (E, Lq, H, B), (1, E * H, E, E * H * Lq), owner=buf)
        jv.sdpa(ctx, dq, dk, dv, None, scale, out=view)
        ctx.synchronize()
        return buf.to_host().reshape(B, Lq, H, E).transpose(0, 2, 1, 3)

    got = run(q, k, v)
    ref = ora.attention_ref(q, k, v, scale)
    assert np.all(np.isfinite(got))
    assert relerr(got, ref) < TOL, describe(got, ref, TOL)
    kb2, vb2 = kb.copy(), vb.copy()
    kb2[1::2] = np.float16(rng.standard_normal(kb2[1::2].shape) * 3)       # disturb every other window
    vb2[1::2] = 7
    got2 = run(q, kb2.transpose(0, 2, 1, 3), vb2.transpose(0, 2, 1, 3))
    assert np.array_equal(got2[0::2], got[0::2])


@pytest.mark.parametrize("B,H,Lq,Lk,E", [(512, 2, 64, 64, 56), (300, 1, 70, 33, 40)])
def test_many_small_windows_dense_fp32_out(ctx, ora, B, H, Lq, Lk, E):
    """The same windows from dense (B,H,L,E) arrays into an fp32 result (the attn_flash! contract)."""
    from .gpu_helpers import qkv_views
    rng = np.random.default_rng(B + Lq + Lk + 1)
    q = np.float16(rng.standard_normal((B, H, Lq, E)))
    k = np.float16(rng.standard_normal((B, H, Lk, E)))
    v = np.float16(rng.standard_normal((B, H, Lk, E)))
    scale = 1 / np.sqrt(E)
    dq, dk, dv = qkv_views(ctx, q, k, v)
    out = ctx.allocate(np.float32, E, Lq, H, B)
    ctx.fill_bytes(out, 0xFF)
    jv.sdpa(ctx, dq, dk, dv, None, scale, out=out)
    ctx.synchronize()
    got = out.to_host()
    ref = ora.attention_ref(q, k, v, scale)
    assert np.all(np.isfinite(got))
    assert relerr(got, ref) < TOL, describe(got, ref, TOL)


@pytest.mark.parametrize("B,H,Lq,Lk,E", [(1, 8, 23, 4096, 64), (2, 3, 1, 4000, 56), (1, 1, 300, 2048, 32), (1, 20, 130, 1500, 64),
                                         (1, 20, 2000, 2000, 64),     # 160 query pairs: the 12 of the last wave are cut, one of them ragged
                                         (1, 39, 1000, 700, 40)])      # 156 pairs, 8 cut three ways, ragged queries and keys
def test_few_queries_many_keys_split_and_merged(ctx, ora, B, H, Lq, Lk, E):
    """Decode-like shapes (flash.jl:298-323: Lq = 23, Lk = 4096): the keys are split over several CTAs
    per query tile and merged (attn_flash_cm_merge!); the values are those of the unsplit computation."""
    rng = np.random.default_rng(Lq + Lk + E)
    q = np.float16(rng.standard_normal((B, H, Lq, E)))
    k = np.float16(rng.standard_normal((B, H, Lk, E)))
    v = np.float16(rng.standard_normal((B, H, Lk, E)))
    k[:, :, Lk // 2] *= 4          # a late key that moves the running maximum of some rows
    scale = 1 / np.sqrt(E)
    ref = ora.attention_ref(q, k, v, scale)
    for out_dtype in (np.float16, np.float32):
        got, plan = attention_gpu(ctx, q, k, v, scale, out_dtype)
        assert isinstance(plan, jv.FlashTCPlan)
        assert relerr(got, ref) < TOL, describe(got, ref, TOL)


# masked, keys contiguous: even and odd row strides of the mask (rows that start in the middle of a word), one key
# more and less than a block, a mask wider than its rows, and shapes whose keys are split and merged
MASKED = [((1, 2, 300, 1500, 64), (1, 1, 300, 1500), 0), ((1, 1, 257, 129, 64), (1, 1, 257, 129), 0),
          ((1, 2, 129, 127, 72), (1, 2, 129, 127), 0), ((1, 1, 130, 1, 64), (1, 1, 130, 1), 0),
          ((2, 2, 140, 383, 128), (2, 1, 140, 383), 3), ((1, 3, 3, 477, 64), (1, 1, 3, 477), 0),
          ((1, 4, 23, 2049, 72), (1, 1, 23, 2049), 1), ((1, 2, 260, 1030, 96), (1, 1, 1, 1030), 0)]


@pytest.mark.parametrize("shape,bshape,extra", MASKED)
def test_masked_blocks_staged_ahead(ctx, ora, shape, bshape, extra):
    B, H, Lq, Lk, E = shape
    rng = np.random.default_rng(sum(shape) + extra)
    q, k, v = (np.float16(rng.standard_normal((B, H, n, E))) for n in (Lq, Lk, Lk))
    bias = np.float16(rng.standard_normal(bshape))
    bias[rng.random(bshape) < 0.2] = -np.inf
    bias[rng.random(bshape) < 0.1] = -65504
    bias[..., -1, :Lk // 2] = -np.inf          # a row that has seen nothing after its first blocks (or split)
    if bshape[2] > 2:
        bias[..., 1, :] = -np.inf
    wide = np.full(bshape[:3] + (Lk + extra,), np.nan, np.float16)      # the mask as a slice of a wider array
    wide[..., :Lk] = bias
    dq, dk, dv = (ctx.toback(a) for a in (q, k, v))
    db = ctx.toback(wide).slice(0, 0, Lk)
    out = ctx.allocate(np.float32, E, Lq, H, B)
    ctx.fill_bytes(out, 0xFF)
    ctx.ws.reset()
    jv.sdpa(ctx, dq, dk, dv, db, 1 / np.sqrt(E), out=out)
    ctx.synchronize()
    got, ref = out.to_host(), ora.attention_ref(q, k, v, 1 / np.sqrt(E), bias=bias)
    assert np.all(np.isfinite(got))
    assert relerr(got, ref) < TOL, describe(got, ref, TOL)
    if bshape[2] > 2:
        assert np.all(got[:, :, 1] == 0)


# (B, H, Lq, Lk, E): the edges of the query tiles (16, 32) and of the key blocks (64), one block and 128 of them, every
# width of head, parts of a cluster that get different numbers of blocks
FEW = [(1, 1, 1, 1, 8), (1, 2, 16, 63, 64), (2, 3, 17, 64, 56), (1, 5, 16, 65, 72), (1, 2, 9, 129, 128), (1, 1, 32, 8192, 64),
       (1, 5, 32, 65, 40), (1, 19, 7, 345, 56), (1, 8, 13, 4096, 80), (3, 4, 5, 1003, 128), (40, 8, 16, 49, 72)]


@pytest.mark.parametrize("B,H,Lq,Lk,E", FEW)
@pytest.mark.parametrize("masked", [False, True])
def test_few_queries_in_one_launch(ctx, ora, B, H, Lq, Lk, E, masked):
    rng = np.random.default_rng(B + H + Lq + Lk + E)
    buf = np.float16(rng.standard_normal((B, Lk, 2, H, E)))              # keys and values side by side
    k, v = (buf[:, :, i].transpose(0, 2, 1, 3) for i in range(2))
    q = np.float16(rng.standard_normal((B, H, Lq, E)))
    bias = None
    if masked:
        bias = np.float16(rng.standard_normal((B, 1, Lq, Lk)))
        bias[rng.random(bias.shape) < 0.2] = -np.inf
        bias[:, :, 0, : Lk // 2] = -np.inf
        bias[:, :, Lq - 1] = -np.inf
    ref = ora.attention_ref(q, k, v, 1 / np.sqrt(E), bias=bias)
    for out_dtype in (np.float16, np.float32):
        n0 = ctx.launch_count()
        got, plan = attention_gpu(ctx, q, k, v, 1 / np.sqrt(E), out_dtype, bias=bias)
        assert isinstance(plan, jv.FlashTCPlan) and ctx.launch_count() - n0 == 1
        assert np.all(np.isfinite(got))
        # P is rounded to fp16 (2^-11 per key, averaged over them) and, for fp16, the result once more
        assert relerr(got, ref) < 2e-3, describe(got, ref, 2e-3)
        if masked:
            assert np.all(got[:, :, Lq - 1] == 0)


# (B, H, Lq, Lk, E) with more than 296 query tiles: one key past the window kernel's, one block and four of them, ragged
# tiles, one query past the few-query kernel's
SHORT = [(150, 2, 65, 65, 64), (300, 1, 33, 129, 32), (100, 3, 130, 200, 56), (75, 4, 256, 256, 64), (160, 2, 100, 64 * 3, 8)]


@pytest.mark.parametrize("B,H,Lq,Lk,E", SHORT)
def test_short_keys_share_an_sm(ctx, ora, B, H, Lq, Lk, E):
    """One query tile per CTA, four CTAs per SM; operands side by side in one projection, result token-major."""
    rng = np.random.default_rng(B + Lq + Lk)
    buf = np.float16(rng.standard_normal((B, max(Lq, Lk), 3, H, E)))
    q, k, v = (buf[:, :n, i].transpose(0, 2, 1, 3) for i, n in enumerate((Lq, Lk, Lk)))
    dq, dk, dv = qkv_views(ctx, q, k, v)
    ref = ora.attention_ref(q, k, v, 1 / np.sqrt(E))
    for dt in (np.float16, np.float32):
        flat = ctx.allocate(dt, E * H, Lq * B)
        ctx.fill_bytes(flat, 0xFF)
        out = jv.DeviceArray(ctx, flat.ptr, dt, (E, Lq, H, B), (1, E * H, E, E * H * Lq), owner=flat)
        ctx.ws.reset()
        jv.sdpa(ctx, dq, dk, dv, None, 1 / np.sqrt(E), out=out)
        ctx.synchronize()
        got = flat.to_host().reshape(B, Lq, H, E).transpose(0, 2, 1, 3)
        assert np.all(np.isfinite(got))
        # P is rounded to fp16 (2^-11 per key, averaged over them) and, for fp16, the result once more
        assert relerr(got, ref) < 2e-3, describe(got, ref, 2e-3)


@pytest.mark.parametrize("first,best", [(3, 5), (3, 64), (63, 127), (10, 100)])
@pytest.mark.parametrize("Lk", [128, 196, 256])
def test_the_heaviest_of_the_first_128_keys_is_not_rounded(ctx, Lk, first, best):
    """One key holds nearly all of a row's weight, another up to 2^8 less, the rest nothing.  The heavy one lies in the
    first 128 keys, so its probability is the reference point of the exponentials and exact: what is left is the
    rounding of the light one (at least 2^-6 of the weight at 2^-11) and of fp32.  Whole tiles, four CTAs per SM."""
    B, H, Lq, E = 160, 2, 128, 64
    rng = np.random.default_rng(Lk + best)
    q, k = np.zeros((B, H, Lq, E), np.float16), np.zeros((B, H, Lk, E), np.float16)
    q[..., 0] = 1
    k[..., 0] = -20                                    # 2^-28 of the first key
    k[:, :, first, 0] = 0
    k[:, :, best, 0] = 4.2 + 1.3 * rng.random((B, H))   # 2^6 to 2^7.95 times the first key
    v = np.float16(rng.standard_normal((B, H, Lk, E)))
    got, _ = attention_gpu(ctx, q, k, v, 1.0, np.float32)
    s = k[..., 0].astype(np.float64)
    p = np.exp(s - s.max(-1, keepdims=True))
    ref = np.einsum("bhk,bhke->bhe", p / p.sum(-1, keepdims=True), v.astype(np.float64))[:, :, None]
    # 2^-6 * 2^-11 of the light key's value, plus a few fp32 roundings, against values of size one
    err = np.abs(got - ref).max() / np.abs(ref).max()
    assert err < 1.2e-5, err


@pytest.mark.parametrize("B,H,Lq,Lk,E,masked", [(1, 2, 300, 1500, 64, True), (1, 3, 40, 2000, 128, True), (1, 36, 32, 4096, 64, False),
                                                (1, 36, 16, 8192, 72, True)])
def test_masked_calls_and_few_queries_do_not_depend_on_the_workspace(ora, B, H, Lq, Lk, E, masked):
    """Shapes whose keys the large kernel splits.  Recorded on a context that has no workspace yet, a masked call and one of
    few queries run (unsplit); run eagerly again and again without a reset, they leave the workspace as they found it."""
    rng = np.random.default_rng(Lq)
    q, k, v = (np.float16(rng.standard_normal((B, H, n, E))) for n in (Lq, Lk, Lk))
    bias = None
    if masked:
        bias = np.float16(rng.standard_normal((1, 1, Lq, Lk)))
        bias[rng.random(bias.shape) < 0.2] = -np.inf
    ref = ora.attention_ref(q, k, v, 1 / np.sqrt(E), bias=bias)
    with jv.Ctx(0) as c:
        dq, dk, dv, db = (None if a is None else c.toback(a) for a in (q, k, v, bias))
        out = c.allocate(np.float32, E, Lq, H, B)
        call = lambda: jv.sdpa(c, dq, dk, dv, db, 1 / np.sqrt(E), out=out)
        c.fill_bytes(out, 0xFF)
        g = c.capture(call)
        assert c.ws.stats()[1] == 0
        g.replay()
        c.synchronize()
        assert relerr(out.to_host(), ref) < 2e-3      # P rounded to fp16
        call()
        cap = c.ws.stats()
        assert cap[0] == 0 and cap[1] > 0             # split, and its scratch given back
        for _ in range(20):
            c.fill_bytes(out, 0xFF)
            call()
        c.synchronize()
        assert c.ws.stats() == cap
        assert relerr(out.to_host(), ref) < 2e-3


@pytest.mark.parametrize("B,H,Lq,Lk,E", FEW)
@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("most", [16, 1])
def test_few_queries_whatever_is_faster(ctx, ora, B, H, Lq, Lk, E, masked, most, monkeypatch):
    """The shapes above on the kernel of few queries also where the large one is the faster, cut as far as the keys
    allow and not at all."""
    monkeypatch.setenv("B200_ATTENTION_PARTS", str(most))
    test_few_queries_in_one_launch(ctx, ora, B, H, Lq, Lk, E, masked)


@pytest.mark.parametrize("B,H,Lq,Lk,E", [(1, 2, 23, 4096, 64), (1, 3, 5, 4500, 128)])
def test_few_queries_with_smaller_clusters(ctx, ora, B, H, Lq, Lk, E, monkeypatch):
    """Clusters of sixteen are more than every device must hold: the same kernel with the keys over eight CTAs and fewer,
    down to one, which walk the ring up to sixteen times as often.  fp32 shows that the split did change."""
    rng = np.random.default_rng(Lk)
    q, k, v = (np.float16(rng.standard_normal((B, H, n, E))) for n in (Lq, Lk, Lk))
    ref = ora.attention_ref(q, k, v, 1 / np.sqrt(E))
    seen = []
    for most in (16, 8, 4, 2, 1):
        monkeypatch.setenv("B200_ATTENTION_PARTS", str(most))
        got, _ = attention_gpu(ctx, q, k, v, 1 / np.sqrt(E), np.float32)
        assert relerr(got, ref) < 2e-3, (most, describe(got, ref, 2e-3))     # P rounded to fp16
        assert not any(np.array_equal(got, s) for s in seen), most
        seen.append(got)


# a CTA each, on either side of the rule's lines (three, four and fourteen units an SM) and of few keys, and walking CTAs of at
# most one unit and of many
@pytest.mark.parametrize("E,Lq,Lk,H,B,dt", [(56, 64, 64, 3, 500, np.float16), (64, 49, 49, 2, 700, np.float16), (8, 70, 5, 3, 333, np.float32),
                                            (40, 16, 64, 5, 601, np.float16), (56, 129, 33, 2, 297, np.float16),
                                            (56, 64, 64, 5, 100, np.float16), (64, 50, 64, 7, 127, np.float16), (40, 65, 33, 4, 40, np.float32),
                                            (56, 64, 64, 4, 111, np.float32), (24, 17, 1, 6, 148, np.float16), (64, 100, 32, 3, 900, np.float16),
                                            (64, 49, 49, 3, 700, np.float16), (8, 70, 33, 4, 300, np.float32), (56, 129, 40, 2, 360, np.float16)])
def test_windows_walked_in_turn(ctx, ora, E, Lq, Lk, H, B, dt):
    """Both forms on either side of their rule: head dims and key counts that leave columns and rows of zeros, buffers used
    again, query tiles of different fill next to each other, and a window of NaN that must not reach its neighbours."""
    rng = np.random.default_rng(E + Lq + Lk)
    q = np.float16(rng.standard_normal((B, H, Lq, E)))
    k, v = (np.float16(rng.standard_normal((B, H, Lk, E))) for _ in range(2))
    q[3] = np.nan
    out = ctx.allocate(dt, E, Lq, H, B)
    ctx.fill_bytes(out, 0xFF)
    ctx.ws.reset()
    jv.sdpa(ctx, ctx.toback(q), ctx.toback(k), ctx.toback(v), None, 1.0 / math.sqrt(E), out=out)
    ctx.synchronize()
    got = out.to_host().astype(np.float64)
    s = np.einsum("bhqe,bhke->bhqk", q.astype(np.float64), k.astype(np.float64)) / math.sqrt(E)
    pr = np.exp(s - s.max(-1, keepdims=True))
    ref = np.einsum("bhqk,bhke->bhqe", pr / pr.sum(-1, keepdims=True), v.astype(np.float64))
    assert np.all(np.isnan(got[3]))
    keep = np.arange(B) != 3
    # P rounded to fp16 (2^-11 relative, against values of order one), and one rounding of the result
    assert np.all(np.isfinite(got[keep])) and np.max(np.abs(got[keep] - ref[keep])) < 5e-3


def test_more_than_2_to_the_30_windows(ctx):
    """Heads x batch past 2^30, which the walk over the windows counts: one query and one key each, so that the result is v,
    out of operands that overlap; 17 GB of results, a few planes of them read back."""
    E, H, B = 8, 65535, 16385
    v = np.float16(np.random.default_rng(30).standard_normal(8 * (H + B)))
    d = ctx.toback(v)
    view = jv.DeviceArray(ctx, d.ptr, np.float16, (E, 1, H, B), (1, 8, 8, 8), owner=d)
    out = ctx.allocate(np.float16, E, 1, H, B)
    ctx.fill_bytes(out, 0xFF)
    jv.sdpa(ctx, view, view, view, None, 1.0, out=out)
    ctx.synchronize()
    for b in (0, 1, 8191, 8192, 16383, 16384):
        plane = jv.DeviceArray(ctx, out.ptr + b * H * E * 2, np.float16, (E, H), owner=out)
        assert np.array_equal(plane.to_host(), v[8 * b:8 * (b + H)].reshape(H, E)), b


@pytest.mark.parametrize("E", [56, 64, 72, 80, 96])
@pytest.mark.parametrize("Lq,Lk", [(300, 33), (129, 97), (128, 128), (257, 225), (1, 700), (300, 1025)])
def test_reference_point_that_moves_in_later_blocks(ctx, E, Lq, Lk):
    """Scores that grow from key block to key block, slowly enough to be let through or by more than 2^8 at once; the
    last 32 keys of a block take another way to the product for some head dims."""
    rng = np.random.default_rng(E + 7 * Lq + Lk)
    q, k, v = (np.float16(rng.standard_normal((2, 3, n, E))) for n in (Lq, Lk, Lk))
    grow = np.where(np.arange(Lk) // 128 % 3 == 2, 1.0 + np.arange(Lk) // 128, 1.0) * np.where(np.arange(Lk) % 128 >= 96, 1.5, 1.0)
    k = np.float16(k * grow[None, None, :, None])
    got, plan = attention_gpu(ctx, q, k, v, 0.5, np.float32)
    assert isinstance(plan, jv.FlashTCPlan)
    s = np.einsum("bhqe,bhke->bhqk", np.float64(q), np.float64(k)) * 0.5
    p = np.exp(s - s.max(-1, keepdims=True))
    ref = np.einsum("bhqk,bhke->bhqe", p / p.sum(-1, keepdims=True), np.float64(v))
    # P is rounded to fp16 (2^-11 of each weight, none rounded further: they lie within 2^8 of the reference point or
    # below 2^-14 of it, 2^-25 each), sums are fp32 over Lk terms
    vmax = np.abs(np.float64(v)).max()
    assert np.abs(got - ref).max() < vmax * (2.0 ** -11 + Lk * 2.0 ** -25 + 1e-5)


@pytest.mark.parametrize("B,H,Lq,Lk,E", [(1, 8, 300, 1001, 64), (2, 6, 513, 640, 56), (1, 20, 129, 1500, 72), (3, 4, 260, 2050, 128), (1, 6, 1000, 127, 64),
                                           (2, 30, 144, 24, 64), (2, 30, 29, 72, 80)])
@pytest.mark.parametrize("planes", ["all", "batch", "head", "keys"])
def test_however_a_mask_lies_the_result_is_the_same(ctx, ora, B, H, Lq, Lk, E, planes):
    """The same mask on 16-byte boundaries (read through a tensor map where its strides allow one), behind an odd number of
    entries, on 8-byte boundaries, and with its keys apart: read in place or by way of a copy, every bit is the same."""
    rng = np.random.default_rng(Lq + Lk + E)
    q, k, v = (np.float16(rng.standard_normal((B, H, n, E))) for n in (Lq, Lk, Lk))
    shape = {"all": (1, 1, Lq, Lk), "batch": (B, 1, Lq, Lk), "head": (1, H, Lq, Lk), "keys": (B, 1, 1, Lk)}[planes]
    bias = np.float16(rng.standard_normal(shape))
    bias[rng.random(shape) < 0.2] = -np.inf
    if planes != "keys":
        bias[..., Lq - 1, : Lk // 2] = -np.inf
        bias[..., 0, :] = -np.inf
    dq, dk, dv = qkv_views(ctx, q, k, v)

    def run(pitch, offset, apart):
        """`bias` in a device array whose rows are `pitch` entries apart (keys apart: whose keys are), `offset` entries in."""
        n0, n1, n2, n3 = shape
        inner, outer = (n2, n3) if apart else (n3, n2)
        flat = np.full(offset + n0 * n1 * outer * pitch, np.nan, np.float16)
        rows = flat[offset:].reshape(n0, n1, outer, pitch)[..., :inner]
        rows[...] = bias.swapaxes(2, 3) if apart else bias
        d = ctx.toback(flat)
        plane = outer * pitch
        st = (pitch, 1) if apart else (1, pitch)
        db = jv.DeviceArray(ctx, d.ptr + 2 * offset, np.float16, (n3, n2, n1, n0), st + (plane, plane * n1), owner=d)
        out = ctx.allocate(np.float32, E, Lq, H, B)
        ctx.fill_bytes(out, 0xFF)
        ctx.ws.reset()
        jv.sdpa(ctx, dq, dk, dv, db, 1 / np.sqrt(E), out=out)
        ctx.synchronize()
        return out.to_host()

    aligned = (Lk + 7) // 8 * 8
    got = run(aligned, 0, False)
    assert np.all(np.isfinite(got))
    ref = ora.attention_ref(q, k, v, 1 / np.sqrt(E), bias=bias)
    assert relerr(got, ref) < TOL, describe(got, ref, TOL)
    if planes != "keys":
        assert np.all(got[:, :, 0] == 0)
    for pitch, offset, apart in ((aligned, 5, False), (aligned + 1, 0, False), (aligned + 4, 4, False), (Lq + 3, 1, True)):
        assert np.array_equal(run(pitch, offset, apart), got), (pitch, offset, apart)


# items of two tiles, few enough to be cut over a cluster's CTAs: 2 to 8 of them, parts of uneven length, shares of rows that do
# not divide 256, a second tile of one row, every width of head
JOINED = [(1, 1, 257, 385, 64), (1, 2, 300, 900, 56), (2, 3, 500, 1700, 64), (1, 1, 256, 1100, 72), (1, 5, 700, 700, 80),
          (1, 2, 1000, 1300, 128), (1, 18, 1020, 1020, 64), (3, 1, 129, 900, 104), (1, 9, 2040, 2040, 32)]


@pytest.mark.parametrize("B,H,Lq,Lk,E", JOINED)
@pytest.mark.parametrize("masked", [False, True])
def test_keys_cut_over_a_cluster(ctx, ora, B, H, Lq, Lk, E, masked):
    rng = np.random.default_rng(B + H + Lq + Lk + E)
    q, k, v = (np.float16(rng.standard_normal((B, H, n, E))) for n in (Lq, Lk, Lk))
    k[:, :, Lk // 3:Lk // 3 + 3] *= 4                                     # the reference points of the parts differ
    bias = None
    if masked:
        bias = np.float16(rng.standard_normal((B, 1, Lq, Lk)))
        bias[rng.random(bias.shape) < 0.2] = -np.inf
        bias[:, :, 0, : Lk // 2] = -np.inf                                # parts that see nothing of a row
        bias[:, :, Lq - 1] = -np.inf
    ref = ora.attention_ref(q, k, v, 1 / np.sqrt(E), bias=bias)
    buf = ctx.allocate(np.float16, H * E, Lq * B)                         # the result token-major as well
    for out in (ctx.allocate(np.float32, E, Lq, H, B),
                jv.DeviceArray(ctx, buf.ptr, np.float16, (E, Lq, H, B), (1, H * E, E, H * E * Lq), owner=buf)):
        dq, dk, dv = qkv_views(ctx, q, k, v)
        db = None if bias is None else ctx.toback(bias)
        ctx.fill_bytes(buf if out.ptr == buf.ptr else out, 0xFF)
        ctx.ws.reset()
        n0 = ctx.launch_count()
        jv.sdpa(ctx, dq, dk, dv, db, 1 / np.sqrt(E), out=out)
        assert ctx.launch_count() - n0 <= (2 if masked else 1) and (masked or ctx.ws.stats()[0] == 0)
        ctx.synchronize()
        got = out.to_host() if out.ptr != buf.ptr else buf.to_host().reshape(B, Lq, H, E).transpose(0, 2, 1, 3)
        assert np.all(np.isfinite(got))
        # P is rounded to fp16 (2^-11 per key, averaged over them) and, for fp16, the result once more
        assert relerr(got, ref) < 2e-3, describe(got, ref, 2e-3)
        if masked:
            assert np.all(got[:, :, Lq - 1] == 0)


# one full round of items and a few (148 SMs), two rounds and 40, most that three CTAs an item leave room for, and every width
@pytest.mark.parametrize("B,H,Lq,Lk,E", [(1, 19, 2040, 900, 64), (3, 14, 1999, 700, 32), (1, 12, 4096, 520, 64), (2, 19, 1100, 1200, 72),
                                         (1, 38, 1024, 1100, 128)])
def test_a_last_round_cut_over_clusters(ctx, ora, B, H, Lq, Lk, E):
    """The items past the last full round are a second launch, whose clusters join their rows: no scratch, every row; and a layer
    norm that is launched early behind it, eagerly and recorded, finds both launches' rows over a poisoned result."""
    rng = np.random.default_rng(H + Lk)
    q, k, v = (np.float16(rng.standard_normal((B, H, n, E))) for n in (Lq, Lk, Lk))
    dq, dk, dv = qkv_views(ctx, q, k, v)
    out, z = ctx.allocate(np.float16, E, Lq, H, B), ctx.allocate(np.float16, E, Lq * H * B)
    mean, rstd = ctx.allocate(np.float32, Lq * H * B), ctx.allocate(np.float32, Lq * H * B)
    flat = jv.DeviceArray(ctx, out.ptr, np.float16, (E, Lq * H * B), owner=out)

    def norm():
        jv.layernorm_(ctx, z, mean, rstd, flat, None, None, E, 1e-5)

    def both():
        ctx.fill_bytes(out, 0xFF)
        jv.sdpa(ctx, dq, dk, dv, None, 1 / np.sqrt(E), out=out)
        norm()

    ctx.ws.reset()
    ctx.fill_bytes(out, 0xFF)
    n0 = ctx.launch_count()
    jv.sdpa(ctx, dq, dk, dv, None, 1 / np.sqrt(E), out=out)
    if ctx.dev.cores == 148:
        assert ctx.launch_count() - n0 == 2 and ctx.ws.stats()[0] == 0
    ctx.synchronize()
    norm()
    ctx.synchronize()
    got, want = out.to_host(), z.to_host()
    ref = ora.attention_ref(q, k, v, 1 / np.sqrt(E))
    # P is rounded to fp16 (2^-11 per key, averaged over them) and the result once more
    assert relerr(got, ref) < 2e-3, describe(got, ref, 2e-3)
    g = ctx.capture(both)
    for run in (both, g.replay) * 3:
        ctx.fill_bytes(z, 0xFF)
        run()
        ctx.synchronize()
        assert np.array_equal(z.to_host(), want) and np.array_equal(out.to_host(), got)
    del g


def test_a_mask_that_is_not_copied_takes_no_workspace(ora):
    """Masks off 16-byte boundaries: a plane a head, which is dearer to copy than to read in place, and one of more entries than are
    ever copied.  The workspace stays as it was found."""
    rng = np.random.default_rng(12)
    with jv.Ctx(0) as c:
        c.scratch(np.float16, 8)
        c.ws.reset()
        found = c.ws.stats()
        B, H, L, E = 2, 8, 1001, 64
        q, k, v = (np.float16(rng.standard_normal((B, H, L, E))) for _ in range(3))
        bias = np.float16(rng.standard_normal((B, H, L, L)))
        bias[rng.random(bias.shape) < 0.2] = -np.inf
        dq, dk, dv = qkv_views(c, q, k, v)
        db, out = c.toback(bias), c.allocate(np.float32, E, L, H, B)
        c.fill_bytes(out, 0xFF)
        jv.sdpa(c, dq, dk, dv, db, 1 / np.sqrt(E), out=out)
        c.synchronize()
        ref = ora.attention_ref(q, k, v, 1 / np.sqrt(E), bias=bias)
        assert relerr(out.to_host(), ref) < TOL, describe(out.to_host(), ref, TOL)
        assert c.ws.stats() == found

        H, L = 3, 11601
        dq, dk, dv = (c.toback(np.float16(rng.standard_normal((1, H, L, E)))) for _ in range(3))
        room = c.allocate(np.float16, L * L + 1)
        c.fill_bytes(room, 0)
        zeros = jv.DeviceArray(c, room.ptr + 2, np.float16, (L, L, 1, 1), owner=room)
        got, ref = (c.allocate(np.float32, E, L, H, 1) for _ in range(2))
        c.fill_bytes(got, 0xFF)
        jv.sdpa(c, dq, dk, dv, zeros, 1 / np.sqrt(E), out=got)
        c.synchronize()
        assert c.ws.stats() == found
        jv.sdpa(c, dq, dk, dv, None, 1 / np.sqrt(E), out=ref)
        c.synchronize()
        # either side rounds P to fp16 about a reference point of its own: 2^-11 of each of 11601 weights
        assert relerr(got.to_host(), ref.to_host()) < 2e-3
