import math
import os

import numpy as np
import pytest

import juliavision_b200 as jv

from .conftest import relerr
from .gpu_helpers import describe, linear_gpu

pytestmark = pytest.mark.gpu
G = os.path.join(os.path.dirname(__file__), "golden")
TOL = 1e-2  # max relative error on fp16 outputs against the fp32-accumulated oracle


def test_golden(ctx):
    g = np.load(os.path.join(G, "linear.npz"))
    for epi, key in (("identity", "y_none"), ("gelu", "y_gelu"), ("relu", "y_relu")):
        got = linear_gpu(ctx, g["X"], g["Wt"], g["b"], epi=epi)
        assert got.shape == g[key].shape
        assert relerr(got, g[key]) < 2e-3, (epi, describe(got, g[key], 2e-3))


def _case(rng, tokens, out, K, scale=0.05):
    X = (rng.standard_normal((tokens, K)) * scale).astype(np.float16)
    Wt = (rng.standard_normal((K, out)) * scale).astype(np.float16)
    b = (rng.standard_normal(out) * scale).astype(np.float16)
    return X, Wt, b


# (tokens, out features, K): aligned, ragged tokens, ragged features, ragged K, tiny, one tile each way
SHAPES = [(256, 256, 128), (128, 64, 64), (1500, 1280, 1280), (100, 1000, 768), (37, 40, 72), (300, 3072, 768),
          (129, 264, 200), (1, 8, 8), (513, 520, 1032), (2000, 112, 448)]


@pytest.mark.parametrize("tokens,out,K", SHAPES)
def test_vs_oracle(ctx, ora, tokens, out, K):
    rng = np.random.default_rng(tokens * 7 + out * 3 + K)
    X, Wt, b = _case(rng, tokens, out, K, scale=0.25)
    plan = jv.mmplan(ctx, ctx.allocate(np.float16, out, tokens), ctx.toback(Wt), ctx.toback(X))
    assert isinstance(plan, jv.MMGemvPlan if tokens == 1 else jv.MMTilePlan), plan
    for epi, bias in (("identity", b), ("gelu", b), ("relu", None)):
        got = linear_gpu(ctx, X, Wt, bias, epi=epi)
        ref = ora.linear(X, Wt, bias, epi=epi if epi != "identity" else "none")
        assert got.shape == (tokens, out)
        assert relerr(got, ref) < TOL, (epi, describe(got, ref, TOL))
        # tighter: the only differences are fp32 summation order, i.e. a last-bit flip here and there
        d = np.abs(got.astype(np.float64) - ref.astype(np.float64))
        assert np.mean(d > 4 * np.spacing(np.abs(ref)).astype(np.float64) + 1e-6) < 1e-3


def test_config1_linear(ctx, ora):
    """X 4096x768, W 3072x768, b 3072, N(0,1)*0.05, fp16 out."""
    rng = np.random.default_rng(20260101)
    X, Wt, b = _case(rng, 4096, 3072, 768)
    got = linear_gpu(ctx, X, Wt, b)
    ref = ora.linear(X, Wt, b)
    assert relerr(got, ref) < TOL, describe(got, ref, TOL)


def test_fp32_output(ctx, ora):
    rng = np.random.default_rng(5)
    X, Wt, b = _case(rng, 200, 136, 264, scale=0.25)
    got = linear_gpu(ctx, X, Wt, b, epi="gelu", out_dtype=np.float32)
    ref = ora.linear(X, Wt, b, epi="gelu", out_dtype=np.float32)
    assert got.dtype == np.float32
    assert relerr(got, ref) < 1e-4, describe(got, ref, 1e-4)


def test_unaligned_operands_take_the_scalar_kernel_bit_exact(ctx, ora):
    """lda = 37 cannot be a tensor-map stride: the scalar kernel runs mm2's arithmetic, so the
    result equals the oracle bit for bit."""
    rng = np.random.default_rng(6)
    X, Wt, b = _case(rng, 50, 37, 96, scale=0.25)
    plan = jv.mmplan(ctx, ctx.allocate(np.float16, 37, 50), ctx.toback(Wt), ctx.toback(X))
    assert isinstance(plan, jv.MMScalarPlan)
    got = linear_gpu(ctx, X, Wt, b, epi="relu")
    assert np.array_equal(got, ora.linear(X, Wt, b, epi="relu"))


# (tokens, out, K) with an odd `out`: one to eight token tiles and a second block of them, fewer columns than one step,
# reductions split over a cluster or staged in several chunks, a leading dimension of the tokens off 8 elements
UNALIGNED = [(2, 65, 512), (5, 4099, 1280), (8, 121, 640), (9, 1001, 72), (17, 1337, 712), (33, 57003, 16), (64, 1001, 1408),
             (65, 333, 403), (130, 113, 2000), (7, 51865, 129)]


@pytest.mark.parametrize("tokens,out,K", UNALIGNED)
@pytest.mark.parametrize("out_dtype,epi", [(np.float16, "gelu"), (np.float32, "identity")])
def test_unaligned_rows_on_the_tensor_cores(ctx, ora, tokens, out, K, out_dtype, epi):
    """Operands no tensor map can express, from 32 k elements of A up: A and the output start one element into an
    allocation whose neighbours hold NaN, so every column has its own offset from a 16-byte boundary."""
    rng = np.random.default_rng(tokens + out + K)
    X, Wt, b = _case(rng, tokens, out, K, scale=0.25)
    pad = np.full(K * out + 16, np.nan, np.float16)
    pad[1:1 + K * out] = Wt.reshape(-1)
    base = ctx.toback(pad)
    A = jv.DeviceArray(ctx, base.ptr + 2, np.float16, (out, K), owner=base)
    es = np.dtype(out_dtype).itemsize
    dest = ctx.allocate(out_dtype, out * tokens + 2)
    ctx.fill_bytes(dest, 0xFF)
    Y = jv.DeviceArray(ctx, dest.ptr + es, out_dtype, (out, tokens), owner=dest)
    jv.matmul_(ctx, Y, A, ctx.toback(X), ctx.toback(b), epi=epi)
    ctx.synchronize()
    flat = dest.to_host()
    got, ref = flat[1:-1].reshape(tokens, out), ora.linear(X, Wt, b, epi=epi, out_dtype=out_dtype)
    assert np.isnan(flat[0]) and np.isnan(flat[-1]), "wrote outside the output"
    # fp32 sums in another order: sqrt(K) eps32 against the sums' own size, one fp16 rounding step for fp16 results
    tol = 2e-3 if out_dtype == np.float16 else 2e-5
    assert relerr(got, ref) < tol, describe(got, ref, tol)


def test_batched(ctx, ora):
    rng = np.random.default_rng(7)
    nb, m, k, n = 6, 70, 64, 136
    a = (rng.standard_normal((nb, m, k)) * 0.25).astype(np.float16)
    b = (rng.standard_normal((nb, k, n)) * 0.25).astype(np.float16)
    A, B = ctx.toback(b), ctx.toback(a)          # reference orientation: A = torch b (n,k,nb), B = torch a (k,m,nb)
    out = ctx.allocate(np.float16, n, m, nb)
    ctx.fill_bytes(out, 0xFF)
    jv.batchedmatmul_(ctx, out, A, B)
    ctx.synchronize()
    got = out.to_host()
    ref = ora.bmm(a, b)
    assert relerr(got, ref) < TOL, describe(got, ref, TOL)


@pytest.mark.parametrize("tile", ["320x2", "256x2s", "128x1"])
def test_batched_under_forced_schedules(ctx, ora, tile, monkeypatch):
    """Several planes through the wide tile, a split along K and single-CTA tiles: the plane index is the third
    coordinate of every tensor map and part of the tile index, whatever the schedule."""
    monkeypatch.setenv("B200_GEMM_TILE", tile)
    rng = np.random.default_rng(17)
    nb, m, k, n = 3, 300, 640, 712
    a = (rng.standard_normal((nb, m, k)) * 0.25).astype(np.float16)
    b = (rng.standard_normal((nb, k, n)) * 0.25).astype(np.float16)
    A, B = ctx.toback(b), ctx.toback(a)
    out = ctx.allocate(np.float16, n, m, nb)
    ctx.fill_bytes(out, 0xFF)
    jv.batchedmatmul_(ctx, out, A, B)
    ctx.synchronize()
    assert relerr(out.to_host(), ora.bmm(a, b)) < TOL


def test_padded_leading_dimensions(ctx, ora):
    """Views into wider buffers (ld > extent): the bytes outside the view stay untouched."""
    rng = np.random.default_rng(8)
    tokens, out, K = 130, 72, 80
    X, Wt, b = _case(rng, tokens, out, K, scale=0.25)
    big = ctx.allocate(np.float16, 96, tokens)
    ctx.fill_bytes(big, 0xFF)
    view = big.slice(0, 0, out)                   # (72, tokens) with ld 96
    jv.matmul_(ctx, view, ctx.toback(Wt), ctx.toback(X), ctx.toback(b))
    ctx.synchronize()
    host = big.to_host()                          # torch (tokens, 96)
    assert relerr(host[:, :out], ora.linear(X, Wt, b)) < TOL
    assert np.all(np.isnan(host[:, out:]))


def test_declines(ctx):
    a32 = ctx.allocate(np.float32, 64, 64)
    a16 = ctx.allocate(np.float16, 64, 64)
    assert jv.mmplan(ctx, a16, a32, a16) == jv.Decline("operands")       # test_batchedmatmul.jl:107-125
    assert jv.mmplan(ctx, a16, a16, ctx.allocate(np.float16, 32, 64)) == jv.Decline("extent")
    with pytest.raises(jv.B200Error):
        jv.matmul_(ctx, a16, a32, a16)
    empty = ctx.allocate(np.float16, 64, 0)
    assert jv.mmplan(ctx, empty, a16, empty) == jv.Decline("extent")


def test_linearity_at_full_size(ctx):
    """Size-independent property at the bench's size: W = [I;0] copies X, and f(X1+X2) = f(X1)+f(X2)
    for operands whose sums are exact in fp16."""
    tokens, K, out = 4096, 768, 3072
    rng = np.random.default_rng(9)
    X = rng.integers(-8, 9, (tokens, K)).astype(np.float16)
    Wt = np.zeros((K, out), np.float16)
    Wt[np.arange(K), np.arange(K)] = 1
    got = linear_gpu(ctx, X, Wt)
    assert np.array_equal(got[:, :K], X) and not got[:, K:].any()
    W2 = rng.integers(-2, 3, (K, out)).astype(np.float16)
    X2 = rng.integers(-2, 3, (tokens, K)).astype(np.float16)
    X1 = rng.integers(-2, 3, (tokens, K)).astype(np.float16)
    y1, y2, y12 = (linear_gpu(ctx, x, W2, out_dtype=np.float32) for x in (X1, X2, X1 + X2))
    assert np.array_equal(y1 + y2, y12)           # integer-valued: every partial sum is exact


@pytest.mark.parametrize("tile", ["256x2", "128x2", "256x1", "128x1", "64x1", "256x2s", "128x2s", "256x1s", "64x1s",
                                  "272x2", "320x2", "384x2", "432x2", "512x2"])
def test_every_tile_shape_and_schedule(ctx, ora, tile, monkeypatch):
    """The planner picks one (tile width, CTAs per tile, schedule) per call; the debugging override
    forces each of them in turn — CTA pairs, single CTAs, whole-tile and stream-K schedules (a
    trailing `s`), the wide single-accumulator tile at several widths (a width above 256) — on shapes
    with ragged tails, several tiles per worker and tiles cut across workers.  All must agree with the oracle like the planner's own choice does."""
    monkeypatch.setenv("B200_GEMM_TILE", tile)
    rng = np.random.default_rng(hash(tile) % 1000)
    for tokens, out, K in ((1500, 1280, 1280), (700, 5120, 640), (300, 1000, 4096), (4096, 3072, 768)):
        X, Wt, b = _case(rng, tokens, out, K, scale=0.25)
        got = linear_gpu(ctx, X, Wt, b, epi="gelu")
        ref = ora.linear(X, Wt, b, epi="gelu")
        assert relerr(got, ref) < TOL, (tile, tokens, out, K, describe(got, ref, TOL))


@pytest.mark.parametrize("tile", ["64x1k2", "64x1k8", "128x1k2", "128x1k3", "128x1k8"])
@pytest.mark.parametrize("tokens,out,K", [(2, 8, 512), (129, 264, 530), (300, 200, 1288), (17, 1000, 4264)])
def test_tiles_shared_by_a_cluster(ctx, ora, tile, tokens, out, K, monkeypatch):
    """K split over a cluster's CTAs: even and uneven parts (one k-block each at the least), ragged tiles both ways,
    fp16 with an activation and fp32; the same bits every time, and two planes at once."""
    monkeypatch.setenv("B200_GEMM_TILE", tile)
    rng = np.random.default_rng(tokens + out + K)
    X, Wt, b = _case(rng, tokens, out, K, scale=0.25)
    got = linear_gpu(ctx, X, Wt, b, epi="gelu")
    assert relerr(got, ora.linear(X, Wt, b, epi="gelu")) < 2e-3          # one rounding step of fp16
    f32 = linear_gpu(ctx, X, Wt, b, out_dtype=np.float32)
    ref = ora.linear(X, Wt, b, out_dtype=np.float32)
    assert relerr(f32, ref) < 2e-5, describe(f32, ref, 2e-5)             # sqrt(K) eps32
    assert np.array_equal(f32, linear_gpu(ctx, X, Wt, b, out_dtype=np.float32))
    A, B = np.stack([Wt, -Wt]), np.stack([X, 2 * X])
    two = ctx.allocate(np.float32, out, tokens, 2)
    ctx.fill_bytes(two, 0xFF)
    jv.batchedmatmul_(ctx, two, ctx.toback(A), ctx.toback(B))
    ctx.synchronize()
    zero = ora.linear(X, Wt, out_dtype=np.float32)
    assert relerr(two.to_host(), np.stack([zero, -2 * zero])) < 2e-5


def _pair_parts(ctx, tokens, out, K, nbatch=1):
    """Over how many CTA pairs the plan cuts a 256 x 256 tile's reduction."""
    import ctypes as C
    from juliavision_b200 import _lib
    p = _lib.GemmPlan()
    _lib.check(_lib.lib().b200_gemm_f16_plan(ctx.handle, out, tokens, K, nbatch, C.byref(p)))
    assert (p.block_m, p.block_n) == (256, 256)
    return p.ctas / (2 * -(-tokens // 256) * -(-out // 256) * nbatch)


# `one`, `two`: the pairs a tile of the product, and of two of them at once, is shared by; 1 where the clusters would not all be
# resident, and the tiles stay whole
@pytest.mark.parametrize("tile,tokens,out,K,one,two", [
    ("256x2k2", 2, 8, 512, 2, 2), ("256x2k2", 129, 264, 530, 2, 2), ("256x2k2", 300, 200, 1288, 2, 2), ("256x2k2", 517, 1000, 4264, 2, 2),
    ("256x2k2", 1000, 1000, 5120, 2, 2), ("256x2k2", 1500, 1280, 5120, 2, 1),
    ("256x2k4", 2, 8, 512, 4, 4), ("256x2k4", 129, 264, 530, 4, 4), ("256x2k4", 300, 200, 1288, 4, 4), ("256x2k4", 300, 700, 4264, 4, 4),
    ("256x2k4", 517, 1000, 4264, 4, 1), ("256x2k4", 1500, 1280, 5120, 1, 1)])
def test_tiles_shared_by_the_pairs_of_a_cluster(ctx, ora, tile, tokens, out, K, one, two, monkeypatch):
    monkeypatch.setenv("B200_GEMM_TILE", tile)
    if ctx.dev.cores == 148:
        assert (_pair_parts(ctx, tokens, out, K), _pair_parts(ctx, tokens, out, K, 2)) == (one, two)
    test_tiles_shared_by_a_cluster(ctx, ora, tile, tokens, out, K, monkeypatch)


@pytest.mark.parametrize("tokens,out,K,parts", [(1500, 1280, 5120, 2), (1500, 1280, 4096, 2), (512, 4096, 4096, 2), (500, 1280, 5120, 4),
                                                (995, 664, 4720, 4)])
def test_the_planner_shares_tiles_of_long_reductions_among_pairs(ctx, ora, tokens, out, K, parts):
    """Its own choice, no override, and what it gives."""
    if ctx.dev.cores == 148:
        assert _pair_parts(ctx, tokens, out, K) == parts
    rng = np.random.default_rng(tokens + K)
    X, Wt, b = _case(rng, tokens, out, K, scale=0.25)
    got, ref = linear_gpu(ctx, X, Wt, b, out_dtype=np.float32), ora.linear(X, Wt, b, out_dtype=np.float32)
    assert relerr(got, ref) < 2e-5, describe(got, ref, 2e-5)             # sqrt(K) eps32


def test_plans_made_by_several_threads_agree(ctx):
    """The plan entry asks the runtime once per device and keeps the answer for every thread."""
    import ctypes as C
    import threading
    from juliavision_b200 import _lib
    shapes = [(768, 160, 3072), (2112, 42, 3152), (304, 18, 2144), (3072, 4096, 768)]
    def plans(c):
        out = []
        for M, N, K in shapes:
            p = _lib.GemmPlan()
            _lib.check(_lib.lib().b200_gemm_f16_plan(c.handle, M, N, K, 1, C.byref(p)))
            out.append((p.block_m, p.block_n, p.ctas))
        return out
    want, got = plans(ctx), []
    ts = [threading.Thread(target=lambda: got.append(plans(ctx))) for _ in range(8)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert got == [want] * 8
    assert any(p[2] > -(-M // p[1]) * -(-N // p[0]) for p, (M, N, K) in zip(want, shapes)), "no shape splits K here"


@pytest.mark.parametrize("tokens,out,K,tile", [
    (57732, 736, 216, (256, 256)),    # several rounds of wide tiles: every width is held to the same share of its epilogue
    (131072, 336, 112, (256, 128)),   # a width that three narrow tiles cover and two wide ones overshoot
    (46572, 2408, 128, (256, 128)),   # rows of results off 32-byte sectors, two k-blocks
    (46572, 2432, 128, (256, 256)),   # the same on sectors
    (7287, 528, 128, (128, 128)),     # one round: no pairs
    (51442, 184, 168, (256, 256)),    # three rounds of one feature tile: pairs
])
def test_tiles_for_short_reductions(ctx, tokens, out, K, tile):
    import ctypes as C
    from juliavision_b200 import _lib
    p = _lib.GemmPlan()
    _lib.check(_lib.lib().b200_gemm_f16_plan(ctx.handle, out, tokens, K, 1, C.byref(p)))
    assert (p.block_m, p.block_n) == tile


def test_streamk_is_deterministic(ctx, monkeypatch):
    monkeypatch.setenv("B200_GEMM_TILE", "256x2s")
    rng = np.random.default_rng(77)
    X, Wt, b = _case(rng, 1500, 1280, 5120, scale=0.25)
    a1 = linear_gpu(ctx, X, Wt, b)
    a2 = linear_gpu(ctx, X, Wt, b)
    assert np.array_equal(a1, a2)


@pytest.mark.parametrize("K", [768, 1280])
@pytest.mark.parametrize("out", [1000, 3072, 5120])
@pytest.mark.parametrize("tokens", [256, 4096, 65536])
def test_sweep_rows_sampled_and_row_shards(ctx, ora, tokens, out, K):
    """The scaling sweep's GEMM shapes (tokens 256..65536, out 1000/3072/5120 with 1000 ragged, K 768/1280).
    A sample of rows against the oracle, and the row split the sharding layer makes: each shard computed on
    its own equals the same rows of the whole product."""
    rng = np.random.default_rng(tokens + out + K)
    X = np.float16(rng.standard_normal((tokens, K), dtype=np.float32) * 0.05)
    Wt = np.float16(rng.standard_normal((K, out), dtype=np.float32) * 0.05)
    b = np.float16(rng.standard_normal(out, dtype=np.float32) * 0.05)
    got = linear_gpu(ctx, X, Wt, b)
    rows = np.sort(rng.choice(tokens, 48, replace=False))
    ref = ora.linear(np.ascontiguousarray(X[rows]), Wt, b)
    assert relerr(got[rows], ref) < TOL, describe(got[rows], ref, TOL)
    world = 8
    for rank in (0, 3, world - 1):
        r0, r1 = jv.shard_range(tokens, world, rank, align=256)
        if r1 > r0:
            part = linear_gpu(ctx, np.ascontiguousarray(X[r0:r1]), Wt, b)
            assert relerr(part, got[r0:r1]) < 1e-3
            assert np.mean(part != got[r0:r1]) < 1e-3      # summation order may differ where a tile was split along K


@pytest.mark.parametrize("dtype", [np.float32, np.float16])
@pytest.mark.parametrize("M,K", [(1280, 1280), (5120, 1280), (1280, 5120), (51865, 1280), (37, 50), (8, 4096), (1000, 3)])
def test_gemv_one_token(ctx, ora, dtype, M, K):
    """The one-token case (MMGemvPlan, matmul.jl:103-137): fp32 operands as in the reference and fp16
    ones; bias and activation in the store; compared with the oracle's fp32-accumulated product."""
    rng = np.random.default_rng(M + K)
    Wt = (rng.standard_normal((K, M)) * 0.05).astype(dtype)          # torch (in, out): column-major (M, K)
    x = (rng.standard_normal((1, K))).astype(dtype)
    b = (rng.standard_normal(M) * 0.05).astype(dtype)
    A, B, bias = ctx.toback(Wt), ctx.toback(x), ctx.toback(b)
    for epi, bb in (("identity", bias), ("gelu", bias), ("relu", None)):
        out = ctx.allocate(dtype, M, 1)
        ctx.fill_bytes(out, 0xFF)
        assert isinstance(jv.mmplan(ctx, out, A, B, bb), jv.MMGemvPlan)
        ctx.ws.reset()
        jv.matmul_(ctx, out, A, B, bb, epi=epi)
        ctx.synchronize()
        got = out.to_host()
        ctx.fill_bytes(out, 0xFF)
        ctx.ws.reset()
        jv.matmul_(ctx, out, A, B, bb, epi=epi)      # the K split's partial sums are added in a fixed order
        ctx.synchronize()
        assert np.array_equal(got.view(np.uint8), out.to_host().view(np.uint8))
        want = x.astype(np.float64) @ Wt.astype(np.float64) + (b.astype(np.float64) if bb is not None else 0)
        if dtype == np.float16:
            ref = ora.linear(x, Wt, b if bb is not None else None, epi=epi if epi != "identity" else "none")
            assert relerr(got, ref) < TOL, describe(got, ref, TOL)
        else:
            from scipy.special import erf
            ref = {"identity": want, "relu": np.maximum(want, 0), "gelu": 0.5 * want * (1 + erf(want / np.sqrt(2)))}[epi]
            assert relerr(got, ref) < 1e-4, describe(got, ref, 1e-4)


@pytest.mark.parametrize("dtype", [np.float32, np.float16])
@pytest.mark.parametrize("M0,lead,rows", [(3, 1000, 251), (1, 264, 1), (5, 4099, 4000), (0, 496, 496), (7, 249, 242)])
def test_gemv_rows_of_a_wider_matrix(ctx, dtype, M0, lead, rows):
    """A is rows M0 .. M0+rows of a (lead, K) matrix: the first element off a 16-byte boundary and a
    leading dimension of any parity, so every column starts at its own offset within an aligned vector.
    The rows outside the view hold huge values, which must not reach the result."""
    K = 300
    rng = np.random.default_rng(lead + rows)
    full = np.full((K, lead), 6.0e4, dtype)                         # torch (in, out): column-major (lead, K)
    full[:, M0:M0 + rows] = (rng.standard_normal((K, rows)) * 0.05).astype(dtype)
    x = rng.standard_normal((1, K)).astype(dtype)
    A = ctx.toback(full).slice(0, M0, M0 + rows)
    B = ctx.toback(x)
    out = ctx.allocate(np.float32, rows, 1)
    ctx.fill_bytes(out, 0xFF)
    assert isinstance(jv.mmplan(ctx, out, A, B, None), jv.MMGemvPlan)
    ctx.ws.reset()
    jv.matmul_(ctx, out, A, B, None)
    ctx.synchronize()
    got = out.to_host().reshape(-1)
    want = (x.astype(np.float64) @ full[:, M0:M0 + rows].astype(np.float64)).reshape(-1)
    assert np.all(np.isfinite(got))
    assert relerr(got, want) < 1e-4, describe(got, want, 1e-4)


def test_gemv_without_a_reduction_axis(ctx):
    """K = 0 through the C ABI: the sum is empty, the result is the bias (or zero)."""
    import ctypes as C
    from juliavision_b200 import _lib
    M = 300
    b = np.float16(np.random.default_rng(3).standard_normal(M))
    bias, out = ctx.toback(b), ctx.allocate(np.float16, M, 1)
    for bp, want in ((bias.ptr, b), (None, np.zeros(M, np.float16))):
        ctx.fill_bytes(out, 0xFF)
        rc = _lib.lib().b200_gemv(ctx.handle, M, 0, None, M, None, bp, _lib.F16, out.ptr, _lib.F16, 0)
        assert rc == _lib.OK
        ctx.synchronize()
        assert np.array_equal(out.to_host().reshape(-1), want)


@pytest.mark.parametrize("M,K", [(7076, 960), (5176, 798), (1051, 417), (2909, 401), (1189, 4174)])
def test_one_token_sums_are_short_chains(ctx, M, K):
    """fp32 against 64 bits.  A chain of n additions of random terms leaves c sqrt(n / 2) of the result's size, c the root
    mean square of a relative fp32 rounding (about 0.6 2^-24): the columns of a warp, or half of them (16 warps, and up to
    eight parts of K where row blocks of 124 leave SMs free), and in pairwise sums one rounding per level."""
    rng = np.random.default_rng(M + K)
    Wt, x = np.float32(rng.standard_normal((K, M)) * 0.05), np.float32(rng.standard_normal((1, K)))
    out = ctx.allocate(np.float32, M, 1)
    ctx.ws.reset()
    jv.matmul_(ctx, out, ctx.toback(Wt), ctx.toback(x), None)
    ctx.synchronize()
    ref = (x.astype(np.float64) @ Wt.astype(np.float64)).ravel()
    err = np.linalg.norm(out.to_host().ravel() - ref) / np.linalg.norm(ref)
    blocks, parts = -(-M // 124), 1
    while parts < 8 and 2 * parts * blocks <= 148 and K >= 2 * parts * 128:
        parts *= 2
    columns = -(-K // (16 * parts))
    chain = columns / 2 if parts == 8 else columns / 2 / 2 + 1      # in pairs while there are fewer than eight parts
    bound = 0.6 * 2.0 ** -24 * np.sqrt(chain + 4 + np.log2(parts) + 1)
    assert err < bound, (err, bound)


def test_timeline_records_time_and_cycles(ctx):
    """b200_timeline: worker 0's events in nanoseconds and in SM cycles; their ratio is a plausible clock,
    the events are in order, every worker's exit is recorded, and nothing is written once it is off."""
    import ctypes as C
    from juliavision_b200 import _lib
    rng = np.random.default_rng(1)
    X = ctx.toback(np.float16(rng.standard_normal((2048, 1024), dtype=np.float32) * 0.05))
    W = ctx.toback(np.float16(rng.standard_normal((1024, 2048), dtype=np.float32) * 0.05))
    out = ctx.allocate(np.float16, 2048, 2048)
    tl = ctx.allocate(np.uint64, 256)
    ctx.fill_bytes(tl, 0)
    jv.matmul_(ctx, out, W, X, None)
    ctx.synchronize()
    _lib.check(_lib.lib().b200_timeline(ctx.handle, tl.ptr))
    jv.matmul_(ctx, out, W, X, None)
    ctx.synchronize()
    _lib.check(_lib.lib().b200_timeline(ctx.handle, None))
    t = tl.to_host().astype(np.int64)
    assert 0 < t[0] <= t[1] <= t[3] <= t[4] <= t[8] <= t[12] <= t[16]          # entry .. exit, in order
    ns, clk = t[16] - t[0], t[64 + 16] - t[64 + 0]
    assert ns > 0 and 500 < clk / ns * 1e3 < 2200                               # MHz
    exits = t[128:128 + 120]
    assert 1 <= np.count_nonzero(exits) <= 120 and np.all(exits[exits > 0] >= t[0])   # one per worker
    ctx.fill_bytes(tl, 0)
    jv.matmul_(ctx, out, W, X, None)
    ctx.synchronize()
    assert not tl.to_host().any()


@pytest.mark.parametrize("tile", ["64x1k2", "128x1k8"])
def test_timeline_of_a_cluster_is_one_cta(ctx, tile, monkeypatch):
    """With a K split the worker is a cluster, and its first CTA records: events in order and a plausible clock from first
    to last, one exit per tile, launch after launch."""
    from juliavision_b200 import _lib
    monkeypatch.setenv("B200_GEMM_TILE", tile)
    rng = np.random.default_rng(2)
    X = ctx.toback(np.float16(rng.standard_normal((128, 2048)) * 0.05))
    W = ctx.toback(np.float16(rng.standard_normal((2048, 512)) * 0.05))
    out = ctx.allocate(np.float16, 512, 128)
    tl = ctx.allocate(np.uint64, 256)
    for _ in range(8):
        ctx.fill_bytes(tl, 0)
        _lib.check(_lib.lib().b200_timeline(ctx.handle, tl.ptr))
        jv.matmul_(ctx, out, W, X, None)
        ctx.synchronize()
        _lib.check(_lib.lib().b200_timeline(ctx.handle, None))
        t = tl.to_host().astype(np.int64)
        assert 0 < t[0] <= t[1] <= t[3] <= t[4] <= t[8] <= t[12] <= t[16]
        for a, b in ((0, 16), (0, 8), (4, 12)):
            ns, clk = t[b] - t[a], t[64 + b] - t[64 + a]
            assert ns >= 0 and abs(clk / 1.4 - ns) < 1000 + 0.8 * ns       # 0.8 to 2.2 GHz, the clock ticks in steps
        assert np.count_nonzero(t[128:]) == 512 // int(tile.split("x")[0])


def test_weight_operand_produced_by_the_previous_launch(ctx):
    """Launches overlap their predecessor's tail (programmatic dependent launch) and must not read an operand
    before the dependency wait.  Here the first product is the second one's A operand (as in a batched
    product of two activations) and changes every round, so a read that came too early would show."""
    rng = np.random.default_rng(31)
    M1, K1, N1 = 512, 256, 384          # Y1 (M1, N1) = W1 (M1, K1) . X1 (K1, N1)
    N2 = 300                            # Y2 (M1, N2) = Y1 (M1, N1) . X2 (N1, N2)
    W1 = ctx.toback(np.float16(rng.standard_normal((K1, M1)) * 0.1))      # torch (K, out)
    X2 = ctx.toback(np.float16(rng.standard_normal((N2, N1)) * 0.1))      # torch (tokens, K)
    Y1 = ctx.allocate(np.float16, M1, N1)
    Y2 = ctx.allocate(np.float16, M1, N2)
    for round_ in range(4):
        x1 = np.float16(rng.standard_normal((N1, K1)) * 0.1)
        X1 = ctx.toback(x1)
        jv.matmul_(ctx, Y1, W1, X1, None)
        jv.matmul_(ctx, Y2, Y1, X2, None)     # A = the output of the launch just before
        ctx.synchronize()
        y1 = Y1.to_host()                                        # torch (N1, M1)
        want = np.float32(X2.to_host()) @ np.float32(y1)         # (N2, N1) @ (N1, M1)
        assert relerr(Y2.to_host(), want) < 5e-3, f"round {round_}"


@pytest.mark.parametrize("tile", ["256x2", "128x2"])
@pytest.mark.parametrize("tokens,out,K", [(300, 8, 64), (700, 24, 1536), (520, 264, 1472), (4100, 1304, 72), (20000, 456, 40), (257, 40, 1528)])
def test_pairs_of_ctas_store_wide_chunks(ctx, ora, tile, tokens, out, K, monkeypatch):
    """Feature counts that end inside a stored chunk, reductions on both sides of the deeper ring's rule, one and many tiles
    a worker with feature tiles that do not divide its step: results by rounding at the store only."""
    monkeypatch.setenv("B200_GEMM_TILE", tile)
    rng = np.random.default_rng(tokens + out + K)
    X, Wt, b = _case(rng, tokens, out, K, scale=0.25)
    for epi, bias in (("identity", b), ("gelu", b), ("relu", None)):
        got = linear_gpu(ctx, X, Wt, bias, epi=epi)
        ref = ora.linear(X, Wt, bias, epi=epi)
        assert relerr(got, ref) < 2e-3, (epi, describe(got, ref, 2e-3))          # one rounding step of fp16


def test_gelu_over_every_half(ctx, ora):
    """The folded activation against the stand-alone op (equal bits) and the oracle (an fp16 step, and what 7.1.26 in fp32
    is off by where it cancels), for every finite fp16 value; infinities and NaN as the formula has them."""
    x = np.arange(65536, dtype=np.uint16).view(np.float16)
    x = np.concatenate([x[np.isfinite(x)], np.float16([np.inf, -np.inf, np.nan, 0, 0, 0, 0, 0])])
    d, o = ctx.toback(x), ctx.allocate(np.float16, x.size)
    jv.act_(ctx, o, d, "gelu")
    alone = o.to_host()
    with np.errstate(over="ignore", invalid="ignore"):
        ref = ora.act(x, "gelu")
        fin = np.isfinite(x)
        step = np.spacing(np.abs(ref[fin])).astype(np.float32)
    assert np.all(np.abs(alone[fin].astype(np.float32) - ref[fin].astype(np.float32)) <= step + 1e-7)
    assert alone[~fin][0] == np.inf and np.isnan(alone[~fin][1]) and np.isnan(alone[~fin][2])
    finite = np.where(fin, x, np.float16(0))
    one = np.zeros((300, 8), np.float16)
    one[:, 0] = 1
    weight = np.zeros((8, x.size), np.float16)
    weight[0] = finite
    got = linear_gpu(ctx, one, weight, None, epi="gelu")       # x * 1 + zeros: the values themselves, exactly
    want = np.where(fin, alone, alone[np.flatnonzero(finite == 0)[0]])
    assert np.all(got == want[None, :])


def test_gelu_of_large_negative_values_goes_to_zero(ctx):
    """fp32 results below -6, from every product's store: no further from x Phi(x) than 0 is (the 7.1.26
    steps give 0 there), but for one step of the smallest float times nine."""
    x = -np.float16(2.0) ** np.linspace(np.log2(6.01), 15.9, 400).astype(np.float16)
    x = np.concatenate([x, np.float16([-6.004, -8.992, -9.0, -9.008, -65504.0])])
    x = np.concatenate([x, np.zeros(-x.size % 8, np.float16)])
    exact = np.array([0.5 * float(t) * math.erfc(-float(t) / math.sqrt(2)) for t in x])
    got = []
    for tokens, out in ((1, x.size), (3, x.size), (300, x.size), (5, x.size - 1)):      # row, few rows, tiles, unaligned rows
        one, weight = np.zeros((tokens, 128), np.float16), np.zeros((128, out), np.float16)
        one[:, 0], weight[0] = 1, x[:out]
        got += list(linear_gpu(ctx, one, weight, None, epi="gelu", out_dtype=np.float32)[[0, -1]])
    for g in got:
        e = exact[:g.size]
        assert np.all(np.abs(g.astype(np.float64) - e) <= np.abs(e) + 2e-44)


# (tokens, out features, K, launches on 148 SMs): what is left past the full rounds is one block, some, exactly half a round, just
# more than that; of a short reduction, which is not split; split in two, four and eight parts, some of those without a step; weights
# that are long, and which the form in tensor memory would take longer for: reductions that leave it a small ring, very many rows
@pytest.mark.parametrize("tokens,out,K,launches", [(2, 35525, 512, 2), (16, 35641, 515, 2), (19, 20001, 1024, 2), (33, 16577, 520, 2),
                                                   (5, 53279, 384, 1), (5, 53279, 512, 2), (5, 53401, 512, 1), (33, 8289, 2100, 2),
                                                   (5, 37001, 3300, 2), (2, 250001, 900, 2), (16, 16801, 5000, 2),
                                                   (20, 17001, 2800, 2), (60, 9001, 1350, 2), (36, 9951, 2199, 2)])
@pytest.mark.parametrize("dt", [np.float16, np.float32])
def test_unaligned_rows_past_the_last_full_round(ctx, ora, tokens, out, K, launches, dt):
    """Row blocks that fill the GPU once or more and leave some: at most half a round of them is a launch of its own, split
    along K; with a bias, every row."""
    rng = np.random.default_rng(tokens + out)
    X, Wt, b = _case(rng, tokens, out, K, scale=0.25)
    before = ctx.launch_count()
    got = linear_gpu(ctx, X, Wt, b, out_dtype=dt)
    if ctx.dev.cores == 148:
        assert ctx.launch_count() - before == launches
    ref = ora.linear(X, Wt, b, out_dtype=dt)
    tol = 2e-3 if dt == np.float16 else 2e-5             # one rounding step of fp16; sqrt(K) eps32
    assert relerr(got, ref) < tol, describe(got, ref, tol)


# (tokens, out features, K, elements between columns, elements off the boundary): a token block of 16, 32, 48 and 64, and more than
# one; the last class without its last column, a reduction that ends inside sixteen of a class, and B off 16 bytes; one row block a
# CTA and several, the last one cut; rows 0 ... 7 elements off in turn, or all the same; few columns to a class, and many
@pytest.mark.parametrize("tokens,out,K,lda,off", [(5, 56251, 801, 56253, 1), (8, 40501, 1112, 40501, 1), (7, 15001, 3072, 15003, 5), (9, 28673, 736, 28675, 7),
                                                  (16, 85001, 257, 85004, 2), (17, 21001, 1024, 21001, 0), (32, 328001, 65, 328002, 5),
                                                  (33, 8291, 1103, 8297, 3), (48, 9001, 1280, 9001, 1), (49, 140001, 66, 140003, 6),
                                                  (64, 9001, 1280, 9003, 0), (50, 11003, 2000, 11005, 4), (70, 9005, 1000, 9006, 3)])
@pytest.mark.parametrize("dt", [np.float16, np.float32])
def test_unaligned_rows_of_long_products(ctx, ora, tokens, out, K, lda, off, dt):
    """Weights that long go to the form in tensor memory: with a bias, every row, and what lies between the columns and around
    them (NaN here) stays out of the results."""
    rng = np.random.default_rng(out)
    X, Wt, b = _case(rng, tokens, out, K, scale=0.25)
    room = np.full(off + K * lda + 8, np.nan, np.float16)
    np.lib.stride_tricks.as_strided(room[off:], (K, out), (2 * lda, 2))[...] = Wt
    base, x, bias = ctx.toback(room), ctx.toback(X), ctx.toback(b)
    w = jv.DeviceArray(ctx, base.ptr + 2 * off, np.float16, (out, K), (1, lda), owner=base)
    y = ctx.allocate(dt, out, tokens)
    ctx.fill_bytes(y, 0xFF)
    jv.matmul_(ctx, y, w, x, bias)
    ctx.synchronize()
    got, ref = y.to_host(), ora.linear(X, Wt, b, out_dtype=dt)
    tol = 2e-3 if dt == np.float16 else 2e-5             # one rounding step of fp16; sqrt(K) eps32
    assert relerr(got, ref) < tol, describe(got, ref, tol)


# a token block of 16, 32, 48 and 64; rows past a last full round of gemm_rows.cu's, which would be a second launch there
@pytest.mark.parametrize("tokens,out,K", [(8, 37601, 1200), (16, 16701, 1280), (27, 16701, 1280), (48, 8403, 1100), (61, 8403, 1100)])
@pytest.mark.parametrize("dt", [np.float16, np.float32])
@pytest.mark.parametrize("epi,with_bias", [("gelu", True), ("relu", False), ("identity", False)])
def test_unaligned_rows_of_long_products_end_in_their_activation(ctx, ora, tokens, out, K, dt, epi, with_bias):
    """In one launch; A and the output one element into allocations whose neighbours hold NaN."""
    rng = np.random.default_rng(out + tokens)
    X, Wt, b = _case(rng, tokens, out, K, scale=0.25)
    pad = np.full(K * out + 16, np.nan, np.float16)
    pad[1:1 + K * out] = Wt.reshape(-1)
    base, x, bias = ctx.toback(pad), ctx.toback(X), ctx.toback(b) if with_bias else None
    w = jv.DeviceArray(ctx, base.ptr + 2, np.float16, (out, K), owner=base)
    dest = ctx.allocate(dt, out * tokens + 2)
    ctx.fill_bytes(dest, 0xFF)
    y = jv.DeviceArray(ctx, dest.ptr + np.dtype(dt).itemsize, dt, (out, tokens), owner=dest)
    before = ctx.launch_count()
    jv.matmul_(ctx, y, w, x, bias, epi=epi)
    if ctx.dev.cores == 148:
        assert ctx.launch_count() - before == 1
    ctx.synchronize()
    flat = dest.to_host()
    got, ref = flat[1:-1].reshape(tokens, out), ora.linear(X, Wt, b if with_bias else None, epi=epi if epi != "identity" else "none", out_dtype=dt)
    assert np.isnan(flat[0]) and np.isnan(flat[-1]), "wrote outside the output"
    tol = 2e-3 if dt == np.float16 else 2e-5             # one rounding step of fp16; sqrt(K) eps32
    assert relerr(got, ref) < tol, describe(got, ref, tol)


def test_what_follows_a_product_in_two_launches_waits_for_both(ctx):
    """A layer norm that is launched early behind the second launch, eagerly and recorded, gives the bits it gives behind a
    finished product, over results that are poisoned before each."""
    rng = np.random.default_rng(8)
    M, K, tokens, C = 35840, 1024, 5, 112
    base = ctx.toback(np.concatenate([np.float16([0]), (rng.standard_normal(M * K, dtype=np.float32) * 0.05).astype(np.float16)]))
    w = jv.DeviceArray(ctx, base.ptr + 2, np.float16, (M, K), owner=base)            # off a 16-byte boundary: by row blocks
    x = ctx.toback((rng.standard_normal((tokens, K)) * 0.25).astype(np.float16))
    y, z = ctx.allocate(np.float16, M, tokens), ctx.allocate(np.float16, M, tokens)
    rows = M * tokens // C
    mean, rstd = ctx.allocate(np.float32, rows), ctx.allocate(np.float32, rows)
    view = lambda a: jv.DeviceArray(ctx, a.ptr, np.float16, (C, rows), owner=a)

    def norm():
        jv.layernorm_(ctx, view(z), mean, rstd, view(y), None, None, C, 1e-5)

    def both():
        ctx.fill_bytes(y, 0xFF)
        jv.matmul_(ctx, y, w, x, None)
        norm()

    ctx.fill_bytes(y, 0xFF)
    before = ctx.launch_count()
    jv.matmul_(ctx, y, w, x, None)
    assert ctx.launch_count() - before == 2
    ctx.synchronize()
    norm()
    ctx.synchronize()
    product, want = y.to_host(), z.to_host()
    assert np.all(np.isfinite(want))
    g = ctx.capture(both)
    for run in (both, g.replay) * 4:
        ctx.fill_bytes(z, 0xFF)
        run()
        ctx.synchronize()
        assert np.array_equal(z.to_host(), want) and np.array_equal(y.to_host(), product)
    del g
