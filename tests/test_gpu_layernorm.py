import os

import numpy as np
import pytest

import juliavision_b200 as jv

from .conftest import relerr
from .gpu_helpers import describe, layernorm_gpu

pytestmark = pytest.mark.gpu
G = os.path.join(os.path.dirname(__file__), "golden")


def test_golden(ctx):
    g = np.load(os.path.join(G, "layernorm.npz"))
    out, mean, rstd = layernorm_gpu(ctx, g["a"], g["gamma"], g["beta"], float(g["eps"]), out_dtype=np.float32)
    assert np.max(np.abs(out - g["out"])) < 5e-6
    assert np.max(np.abs(mean - g["mean"])) < 1e-6 and relerr(rstd, g["rstd"]) < 1e-6


@pytest.mark.parametrize("groups,C", [(1500, 1280), (4096, 112), (64, 144), (333, 576), (7, 100), (5, 4104),
                                      (3, 8200), (1, 8), (65536, 112), (999, 112), (1001, 64), (7, 56), (130, 128)])
@pytest.mark.parametrize("dt_in,dt_out", [(np.float16, np.float16), (np.float16, np.float32),
                                          (np.float32, np.float32), (np.float32, np.float16)])
def test_vs_oracle(ctx, ora, groups, C, dt_in, dt_out):
    if groups * C > 2_000_000 and dt_in != np.float16:
        pytest.skip("large case runs once")
    rng = np.random.default_rng(groups * 131 + C)
    a = (rng.standard_normal((groups, C)) * 2 + 0.5).astype(dt_in)
    gam = (1 + 0.1 * rng.standard_normal(C)).astype(dt_in)
    bet = (0.1 * rng.standard_normal(C)).astype(dt_in)
    for g, b in ((gam, bet), (None, None), (gam, None)):
        got, mean, rstd = layernorm_gpu(ctx, a, g, b, 1e-5, out_dtype=dt_out)
        ref, rmean, rrstd = ora.layernorm(a, g, b, 1e-5, out_dtype=dt_out)
        assert got.dtype == dt_out and got.shape == ref.shape
        # fp32 statistics in a different summation order: a few fp32 ulps, at most one output ulp
        tol = 1.5e-3 if dt_out == np.float16 else 2e-6
        assert np.all(np.isfinite(got)), describe(got, ref, tol)          # poison fully overwritten
        assert relerr(got, ref) < tol, describe(got, ref, tol)
        assert np.max(np.abs(mean - rmean)) < 1e-5 and relerr(rstd, rrstd) < 1e-5


@pytest.mark.parametrize("dt,C", [(np.float16, 4104), (np.float16, 8192), (np.float16, 8200), (np.float16, 16384),
                                  (np.float16, 16392), (np.float32, 2052), (np.float32, 4096), (np.float32, 4280),
                                  (np.float32, 8192), (np.float32, 8196)])
def test_rows_wider_than_a_warp_holds(ctx, ora, dt, C):
    """A block per row: the smallest and largest widths of its two forms, and the next ones on either side."""
    rng = np.random.default_rng(C)
    a = (rng.standard_normal((37, C)) * 2 + 0.5).astype(dt)
    gam, bet = ((o + 0.1 * rng.standard_normal(C)).astype(dt) for o in (1, 0))
    got, mean, rstd = layernorm_gpu(ctx, a, gam, bet, 1e-5)
    ref, rmean, rrstd = ora.layernorm(a, gam, bet, 1e-5, out_dtype=dt)
    tol = 1.5e-3 if dt == np.float16 else 2e-6      # as above: a few fp32 ulps of the sums, at most one output ulp
    assert relerr(got, ref) < tol, describe(got, ref, tol)
    assert np.max(np.abs(mean - rmean)) < 1e-5 and relerr(rstd, rrstd) < 1e-5


@pytest.mark.parametrize("C", [2052, 4280, 8192, 8196])
def test_rows_wider_than_a_warp_holds_round_gamma_and_beta_once(ctx, C):
    """fp32, where it shows: y gamma + beta is one rounding of the row's own y = (x - mean) rstd, in the form of a block
    per row as in the general one (C = 8196).  64 bits hold the product of two fp32 numbers exactly."""
    rng = np.random.default_rng(C)
    a = np.float32(rng.standard_normal((37, C)) * 2 + 0.5)
    gam, bet = np.float32(1 + 0.1 * rng.standard_normal(C)), np.float32(rng.standard_normal(C))
    got, mean, rstd = layernorm_gpu(ctx, a, gam, bet, 1e-5)
    y = (a - mean.reshape(-1, 1)) * rstd.reshape(-1, 1)
    once = np.float32(y.astype(np.float64) * gam + bet)
    assert np.mean(got != once) < 1e-4      # a double rounding where 64 bits end on a tie
    got, mean, rstd = layernorm_gpu(ctx, a, None, bet, 1e-5)      # beta alone: added to the product with rstd
    once = np.float32((a - mean.reshape(-1, 1)).astype(np.float64) * rstd.reshape(-1, 1) + bet)
    assert np.mean(got != once) < 1e-4


def test_mean_dominates_variance(ctx, ora):
    a = (np.float32(1000.0) + np.float32(0.5) * np.sin(np.arange(4 * 256, dtype=np.float32))).reshape(4, 256)
    got, _, _ = layernorm_gpu(ctx, a, eps=1e-5)
    ref, _, _ = ora.layernorm(a, eps=1e-5)
    assert np.max(np.abs(got - ref)) < 2e-3


def test_empty_and_errors(ctx):
    import juliavision_b200 as jv
    a = ctx.allocate(np.float16, 16, 0)
    out = ctx.allocate(np.float16, 16, 0)
    m = ctx.allocate(np.float32, 1)
    jv.layernorm_(ctx, out, m, m, a, None, None, 16, 1e-5)  # zero groups: no launch, no error
    b = ctx.allocate(np.float16, 10, 3)
    with pytest.raises(jv.B200Error):
        jv.layernorm_(ctx, b, m, m, b, None, None, 7, 1e-5)  # 30 is not a multiple of 7


PACKED = [1000, 1024, 1176, 1480, 1800, 2048]    # 4, 4, 5, 6 and 8 vectors per lane, the last one ragged or full; 5 and 6 pack


def _packed_rows(C):
    """Rows just past the 48 Mi elements from which fp16 launches take the packed form, the last block of four ragged."""
    groups = ((48 << 20) + C - 1) // C + 1
    return groups + (groups % 4 == 0)


@pytest.mark.parametrize("C", PACKED)
def test_rows_the_cache_does_not_hold(ctx, ora, C):
    """The packed form and its neighbours: first and last rows and a sample, with gamma and beta, one of them and neither."""
    groups = _packed_rows(C)
    rng = np.random.default_rng(C)
    a = np.float16(rng.standard_normal((groups, C), dtype=np.float32) * 2 + 0.5)
    gam, bet = (np.float16(o + 0.1 * rng.standard_normal(C)) for o in (1, 0))
    rows = np.unique(np.concatenate([np.arange(9), groups - 1 - np.arange(9), rng.integers(0, groups, 400)]))
    for g, b in ((gam, bet), (gam, None), (None, bet), (None, None)):
        got, mean, rstd = layernorm_gpu(ctx, a, g, b, 1e-5)
        ref, rmean, rrstd = ora.layernorm(a[rows], g, b, 1e-5)
        assert np.all(np.isfinite(got)) and np.all(np.isfinite(mean)) and np.all(np.isfinite(rstd))
        assert relerr(got[rows], ref) < 1.5e-3, describe(got[rows], ref, 1.5e-3)    # as above: at most one output ulp
        assert np.max(np.abs(mean[rows] - rmean)) < 1e-5 and relerr(rstd[rows], rrstd) < 1e-5


@pytest.mark.parametrize("C", [1000, 1176, 1480, 1800])
def test_add_layernorm_equals_the_three_ops_where_the_cache_does_not_hold_them(ctx, C):
    """The promise of equal bits at the size where both take the packed form, and one row short of it, where neither does."""
    rng = np.random.default_rng(C)
    least = ((48 << 20) + C - 1) // C
    g, b = (ctx.toback(np.float16(o + 0.1 * rng.standard_normal(C))) for o in (1, 0))
    for groups, clamp, gb in ((_packed_rows(C), (-500.0, 500.0), (g, b)), (least, None, (g, None)), (least, None, (None, b)),
                              (least - 1, None, (g, b)), (least - 1, None, (None, b))):
        x0, h0 = (np.float16(rng.standard_normal((groups, C), dtype=np.float32) * 300) for _ in range(2))
        mean, rstd, m2, r2 = (ctx.allocate(np.float32, groups) for _ in range(4))
        xa, ha, oa = ctx.toback(x0), ctx.toback(h0), ctx.allocate(np.float16, C, groups)
        jv.add_(ctx, xa, xa, ha)
        if clamp:
            jv.clamp_(ctx, xa, xa, *clamp)
        jv.layernorm_(ctx, oa, mean, rstd, xa, *gb, C, 1e-5)
        xb, ob = ctx.toback(x0), ctx.allocate(np.float16, C, groups)
        ctx.fill_bytes(ob, 0xFF)
        jv.add_layernorm_(ctx, ob, m2, r2, xb, ha, *gb, C, 1e-5, clamp=clamp)
        ctx.synchronize()
        for one, other in ((xa, xb), (oa, ob), (mean, m2), (rstd, r2)):
            assert np.array_equal(one.to_host(), other.to_host()), (groups, C)


@pytest.mark.parametrize("C,same", [(1000, True), (1024, True), (1176, False), (1480, False), (1800, True), (2048, True)])
def test_only_the_widths_that_gain_take_the_packed_form(ctx, C, same):
    """Five and six vectors per lane are faster packed, four and eight slower: there a row keeps its bits whatever the launch."""
    rng = np.random.default_rng(C)
    part = np.float16(rng.standard_normal((4096, C)) * 2 + 0.5)
    gam, bet = (np.float16(o + 0.1 * rng.standard_normal(C)) for o in (1, 0))
    small = layernorm_gpu(ctx, part, gam, bet, 1e-5)
    large = layernorm_gpu(ctx, np.tile(part, (-(-_packed_rows(C) // 4096), 1)), gam, bet, 1e-5)
    equal = [np.array_equal(a, b[:len(a)]) for a, b in zip(small, large)]
    assert equal == [True] * 3 if same else not all(equal)


@pytest.mark.parametrize("dt,C,groups", [(np.float16, 8, 2369), (np.float16, 64, 75779), (np.float16, 72, 37887), (np.float16, 112, 37891),
                                         (np.float16, 128, 2371), (np.float16, 136, 18943), (np.float16, 256, 18947),
                                         (np.float32, 28, 37889), (np.float32, 128, 18945), (np.float16, 264, 2369),
                                         (np.float16, 512, 2370),
                                         # two and four rows on either side of their rules, alone and behind the add
                                         (np.float16, 8, 113665), (np.float16, 56, 227331), (np.float16, 120, 56831), (np.float16, 128, 113667),
                                         (np.float16, 248, 28419), (np.float16, 256, 56835), (np.float32, 28, 113667), (np.float32, 60, 23681),
                                         (np.float32, 128, 28417), (np.float16, 264, 11841), (np.float16, 512, 11845)])
def test_several_narrow_rows_at_a_time(ctx, ora, dt, C, groups):
    """Widths at both ends of a row's lanes, row counts that leave a last group short and on either side of the rules for
    two and four rows: the oracle's values, and bit for bit what one row at a time (a launch of few rows) gives; with fp16 also
    behind the residual add."""
    rng = np.random.default_rng(C + groups)
    a = (rng.standard_normal((groups, C), dtype=np.float32) * 2 + 0.5).astype(dt)
    gam, bet = ((o + 0.1 * rng.standard_normal(C)).astype(dt) for o in (1, 0))
    part = slice(groups - 1999, groups)
    for g, b in ((gam, bet), (gam, None), (None, bet)):
        got, mean, rstd = layernorm_gpu(ctx, a, g, b, 1e-5)
        few, fmean, frstd = layernorm_gpu(ctx, np.ascontiguousarray(a[part]), g, b, 1e-5)
        assert np.array_equal(got[part], few) and np.array_equal(mean[part], fmean) and np.array_equal(rstd[part], frstd)
    ref, rmean, rrstd = ora.layernorm(a[part], None, bet, 1e-5, out_dtype=dt)
    tol = 1.5e-3 if dt == np.float16 else 2e-6      # as above: a few fp32 ulps of the sums, at most one output ulp
    assert relerr(few, ref) < tol, describe(few, ref, tol)
    assert np.max(np.abs(fmean - rmean)) < 1e-5 and relerr(frstd, rrstd) < 1e-5
    if dt != np.float16:
        return
    h0 = rng.standard_normal((groups, C), dtype=np.float32).astype(dt)
    gd, bd = ctx.toback(gam), ctx.toback(bet)
    for clamp in (None, (-1.5, 2.0)):
        xa, xb, ha = ctx.toback(a), ctx.toback(a), ctx.toback(h0)
        m1, r1, m2, r2 = (ctx.allocate(np.float32, groups) for _ in range(4))
        oa, ob = ctx.allocate(dt, C, groups), ctx.allocate(dt, C, groups)
        jv.add_(ctx, xa, xa, ha)
        if clamp:
            jv.clamp_(ctx, xa, xa, *clamp)
        jv.layernorm_(ctx, oa, m1, r1, xa, gd, bd, C, 1e-5)
        ctx.fill_bytes(ob, 0xFF)
        jv.add_layernorm_(ctx, ob, m2, r2, xb, ha, gd, bd, C, 1e-5, clamp=clamp)
        ctx.synchronize()
        for one, other in ((xa, xb), (oa, ob), (m1, m2), (r1, r2)):
            assert np.array_equal(one.to_host(), other.to_host())


# the narrowest and widest rows of the form of a block a row, those next to them, four and five vectors a thread, idle lanes
SPLIT = [(np.float16, 1792, 70), (np.float16, 1800, 70), (np.float16, 2056, 600), (np.float16, 2560, 70), (np.float16, 3080, 70),
         (np.float16, 4096, 2400), (np.float16, 4104, 592), (np.float16, 4104, 593), (np.float16, 5120, 600), (np.float16, 16384, 600),
         (np.float32, 1024, 70), (np.float32, 1028, 70), (np.float32, 1540, 600), (np.float32, 2048, 70)]


@pytest.mark.parametrize("dt,C,groups", SPLIT)
def test_a_block_a_row(ctx, ora, dt, C, groups):
    rng = np.random.default_rng(C + groups)
    a = (rng.standard_normal((groups, C), dtype=np.float32) * 2 + 0.5).astype(dt)
    gam, bet = ((o + 0.1 * rng.standard_normal(C)).astype(dt) for o in (1, 0))
    tol = 1.5e-3 if dt == np.float16 else 2e-6      # as above: a few fp32 ulps of the sums, at most one output ulp
    for g, b in ((gam, bet), (gam, None), (None, bet), (None, None)):
        got, mean, rstd = layernorm_gpu(ctx, a, g, b, 1e-5)
        ref, rmean, rrstd = ora.layernorm(a, g, b, 1e-5, out_dtype=dt)
        assert relerr(got, ref) < tol, describe(got, ref, tol)
        assert np.max(np.abs(mean - rmean)) < 1e-5 and relerr(rstd, rrstd) < 1e-5
    if dt != np.float16:
        return
    h = (rng.standard_normal((groups, C), dtype=np.float32)).astype(dt)     # behind the add: the three ops, bit for bit
    for clamp in (None, (-1.5, 2.0)):
        xa, xb, dh, dg, db = (ctx.toback(t) for t in (a, a, h, gam, bet))
        m1, r1, m2, r2 = (ctx.allocate(np.float32, groups) for _ in range(4))
        oa, ob = ctx.allocate(dt, C, groups), ctx.allocate(dt, C, groups)
        jv.add_(ctx, xa, xa, dh)
        if clamp:
            jv.clamp_(ctx, xa, xa, *clamp)
        jv.layernorm_(ctx, oa, m1, r1, xa, dg, db, C, 1e-5)
        ctx.fill_bytes(ob, 0xFF)
        jv.add_layernorm_(ctx, ob, m2, r2, xb, dh, dg, db, C, 1e-5, clamp=clamp)
        ctx.synchronize()
        for one, other in ((xa, xb), (oa, ob), (m1, m2), (r1, r2)):
            assert np.array_equal(one.to_host(), other.to_host())


@pytest.mark.parametrize("dt,C,groups", [(np.float16, 1800, 800), (np.float16, 4096, 800), (np.float16, 4104, 800), (np.float16, 5120, 800),
                                         (np.float16, 6152, 800), (np.float16, 8200, 800), (np.float16, 16384, 600), (np.float32, 2048, 600),
                                         (np.float32, 3076, 600)])
def test_a_wide_rows_bits_do_not_depend_on_the_rows_beside_it(ctx, dt, C, groups):
    """The rows of a shard are those of the whole: below and above four rows an SM, and one alone."""
    rng = np.random.default_rng(C)
    a = (rng.standard_normal((groups, C), dtype=np.float32) * 2 + 0.5).astype(dt)
    gam, bet = ((o + 0.1 * rng.standard_normal(C)).astype(dt) for o in (1, 0))
    whole = layernorm_gpu(ctx, a, gam, bet, 1e-5)
    for n in (1, 148, 592):
        for one, other in zip(layernorm_gpu(ctx, a[:n], gam, bet, 1e-5), whole):
            assert np.array_equal(one, other[:n])
