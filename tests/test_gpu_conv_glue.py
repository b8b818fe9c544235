import os

import numpy as np
import pytest
import torch

import juliavision_b200 as jv

from .conftest import relerr
from .gpu_helpers import describe

pytestmark = pytest.mark.gpu
G = os.path.join(os.path.dirname(__file__), "golden")


def conv_gpu(ctx, x, w, b, stride, padding, act="identity", out_dtype=np.float16):
    """x torch (N,Cin,H,W), w torch (Cout,Cin,KH,KW); stride/padding torch (h,w) order."""
    dx, dw = ctx.toback(x), ctx.toback(w)
    db = None if b is None else ctx.toback(b)
    N, Cin, H, W = x.shape
    Cout, _, KH, KW = w.shape
    OW = jv.convsize(W, KW, stride[1], padding[1], 1)
    OH = jv.convsize(H, KH, stride[0], padding[0], 1)
    out = ctx.allocate(out_dtype, OW, OH, Cout, N)
    ctx.fill_bytes(out, 0xFF)
    ctx.ws.reset()
    jv.convolution_(ctx, out, dx, dw, db, (stride[1], stride[0]), (padding[1], padding[0]), (1, 1), 1, act=act)
    ctx.synchronize()
    return out.to_host()


def test_conv_golden(ctx):
    g = np.load(os.path.join(G, "conv.npz"))
    W, H, Cin, Cout, KW, KH, st, pd = (int(t) for t in g["geom"])
    x = np.float16(0.4 * np.sin(np.linspace(0, 9, W * H * Cin))).reshape(1, Cin, H, W)
    w = np.float16(0.3 * np.cos(np.linspace(0, 7, KW * KH * Cin * Cout))).reshape(Cout, Cin, KH, KW)
    got = conv_gpu(ctx, x, w, None, (st, st), (pd, pd), out_dtype=np.float32)
    assert relerr(got[0], g["out"]) < 5e-3, describe(got[0], g["out"], 5e-3)   # test_convtranspose_gemm.jl:154-200


# (W,H,Cin,Cout,KW,KH,s,p): the reference's CRS-padding cases plus the Hiera stem geometry at 256^2
@pytest.mark.parametrize("W,H,Cin,Cout,KW,KH,s,p", [(64, 64, 5, 32, 3, 3, 1, 1), (48, 48, 7, 48, 5, 5, 2, 2),
                                                     (32, 32, 32, 64, 3, 3, 1, 1), (256, 256, 3, 112, 7, 7, 4, 3),
                                                     (30, 22, 4, 24, 3, 3, 1, 1)])
def test_conv_vs_oracle(ctx, ora, W, H, Cin, Cout, KW, KH, s, p):
    rng = np.random.default_rng(W + Cin + Cout)
    x = np.float16(rng.standard_normal((2, Cin, H, W)) * 0.5)
    w = np.float16(rng.standard_normal((Cout, Cin, KH, KW)) * 0.1)
    b = np.float16(rng.standard_normal(Cout) * 0.1)
    got = conv_gpu(ctx, x, w, b, (s, s), (p, p), act="relu")
    ref = ora.conv2d(x, w, b, (s, s), (p, p), (1, 1), epi="relu")
    assert got.shape == ref.shape
    assert relerr(got, ref) < 5e-3, describe(got, ref, 5e-3)


@pytest.mark.parametrize("W,H,Cin,Cout", [(64, 64, 144, 256), (32, 32, 32, 48), (16, 24, 8, 8)])
def test_conv_1x1_is_a_gemm(ctx, ora, W, H, Cin, Cout):
    rng = np.random.default_rng(W * Cin)
    x = np.float16(rng.standard_normal((1, Cin, H, W)) * 0.5)
    w = np.float16(rng.standard_normal((Cout, Cin, 1, 1)) * 0.1)
    b = np.float16(rng.standard_normal(Cout) * 0.1)
    got = conv_gpu(ctx, x, w, b, (1, 1), (0, 0))
    ref = ora.conv2d(x, w, b)
    assert relerr(got, ref) < 5e-3, describe(got, ref, 5e-3)


# (N, Cin, H, W, Cout, KH, KW, stride, padding, dilation), torch order: pixel counts off 8 and 128, rows shorter than a
# chunk of 8 pixels, channel counts on both sides of a tile, every stride form, dilation, wide padding, a 1x1 of odd size
IMPLICIT = [(1, 3, 33, 41, 40, 7, 7, (4, 4), (3, 3), (1, 1)), (2, 8, 5, 6, 33, 3, 3, (1, 1), (1, 1), (1, 1)),
            (1, 16, 31, 29, 130, 3, 3, (2, 2), (1, 1), (1, 1)), (1, 24, 17, 19, 257, 1, 1, (1, 1), (0, 0), (1, 1)),
            (1, 5, 40, 37, 64, 3, 5, (3, 1), (2, 4), (2, 2)), (3, 8, 64, 128, 64, 3, 3, (1, 1), (1, 1), (1, 1)),
            (1, 200, 13, 150, 300, 3, 3, (1, 3), (1, 1), (1, 1)), (1, 1, 9, 200, 16, 2, 2, (1, 1), (5, 9), (1, 1))]


@pytest.mark.parametrize("N,Cin,H,W,Cout,KH,KW,stride,padding,dilation", IMPLICIT)
@pytest.mark.parametrize("dt", [np.float16, np.float32])
def test_conv_gathered_into_the_tiles(ctx, ora, N, Cin, H, W, Cout, KH, KW, stride, padding, dilation, dt):
    rng = np.random.default_rng(Cin + Cout + W)
    x = np.float16(rng.standard_normal((N, Cin, H, W)) * 0.5)
    w = np.float16(rng.standard_normal((Cout, Cin, KH, KW)) * 0.2)
    b = np.float16(rng.standard_normal(Cout) * 0.2)
    ref = ora.conv2d(x, w, b, stride, padding, dilation, epi="relu", out_dtype=dt)
    flat = ctx.allocate(dt, ref.size + 1)      # the output one element off its allocation's alignment
    ctx.fill_bytes(flat, 0xFF)
    out = jv.DeviceArray(ctx, flat.ptr + np.dtype(dt).itemsize, dt, tuple(reversed(ref.shape)), owner=flat)
    ctx.ws.reset()
    jv.convolution_(ctx, out, ctx.toback(x), ctx.toback(w), ctx.toback(b), stride[::-1], padding[::-1], dilation[::-1], act="relu")
    ctx.synchronize()
    host = flat.to_host()
    assert np.isnan(host[0]), "wrote before the output"
    got = host[1:].reshape(ref.shape)
    # fp32 sums in another order (sqrt(CRS) eps32), then one fp16 rounding step
    tol = 2e-3 if dt == np.float16 else 2e-5
    assert relerr(got, ref) < tol, describe(got, ref, tol)


@pytest.mark.parametrize("Cin,Cout,H,W", [(136, 40, 17, 19), (72, 257, 33, 31)])
def test_a_weight_off_its_boundary_does_not_depend_on_the_workspace(ora, Cin, Cout, H, W):
    """A 1x1 convolution of an odd image needs no scratch but for a weight that starts off a 16-byte boundary, which the
    implicit kernel wants copied.  Recorded on a context that has no workspace yet it runs all the same; in a loop
    without a reset it leaves the workspace as it found it."""
    rng = np.random.default_rng(Cout)
    x = np.float16(rng.standard_normal((1, Cin, H, W)) * 0.5)
    w = np.float16(rng.standard_normal((Cout, Cin, 1, 1)) * 0.2)
    ref = ora.conv2d(x, w, None, out_dtype=np.float32)
    with jv.Ctx(0) as c:
        dx, base = c.toback(x), c.toback(np.concatenate([np.float16([0]), w.reshape(-1)]))
        dw = jv.DeviceArray(c, base.ptr + 2, np.float16, (1, 1, Cin, Cout), owner=base)
        out = c.allocate(np.float32, W, H, Cout, 1)
        call = lambda: jv.convolution_(c, out, dx, dw, None, (1, 1), (0, 0), (1, 1))
        c.fill_bytes(out, 0xFF)
        g = c.capture(call)
        assert c.ws.stats()[1] == 0
        g.replay()
        c.synchronize()
        assert relerr(out.to_host(), ref) < 2e-5      # fp32 sums in another order
        c.fill_bytes(out, 0xFF)
        call()
        cap = c.ws.stats()
        assert cap[0] == 0 and cap[1] > 0
        for _ in range(20):
            call()
        c.synchronize()
        assert c.ws.stats() == cap
        assert relerr(out.to_host(), ref) < 2e-5


@pytest.mark.parametrize("side", [16, 17])      # an image the GEMM can store, one it cannot
@pytest.mark.parametrize("epilogue", [-1, 4])
def test_an_epilogue_that_does_not_exist_is_refused(ctx, side, epilogue):
    from juliavision_b200 import _lib
    x, w = ctx.toback(np.zeros((1, 8, side, side), np.float16)), ctx.toback(np.zeros((8, 8, 1, 1), np.float16))
    out = ctx.allocate(np.float16, side, side, 8, 1)
    rc = _lib.lib().b200_conv2d_f16(ctx.handle, side, side, 8, 1, 1, 1, 8, 1, 1, 0, 0, 1, 1, x.ptr, w.ptr, None, out.ptr, 0, epilogue)
    assert rc == _lib.lib().b200_conv2d_f16(ctx.handle, side, side, 8, 1, 1, 1, 8, 0, 1, 0, 0, 1, 1, x.ptr, w.ptr, None, out.ptr, 0, 0) != 0


# 1x1 convolutions of odd images: (N, Cin, H, W, Cout, whether the scalar GEMM takes them, a launch per image, rather than the
# implicit kernel)
@pytest.mark.parametrize("N,Cin,H,W,Cout,scalar", [(1, 1, 15, 21, 88, True), (1, 16, 45, 53, 96, True), (1, 40, 7, 9, 512, True),
                                                   (2, 3, 321, 235, 8, True), (1, 40, 21, 25, 24, False), (4, 8, 7, 7, 64, False),
                                                   (1, 512, 9, 11, 88, False), (1, 128, 51, 37, 64, False)])
@pytest.mark.parametrize("dt", [np.float16, np.float32])
def test_conv_1x1_of_odd_images(ctx, ora, N, Cin, H, W, Cout, scalar, dt):
    rng = np.random.default_rng(Cin + Cout + W)
    x = np.float16(rng.standard_normal((N, Cin, H, W)) * 0.5)
    w = np.float16(rng.standard_normal((Cout, Cin, 1, 1)) * 0.2)
    b = np.float16(rng.standard_normal(Cout) * 0.2)
    before = ctx.launch_count()
    got = conv_gpu(ctx, x, w, b, (1, 1), (0, 0), out_dtype=dt)
    assert ctx.launch_count() - before == (N if scalar else 1)
    # fp32 sums in another order (sqrt(Cin) eps32), then one fp16 rounding step
    tol = 2e-3 if dt == np.float16 else 2e-5
    ref = ora.conv2d(x, w, b, out_dtype=dt)
    assert relerr(got, ref) < tol, describe(got, ref, tol)


def test_im2col_bit_exact(ctx, ora):
    import ctypes as C
    from juliavision_b200 import _lib
    rng = np.random.default_rng(3)
    x = np.float16(rng.standard_normal((2, 5, 20, 24)))
    N, Cin, H, W = x.shape
    KH = KW = 3
    OW, OH = jv.convsize(W, KW, 2, 1, 1), jv.convsize(H, KH, 2, 1, 1)
    NPQ, CRS = OW * OH * N, KW * KH * Cin
    MP, CRSP = (NPQ + 15) // 16 * 16, (CRS + 15) // 16 * 16
    col = ctx.allocate(np.float16, MP, CRSP)
    ctx.fill_bytes(col, 0xFF)
    _lib.check(_lib.lib().b200_im2col_f16(ctx.handle, W, H, Cin, N, KW, KH, 2, 2, 1, 1, 1, 1, MP, CRSP,
                                          ctx.toback(x).ptr, col.ptr))
    ctx.synchronize()
    assert np.array_equal(col.to_host(), ora.im2col(x, KH, KW, (2, 2), (1, 1), (1, 1), MP, CRSP))


def test_glue_bit_exact(ctx, ora):
    rng = np.random.default_rng(4)
    for n in (1, 7, 8, 1000, 1500 * 1280 + 3):
        a = np.float16(rng.standard_normal(n) * 4)
        b = np.float16(rng.standard_normal(n) * 4)
        da, db, do = ctx.toback(a), ctx.toback(b), ctx.allocate(np.float16, n)
        jv.add_(ctx, do, da, db)
        assert np.array_equal(do.to_host(), ora.add(a, b))
        jv.clamp_(ctx, do, da, -1.5, 2.25)
        assert np.array_equal(do.to_host(), ora.clamp(a, -1.5, 2.25))
        jv.act_(ctx, do, da, "relu")
        assert np.array_equal(do.to_host(), ora.act(a, "relu"))
        jv.act_(ctx, do, da, "gelu")
        ref = ora.act(a, "gelu")
        d = np.abs(do.to_host().astype(np.float32) - ref.astype(np.float32))
        assert np.all(d <= np.spacing(np.abs(ref)).astype(np.float32) + 1e-7)   # fast exp: one fp16 ulp at most


# (N, Cin, H, W, Cout, KH, KW, stride, padding, dilation): 8 and 4 columns a kernel row, each with tiles of 64, 128 and 256
# channels and two channel tiles; taps before and behind the words' ends, one and several k-blocks and images, clusters of 1, 2,
# 4 and 8 parts, odd kernel-row counts, dilated rows, strides past a word, pixels past the last tile
WORDS = [(1, 3, 75, 100, 112, 7, 7, (4, 4), (3, 3), (1, 1)), (2, 3, 40, 44, 24, 7, 5, (3, 4), (2, 2), (2, 1)),
         (1, 3, 90, 132, 200, 7, 7, (4, 4), (3, 3), (1, 1)), (1, 5, 70, 104, 66, 4, 8, (1, 8), (0, 0), (1, 1)),
         (1, 20, 51, 52, 40, 7, 6, (4, 4), (3, 3), (1, 1)), (1, 40, 83, 88, 112, 7, 7, (4, 4), (3, 3), (1, 1)),
         (3, 1, 50, 52, 16, 3, 5, (2, 4), (0, 5), (3, 1)), (2, 17, 31, 30, 64, 3, 3, (2, 2), (1, 1), (1, 1)),
         (1, 64, 20, 26, 40, 3, 3, (2, 6), (1, 1), (1, 1)), (1, 24, 45, 62, 104, 3, 3, (2, 2), (1, 1), (1, 1)),
         (1, 15, 61, 66, 300, 3, 3, (2, 2), (1, 1), (1, 1)), (1, 48, 45, 50, 130, 3, 3, (2, 2), (1, 1), (1, 1)),
         (1, 172, 44, 30, 72, 3, 3, (2, 2), (1, 1), (1, 1)), (1, 16, 64, 64, 128, 3, 3, (2, 2), (1, 1), (1, 1)),
         (1, 96, 33, 38, 24, 1, 4, (2, 2), (0, 4), (1, 1))]
# the same kernels where reading in words does not gain: a weight larger than the image, half of the columns zeros on a short
# reduction, a long chain a CTA against a small im2col matrix
NOT_WORDS = [(1, 3, 37, 64, 112, 7, 7, (4, 4), (3, 3), (1, 1)), (1, 16, 37, 38, 8, 2, 2, (2, 2), (1, 1), (1, 1)),
             (1, 64, 60, 64, 256, 3, 3, (2, 2), (1, 1), (1, 1))]


@pytest.mark.parametrize("N,Cin,H,W,Cout,KH,KW,stride,padding,dilation", WORDS + NOT_WORDS)
@pytest.mark.parametrize("dt", [np.float16, np.float32])
def test_conv_of_even_stride_reads_whole_words(ctx, ora, N, Cin, H, W, Cout, KH, KW, stride, padding, dilation, dt):
    rng = np.random.default_rng(Cin + Cout + W)
    x = np.float16(rng.standard_normal((N, Cin, H, W)) * 0.5)
    w = np.float16(rng.standard_normal((Cout, Cin, KH, KW)) * 0.2)
    b = np.float16(rng.standard_normal(Cout) * 0.2)
    ref = ora.conv2d(x, w, b, stride, padding, dilation, out_dtype=dt)
    out = ctx.allocate(dt, *reversed(ref.shape))
    ctx.fill_bytes(out, 0xFF)
    ctx.ws.reset()
    args = ctx.toback(x), ctx.toback(w), ctx.toback(b)
    before = ctx.launch_count()
    jv.convolution_(ctx, out, *args, stride[::-1], padding[::-1], dilation[::-1])
    # in words: the weight laid out and the convolution, whose scratch is given back; by taps no scratch and one launch, or, as
    # by an im2col matrix, scratch that stays until the reset
    route = ctx.launch_count() - before, ctx.ws.stats()[0]
    assert (route == (2, 0)) == ((N, Cin, H, W, Cout, KH, KW, stride, padding, dilation) in WORDS), route
    ctx.synchronize()
    got = out.to_host()
    tol = 2e-3 if dt == np.float16 else 2e-5      # as for the taps
    assert relerr(got, ref) < tol, describe(got, ref, tol)


@pytest.mark.parametrize("Cin,Cout,H,W,scratch", [(24, 104, 45, 62, 0), (3, 64, 90, 132, None), (16, 64, 64, 64, None)])
def test_conv_in_words_does_not_depend_on_the_workspace(ora, Cin, Cout, H, W, scratch):
    """Recorded on a context that has no workspace yet, the laid-out weight is refused: the call goes by taps as it would have
    without the words, or says that it has no room where that route wants scratch of its own; then in words all the same."""
    rng = np.random.default_rng(Cout + W)
    x = np.float16(rng.standard_normal((1, Cin, H, W)) * 0.5)
    w = np.float16(rng.standard_normal((Cout, Cin, 3, 3)) * 0.2)
    ref = ora.conv2d(x, w, None, (2, 2), (1, 1), out_dtype=np.float32)
    with jv.Ctx(0) as c:
        dx, dw = c.toback(x), c.toback(w)
        out = c.allocate(np.float32, *reversed(ref.shape))
        c.fill_bytes(out, 0xFF)
        c.synchronize()
        call = lambda: jv.convolution_(c, out, dx, dw, None, (2, 2), (1, 1), (1, 1))
        before = c.launch_count()
        if scratch == 0:
            g = c.capture(call)
            assert c.launch_count() - before == 1 and c.ws.stats()[1] == 0
            g.replay()
            c.synchronize()
            assert relerr(out.to_host(), ref) < 2e-5
            del g
        else:
            with pytest.raises(jv.B200Error):
                c.capture(call)
        c.fill_bytes(out, 0xFF)
        before = c.launch_count()
        call()
        assert c.launch_count() - before == 2
        g = c.capture(call)
        c.fill_bytes(out, 0xFF)
        g.replay()
        c.synchronize()
        assert relerr(out.to_host(), ref) < 2e-5
        del g


# (N, Cin, H, W, Cout, (KH, KW), (py, px), (dy, dx)), every row of results as long as the image's: the narrowest image, one and two
# k-blocks' ends inside sixteen rows, more pixel tiles than two CTAs an SM take (64 and 128 channels), a split reduction, 256 channels
# a CTA, 1 x 1, four taps and two (dilated, so that the lengths agree), an image the GEMM could store as well
RUNS = [(1, 3, 9, 8, 5, (3, 3), (1, 1), (1, 1)), (2, 5, 17, 11, 70, (3, 3), (1, 1), (1, 1)), (1, 40, 37, 131, 200, (1, 1), (0, 0), (1, 1)),
        (2, 8, 201, 255, 40, (3, 3), (1, 1), (1, 1)), (1, 9, 261, 255, 100, (3, 3), (1, 1), (1, 1)), (1, 200, 33, 31, 300, (3, 3), (1, 1), (1, 1)),
        (1, 16, 51, 49, 24, (4, 2), (0, 1), (1, 2)), (3, 7, 21, 23, 16, (2, 4), (3, 3), (5, 2)), (1, 64, 60, 64, 64, (3, 3), (1, 1), (1, 1)),
        (1, 12, 40, 45, 72, (3, 3), (2, 9), (1, 9))]


@pytest.mark.parametrize("N,Cin,H,W,Cout,K,pad,dil", RUNS)
@pytest.mark.parametrize("off", [0, 1, 6])
def test_conv_in_runs(ctx, ora, N, Cin, H, W, Cout, K, pad, dil, off):
    """Stride one and rows of the same length, the image at any distance from 16 bytes, NaN before and behind it."""
    rng = np.random.default_rng(Cin + Cout + W)
    x = np.float16(rng.standard_normal((N, Cin, H, W)) * 0.5)
    w = np.float16(rng.standard_normal((Cout, Cin) + K) * 0.2)
    b = np.float16(rng.standard_normal(Cout) * 0.2)
    ref = torch.nn.functional.conv2d(*(torch.from_numpy(a).double() for a in (x, w, b)), padding=pad, dilation=dil).numpy()
    assert ref.shape[-1] == W
    base = ctx.toback(np.concatenate([np.full(off, np.nan, np.float16), x.reshape(-1), np.full(8, np.nan, np.float16)]))
    dx = jv.DeviceArray(ctx, base.ptr + 2 * off, np.float16, (W, H, Cin, N), owner=base)
    dw, db = ctx.toback(w), ctx.toback(b)
    for dt, tol in ((np.float16, 2e-3), (np.float32, 2e-5)):      # one rounding step of fp16; sqrt(CRS) eps32
        out = ctx.allocate(dt, *reversed(ref.shape))
        ctx.fill_bytes(out, 0xFF)
        jv.convolution_(ctx, out, dx, dw, db, (1, 1), pad[::-1], dil[::-1], 1)
        ctx.synchronize()
        assert relerr(out.to_host(), ref) < tol, describe(out.to_host(), ref, tol)


@pytest.mark.parametrize("N,Cin,H,W,K,pad", [(2, 5, 17, 11, (3, 3), (1, 1)), (2, 9, 201, 255, (3, 3), (1, 1)), (1, 33, 21, 25, (3, 3), (1, 1)),
                                             (1, 6, 19, 13, (1, 3), (0, 1))])
@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_conv_in_runs_keeps_to_its_taps(ctx, N, Cin, H, W, K, pad, bad):
    """What a run crosses and a pixel's taps do not reach stays out of it: the other end of the row above or below, the next channel's
    first row, the last row of the one before, another image.  The rest has the bits it has with zeros there."""
    rng = np.random.default_rng(W)
    x = np.float16(rng.standard_normal((N, Cin, H, W)) * 0.5)
    w = np.float16((0.1 + rng.random((24, Cin) + K)) * 0.2)
    for where in (np.s_[:, :, :, 0], np.s_[:, :, :, W - 1], np.s_[:, :, 0], np.s_[:, 1, H - 1]) + (np.s_[0],) * (N > 1):
        spoilt, clean, marks = x.copy(), x.copy(), np.zeros_like(x)
        spoilt[where], clean[where], marks[where] = bad, 0, 1
        reached = torch.nn.functional.conv2d(torch.from_numpy(marks).float(), torch.ones((1, Cin) + K), padding=pad).numpy() > 0
        reached = np.broadcast_to(reached, (N, 24) + reached.shape[2:])
        got, want = conv_gpu(ctx, spoilt, w, None, (1, 1), pad), conv_gpu(ctx, clean, w, None, (1, 1), pad)
        assert np.all(np.isfinite(want)) and not np.any(np.isfinite(got[reached]))
        assert not np.all(reached) and np.array_equal(got[~reached], want[~reached])


# more pixel tiles than two CTAs an SM take: 64 and 128 channels a CTA, ragged, one and several k-blocks, words of 4 and 2, two images
@pytest.mark.parametrize("N,Cin,H,W,Cout,K,stride", [(1, 3, 808, 804, 112, 7, 4), (2, 3, 600, 608, 40, 7, 4), (1, 5, 395, 396, 72, 3, 2), (1, 24, 390, 400, 64, 3, 2)])
@pytest.mark.parametrize("dt", [np.float16, np.float32])
@pytest.mark.parametrize("act", ["identity", "gelu"])
def test_conv_in_words_of_many_tiles(ctx, ora, N, Cin, H, W, Cout, K, stride, dt, act):
    rng = np.random.default_rng(Cin + Cout + W)
    x = np.float16(rng.standard_normal((N, Cin, H, W)) * 0.5)
    w = np.float16(rng.standard_normal((Cout, Cin, K, K)) * 0.2)
    b = np.float16(rng.standard_normal(Cout) * 0.2)
    ref = ora.conv2d(x, w, b, (stride,) * 2, (K // 2,) * 2, epi={"identity": "none"}.get(act, act), out_dtype=dt)
    out = ctx.allocate(dt, *reversed(ref.shape))
    ctx.fill_bytes(out, 0xFF)
    ctx.ws.reset()
    half, dx, dw, db = ctx.toback(x * np.float16(0.5)), ctx.allocate(np.float16, W, H, Cin, N), ctx.toback(w), ctx.toback(b)
    ctx.fill_bytes(dx, 0xFF)
    jv.add_(ctx, dx, half, half)          # the image is the output of the kernel right before
    jv.convolution_(ctx, out, dx, dw, db, (stride,) * 2, (K // 2,) * 2, (1, 1), 1, act=act)
    ctx.synchronize()
    tol = 2e-3 if dt == np.float16 else 2e-5      # as above
    assert relerr(out.to_host(), ref) < tol, describe(out.to_host(), ref, tol)


# 64, 128 and 256 channels a CTA: up to a CTA an SM and more of them, four smaller CTAs an SM among them, words of 4 and 2
@pytest.mark.parametrize("N,Cin,H,W,Cout,K,stride", [(1, 3, 256, 256, 64, 7, 4), (1, 3, 808, 804, 112, 7, 4), (1, 16, 130, 132, 100, 3, 2),
                                                     (1, 16, 180, 180, 200, 3, 2), (1, 3, 512, 512, 160, 7, 4), (1, 3, 700, 700, 200, 7, 4)])
def test_conv_in_words_reads_what_was_written_last(ctx, ora, N, Cin, H, W, Cout, K, stride):
    """One buffer, rewritten by the kernel right before and convolved again and again: every result is that of the image and bias
    it was called on, eagerly and recorded."""
    rng = np.random.default_rng(Cin + Cout + W)
    images = [np.float16(rng.standard_normal((N, Cin, H, W)) * 0.5) for _ in range(3)]
    w = np.float16(rng.standard_normal((Cout, Cin, K, K)) * 0.2)
    biases = [np.float16(rng.standard_normal(Cout) * 0.2) for _ in images]
    dw, x, b = ctx.toback(w), ctx.allocate(np.float16, W, H, Cin, N), ctx.allocate(np.float16, Cout)
    hx, hb = ([ctx.toback(a * np.float16(0.5)) for a in part] for part in (images, biases))
    refs = [ora.conv2d(a, w, v, (stride,) * 2, (K // 2,) * 2, out_dtype=np.float32) for a, v in zip(images, biases)]
    outs = [ctx.allocate(np.float32, *reversed(refs[0].shape)) for _ in range(6)]

    def rounds():
        for i, out in enumerate(outs):
            jv.add_(ctx, b, hb[i % 3], hb[i % 3])
            jv.add_(ctx, x, hx[i % 3], hx[i % 3])
            jv.convolution_(ctx, out, x, dw, b, (stride,) * 2, (K // 2,) * 2, (1, 1), 1)

    ctx.ws.reset()
    before = ctx.launch_count()
    rounds()
    assert ctx.launch_count() - before == 4 * len(outs)     # two sums, the weight laid out, the convolution in words
    g = ctx.capture(rounds)
    for run in (rounds, g.replay):
        for out in outs:
            ctx.fill_bytes(out, 0xFF)
        run()
        ctx.synchronize()
        for i, out in enumerate(outs):
            assert relerr(out.to_host(), refs[i % 3]) < 2e-5, i      # as above
    del g


def test_conv_in_words_keeps_to_its_taps(ctx, ora):
    """An infinity or NaN beside a pixel's taps, inside the words that hold them, does not reach it."""
    x = np.float16(np.random.default_rng(3).standard_normal((1, 2, 16, 64)))
    w = np.float16(np.random.default_rng(4).standard_normal((8, 2, 3, 5)))
    x[0, 0, :, 0::8] = np.inf
    x[0, 1, :, 7::8] = np.nan
    got = conv_gpu(ctx, x, w, None, (1, 8), (1, 0))         # taps 0..4 of words of 8: 0 is one, 7 is none
    clean = x.copy()
    clean[0, 1, :, 7::8] = 0
    assert not np.isnan(got).all() and np.array_equal(np.isnan(got), np.isnan(conv_gpu(ctx, clean, w, None, (1, 8), (1, 0))))
    got = conv_gpu(ctx, np.ascontiguousarray(x[:, 1:]), np.ascontiguousarray(w[:, 1:]), None, (1, 8), (1, 0))
    ref = ora.conv2d(np.ascontiguousarray(clean[:, 1:]), np.ascontiguousarray(w[:, 1:]), None, (1, 8), (1, 0))
    assert np.all(np.isfinite(got)) and relerr(got, ref) < 2e-3


@pytest.mark.parametrize("n,d0,d1", [(2, 112, 264), (1, 8, 8), (3, 72, 56), (1, 64, 64), (1, 200, 4096)])
def test_transposed_copy_in_words_is_exact(ctx, n, d0, d1):
    """Tiles cut on either side, against numpy; a source one element off its boundary takes the narrow kernel, same result."""
    a = np.float16(np.random.default_rng(d0 + d1).standard_normal((n, d0, d1)))
    got = ctx.contiguous(ctx.toback(a).permute((1, 0, 2))).to_host()
    assert np.array_equal(got, a.transpose(0, 2, 1))
    flat = ctx.toback(np.concatenate([np.float16([0]), a.ravel()]))
    off = jv.DeviceArray(ctx, flat.ptr + 2, np.float16, (d1, d0, n), owner=flat)
    assert np.array_equal(ctx.contiguous(off.permute((1, 0, 2))).to_host(), a.transpose(0, 2, 1))


def test_permute_bit_exact(ctx):
    rng = np.random.default_rng(5)
    a = np.float16(rng.standard_normal((2, 37, 5, 24)))         # torch (B,L,H,E) -> device (E,H,L,B)
    d = ctx.toback(a)
    v = d.permute((0, 2, 1, 3))                                  # (E,L,H,B) view
    assert np.array_equal(ctx.contiguous(v).to_host(), a.transpose(0, 2, 1, 3))
    t = d.permute((2, 0, 1, 3))                                  # (L,E,H,B): source contiguous along output axis 1
    assert np.array_equal(ctx.contiguous(t).to_host(), a.transpose(0, 2, 3, 1))
    f = np.float32(rng.standard_normal((3, 4, 50, 33)))
    df = ctx.toback(f)
    assert np.array_equal(ctx.contiguous(df.permute((1, 0, 3, 2))).to_host(), f.transpose(1, 0, 3, 2))
    # axis 0 kept in front: 16-byte pieces when its extent and the strides allow, element by element when not
    for shape, dt in (((4, 9, 6, 64), np.float16), ((2, 5, 7, 20), np.float16), ((3, 6, 5, 8), np.float32), ((2, 3, 4, 6), np.float32)):
        g = rng.standard_normal(shape).astype(dt)
        dg = ctx.toback(g)
        assert np.array_equal(ctx.contiguous(dg.permute((0, 2, 1, 3))).to_host(), g.transpose(0, 2, 1, 3))
        assert np.array_equal(ctx.contiguous(dg.permute((0, 3, 2, 1))).to_host(), g.transpose(2, 1, 0, 3))


def test_pool_and_workspace(ctx):
    from juliavision_b200 import _lib
    import ctypes as C
    ctx.ws.reset()
    a = ctx.scratch(np.float16, 1000)
    b = ctx.scratch(np.float32, 10)
    assert a.ptr % 256 == 0 and b.ptr % 256 == 0 and b.ptr >= a.ptr + 2000     # workspace.jl:63-66
    used, cap, retired = ctx.ws.stats()
    assert cap >= 1 << 20                                                      # min 1 MiB (workspace.jl:85)
    big = ctx.scratch(np.uint8, cap + 5)                                       # forces a grow: old block retired
    assert ctx.ws.stats()[2] == 1 and ctx.ws.stats()[1] >= int(1.5 * (cap + 5)) - 512
    ctx.ws.reset()
    assert ctx.ws.stats()[0] == 0 and ctx.ws.stats()[2] == 0
    def reserved():
        use, res = C.c_size_t(), C.c_size_t()
        _lib.check(_lib.lib().b200_pool_stats(ctx.handle, C.byref(use), C.byref(res)))
        return res.value
    x = ctx.allocate(np.float32, 1024)
    assert x.ptr % 256 == 0
    before = reserved()
    del x
    y = ctx.allocate(np.float32, 1024)                                         # a freed block of the size class is reused:
    assert reserved() == before                                                # nothing new is taken from the driver
    with pytest.raises(jv.B200Error):
        _lib.check(_lib.lib().b200_pool_free(ctx.handle, C.c_void_p(12345)))


# (N, Cin, H, W, Cout, KH, KW, stride, padding, dilation, groups) in torch order
GROUPED = [(2, 16, 20, 24, 32, 3, 3, (1, 1), (1, 1), (1, 1), 2),     # aligned slices: tensor-core GEMM per group
           (1, 6, 9, 8, 8, 3, 3, (2, 1), (1, 1), (1, 1), 2),         # unaligned slices: the scalar GEMM
           (2, 8, 12, 12, 8, 3, 3, (1, 1), (1, 1), (1, 1), 8),       # depthwise
           (1, 32, 16, 16, 64, 1, 1, (1, 1), (0, 0), (1, 1), 4)]     # grouped 1x1: no gather


@pytest.mark.parametrize("N,Cin,H,W,Cout,KH,KW,stride,padding,dilation,groups", GROUPED)
def test_grouped_conv_vs_oracle(ctx, ora, N, Cin, H, W, Cout, KH, KW, stride, padding, dilation, groups):
    """conv2d with GROUPS > 1 (conv.jl:26-51): every group lowered like the ungrouped convolution."""
    rng = np.random.default_rng(Cin * 13 + groups)
    x = np.float16(rng.standard_normal((N, Cin, H, W)) * 0.5)
    w = np.float16(rng.standard_normal((Cout, Cin // groups, KH, KW)) * 0.2)
    b = np.float16(rng.standard_normal(Cout) * 0.2)
    ref = ora.conv2d_grouped(x, w, b, stride, padding, dilation, groups, epi="relu")
    out = ctx.allocate(np.float16, ref.shape[3], ref.shape[2], Cout, N)
    ctx.fill_bytes(out, 0xFF)
    ctx.ws.reset()
    jv.convolution_(ctx, out, ctx.toback(x), ctx.toback(w), ctx.toback(b), stride[::-1], padding[::-1], dilation[::-1],
                    groups, act="relu")
    ctx.synchronize()
    got = out.to_host()
    assert np.all(np.isfinite(got))
    assert relerr(got, ref) < 5e-3, describe(got, ref, 5e-3)


# (N, Cin, H, W, Cout, KH, KW, stride, padding, dilation, output_padding, groups)
TRANSPOSED = [(1, 64, 16, 16, 32, 2, 2, (2, 2), (0, 0), (1, 1), (0, 0), 1),      # SAM 2's upsampler: shufflecase -> GEMM
              (2, 24, 9, 7, 16, 2, 3, (2, 3), (0, 0), (1, 1), (0, 0), 1),        # shufflecase, odd extents, two images
              (2, 4, 5, 6, 6, 3, 2, (2, 3), (1, 0), (1, 2), (1, 1), 2),          # grouped, padded, dilated, output padding
              (1, 8, 10, 10, 8, 3, 3, (1, 1), (1, 1), (1, 1), (0, 0), 8),        # depthwise (Kokoro's upsampler form)
              (1, 16, 8, 8, 8, 4, 4, (2, 2), (1, 1), (1, 1), (0, 0), 1)]         # overlapping receptive fields: the gather


@pytest.mark.parametrize("N,Cin,H,W,Cout,KH,KW,stride,padding,dilation,outpad,groups", TRANSPOSED)
def test_transposed_conv_vs_oracle(ctx, ora, N, Cin, H, W, Cout, KH, KW, stride, padding, dilation, outpad, groups):
    """convolutiontranspose! (conv.jl:247-290): the GEMM + shuffle route where the receptive fields tile the output,
    the deterministic gather elsewhere; both against the oracle's gather (conv.jl:147-190)."""
    rng = np.random.default_rng(Cin * 7 + Cout)
    x = np.float16(rng.standard_normal((N, Cin, H, W)) * 0.5)
    w = np.float16(rng.standard_normal((Cin, Cout // groups, KH, KW)) * 0.2)
    b = np.float16(rng.standard_normal(Cout) * 0.2)
    for out_dtype in (np.float16, np.float32):
        ref = ora.convtranspose2d(x, w, b, stride, padding, dilation, outpad, groups, out_dtype=np.float32)
        out = ctx.allocate(out_dtype, ref.shape[3], ref.shape[2], Cout, N)
        ctx.fill_bytes(out, 0xFF)
        ctx.ws.reset()
        dw = ctx.toback(w)
        assert jv.shufflecase(dw, stride[::-1], padding[::-1], dilation[::-1], outpad[::-1], groups) == \
            (groups == 1 and (KH, KW) == stride and padding == (0, 0) and outpad == (0, 0) and dilation == (1, 1))
        jv.convolutiontranspose_(ctx, out, ctx.toback(x), dw, ctx.toback(b), stride[::-1], padding[::-1], dilation[::-1],
                                 outpad[::-1], groups)
        ctx.synchronize()
        got = out.to_host()
        assert got.shape == ref.shape and np.all(np.isfinite(got))
        assert relerr(got, ref) < 5e-3, describe(got, ref, 5e-3)
