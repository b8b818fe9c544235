"""The native host side of the entry points against the Python one: whatever it takes, it hands the library the very
arguments the Python route would; whatever the Python route refuses, it leaves alone.  No GPU: both call recorders."""
import ctypes as C
import itertools
import random

import numpy as np
import pytest

import juliavision_b200 as jv
from juliavision_b200 import _lib

NAMES = ("b200_gemm_f16", "b200_gemv", "b200_attention_f16_bias", "b200_layernorm", "b200_conv2d_grouped_f16")


class FakeCtx:
    handle = 4096


class NoHost:
    """The native module answering None to everything: the Python route runs."""
    def __getattr__(self, name):
        return lambda *a: None


def plain(v):
    if isinstance(v, C._Pointer):
        v = v.contents if v else None
    elif hasattr(v, "_obj"):          # byref
        v = v._obj
    if isinstance(v, _lib.Strided4):
        return (v.ptr or 0,) + tuple(v.stride)
    return np.float32(v) if isinstance(v, float) else (v or 0)


class Recorder:
    """Stands for the library: the five entry points note their arguments, the planning calls are the library's own."""
    def __init__(self, real):
        self.real, self.calls = real, []
        for n in NAMES:
            setattr(self, n, lambda *a, n=n: self.calls.append((n,) + tuple(plain(v) for v in a)) or 0)

    def b200_gemm_f16_plan(self, *a):
        return 0

    def __getattr__(self, name):
        return getattr(self.real, name)


@pytest.fixture
def both(monkeypatch):
    real = _lib.lib()
    rec = Recorder(real)
    keep = [C.CFUNCTYPE(_lib.SIGNATURES[n][0], *_lib.SIGNATURES[n][1])(getattr(rec, n)) for n in NAMES]
    native = _lib.host()
    native.bind(*(C.cast(f, C.c_void_p).value for f in keep))
    monkeypatch.setattr(_lib, "_lib", rec)

    def run(fn, *args, **kw):
        """(native call or None, Python call or the exception's type) for one set of operands."""
        seen = []
        for host in (native, NoHost()):
            monkeypatch.setattr(_lib, "_host", host)
            rec.calls.clear()
            try:
                fn(FakeCtx, *args, **kw)
                seen.append(list(rec.calls))
            except Exception as e:
                seen.append(type(e))
        return seen
    yield run
    monkeypatch.undo()
    _lib._host = None
    _lib.host()                       # bound to the library again


def arr(dt, shape, strides=None, ptr=None):
    return jv.DeviceArray(FakeCtx, ptr or random.randrange(1, 1 << 40) * 2, dt, shape, strides)


def agree(seen):
    assert seen[0] == seen[1], seen
    return isinstance(seen[0], list) and len(seen[0]) == 1


def test_matmul(both):
    random.seed(1)
    f16, f32, taken = np.float16, np.float32, 0
    for M, N, K in itertools.product((1, 8, 37, 51865), (1, 2, 300), (1, 7, 64)):
        for ta, tb, to in ((f16, f16, f16), (f16, f16, f32), (f32, f32, f32), (f32, f32, f16), (f16, f32, f16), (np.uint8, f16, f16)):
            for pad, bias, epi in ((0, None, "identity"), (3, (ta, M), "gelu"), (0, (f32, M), "relu"), (0, (ta, M + 1), "none"), (0, (ta, M), None)):
                A, B, out = (arr(t, s, (1, s[0] + pad)) for t, s in ((ta, (M, K)), (tb, (K, N)), (to, (M, N))))
                b = arr(bias[0], (bias[1],)) if bias else None
                taken += agree(both(jv.matmul_, out, A, B, b, epi=epi))
    for A, B, out in ((arr(f16, (8, 4), (2, 16)), arr(f16, (4, 3)), arr(f16, (8, 3))), (arr(f16, (8, 4), (1, 4)), arr(f16, (4, 3)), arr(f16, (8, 3))),
                      (arr(f16, (8, 4)), arr(f16, (5, 3)), arr(f16, (8, 3))), (arr(f16, (8, 4)), arr(f16, (4, 1), (4, 4)), arr(f16, (8, 1))),
                      (arr(f16, (8, 4)), arr(f16, (4, 3)), arr(f16, (8, 3, 1))), (arr(f16, (0, 4)), arr(f16, (4, 3)), arr(f16, (0, 3)))):
        agree(both(jv.matmul_, out, A, B, None))
    agree(both(jv.matmul_, arr(f16, (8, 3)), arr(f16, (8, 4)), arr(f16, (4, 3)), arr(f16, (2, 4))))      # a bias of two axes
    agree(both(jv.matmul_, arr(f16, (8, 3)), arr(f16, (8, 4)), arr(f16, (4, 3)), arr(f16, (8,), (2,))))  # a strided bias
    agree(both(jv.matmul_, arr(f16, (8, 3)), arr(f16, (8, 4)), arr(f16, (4, 3)), None, epi="tanh"))
    agree(both(jv.matmul_, arr(f16, (8, 3)), arr(f16, (8, 4), ptr=1 << 63), arr(f16, (4, 3)), None))     # past a signed 64-bit integer
    assert taken > 100


def test_sdpa(both):
    random.seed(2)
    f16, taken = np.float16, 0
    for E, Lq, Lk, H, B in itertools.product((7, 8, 64, 128, 136), (1, 5), (1, 9), (1, 3), (1, 2)):
        for layout, dt in ((None, f16), ("packed", f16), (None, np.float32)):
            st = lambda L: None if layout is None else (1, 3 * E * H, E, 3 * E * H * L)
            q, k, v = arr(dt, (E, Lq, H, B), st(Lq)), arr(f16, (E, Lk, H, B), st(Lk)), arr(f16, (E, Lk, H, B))
            for mask in (None, (Lk, Lq, H, B), (Lk, 1, 1, B), (1, Lq, 1, 1), (Lk + 1, Lq, 1, 1)):
                m = arr(f16, mask) if mask else None
                for out in (arr(f16, (E, Lq, H, B)), arr(np.float32, (E, Lq, H, B), (1, E * H, E, E * H * Lq))):
                    taken += agree(both(jv.sdpa, q, k, v, m, 0.25, out=out))
    q = arr(f16, (64, 5, 2, 1))
    for k, v, out in ((arr(f16, (64, 9, 3, 1)), arr(f16, (64, 9, 3, 1)), q), (arr(f16, (64, 9, 2, 1)), arr(f16, (64, 8, 2, 1)), q),
                      (q, q, arr(f16, (64, 4, 2, 1))), (q, q, arr(f16, (64, 5, 2, 1), (2, 128, 640, 1280))),
                      (arr(f16, (64, 5, 2, 1), (2, 128, 640, 1280)), q, q), (arr(f16, (64, 0, 2, 1)), arr(f16, (64, 0, 2, 1)), q)):
        agree(both(jv.sdpa, q, k, v, None, None, out=out))
    agree(both(jv.sdpa, q, q, q, None, 1, out=q))
    agree(both(jv.sdpa, q, q, q, arr(f16, (5, 5)), 0.5, out=q))
    assert taken > 100


def test_layernorm(both):
    random.seed(3)
    f16, f32, taken = np.float16, np.float32, 0
    for C, rows, ti, to in itertools.product((1, 8, 13, 1280), (0, 1, 7), (f16, f32, np.uint8), (f16, f32, np.uint8)):
        for g, b in ((None, None), ((ti, C), (ti, C)), ((f32, C), None), ((ti, C), (ti, C + 1))):
            vec = lambda d: arr(d[0], (d[1],)) if d else None
            taken += agree(both(jv.layernorm_, arr(to, (C, rows)), arr(f32, (rows,)), arr(f32, (rows + 1,)), arr(ti, (C, rows)), vec(g), vec(b), C, 1e-5))
    a = arr(f16, (8, 6))
    for out, mean, rstd, C, eps in ((arr(f16, (8, 5)), arr(f32, (6,)), arr(f32, (6,)), 8, 1e-5), (a, arr(f16, (6,)), arr(f32, (6,)), 8, 1e-5),
                                    (a, arr(f32, (5,)), arr(f32, (6,)), 8, 1e-5), (a, arr(f32, (6,)), arr(f32, (6,)), 7, 1e-5),
                                    (a, arr(f32, (6,)), arr(f32, (6,)), 8, 1), (arr(f16, (8, 6), (1, 9)), arr(f32, (6,)), arr(f32, (6,)), 8, 1e-5),
                                    (a, arr(f32, (1,)), arr(f32, (1,)), 48, 1e-5)):
        agree(both(jv.layernorm_, out, mean, rstd, a, None, None, C, eps))
    assert taken > 50


def test_convolution(both):
    random.seed(4)
    f16, taken = np.float16, 0
    for W, H, k, s, p, d, groups in itertools.product((1, 9), (4, 17), (1, 3), (1, 2), (0, 1), (1, 2), (1, 2, 3)):
        OW, OH = jv.convsize(W, k, s, p, d), jv.convsize(H, k, s, p, d)
        x, w = arr(f16, (W, H, 6, 2)), arr(f16, (k, k, 6 // groups, 12))
        for dt, bias in ((f16, arr(f16, (12,))), (np.float32, None), (np.uint8, None)):
            taken += agree(both(jv.convolution_, arr(dt, (OW, OH, 12, 2)), x, w, bias, (s, s), (p, p), (d, d), groups, act="relu"))
    x, w, out = arr(f16, (9, 9, 4, 1)), arr(f16, (3, 3, 4, 8)), arr(f16, (7, 7, 8, 1))
    for o, xx, ww, st, g, act in ((out, x, w, [1, 1], 1, "relu"), (arr(f16, (7, 8, 8, 1)), x, w, (1, 1), 1, "relu"), (out, x, w, (1, 1), 0, "relu"),
                                  (out, arr(np.float32, (9, 9, 4, 1)), w, (1, 1), 1, "relu"), (out, x, w, (1, 1), 1, "swish"),
                                  (out, arr(f16, (9, 9, 4, 1), (1, 9, 90, 400)), w, (1, 1), 1, None), (out, x, arr(f16, (3, 3, 5, 8)), (1, 1), 1, None)):
        agree(both(jv.convolution_, o, xx, ww, None, st, (0, 0), (1, 1), g, act=act))
    assert taken > 50


def test_convolution_bias(both, monkeypatch):
    """One fp16 value per channel, side by side: any other type, fewer of them or a stride is refused on both routes, and
    in the transposed form; a vector of more axes, or one that goes on behind the channels, is read as it always was."""
    f16, f32 = np.float16, np.float32
    x, w, out = arr(f16, (9, 9, 4, 1)), arr(f16, (3, 3, 4, 8)), arr(f16, (7, 7, 8, 1))
    args = ((1, 1), (0, 0), (1, 1))
    for b in (arr(f32, (8,)), arr(np.uint8, (8,)), arr(f16, (7,)), arr(f16, (8,), (2,)), arr(f16, (1,))):
        assert both(jv.convolution_, out, x, w, b, *args) == [jv.B200Error, jv.B200Error], b
    for b in (arr(f16, (8,)), arr(f16, (1, 1, 8, 1)), arr(f16, (8,), ptr=2), arr(f16, (9,)), None):
        assert agree(both(jv.convolution_, out, x, w, b, *args)), b
    wt, wide = arr(f16, (3, 3, 8, 4)), arr(f16, (11, 11, 8, 1))
    monkeypatch.setattr(_lib._lib, "b200_convtranspose2d_f16", lambda *a: 0, raising=False)
    for b in (arr(f32, (8,)), arr(f16, (7,)), arr(f16, (8,), (2,))):
        with pytest.raises(jv.B200Error):
            jv.convolutiontranspose_(FakeCtx, wide, x, wt, b, *args)
    jv.convolutiontranspose_(FakeCtx, wide, x, wt, arr(f16, (8,)), *args)


def test_an_array_has_one_element_type(both):
    """The native route reads the dtype the array shows, as the Python route does: also after it was assigned."""
    f16, f32 = np.float16, np.float32
    A, B, out = arr(f32, (8, 4)), arr(f32, (4, 3)), arr(f16, (8, 3))
    assert not agree(both(jv.matmul_, out, A, B, None))                # fp32 products of several tokens are declined
    A.dtype = B.dtype = np.dtype(f16)
    assert agree(both(jv.matmul_, out, A, B, None))
    out.dtype = np.dtype(f32)
    assert agree(both(jv.matmul_, out, A, B, None))
    for d in (">f2", "i2", "f8"):
        A.dtype = np.dtype(d)
        assert not agree(both(jv.matmul_, out, A, B, None)), d


def test_numbers_that_wrap_in_64_bits_go_the_python_route(both):
    """Python's integers do not wrap: what it refuses for its size must not be read as a small number."""
    f16, f32, big = np.float16, np.float32, 1 << 32
    a, m = arr(f16, (big, big)), arr(f32, (4,))
    assert both(jv.layernorm_, arr(f16, (big, big)), m, m, a, None, None, 1, 1e-5) == [jv.B200Error] * 2     # 2^64 elements
    x, w = arr(f16, (9, 9, 4, 1)), arr(f16, (3, 3, 4, 8))
    for out, p, d in ((arr(f16, (5, 5, 8, 1)), (1 << 63) - 1, 1), (arr(f16, (7, 7, 8, 1)), 0, (1 << 63) + 1), (arr(f16, (5, 5, 8, 1)), 1, (1 << 62) + 2)):
        assert not agree(both(jv.convolution_, out, x, w, None, (1, 1), (p, p), (d, d))), (p, d)
    assert agree(both(jv.convolution_, arr(f16, (7, 7, 8, 1)), x, w, None, (1, 1), (0, 0), (1, 1)))
