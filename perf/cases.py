"""The work a user of this package has it do, as cases that can be timed and compared.

`listed()` names them, `draw()` gives more of the same ranges, `prepare()` makes what a program holds before
the call (device arrays, weights, a recorded pass), `run()` is one pass through the public entry points.
Inputs are made on the GPU from the seed alone; a result is handed back as a tensor over the library's own
output buffer.
"""
import math

import numpy as np
import torch

import juliavision_b200 as jv
from juliavision_b200.encoder import Encoder, EncoderConfig
from juliavision_b200.hiera import Hiera, HieraConfig

NP = {"f16": np.float16, "f32": np.float32}
TORCH = {"f16": torch.float16, "f32": torch.float32}
SIZE = {"f16": 2, "f32": 4}
_ctx = None


def context():
    """The one context a program keeps for its GPU."""
    global _ctx
    if _ctx is None:
        _ctx = jv.Ctx(0)
    return _ctx


# ------------------------------------------------------------------------------------- the cases
def listed():
    return [
        # One token through a 1280-wide projection: the smallest call a decoder makes, many times per token.
        dict(name="token_1280x1280", kind="linear", tokens=1, features=1280, k=1280, epi="none", dtype="f16"),
        # The vocabulary projection for a beam of five: 51865 rows, a leading dimension no 16-byte boundary divides.
        dict(name="logits_5x51865x1280", kind="linear", tokens=5, features=51865, k=1280, epi="none", dtype="f16"),
        # An ordinary linear layer with a bias.
        dict(name="linear_4096x3072x768", kind="linear", tokens=4096, features=3072, k=768, epi="none", dtype="f16"),
        # The largest product of the row-sharded sweep.
        dict(name="linear_65536x5120x1280", kind="linear", tokens=65536, features=5120, k=1280, epi="none", dtype="f16"),
        # Self attention at the head dim and length of a long encoder, batch 1.
        dict(name="attention_4096_e64_h12", kind="attention", batch=1, heads=12, queries=4096, keys=4096, head_dim=64,
             mask=False, packed=False),
        # The image model's global attention: 72-wide heads.
        dict(name="attention_4096_e72_h8", kind="attention", batch=1, heads=8, queries=4096, keys=4096, head_dim=72,
             mask=False, packed=False),
        # The mem-efficient variant with its additive mask, one (queries, keys) plane for all heads.
        dict(name="attention_masked_1500_h20", kind="attention", batch=1, heads=20, queries=1500, keys=1500, head_dim=64,
             mask=True, packed=False),
        # A decoder's few queries over a long memory.
        dict(name="attention_23x4096_h8", kind="attention", batch=1, heads=8, queries=23, keys=4096, head_dim=64,
             mask=False, packed=False),
        # A layer norm over a tensor larger than the L2 cache.
        dict(name="layernorm_65536x1280", kind="layernorm", rows=65536, width=1280, dtype="f16"),
        # The stem of an image encoder: 1024 x 1024 x 3, 7x7 kernel, stride 4, 112 channels.
        dict(name="conv_stem_1024", kind="conv", width=1024, height=1024, cin=3, cout=112, kernel=7, stride=4, pad=3, images=1,
             act="identity"),
        # The whole 32-layer encoder on one 1500-token input, recorded once and replayed.
        dict(name="encoder_32x1280_1500", kind="encoder", layers=32, d_model=1280, heads=20, ffn=5120, tokens=1500),
        # The whole hierarchical image encoder, eight 1024 x 1024 images per pass, recorded once and replayed.
        dict(name="hiera_8x1024", kind="hiera", images=8, side=1024),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["linear", "linear", "linear", "token", "logits", "attention", "attention", "few", "windows", "layernorm",
                       "conv", "encoder", "hiera"])
    if kind == "linear":
        while True:
            tokens, features, k = _log(rng, 2, 65536), 8 * _log(rng, 14, 640), 8 * _log(rng, 14, 640)
            if tokens * features * k <= 65536 * 5120 * 1280:
                return dict(kind="linear", tokens=tokens, features=features, k=k, epi=rng.choice(["none", "none", "gelu", "relu"]),
                            dtype="f16")
    if kind == "token":
        return dict(kind="linear", tokens=1, features=_log(rng, 256, 51865), k=_log(rng, 256, 5120),
                    epi=rng.choice(["none", "gelu"]), dtype=rng.choice(["f16", "f32"]))
    if kind == "logits":
        return dict(kind="linear", tokens=_log(rng, 2, 64), features=2 * _log(rng, 500, 26000) + 1, k=8 * _log(rng, 48, 160),
                    epi="none", dtype="f16")
    if kind == "attention":
        while True:
            c = dict(kind="attention", batch=rng.choice([1, 1, 2, 4]), heads=rng.randint(2, 20), queries=_log(rng, 64, 4096),
                     keys=0, head_dim=rng.choice([32, 56, 64, 64, 72, 80, 96, 128]), mask=rng.random() < 0.25,
                     packed=rng.random() < 0.5)
            c["keys"] = c["queries"]
            if c["batch"] * c["heads"] * c["queries"] ** 2 * c["head_dim"] <= 4096 * 4096 * 64 * 24:
                return c
    if kind == "few":
        return dict(kind="attention", batch=rng.choice([1, 1, 2]), heads=rng.randint(4, 20), queries=_log(rng, 1, 64),
                    keys=_log(rng, 256, 8192), head_dim=rng.choice([56, 64, 64, 72, 128]), mask=rng.random() < 0.25, packed=False)
    if kind == "windows":
        side = rng.choice([4, 7, 8, 8, 14, 16])
        return dict(kind="attention", batch=_log(rng, 32, 262144 // side ** 3 // 2), heads=rng.randint(2, 8), queries=side * side,
                    keys=side * side, head_dim=rng.choice([56, 56, 64]), mask=False, packed=True)
    if kind == "layernorm":
        while True:
            rows, width = _log(rng, 64, 262144), 8 * _log(rng, 14, 640)
            if rows * width <= 65536 * 1280:
                return dict(kind="layernorm", rows=rows, width=width, dtype=rng.choice(["f16", "f16", "f32"]))
    if kind == "conv":
        side, stride = _log(rng, 32, 1024), rng.choice([1, 1, 2, 4])
        kernel = {1: rng.choice([1, 3]), 2: 3, 4: 7}[stride]
        cin = 3 if stride == 4 else 8 * _log(rng, 2, 32)
        cout = 8 * _log(rng, 4, 32)
        while side * side * cin * max(1, kernel * kernel // stride ** 2) > 1024 * 1024 * 16:
            side //= 2
        return dict(kind="conv", width=side, height=max(16, side - rng.randint(0, 9)), cin=cin, cout=cout, kernel=kernel,
                    stride=stride, pad=kernel // 2, images=rng.choice([1, 1, 2]), act=rng.choice(["identity", "relu"]))
    if kind == "encoder":
        heads = rng.choice([6, 8, 12, 16, 20])
        return dict(kind="encoder", layers=rng.randint(1, 8), d_model=64 * heads, heads=heads, ffn=256 * heads,
                    tokens=_log(rng, 50, 3000))
    return dict(kind="hiera", images=rng.randint(1, 8), side=rng.choice([512, 1024]))


# ----------------------------------------------------------------------------------- preparation
def _randn(gen, shape, scale, dtype=torch.float16):
    return torch.randn(shape, generator=gen, device="cuda", dtype=torch.float32).mul_(scale).to(dtype)


def _array(t):
    """A dense tensor as the device array of the reversed shape."""
    return jv.DeviceArray(context(), t.data_ptr(), {torch.float16: np.float16, torch.float32: np.float32}[t.dtype],
                          tuple(reversed(t.shape)), owner=t)


class _Interface:
    def __init__(self, a):
        self.owner = a
        self.__cuda_array_interface__ = dict(version=3, data=(a.ptr, False), shape=tuple(reversed(a.shape)),
                                             typestr={2: "<f2", 4: "<f4"}[a.dtype.itemsize], strides=None)


def _tensor(a):
    """A dense device array as a tensor over the same memory, in the reversed (torch) order."""
    return torch.as_tensor(_Interface(a), device="cuda")


def _host_linear(gen, out, inp, scale):
    """A host (out, in) weight whose memory holds (in, out): the transposed copy the upload asks for is then a view."""
    return _randn(gen, (inp, out), scale).cpu().numpy().T


def _host(gen, *shape, scale=0.02):
    return _randn(gen, shape, scale).cpu().numpy()


def prepare(case, seed):
    ctx = context()
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    return globals()["_prepare_" + case["kind"]](ctx, case, gen)


def _prepare_linear(ctx, c, gen):
    dt = TORCH[c["dtype"]]
    x = _array(_randn(gen, (c["tokens"], c["k"]), 1.0, dt))
    w = _array(_randn(gen, (c["k"], c["features"]), 0.05, dt))
    b = _array(_randn(gen, (c["features"],), 0.05, dt))
    out = ctx.allocate(NP[c["dtype"]], c["features"], c["tokens"])
    epi = {"none": "identity"}.get(c["epi"], c["epi"])
    return dict(run=_run_linear, ctx=ctx, x=x, w=w, b=b, epi=epi, out=out, result=_tensor(out))


def _prepare_attention(ctx, c, gen):
    B, H, Lq, Lk, E = c["batch"], c["heads"], c["queries"], c["keys"], c["head_dim"]
    if c["packed"]:      # q, k and v side by side in one projection, tokens outermost; the result token-major as well
        d = H * E
        qkv = _randn(gen, (B * Lk, 3 * d), 1.0)
        q, k, v = (jv.DeviceArray(ctx, qkv.data_ptr() + 2 * i * d, np.float16, (E, Lk, H, B), (1, 3 * d, E, 3 * d * Lk), owner=qkv)
                   for i in range(3))
        buf = ctx.allocate(np.float16, d, Lq * B)
        out = jv.DeviceArray(ctx, buf.ptr, np.float16, (E, Lq, H, B), (1, d, E, d * Lq), owner=buf)
    else:
        q = _array(_randn(gen, (B, H, Lq, E), 1.0))
        k, v = (_array(_randn(gen, (B, H, Lk, E), 1.0)) for _ in range(2))
        out = buf = ctx.allocate(np.float16, E, Lq, H, B)
    mask = None
    if c["mask"]:        # a finite bias, and a tenth of the keys hidden from each query
        m = _randn(gen, (1, 1, Lq, Lk), 0.5)
        m.masked_fill_(torch.rand((1, 1, Lq, Lk), generator=gen, device="cuda") < 0.1, float("-inf"))
        mask = _array(m)
    return dict(run=_run_attention, ctx=ctx, q=q, k=k, v=v, mask=mask, scale=1.0 / math.sqrt(E), out=out, result=_tensor(buf))


def _prepare_layernorm(ctx, c, gen):
    dt = TORCH[c["dtype"]]
    a = _array(_randn(gen, (c["rows"], c["width"]), 1.0, dt))
    g, b = (_array((_randn(gen, (c["width"],), 0.1, torch.float32) + o).to(dt)) for o in (1.0, 0.0))
    out = ctx.allocate(NP[c["dtype"]], c["width"], c["rows"])
    mean, rstd = ctx.allocate(np.float32, c["rows"]), ctx.allocate(np.float32, c["rows"])
    return dict(run=_run_layernorm, ctx=ctx, a=a, g=g, b=b, out=out, mean=mean, rstd=rstd, width=c["width"],
                result=[_tensor(t) for t in (out, mean, rstd)])


def _conv_out(c):
    return [(n + 2 * c["pad"] - c["kernel"]) // c["stride"] + 1 for n in (c["width"], c["height"])]


def _prepare_conv(ctx, c, gen):
    x = _array(torch.rand((c["images"], c["cin"], c["height"], c["width"]), generator=gen, device="cuda").half())
    w = _array(_randn(gen, (c["cout"], c["cin"], c["kernel"], c["kernel"]), 0.05))
    b = _array(_randn(gen, (c["cout"],), 0.05))
    ow, oh = _conv_out(c)
    out = ctx.allocate(np.float16, ow, oh, c["cout"], c["images"])
    return dict(run=_run_conv, ctx=ctx, x=x, w=w, b=b, out=out, stride=(c["stride"],) * 2, pad=(c["pad"],) * 2, act=c["act"],
                result=_tensor(out))


def _prepare_encoder(ctx, c, gen):
    cfg = EncoderConfig(layers=c["layers"], d_model=c["d_model"], heads=c["heads"], ffn=c["ffn"], tokens=c["tokens"])
    d, f = cfg.d_model, cfg.ffn
    ones, zeros = np.ones(d, np.float16), np.zeros(d, np.float16)
    w = lambda o, i: _host_linear(gen, o, i, 0.02)
    weights = [dict(ln1_g=ones, ln1_b=zeros, wq=w(d, d), bq=_host(gen, d), wk=w(d, d), wv=w(d, d), bv=_host(gen, d), wo=w(d, d),
                    bo=_host(gen, d), ln2_g=ones, ln2_b=zeros, w1=w(f, d), b1=_host(gen, f), w2=w(d, f), b2=_host(gen, d))
               for _ in range(cfg.layers)] + [dict(lnf_g=ones, lnf_b=zeros)]
    enc = Encoder(ctx, cfg, weights)
    _tensor(enc.xin).copy_(_randn(gen, (cfg.tokens, d), 1.0))
    torch.cuda.synchronize()
    return dict(run=_run_recorded, model=enc, graph=enc.capture(), result=[_tensor(enc.x), _tensor(enc.y)])


def _prepare_hiera(ctx, c, gen):
    cfg = HieraConfig(image=c["side"])
    n, lin, k = (lambda *s: _host(gen, *s)), (lambda o, i: _host_linear(gen, o, i, 0.02)), cfg.patch[0]
    S0 = cfg.side(0)
    weights = dict(stem_w=n(cfg.embed, cfg.in_ch, k, k), stem_b=n(cfg.embed), pos=n(S0, S0, cfg.embed), blocks=[])
    for b in cfg.blocks():
        di, d, f = b["dim_in"], b["dim"], b["dim"] * cfg.mlp_ratio
        bw = dict(ln1_g=np.ones(di, np.float16), ln1_b=np.zeros(di, np.float16), wqkv=lin(3 * d, di), bqkv=n(3 * d), wo=lin(d, d),
                  bo=n(d), ln2_g=np.ones(d, np.float16), ln2_b=np.zeros(d, np.float16), w1=lin(f, d), b1=n(f), w2=lin(d, f), b2=n(d))
        if b["pool"]:
            bw.update(wproj=lin(d, di), bproj=n(d))
        weights["blocks"].append(bw)
    model = Hiera(ctx, cfg, weights, batch=c["images"])
    image = _tensor(model.image)
    image.copy_(torch.rand(image.shape, generator=gen, device="cuda"))
    torch.cuda.synchronize()
    return dict(run=_run_recorded, model=model, graph=model.capture(), result=_tensor(model.y))


# ------------------------------------------------------------------------------------- one pass
def run(state):
    state["run"](state)
    return state["result"]


def _run_linear(s):
    s["ctx"].ws.reset()
    jv.matmul_(s["ctx"], s["out"], s["w"], s["x"], s["b"], epi=s["epi"])


def _run_attention(s):
    s["ctx"].ws.reset()
    jv.sdpa(s["ctx"], s["q"], s["k"], s["v"], s["mask"], s["scale"], out=s["out"])


def _run_layernorm(s):
    jv.layernorm_(s["ctx"], s["out"], s["mean"], s["rstd"], s["a"], s["g"], s["b"], s["width"], 1e-5)


def _run_conv(s):
    s["ctx"].ws.reset()
    jv.convolution_(s["ctx"], s["out"], s["x"], s["w"], s["b"], s["stride"], s["pad"], (1, 1), 1, act=s["act"])


def _run_recorded(s):
    s["graph"].replay()


# ------------------------------------------------------------------- what a pass cannot do without
def work(case):
    c = case
    if c["kind"] == "linear":
        t, f, k = c["tokens"], c["features"], c["k"]
        return dict(bytes=SIZE[c["dtype"]] * (t * k + k * f + f + t * f), flops=2.0 * t * f * k)
    if c["kind"] == "attention":
        B, H, Lq, Lk, E = c["batch"], c["heads"], c["queries"], c["keys"], c["head_dim"]
        return dict(bytes=2 * (B * H * E * (2 * Lq + 2 * Lk) + (Lq * Lk if c["mask"] else 0)), flops=4.0 * B * H * Lq * Lk * E)
    if c["kind"] == "layernorm":
        return dict(bytes=SIZE[c["dtype"]] * (2 * c["rows"] * c["width"] + 2 * c["width"]) + 8 * c["rows"],
                    flops=8.0 * c["rows"] * c["width"])
    if c["kind"] == "conv":
        ow, oh = _conv_out(c)
        crs = c["cin"] * c["kernel"] ** 2
        return dict(bytes=2 * (c["images"] * (c["width"] * c["height"] * c["cin"] + ow * oh * c["cout"]) + crs * c["cout"] + c["cout"]),
                    flops=2.0 * c["images"] * ow * oh * crs * c["cout"])
    if c["kind"] == "encoder":
        cfg = EncoderConfig(layers=c["layers"], d_model=c["d_model"], heads=c["heads"], ffn=c["ffn"], tokens=c["tokens"])
        d, f = cfg.d_model, cfg.ffn
        return dict(bytes=2 * (c["layers"] * (4 * d * d + 2 * d * f + 9 * d + f) + 3 * d * c["tokens"]), flops=cfg.flops())
    cfg = HieraConfig(image=c["side"])
    weights = cfg.embed * cfg.in_ch * cfg.patch[0] ** 2 + cfg.side(0) ** 2 * cfg.embed
    for b in cfg.blocks():
        weights += 3 * b["dim"] * b["dim_in"] + (1 + 2 * cfg.mlp_ratio) * b["dim"] ** 2 + (b["dim"] * b["dim_in"] if b["pool"] else 0)
    last = cfg.blocks()[-1]
    return dict(bytes=2 * (weights + c["images"] * (3 * c["side"] ** 2 + last["side"] ** 2 * last["dim"])), flops=cfg.flops(c["images"]))


def tolerance(case):
    """About four times what the path differs by from the same computation in 64 bits: 1.8e-3 over the 32 layers,
    2.9e-4 for attention (P is rounded to fp16), 2.1e-4 for one rounding to fp16 (3.0e-4 behind a GELU), 1.7e-7 in fp32."""
    if case["kind"] in ("encoder", "hiera"):
        return dict(rel=6e-3)
    if case["kind"] == "attention":
        return dict(rel=1.2e-3)
    if case.get("dtype") == "f32":
        return dict(rel=2e-6)
    return dict(rel=8e-4)
