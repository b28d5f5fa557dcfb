"""What the speed of this framework is measured on: the work a user has it do, through its public entry points.

A case is a dict of plain values.  Its ``"kind"`` is one of

* ``frame``   ``Engine.gen_frame``: one generated latent frame (4 denoising passes and the commit pass) of a session
* ``append``  ``Engine.append_frame``: one given latent frame committed to the caches of a session (one pass, eager)
* ``attn``    ``qf.kv_cache_update`` then ``qf.owl_attn``: one layer's append and attention, for a program with its own wiring
* ``gemm``    ``qf.gemm`` with its epilogues
* ``moe``     ``nn.MoE``: the mixture-of-experts MLP of one layer
* ``glue``    one norm, elementwise or narrowing call of ``qf.*``

``listed()`` gives the cases that are always measured, ``draw(rng)`` one more of the same ranges.  ``prepare`` builds on the
GPU what the user's program holds before the call, ``run`` makes one pass, ``work`` and ``tolerance`` say what the pass cannot
do without and how close another correct implementation at the same precision comes.
"""

from __future__ import annotations

import math

import numpy as np
import torch

import quark_b200 as qb
from quark_b200 import nn, qf
from quark_b200.engine import CtrlInput
from quark_b200.models.waypoint_15 import QuantConfig, Waypoint15Config

BYTES = {"bf16": 2, "e4m3": 1, "f32": 4}
TORCH = {"bf16": torch.bfloat16, "e4m3": torch.float8_e4m3fn, "f32": torch.float32}


# --------------------------------------------------------------------------------------------------------------- the cases


def _session(kind, name, height, width, layers, linear, kv, attn, *, d_model=2048, ctrl=False, scales=False, quilt=1):
    c = dict(kind=kind, height=height, width=width, layers=layers, d_model=d_model, linear=linear, kv=kv, attn=attn, ctrl=ctrl, scales=scales, quilt=quilt)
    return dict(c, name=name) if name else c


def _attn(name, height, width, buckets, kv_heads, gqa, dtype, *, packed=True, dilation=1, quilt=1, frame_t=1000):
    c = dict(kind="attn", height=height, width=width, buckets=buckets, kv_heads=kv_heads, gqa=gqa, dtype=dtype, packed=packed, dilation=dilation,
             quilt=quilt, frame_t=frame_t)  # fmt: skip
    return dict(c, name=name) if name else c


def _gemm(name, M, N, K, a, b, out, epilogue="none", groups=1):
    c = dict(kind="gemm", M=M, N=N, K=K, a=a, b=b, out=out, epilogue=epilogue, groups=groups)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the headline: a 720p session (32 x 16 tokens, 24 layers) with linears, caches and attention in e4m3
        _session("frame", "frame-720p-fp8", 32, 16, 24, "fp8", "fp8", "fp8"),
        # the same session without quantisation
        _session("frame", "frame-720p-bf16", 32, 16, 24, "bf16", "bf16", "bf16"),
        # the small resolution (16 x 8 tokens), where every GEMM streams its weights for 128 rows
        _session("frame", "frame-360p-bf16", 16, 8, 24, "bf16", "bf16", "bf16"),
        # a recorded clip being fed into a session before generation starts: one eager pass per frame
        _session("append", "append-360p-fp8", 16, 8, 24, "fp8", "fp8", "fp8"),
        # a smaller model with a controller, an odd grid (240 tokens) and e4m3 caches read by bf16 attention
        _session("frame", "frame-ctrl-mixed", 12, 20, 6, "fp8", "fp8", "bf16", d_model=1024, ctrl=True),
        # one mixture-of-experts MLP at 720p: 8 experts of half the MLP's width, 2 per token
        dict(kind="moe", name="moe-720p-fp8", M=512, D=2048, H=4096, experts=8, top_k=2, fp8=True),
        # the controller row through its first linear: the smallest matrix product of a frame
        _gemm("gemm-row-bf16", 1, 8192, 272, "bf16", "bf16", "bf16", "silu"),
        # a product whose sizes fit no tile
        _gemm("gemm-ragged-bf16", 777, 1096, 1296, "bf16", "bf16", "f32", "bias_silu"),
        # the square product by which the e4m3 rate of the library is quoted
        _gemm("gemm-8192-fp8", 8192, 8192, 8192, "e4m3", "e4m3", "bf16"),
        # attention over a long history: 720p, 128 buckets of 512 keys, e4m3
        _attn("attn-720p-long-fp8", 32, 16, 128, 16, 2, "e4m3", dilation=8),
        # append and attention of a 360p layer in the head-major layout, the functional default
        _attn("attn-360p-bf16", 16, 8, 16, 16, 2, "bf16", packed=False),
        # the norm before a linear at 360p: the smallest call of a frame
        dict(kind="glue", name="norm-360p", op="ada_rmsnorm", rows=128, D=2048),
    ]


def _log(rng, lo, hi, step=1):
    """A multiple of ``step`` in ``[lo, hi]``, spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(hi // step * step, max(-(-lo // step) * step, int(v / step + 0.5) * step))


def _draw_grid(rng, quilt):
    """A token grid of 64 to 512 tokens whose cached frame is a multiple of 16 tokens."""
    while True:
        h, w = rng.randint(4, 32), rng.randint(4, 32)
        if 64 <= h * w <= 512 and h * w % (16 * quilt) == 0:
            return h, w


def draw(rng):
    kind = rng.choice(["frame", "frame", "append", "attn", "attn", "gemm", "gemm", "gemm", "moe", "glue"])
    if kind in ("frame", "append"):
        quilt = rng.choice([1, 1, 1, 2])
        h, w = _draw_grid(rng, quilt)
        linear, kv, attn = rng.choice([("fp8", "fp8", "fp8"), ("fp8", "fp8", "fp8"), ("bf16", "bf16", "bf16"), ("fp8", "bf16", "bf16"), ("bf16", "fp8", "fp8"), ("fp8", "fp8", "bf16")])  # fmt: skip
        scales = attn == "fp8" and rng.random() < 0.25
        return _session(kind, None, h, w, _log(rng, 2, 24), linear, kv, attn, d_model=rng.choice([512, 1024, 1536, 2048, 2048]), ctrl=rng.random() < 0.3,
                        scales=scales, quilt=quilt)  # fmt: skip
    if kind == "attn":
        quilt = rng.choice([1, 1, 2])
        h, w = _draw_grid(rng, quilt)
        buckets, dilation = _log(rng, 2, 128), rng.choice([1, 1, 8])
        return _attn(None, h, w, buckets, rng.choice([1, 2, 4, 8, 16, 16]), rng.choice([1, 2, 2, 4]), rng.choice(["bf16", "e4m3"]), packed=rng.random() < 0.6,
                     dilation=dilation, quilt=quilt, frame_t=_log(rng, 1, 4 * buckets * dilation))  # fmt: skip
    if kind == "gemm":
        a, b = rng.choice([("bf16", "bf16"), ("e4m3", "e4m3"), ("bf16", "e4m3")])
        M, N, K = _log(rng, 1, 8192), _log(rng, 64, 8192, 8), _log(rng, 64, 8192, 16)
        epilogue = rng.choice(["none", "silu", "bias_silu", "gate"])
        out = rng.choice(["bf16", "bf16", "f32", "e4m3"]) if epilogue != "gate" else "bf16"
        groups = 2 if epilogue == "gate" and M % 2 == 0 and rng.random() < 0.3 else 1
        return _gemm(None, M, N, K, a, b, out, epilogue, groups)
    if kind == "moe":
        return dict(kind="moe", M=_log(rng, 16, 512), D=_log(rng, 256, 2048, 64), H=_log(rng, 256, 4096, 64), experts=rng.choice([8, 16]),
                    top_k=rng.choice([1, 2, 4]), fp8=rng.random() < 0.5)  # fmt: skip
    op = rng.choice(["ada_rmsnorm", "ada_rmsnorm_q", "rmsnorm", "head_rmsnorm", "silu", "gate_residual", "add", "euler", "quantize", "dequantize"])
    D = 64 * rng.choice([4, 8, 16, 32, 64]) if op == "head_rmsnorm" else _log(rng, 64, 8192, 8)
    return dict(kind="glue", op=op, rows=_log(rng, 1, 8192), D=D)


# ------------------------------------------------------------------------------------------------------------------ inputs


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _randn(g, shape, dtype="bf16", std=1.0):
    if dtype == "e4m3":
        return (torch.randn(shape, device="cuda", generator=g) * std).to(torch.float8_e4m3fn)
    return torch.randn(shape, device="cuda", generator=g, dtype=TORCH[dtype]) * std


def _q(t, shape=None):
    """The framework's tensor over a torch tensor's memory."""
    names = {torch.bfloat16: "bf16", torch.float8_e4m3fn: "e4m3", torch.float32: "f32", torch.int32: "s32"}
    return qb.QuarkTensor.borrow(t.data_ptr(), tuple(t.shape) if shape is None else shape, names[t.dtype], keepalive=t)


def _config(c):
    quant = QuantConfig(linear=c["linear"], kv_cache=c["kv"], attn_compute=c["attn"], moe="bf16")
    heads = c["d_model"] // 64
    return Waypoint15Config(d_model=c["d_model"], n_layers=c["layers"], n_heads=heads, n_kv_heads=heads // 2, height=c["height"], width=c["width"],
                            ctrl_conditioning=c["ctrl"], fp8_scales=c["scales"], quilt_factor=c["quilt"], quant=quant)  # fmt: skip


def _load_weights(model, cfg, g):
    """Random weights and conditioning rows, made on the GPU: linears N(0, 0.02), a patch embedding of unit variance, scales
    and biases N(0, 0.2), gates N(0, 0.05), so that a block adds some per cent to the residual stream, as in a trained model."""
    weights = {}
    for name, p in model.named_parameters():
        if not name.endswith("lamb"):  # the value residual keeps its initial 0.5
            shape = tuple(p.data.shape)
            weights[name] = _q(_randn(g, shape, std=shape[1] ** -0.5 if name == "patchify.weight" else 0.02))
    model.load_state_dict(weights, strict=False)
    sigmas, d = len(cfg.scheduler_sigmas), cfg.d_model
    rows = _randn(g, (cfg.n_layers, sigmas, 6, 1, d), std=0.2)  # scale, bias, gate of the attention, then of the MLP
    rows[:, :, 2::3] *= 0.25
    for blk, per_sigma in zip(model.blocks, rows):
        blk._cond_lut = [tuple(_q(r) for r in six) for six in per_sigma]
    model._out_norm_luts = [tuple(_q(r) for r in two) for two in _randn(g, (sigmas, 2, 1, d), std=0.2)]
    torch.cuda.synchronize()
    model.prepare()


def _fill_caches(model, cfg, g):
    """Every layer's caches in one piece of memory each, filled with N(0, 1) keys and values as after 128 frames."""
    dt = "e4m3" if cfg.quant.kv_cache == "fp8" else "bf16"
    sizes = [blk.kv_cache.K_cache.numel for blk in model.blocks]
    K, V = (torch.empty(sum(sizes), device="cuda", dtype=TORCH[dt]) for _ in range(2))
    at = 0
    for blk, n in zip(model.blocks, sizes):
        kc = blk.kv_cache
        std_k = std_v = 1.0
        if cfg.fp8_scales and dt == "e4m3":  # the caches then hold the values divided by their head's scale
            heads = np.ones(cfg.n_kv_heads, np.float32)
            kc.set_scales(heads * (8.0 / 448.0), heads * (6.0 / 448.0))
            std_k, std_v = 448.0 / 8.0, 448.0 / 6.0
        for whole, std, name in ((K, std_k, "K_cache"), (V, std_v, "Vt_cache")):
            part = whole[at : at + n]
            part.copy_(torch.randn(n, device="cuda", generator=g) * std)
            setattr(kc, name, _q(part, getattr(kc, name).shape))
        at += n
    torch.cuda.synchronize()
    return K, V


def _prepare_session(c, seed):
    cfg = _config(c)
    g = _gen(seed)
    engine = qb.Engine(cfg=cfg, quant=cfg.quant, load_weights=False)
    _load_weights(engine.model, cfg, g)
    K, V = _fill_caches(engine.model, cfg, g)
    engine.set_frame_t(128)
    r = np.random.default_rng(seed)
    latent = r.standard_normal((1, cfg.channels, cfg.height * cfg.patch[0], cfg.width * cfg.patch[1]), dtype=np.float32)
    ctrl = CtrlInput(button={3, 17, 40}, mouse=(float(r.normal()), float(r.normal())), scroll_wheel=1) if c["ctrl"] else None
    s = dict(c=c, engine=engine, latent=latent, ctrl=ctrl, K=K, V=V)
    _run_session(s)  # a session's first frame makes its buffers and captures its graph; the ones after it are what counts
    return s


def _run_session(s):
    if s["c"]["kind"] == "append":
        s["engine"].append_frame(s["latent"], s["ctrl"])
        return [s["K"], s["V"]]
    out = s["engine"].gen_frame(s["ctrl"], noise=s["latent"])
    return [torch.from_numpy(out.view(np.int16)).view(torch.bfloat16), s["K"], s["V"]]


def _prepare_attn(c, seed):
    g = _gen(seed)
    tpf, Hk, Hq = c["height"] * c["width"], c["kv_heads"], c["kv_heads"] * c["gqa"]
    kept = tpf // c["quilt"]
    cap = (c["buckets"] + 1) * kept
    es = c["dtype"]
    # values of a channel share an offset, as a projection's do
    offset = 0.5 * torch.randn((Hk, 64), device="cuda", generator=g)
    if c["packed"]:
        q = _randn(g, (tpf, (Hq + 2 * Hk) * 64))
        q[:, (Hq + Hk) * 64 :] += offset.reshape(1, -1).to(torch.bfloat16)
        k = v = None
    else:
        q, k, v = _randn(g, (Hq * tpf, 64)), _randn(g, (Hk * tpf, 64)), _randn(g, (Hk * tpf, 64))
        v += offset.repeat_interleave(tpf, 0).to(torch.bfloat16)
    K = _randn(g, (Hk * cap, 64), es)
    V = (torch.randn((Hk * 64, cap), device="cuda", generator=g) + offset.reshape(-1, 1)).to(TORCH[es])
    out = torch.zeros((tpf, Hq * 64) if c["packed"] else (Hq * tpf, 64), device="cuda", dtype=torch.bfloat16)
    ints = torch.tensor([c["frame_t"], 0, 0, 0, 0, 0, 0, 0, 0], device="cuda", dtype=torch.int32)
    geo = dict(B=1, n_kv_heads=Hk, H_spatial=c["height"], W_spatial=c["width"], num_buckets=c["buckets"], pinned_dilation=c["dilation"], packed_qkv=c["packed"],
               quilt_factor=c["quilt"], quilt_offset=c["quilt"] - 1)  # fmt: skip
    s = dict(c=c, geo=geo, Hq=Hq, q=_q(q), k=None if k is None else _q(k), v=None if v is None else _q(v), K=_q(K), V=_q(V), out=_q(out), frame_t=_q(ints[0:1]),
             frozen=_q(ints[1:2]), segments=_q(ints[2:8]), n_segments=_q(ints[8:9]), result=[out, K, V, ints])  # fmt: skip
    torch.cuda.synchronize()
    return s


def _run_attn(s):
    c, geo = s["c"], s["geo"]
    k, v = (s["q"], s["q"]) if c["packed"] else (s["k"], s["v"])
    qf.kv_cache_update(k, v, s["frame_t"], s["frozen"], s["V"], s["segments"], s["n_segments"], s["K"], n_q_heads=s["Hq"], **geo)
    qf.owl_attn(s["q"], s["K"], s["V"], s["segments"], s["n_segments"], gqa_ratio=c["gqa"], compute_dtype=c["dtype"], frame_t=s["frame_t"], out=s["out"], **geo)
    return s["result"]


def _prepare_gemm(c, seed):
    g = _gen(seed)
    M, N, K = c["M"], c["N"], c["K"]
    kw = dict(out_dtype=c["out"], compute_dtype=c["b"])
    if "silu" in c["epilogue"]:
        kw["activation"] = "silu"
    if "bias" in c["epilogue"]:
        kw["bias"] = _q(_randn(g, (N,)))
    if c["epilogue"] == "gate":
        kw.update(gate=_q(_randn(g, (c["groups"], N), std=0.2)), residual=_q(_randn(g, (M, N))), gate_groups=c["groups"])
    out = torch.zeros((M, N), device="cuda", dtype=TORCH[c["out"]])
    s = dict(c=c, A=_q(_randn(g, (M, K), c["a"])), B=_q(_randn(g, (N, K), c["b"], std=K**-0.5 if c["b"] == "bf16" else 0.05)), kw=dict(kw, out=_q(out)), out=out)
    torch.cuda.synchronize()
    return s


def _run_gemm(s):
    qf.gemm(s["A"], s["B"], **s["kw"])
    return s["out"]


def _prepare_moe(c, seed):
    g = _gen(seed)
    layer = nn.MoE(c["M"], c["D"], c["H"], c["experts"], c["top_k"])
    layer.router.weight.data = _q(_randn(g, (c["experts"], c["D"]), std=0.2))
    layer.expert_in.data = _q(_randn(g, (c["experts"] * c["H"], c["D"]), std=0.02))
    layer.expert_out.data = _q(_randn(g, (c["experts"] * c["D"], c["H"]), std=0.02))
    torch.cuda.synchronize()
    layer.prepare(fp8=c["fp8"])
    x = _q(_randn(g, (c["M"], c["D"])))
    torch.cuda.synchronize()
    y = layer(x)  # the layer's buffers
    qb.runtime.synchronize()
    return dict(c=c, layer=layer, x=x, out=_view(y))


class _Memory:
    def __init__(self, t):
        self.__cuda_array_interface__ = dict(shape=t.shape, typestr="<i2", data=(t.data_ptr(), False), version=3)
        self.keep = t


def _view(t):
    """The torch tensor over a bf16 tensor of the framework."""
    return torch.as_tensor(_Memory(t), device="cuda").view(torch.bfloat16)


def _run_moe(s):
    s["layer"](s["x"])
    return s["out"]  # the layer's own output buffer


def _prepare_glue(c, seed):
    g = _gen(seed)
    op, rows, D = c["op"], c["rows"], c["D"]
    x = _randn(g, (rows, D), "e4m3" if op == "dequantize" else "bf16")
    out = torch.zeros((rows, D), device="cuda", dtype=TORCH["e4m3" if op in ("quantize", "ada_rmsnorm_q") else "bf16"])
    X, O = _q(x), _q(out)
    if op in ("ada_rmsnorm", "ada_rmsnorm_q"):
        scale, bias = _q(_randn(g, (1, D), std=0.2)), _q(_randn(g, (1, D), std=0.2))
        call = (lambda: qf.ada_rmsnorm(X, scale, bias, out=O)) if op == "ada_rmsnorm" else (lambda: qf.ada_rmsnorm(X, scale, bias, out_q=O, only_q=True))
    elif op == "rmsnorm":
        call = lambda: qf.rmsnorm(X, out=O)  # noqa: E731
    elif op == "head_rmsnorm":
        heads = D // 64
        call = lambda: qf.head_rmsnorm(X, heads // 2, heads // 4, 64, out=O)  # noqa: E731
    elif op == "silu":
        call = lambda: qf.silu(X, out=O)  # noqa: E731
    elif op == "gate_residual":
        y, gate = _q(_randn(g, (rows, D))), _q(_randn(g, (1, D), std=0.2))
        call = lambda: qf.ada_gate_residual(X, y, gate, out=O)  # noqa: E731
    elif op == "add":
        y = _q(_randn(g, (rows, D)))
        call = lambda: qf.add(X, y, out=O)  # noqa: E731
    elif op == "euler":
        y, dsig = _q(_randn(g, (rows, D))), _q(torch.full((1,), -0.15, device="cuda"))
        call = lambda: qf.euler_step(X, y, dsig, out=O)  # noqa: E731
    elif op == "quantize":
        call = lambda: qf.quantize_e4m3(X, out=O)  # noqa: E731
    elif op == "dequantize":
        call = lambda: qf.dequantize_e4m3(X, out=O)  # noqa: E731
    else:
        raise ValueError(op)
    torch.cuda.synchronize()
    return dict(c=c, call=call, out=out)


def _run_glue(s):
    s["call"]()
    return s["out"]


_PREPARE = {"frame": _prepare_session, "append": _prepare_session, "attn": _prepare_attn, "gemm": _prepare_gemm, "moe": _prepare_moe, "glue": _prepare_glue}
_RUN = {"frame": _run_session, "append": _run_session, "attn": _run_attn, "gemm": _run_gemm, "moe": _run_moe, "glue": _run_glue}


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, int(seed))


def run(state):
    return _RUN[state["c"]["kind"]](state)


# ------------------------------------------------------------------------------------------------- what a pass cannot do without


def _session_work(c):
    cfg = _config(c)
    tpf, d, mlp, qkv = cfg.tpf, cfg.d_model, cfg.mlp_dim, cfg.qkv_dim
    lin, kv = (1 if c["linear"] == "fp8" else 2), (1 if c["kv"] == "fp8" else 2)
    keys = (16 + 1) * (tpf // c["quilt"])  # full windows and the frame itself
    layer_weights = qkv * d + d * d + 2 * d * mlp
    ctrl_weights = 3 * d * d if c["ctrl"] else 0
    patch = 2 * d * cfg.channels * 4
    flops = c["layers"] * (2 * tpf * layer_weights + 4 * cfg.n_heads * tpf * keys * 64) + 2 * tpf * patch
    read = c["layers"] * (layer_weights * lin + 2 * keys * cfg.n_kv_heads * 64 * kv) + patch * 2
    for layer in range(c["layers"]):
        if cfg.has_ctrl(layer):
            flops += 2 * tpf * 2 * d * d + 2 * d * d
            read += ctrl_weights * 2
    # the passes of a frame follow one another and a model's weights do not stay on the chip between them
    passes = 1 if c["kind"] == "append" else len(cfg.scheduler_sigmas)
    return dict(bytes=passes * read + 2 * 2 * cfg.latent_numel, flops=passes * flops)


def work(case):
    c = case
    if c["kind"] in ("frame", "append"):
        return _session_work(c)
    if c["kind"] == "attn":
        tpf, es = c["height"] * c["width"], BYTES[c["dtype"]]
        kept, Hk, Hq = tpf // c["quilt"], c["kv_heads"], c["kv_heads"] * c["gqa"]
        used = min((c["frame_t"] + c["dilation"] - 1) // c["dilation"], c["buckets"])
        keys = (used + 1) * kept
        return dict(bytes=2 * tpf * (Hq + 2 * Hk) * 64 + 2 * Hk * 64 * (keys + 2 * kept) * es + 2 * tpf * Hq * 64, flops=4 * Hq * tpf * keys * 64)
    if c["kind"] == "gemm":
        M, N, K = c["M"], c["N"], c["K"]
        extra = 2 * N if "bias" in c["epilogue"] else 2 * M * N + 2 * N if c["epilogue"] == "gate" else 0
        return dict(bytes=M * K * BYTES[c["a"]] + N * K * BYTES[c["b"]] + M * N * BYTES[c["out"]] + extra, flops=2 * M * N * K)
    if c["kind"] == "moe":
        used = min(c["experts"], c["M"] * c["top_k"])
        return dict(bytes=4 * c["M"] * c["D"] + 2 * c["experts"] * c["D"] + used * 2 * c["D"] * c["H"] * (1 if c["fp8"] else 2),
                    flops=4 * c["M"] * c["top_k"] * c["D"] * c["H"] + 2 * c["M"] * c["D"] * c["experts"])  # fmt: skip
    n = c["rows"] * c["D"]
    per = {"ada_rmsnorm": 4, "ada_rmsnorm_q": 3, "rmsnorm": 4, "head_rmsnorm": 4, "silu": 4, "gate_residual": 6, "add": 6, "euler": 6, "quantize": 3, "dequantize": 3}
    return dict(bytes=n * per[c["op"]], flops=4 * n)


def tolerance(case):
    c = case
    if c["kind"] in ("frame", "append"):
        # e4m3 keeps 3 mantissa bits, so a last-bit difference of a sum becomes a code's difference in the next layer's input;
        # five passes through the layers leave bf16 results about 1e-2 and e4m3 results a few 1e-2 apart
        return {"rel": 0.03 if "fp8" in (c["linear"], c["kv"], c["attn"]) else 0.01, "max": 0.5}
    if c["kind"] == "attn":
        return {"rel": 0.01 if c["dtype"] == "e4m3" else 0.005, "max": 0.2}  # probabilities rounded to e4m3 | bf16
    if c["kind"] == "gemm":
        if c["out"] == "e4m3":
            return {"rel": 0.02, "max": 0.2}  # a sum on the edge of two codes
        if c["out"] == "bf16":
            return {"rel": 0.004, "max": 0.02}
        return {"rel": 5e-4 if "silu" in c["epilogue"] else 2e-5}  # SiLU through the hardware's tanh (2^-11)
    if c["kind"] == "moe":
        return {"rel": 0.02 if c["fp8"] else 0.006, "max": 0.5}  # hidden activations rounded to e4m3 | bf16
    if c["op"] in ("quantize", "dequantize", "add"):
        return "exact"
    return {"rel": 0.02, "max": 0.2} if c["op"] == "ada_rmsnorm_q" else {"rel": 0.004, "max": 0.02}
