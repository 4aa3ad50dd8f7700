"""The calls this library is timed by: inputs, the call, its minimum work and the result in 64 bits.

Every case is one pass through the public entry points (``kudnn_b200.Linear``, ``kudnn_b200.rmsnorm`` and the
``kudnn_b200.torch_ops.Linear`` module) on inputs that are already on the GPU, with the weights pre-packed as a serving
program keeps them.  Kinds:

  linear   one Linear primitive: c = act(a . b + bias), out = c (+) res
  int8     the 8-bit integer product with 32-bit results
  block    RMS normalisation, up-projection with SiLU, down-projection with the residual added (a transformer's
           feed-forward block), the two projections through the torch module
"""
import math

import torch

import kudnn_b200 as kb
from kudnn_b200 import torch_ops

_CODE = {"f32": kb.F32, "f16": kb.F16, "bf16": kb.BF16, "s8": kb.S8}
_TORCH = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16, "s8": torch.int8}
_SIZE = {"f32": 4, "f16": 2, "bf16": 2, "s8": 1}
_ACT = {"none": kb.ACT_NONE, "relu": kb.ACT_RELU, "silu": kb.ACT_SWISH, "gelu_tanh": kb.ACT_GELU_TANH, "gelu_erf": kb.ACT_GELU_ERF}
_RES = {"none": kb.RES_NONE, "add": kb.RES_IDENTICAL, "mul": kb.RES_ELTWISE_MUL}
_EPS = 1e-6


def _linear(m, n, k, a, b=None, act="none", bias=True, res="none", wlayout="BA"):
    """wlayout BA: weights [n, k], k contiguous (torch.nn.Linear's); AB: [k, n], n contiguous."""
    return {"kind": "linear", "m": m, "n": n, "k": k, "a": a, "b": b or a, "act": act, "bias": bias, "res": res,
            "wlayout": wlayout}


def _block(m, hidden, ffn, a):
    return {"kind": "block", "m": m, "hidden": hidden, "ffn": ffn, "a": a}


def listed():
    def named(name, case):
        return dict(case, name=name)

    return [
        # a small fp32 layer as the reference's unit tests call it: one call is launches and latency
        named("fp32_small", _linear(128, 1024, 1024, "f32", act="relu")),
        # the fp32 sizes of the reference's matrix-product benchmark (4096 rows, 1152 to 5120 columns)
        named("fp32_large", _linear(4096, 4608, 2304, "f32", act="relu")),
        # prompt processing: the up-projection of a feed-forward block
        named("prefill_silu", _linear(4096, 11008, 4096, "bf16", act="silu")),
        # prompt processing: GELU and a residual in one call
        named("prefill_gelu_res", _linear(8192, 4096, 4096, "f16", act="gelu_tanh", res="add")),
        # one token of one sequence, the product gated element by element
        named("decode_1", _linear(1, 28672, 8192, "bf16", bias=False, res="mul")),
        # one token of sixteen sequences
        named("decode_16", _linear(16, 28672, 8192, "bf16", bias=False, res="mul")),
        # 8-bit weights with fp16 activations, four sequences
        named("decode_w8_4", _linear(4, 28672, 8192, "f16", b="s8", act="none")),
        # a server's batch of one token each, too many rows for a decode kernel and too few for a prompt
        named("batch_64", _linear(64, 11008, 4096, "bf16", act="silu")),
        # nothing a multiple of anything, weights stored [k, n] with n contiguous
        named("ragged", _linear(333, 3001, 2050, "bf16", act="gelu_erf", wlayout="AB")),
        # the 8-bit integer product at the up-projection's size
        named("int8", {"kind": "int8", "m": 4096, "n": 11008, "k": 4096, "bias": False}),
        # the largest layer: all rows of a long batch of prompts on one GPU
        named("prefill_large", _linear(32768, 28672, 8192, "bf16", act="silu")),
        # a feed-forward block on a prompt of odd length through the torch module
        named("block", _block(1027, 4096, 11008, "f16")),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi, step):
    """Spread over the logarithm of [lo, hi]; three of four are a multiple of `step`, the rest only of 8."""
    step = step if rng.random() < 0.75 else 8
    return max(step, _log(rng, lo, hi) // step * step)


def draw(rng):
    kind = rng.choice(["fp32_small", "fp32_large", "prefill", "gelu_res", "decode", "w8", "batch", "ragged", "int8", "large", "block"])
    act = rng.choice(["none", "relu", "silu", "gelu_tanh"])
    half = rng.choice(["bf16", "f16"])
    if kind == "fp32_small":
        return _linear(_log(rng, 17, 256), _log(rng, 64, 2048), _log(rng, 20, 2048), "f32", act=act, wlayout=rng.choice(["BA", "AB"]))
    if kind == "fp32_large":
        return _linear(_log(rng, 512, 8192), _size(rng, 1152, 5120, 128), _size(rng, 1152, 5120, 128), "f32", act=act)
    if kind == "prefill":
        return _linear(_log(rng, 256, 8192), _size(rng, 1024, 16384, 256), _size(rng, 1024, 8192, 128), half, act=act, bias=rng.random() < 0.7)
    if kind == "gelu_res":
        return _linear(_log(rng, 256, 8192), _size(rng, 1024, 8192, 256), _size(rng, 1024, 8192, 128), half, act="gelu_tanh",
                       res=rng.choice(["add", "mul"]))
    if kind == "decode":
        return _linear(rng.randint(1, 16), _size(rng, 1024, 28672, 256), _size(rng, 1024, 8192, 256), half, act=act,
                       bias=rng.random() < 0.5, res=rng.choice(["none", "add", "mul"]))
    if kind == "w8":
        return _linear(rng.randint(1, 16), _size(rng, 1024, 28672, 256), _log(rng, 1024, 8192) // 16 * 16, "f16", b="s8", act=act,
                       bias=rng.random() < 0.5)
    if kind == "batch":
        return _linear(_log(rng, 17, 255), _size(rng, 1024, 28672, 256), _size(rng, 1024, 8192, 256), half, act=act)
    if kind == "ragged":
        return _linear(_log(rng, 17, 2048), _log(rng, 500, 8000), _log(rng, 500, 4100), half,
                       act=rng.choice(["none", "relu", "gelu_tanh", "gelu_erf"]), res=rng.choice(["none", "add"]),
                       wlayout=rng.choice(["BA", "AB"]))
    if kind == "int8":
        return {"kind": "int8", "m": _log(rng, 128, 8192), "n": _size(rng, 1024, 11008, 128), "k": _size(rng, 1024, 8192, 128),
                "bias": rng.random() < 0.5}
    if kind == "large":
        return _linear(_log(rng, 8192, 32768), _size(rng, 8192, 28672, 256), _size(rng, 4096, 8192, 256), half, act=act)
    return _block(_log(rng, 17, 4096), _size(rng, 1024, 5120, 256), _size(rng, 2816, 13824, 256), half)


# ---- inputs


def _normal(gen, shape, dtype, std=1.0):
    t = torch.empty(shape, dtype=dtype, device="cuda")
    # by rows, so that no input needs a second copy of itself in fp32
    flat = t.view(shape[0], -1) if t.dim() > 1 else t.view(1, -1)
    step = max(1, (1 << 26) // flat.shape[1])
    for r in range(0, flat.shape[0], step):
        part = flat[r:r + step]
        part.copy_(torch.randn(part.shape, generator=gen, device="cuda", dtype=torch.float32).mul_(std))
    return t


def _inputs(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    if case["kind"] == "block":
        dt, m, h, f = _TORCH[case["a"]], case["m"], case["hidden"], case["ffn"]
        return {"x": _normal(gen, (m, h), dt), "g": (1.0 + 0.1 * torch.randn(h, generator=gen, device="cuda")).to(dt),
                "w1": _normal(gen, (f, h), dt, 0.02), "b1": _normal(gen, (f,), dt, 0.02),
                "w2": _normal(gen, (h, f), dt, 0.02), "b2": _normal(gen, (h,), dt, 0.02)}
    m, n, k = case["m"], case["n"], case["k"]
    if case["kind"] == "int8":
        got = {"a": torch.randint(-128, 128, (m, k), generator=gen, device="cuda", dtype=torch.int8),
               "b": torch.randint(-128, 128, (n, k), generator=gen, device="cuda", dtype=torch.int8), "bias": None}
        if case["bias"]:
            got["bias"] = torch.randint(-100000, 100000, (n,), generator=gen, device="cuda", dtype=torch.int32)
        return got
    dt = _TORCH[case["a"]]
    wshape = (n, k) if case["wlayout"] == "BA" else (k, n)
    got = {"a": _normal(gen, (m, k), dt), "bias": None, "res": None}
    if case["b"] == "s8":
        got["b"] = torch.randint(-127, 128, wshape, generator=gen, device="cuda", dtype=torch.int8)
    else:
        got["b"] = _normal(gen, wshape, dt, 0.02)
    if case["bias"]:
        got["bias"] = _normal(gen, (n,), dt, 0.02)
    if case["res"] != "none":
        got["res"] = _normal(gen, (m, n), dt)
    return got


def prepare(case, seed):
    s = _inputs(case, seed)
    s["case"] = case
    if case["kind"] == "block":
        dt, h, f = _TORCH[case["a"]], case["hidden"], case["ffn"]
        up = torch.nn.Linear(h, f, device="meta", dtype=dt)
        down = torch.nn.Linear(f, h, device="meta", dtype=dt)
        for layer, w, b in ((up, s["w1"], s["b1"]), (down, s["w2"], s["b2"])):
            layer.weight = torch.nn.Parameter(w, requires_grad=False)
            layer.bias = torch.nn.Parameter(b, requires_grad=False)
        s["up"] = torch_ops.Linear.from_torch(up, act="silu")
        s["down"] = torch_ops.Linear.from_torch(down, residual="add")
        s["h"] = torch.empty_like(s["x"])
        return s
    m, n, k = case["m"], case["n"], case["k"]
    stream = torch.cuda.current_stream().cuda_stream
    if case["kind"] == "int8":
        desc = kb.make_desc(m, n, k, kb.S8, c_dtype=kb.S32, has_bias=case["bias"], bias_dtype=kb.S32)
        s["y"] = torch.empty((m, n), dtype=torch.int32, device="cuda")
    else:
        desc = kb.make_desc(m, n, k, _CODE[case["a"]], b_dtype=_CODE[case["b"]], b_strides=(1, k) if case["wlayout"] == "BA" else (n, 1),
                            has_bias=case["bias"], act=_ACT[case["act"]], act_alpha=0.0 if case["act"] == "relu" else 1.0,
                            res_op=_RES[case["res"]])
        s["y"] = torch.empty((m, n), dtype=_TORCH[case["a"]], device="cuda")
    s["lin"] = kb.Linear(desc)
    s["lin"].prepack(s["b"], stream=stream)
    return s


def run(state):
    s, case = state, state["case"]
    stream = torch.cuda.current_stream().cuda_stream
    if case["kind"] == "block":
        x = s["x"]
        with torch.no_grad():
            kb.rmsnorm(x, s["h"], x.shape[0], x.shape[1], _CODE[case["a"]], scale=s["g"], flags=kb.NORM_USE_SCALE, eps=_EPS, stream=stream)
            return s["down"](s["up"](s["h"]), x)
    if case["kind"] == "int8" or case["res"] == "none":
        s["lin"].run(s["a"], s["b"], s["y"], s["bias"], stream=stream)
    else:
        s["lin"].run(s["a"], s["b"], None, s["bias"], s["res"], s["y"], stream=stream)
    return s["y"]


# ---- what a pass cannot do without, and what it computes


def work(case):
    if case["kind"] == "block":
        m, h, f, e = case["m"], case["hidden"], case["ffn"], _SIZE[case["a"]]
        return {"bytes": e * (2 * m * h + 2 * h * f + 2 * h + f), "flops": 4 * m * h * f}
    m, n, k = case["m"], case["n"], case["k"]
    if case["kind"] == "int8":
        return {"bytes": m * k + n * k + 4 * m * n + (4 * n if case["bias"] else 0), "flops": 2 * m * n * k}
    e = _SIZE[case["a"]]
    outs = 1 + (1 if case["res"] != "none" else 0)
    return {"bytes": e * (m * k + outs * m * n + (n if case["bias"] else 0)) + _SIZE[case["b"]] * n * k, "flops": 2 * m * n * k}


def tolerance(case):
    if case["kind"] == "int8":
        return "exact"
    # about four times the distance of one run from the 64-bit result
    if case["a"] == "f32":
        return {"rel": 1e-5, "max": 1e-4}
    if case["a"] == "bf16":
        return {"rel": 1.2e-2, "max": 8e-2}
    return {"rel": 3e-3, "max": 3e-2}


def _act64(v, act):
    if act == "relu":
        return v.relu_()
    if act == "silu":
        return v.mul_(torch.sigmoid(v))
    if act == "gelu_tanh":
        return torch.nn.functional.gelu(v, approximate="tanh")
    if act == "gelu_erf":
        return torch.nn.functional.gelu(v)
    return v


def exact(case, seed):
    s = _inputs(case, seed)
    if case["kind"] == "int8":
        y = torch.empty((case["m"], case["n"]), dtype=torch.int32, device="cuda")
        bt = s["b"].double().t()
        for r in range(0, case["m"], 4096):
            part = s["a"][r:r + 4096].double() @ bt  # whole numbers far below 2^53
            y[r:r + 4096] = (part if s["bias"] is None else part + s["bias"]).to(torch.int32)
        return y
    if case["kind"] == "block":
        x = s["x"].double()
        h = x * torch.rsqrt(x.square().mean(dim=1, keepdim=True) + _EPS) * s["g"].double()
        u = _act64(h @ s["w1"].double().t() + s["b1"].double(), "silu")
        return x + u @ s["w2"].double().t() + s["b2"].double()
    b = s["b"].double()
    b = b.t() if case["wlayout"] == "BA" else b
    y = torch.empty((case["m"], case["n"]), dtype=torch.float64, device="cuda")
    for r in range(0, case["m"], 8192):
        part = s["a"][r:r + 8192].double() @ b
        if s["bias"] is not None:
            part += s["bias"].double()
        part = _act64(part, case["act"])
        if case["res"] == "add":
            part += s["res"][r:r + 8192]
        elif case["res"] == "mul":
            part *= s["res"][r:r + 8192]
        y[r:r + 8192] = part
    return y
