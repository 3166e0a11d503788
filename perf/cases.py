"""Performance cases of the quantized-linear path, each one call of a public entry point.

A case names its kind -- ``woq`` (int4 weight-only linear), ``dyn`` (per-token dynamic int8 linear), ``static``
(per-tensor static int8 linear) or ``moe`` (int4 mixture-of-experts FFN) -- and its sizes and options.  Inputs are
synthetic: activations N(0, 1), weights N(0, 0.02) quantised per group or per channel, biases N(0, 0.01), the
distributions of the benchmark.  ``exact`` evaluates the operator's definition in 64 bits; the 8-bit rounding of
activations is part of that definition (IEEE single-precision division, round half to even) and is done as such.
"""
import sys
from pathlib import Path

import torch

sys.path.insert(0, str(Path.cwd() / "zendnn-pytorch-plugin_b200"))   # the working folder is the repository's root

import zentorch_b200  # noqa: E402,F401  (registers torch.ops.zentorch)
from zentorch_b200 import _capi  # noqa: E402

_OPS = torch.ops.zentorch
_DTYPES = {"bf16": torch.bfloat16, "f32": torch.float32, "u8": torch.uint8, "s8": torch.int8}


def _woq(name, m, k, n, gs=128, asym=False, scales="f32", post="none"):
    return dict(name=name, kind="woq", m=m, k=k, n=n, gs=gs, asym=asym, scales=scales, post=post)


def listed():
    return [
        # one token through a square attention projection: the smallest call of a decode step, latency counts
        _woq("woq_decode_4096", 1, 4096, 4096),
        # one token through a wide up projection: a decode step bound by the weight stream
        _woq("woq_decode_wide", 1, 8192, 28672),
        # eight concurrent requests through a down projection, checkpoint with zero points and bf16 scales
        _woq("woq_decode_8rows", 8, 14336, 4096, asym=True, scales="bf16"),
        # a decode batch of 32 through an up projection
        _woq("woq_batch_32", 32, 4096, 14336),
        # a larger decode batch, zero points, gated and added to a residual
        _woq("woq_batch_128", 128, 8192, 8192, asym=True, scales="bf16", post="mul_add"),
        # a short prompt through a layer whose sizes fit no tile: odd rows and columns, small groups
        _woq("woq_ragged", 77, 2816, 5003, gs=64, post="gelu_tanh"),
        # prompt processing: 2048 tokens through an up projection
        _woq("woq_prefill_2048", 2048, 4096, 14336),
        # one token through a fused q/k/v projection in int8
        dict(name="dyn_decode", kind="dyn", m=1, k=8192, n=10240, x="bf16", act="s8_sym", post="none"),
        # the benchmark's dynamic linear: unsigned activations with zero points, fused SiLU
        dict(name="dyn_512_silu", kind="dyn", m=512, k=4096, n=11008, x="bf16", act="u8_asym", post="silu"),
        # prompt processing in int8: 4096 tokens through a wide up projection, the largest call
        dict(name="dyn_prefill_4096", kind="dyn", m=4096, k=8192, n=28672, x="bf16", act="s8_sym", post="none"),
        # an encoder layer's feed-forward input projection, calibrated int8, output requantised for the next layer
        dict(name="static_encoder", kind="static", m=384, k=1024, n=4096, x="f32", y="u8"),
        # a top-2 mixture-of-experts FFN over a batch of 256 tokens
        dict(name="moe_256", kind="moe", t=256, h=4096, i=14336, experts=8, top_k=2, gs=128),
    ]


def _log_int(rng, lo, hi, step=1):
    """A multiple of `step` in [lo, hi], uniform over the logarithm."""
    v = lo * (hi / lo) ** rng.random()
    return min(hi, max(lo, int(round(v / step)) * step))


def draw(rng):
    kind = rng.choice(["woq", "woq", "woq", "woq", "dyn", "dyn", "dyn", "static", "moe", "moe"])
    if kind == "woq":
        m, k = _log_int(rng, 1, 2048), _log_int(rng, 512, 14336, 64)
        n = _log_int(rng, 512, 28672, rng.choice([1, 8, 64, 128]))
        while m * n * k > 2048 * 4096 * 14336:
            m = max(1, m // 2)
        gs = rng.choice([g for g in (32, 64, 128, 128, 256, k) if k % g == 0])
        case = _woq("", m, k, n, gs, rng.random() < 0.4, rng.choice(["f32", "bf16"]),
                    rng.choice(["none", "none", "gelu_tanh", "mul_add", "add", "relu"]))
        del case["name"]
        return case
    if kind == "dyn":
        return dict(kind="dyn", m=_log_int(rng, 1, 4096), k=_log_int(rng, 512, 8192, 16),
                    n=_log_int(rng, 512, 28672, rng.choice([1, 8, 64])), x=rng.choice(["bf16", "bf16", "f32"]),
                    act=rng.choice(["s8_sym", "s8_sym", "u8_asym"]), post=rng.choice(["none", "none", "silu", "gelu_erf"]))
    if kind == "static":
        x = rng.choice(["f32", "bf16", "u8"])
        return dict(kind="static", m=_log_int(rng, 1, 2048), k=_log_int(rng, 256, 4096, 16),
                    n=_log_int(rng, 256, 8192, rng.choice([1, 16])), x=x, y=rng.choice(["f32", "bf16", "u8"]))
    gs = rng.choice([32, 64, 128])
    return dict(kind="moe", t=_log_int(rng, 8, 512), h=_log_int(rng, 512, 4096, 128), i=_log_int(rng, 512, 14336, 128),
                experts=rng.choice([4, 8]), top_k=rng.choice([1, 2, 2]), gs=gs)


# ---- inputs --------------------------------------------------------------------------------------------
def _rng(seed):
    return torch.Generator(device="cuda").manual_seed(seed * 7919 + 17)


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda")


def _int4_weight(g, n, k, gs, asym=False, scale_dtype=torch.float32):
    """q [n, k] int8, scales and zero points [k / gs, n]."""
    w = (_randn(g, n, k) * 0.02).view(n, k // gs, gs)
    if asym:
        lo, hi = w.amin(2), w.amax(2)
        s = ((hi - lo) / 15).clamp(min=1e-6)
        q = torch.round((w - lo.unsqueeze(2)) / s.unsqueeze(2)).clamp_(0, 15)
        zeros = (lo + 8 * s).t().contiguous().to(scale_dtype)
    else:
        s = (w.abs().amax(2) / 7).clamp(min=1e-8)
        q, zeros = torch.round(w / s.unsqueeze(2)).clamp_(-8, 7), None
    return q.to(torch.int8).view(n, k), s.t().contiguous().to(scale_dtype), zeros


def _int8_weight(g, n, k):
    w = _randn(g, n, k) * 0.02
    s = (w.abs().amax(1) / 127).clamp(min=1e-12)
    return torch.round(w / s.unsqueeze(1)).clamp_(-127, 127).to(torch.int8), s


def _inputs(c, seed):
    """The tensors of a case, weights still unpacked."""
    g = _rng(seed)
    d = {}
    if c["kind"] == "woq":
        d["x"] = _randn(g, c["m"], c["k"]).to(torch.bfloat16)
        d["q"], d["s"], d["z"] = _int4_weight(g, c["n"], c["k"], c["gs"], c["asym"], _DTYPES[c["scales"]])
        d["b"] = (_randn(g, c["n"]) * 0.01).to(torch.bfloat16)
        operands = {"add": 1, "mul_add": 2}.get(c["post"], 0)
        d["binary"] = [_randn(g, c["m"], c["n"]).to(torch.bfloat16) for _ in range(operands)]
    elif c["kind"] == "dyn":
        d["x"] = _randn(g, c["m"], c["k"]).to(_DTYPES[c["x"]])
        d["q"], d["s"] = _int8_weight(g, c["n"], c["k"])
        d["b"] = _randn(g, c["n"]) * 0.01
    elif c["kind"] == "static":
        x = _randn(g, c["m"], c["k"])
        d["xs"], d["xz"] = torch.tensor([0.035], device="cuda"), torch.tensor([121], dtype=torch.int32, device="cuda")
        d["x"] = torch.round(x / 0.035 + 121).clamp_(0, 255).to(torch.uint8) if c["x"] == "u8" else x.to(_DTYPES[c["x"]])
        d["q"], d["s"] = _int8_weight(g, c["n"], c["k"])
        d["b"] = _randn(g, c["n"]) * 0.01
        spread = 0.02 * c["k"] ** 0.5 * 6 / 255      # the calibrated range: three standard deviations to either side
        d["os"] = torch.tensor([spread], device="cuda") if c["y"] == "u8" else None
        d["oz"] = torch.tensor([128], dtype=torch.int32, device="cuda") if c["y"] == "u8" else None
    else:
        d["x"] = _randn(g, c["t"], c["h"]).to(torch.bfloat16)
        p, ids = torch.softmax(_randn(g, c["t"], c["experts"]), 1).topk(c["top_k"], 1)
        d["ids"], d["tw"] = ids.to(torch.int32).contiguous(), (p / p.sum(1, keepdim=True)).contiguous()
        d["w13"] = [_int4_weight(g, 2 * c["i"], c["h"], c["gs"])[:2] for _ in range(c["experts"])]
        d["w2"] = [_int4_weight(g, c["h"], c["i"], c["gs"])[:2] for _ in range(c["experts"])]
    return d


def prepare(case, seed):
    """Activations and the weights as a loaded model holds them (packed once at load)."""
    d = _inputs(case, seed)
    s = {"case": case}
    if case["kind"] == "woq":
        packed = _OPS.zentorch_woq_repack_weight(d["q"])
        s["args"] = [d["x"], packed.t(), d["s"], d["z"]]
        s["bias"], s["binary"] = d["b"], d["binary"]
    elif case["kind"] == "moe":
        s["args"] = [d["x"], d["tw"], d["ids"]]
        for name in ("w13", "w2"):
            s["args"].append(torch.stack([_OPS.zentorch_woq_repack_weight(q) for q, _ in d[name]]))
            s["args"].append(torch.stack([sc for _, sc in d[name]]))
    else:
        s.update(d)
    return s


def run(state):
    c = state["case"]
    if c["kind"] == "woq":
        a, b = state["args"], state["bias"]
        if c["post"] == "none":
            return _OPS.zentorch_woq_linear(*a, b)
        if c["post"] == "relu":
            return _OPS.zentorch_woq_linear_relu(*a, b)
        if c["post"] == "gelu_tanh":
            return _OPS.zentorch_woq_linear_gelu_tanh(*a, b)
        if c["post"] == "add":
            return _OPS.zentorch_woq_linear_add(*a, *state["binary"], b)
        return _OPS.zentorch_woq_linear_mul_add(*a, *state["binary"], b)
    if c["kind"] == "dyn":
        if c["act"] == "s8_sym" and c["post"] == "none":
            return _OPS.zentorch_dynamic_qlinear(state["x"], state["q"], state["s"], state["b"])
        return _OPS.zentorch_dynamic_qlinear_ext(state["x"], state["q"], state["s"], state["b"],
                                                 act_quant=c["act"], post_op=c["post"])
    if c["kind"] == "static":
        return _OPS.zentorch_qlinear(state["x"], state["q"], state["xs"], state["xz"], state["s"], None, state["b"],
                                     state["os"], state["oz"], _DTYPES[c["y"]])
    return _capi.moe_woq(*state["args"])


# ---- the work a pass cannot do without --------------------------------------------------------------------
_BYTES = {"bf16": 2, "f32": 4, "u8": 1, "s8": 1}


def work(case):
    c = case
    if c["kind"] == "moe":
        t, h, i, e = c["t"], c["h"], c["i"], min(c["experts"], c["t"] * c["top_k"])
        weights = 3 * h * i * e // 2 + 3 * h * i * e // c["gs"] * 4
        return {"bytes": weights + 2 * t * h * 2 + t * c["top_k"] * 8, "flops": 6 * t * c["top_k"] * h * i}
    m, k, n = c["m"], c["k"], c["n"]
    flops = 2 * m * k * n
    if c["kind"] == "woq":
        tables = k // c["gs"] * n * _BYTES[c["scales"]] * (2 if c["asym"] else 1)
        operands = {"add": 1, "mul_add": 2}.get(c["post"], 0)
        return {"bytes": n * k // 2 + tables + 2 * m * k + 2 * n + 2 * m * n * (1 + operands), "flops": flops}
    out = _BYTES[c["y"]] if c["kind"] == "static" else _BYTES[c["x"]]
    return {"bytes": n * k + m * k * _BYTES[c["x"]] + 8 * n + m * n * out, "flops": flops}


def tolerance(case):
    c = case
    if c["kind"] == "woq":
        # bf16 rounding of the result and, in the tensor-core form, of the dequantised weight: 1.7e-3 - 2.4e-3 of exact
        return {"rel": 8e-3, "max": 0.05}
    if c["kind"] == "moe":
        # two linears as above and a bf16 hidden activation between them
        return {"rel": 1.5e-2, "max": 0.1}
    out = c["y"] if c["kind"] == "static" else c["x"]
    if out == "u8":
        return {"rel": 0.0, "differ": 1e-3}      # ties of the requantisation
    # integer sums are exact: a float result carries the epilogue's rounding, a bf16 one that of its own type
    return {"rel": 1e-5, "max": 1e-4} if out == "f32" else {"rel": 6e-3, "max": 0.03}


# ---- 64-bit evaluation -----------------------------------------------------------------------------------
def _dequant(q, s, z=None):
    n, k = q.shape
    groups = s.shape[0]
    w = q.double().view(n, groups, k // groups)
    if z is not None:
        w = (w - 8) * s.double().t().unsqueeze(2) + z.double().t().unsqueeze(2)
    else:
        w = w * s.double().t().unsqueeze(2)
    return w.view(n, k)


def _post64(y, name):
    if name == "relu":
        return y.clamp(min=0)
    if name == "silu":
        return torch.nn.functional.silu(y)
    if name.startswith("gelu"):
        return torch.nn.functional.gelu(y, approximate="tanh" if name == "gelu_tanh" else "none")
    return y


def exact(case, seed):
    c, d = case, _inputs(case, seed)
    if c["kind"] == "woq":
        y = d["x"].double() @ _dequant(d["q"], d["s"], d["z"]).t() + d["b"].double()
        if c["post"] == "add":
            return y + d["binary"][0].double()
        return y * d["binary"][0].double() + d["binary"][1].double() if c["post"] == "mul_add" else _post64(y, c["post"])
    if c["kind"] == "dyn":
        x = d["x"].float()
        if c["act"] == "u8_asym":
            lo, hi = x.amin(1, keepdim=True).clamp(max=0), x.amax(1, keepdim=True).clamp(min=0)
            s = (hi - lo).clamp(min=1e-12) / 255
            z = torch.round(-lo / s).clamp(0, 255)
            qx = (torch.round(x / s) + z).clamp(0, 255).double() - z.double()
        else:
            s = x.abs().amax(1, keepdim=True).clamp(min=1e-12) / 127
            qx = torch.round(x / s).clamp(-128, 127).double()
        y = (qx @ d["q"].double().t()) * s.double() * d["s"].double() + d["b"].double()
        return _post64(y, c["post"])
    if c["kind"] == "static":
        if c["x"] == "u8":
            qx = d["x"].double()
        else:
            qx = (torch.round(d["x"].float() * (1.0 / d["xs"])) + d["xz"]).clamp(0, 255).double()
        y = ((qx - d["xz"].double()) @ d["q"].double().t()) * d["xs"].double() * d["s"].double() + d["b"].double()
        if c["y"] == "u8":
            return (torch.round(y / d["os"].double()) + d["oz"]).clamp(0, 255).to(torch.uint8)
        return y
    x, y = d["x"].double(), torch.zeros(c["t"], c["h"], dtype=torch.float64, device="cuda")
    for e in range(c["experts"]):
        rows, slot = (d["ids"] == e).nonzero(as_tuple=True)
        if rows.numel():
            hidden = x[rows] @ _dequant(*d["w13"][e]).t()
            act = torch.nn.functional.silu(hidden[:, :c["i"]]) * hidden[:, c["i"]:]
            y.index_add_(0, rows, (act @ _dequant(*d["w2"][e]).t()) * d["tw"][rows, slot].double().unsqueeze(1))
    return y
