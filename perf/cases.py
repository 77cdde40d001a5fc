"""The workloads this library's speed is judged by: what each stands for in use, how its inputs are
made, one pass through the public entry points, the work the pass cannot do without, and how close
two correct implementations come.

A case is a dict of plain values; ``op`` names the entry point:

    linear   ops.gemm_i8 over [M, K] x [N, K]: s8/u8 activations, s8 weights, every destination
    matmul   ops.gemm_i8 over a batch of matrices in MatMul's operand poses
    q4_1     ops.linear_q4_1: f16/f32 activations against llama.cpp Q4_1 blocks
    qdq      ops.quantize_linear followed by ops.dequantize_linear
    fp_act   ops.linear_fp_act: floating activations quantised on the way into the s8 product
    conv     ops.conv2d_i8, one layer or a chain of two, with the filters packed once

Sizes come from the benchmark's configurations and the tests' shape tables, or are generic.
"""
from __future__ import annotations

import math

import torch

from nnops_b200 import ops

_BYTES = {"s32": 4, "s8": 1, "u8": 1, "f32": 4, "f16": 2}
_DTYPE = {"f32": torch.float32, "f16": torch.float16}
# The largest listed product (4096 x 28672 x 8192 multiply-adds) and weight; draws stay within both.
_MOST_MACS = 4096 * 28672 * 8192
_MOST_WEIGHTS = 28672 * 8192


def _linear(name, m, n, k, out, **kw):
    case = {"name": name, "op": "linear", "m": m, "n": n, "k": k, "out": out, "a": "s8", "zp_a": "none", "zp_w": False,
            "act": "none", "packed": False}
    case.update(kw)
    return case


def listed():
    return [
        # One token through an attention projection: the smallest call, a latency.
        _linear("i8_decode_1row", 1, 4096, 4096, "f16"),
        # A serving batch of single tokens through an MLP up-projection: the weights are streamed once.
        _linear("i8_decode_24rows", 24, 11008, 4096, "s8", act="relu"),
        # A prompt chunk through the same layer, requantised for the next one.
        _linear("i8_prefill_512rows", 512, 11008, 4096, "s8", act="relu"),
        # The headline layer, a long prompt: the largest call.
        _linear("i8_prefill_4096rows", 4096, 28672, 8192, "s8", act="relu"),
        # Dynamically quantised activations (a scale and a zero point per token) over sizes that
        # no tile divides: an encoder's classifier or a feature projection.
        _linear("i8_ragged_asymmetric", 333, 1000, 1500, "f32", a="u8", zp_a="token", act="gelu"),
        # Attention scores times values, one product per head, the second operand stored [K, N].
        {"name": "i8_matmul_32heads", "op": "matmul", "batch": 32, "m": 512, "n": 128, "k": 512, "out": "f32", "pose": "nn",
         "shared_w": False},
        # One token against 4-bit weights.
        {"name": "q4_1_decode_1row", "op": "q4_1", "m": 1, "n": 4096, "k": 4096, "a": "f16", "out": "f32", "packed": False,
         "act": "none"},
        # A serving batch against 4-bit weights.
        {"name": "q4_1_decode_16rows", "op": "q4_1", "m": 16, "n": 14336, "k": 4096, "a": "f16", "out": "f16", "packed": False,
         "act": "none"},
        # A prompt against 4-bit weights.
        {"name": "q4_1_prefill_2048rows", "op": "q4_1", "m": 2048, "n": 14336, "k": 4096, "a": "f16", "out": "f16",
         "packed": False, "act": "none"},
        # The elementwise steps around an int8 layer: encode per token, decode.
        {"name": "qdq_per_token", "op": "qdq", "rows": 4096, "cols": 8192, "x": "f16", "q": "s8", "axis": -1},
        # A quantised layer inside a floating-point model, per-token scales.
        {"name": "fp_act_64rows", "op": "fp_act", "m": 64, "n": 4096, "k": 4096, "x": "f16", "per_token": True},
        # Two layers of a convolutional body at batch 32: a 3x3 and the 1x1 that widens its result.
        {"name": "conv_3x3_then_1x1", "op": "conv", "batch": 32, "h": 56, "w": 56, "ic": 256, "oc": 256, "ks": 3, "stride": 1,
         "dil": 1, "pad": 1, "groups": 1, "a": "u8", "out": "s8", "zp_w": False, "oc2": 1024},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi, step, ragged=0.25):
    """Log-uniform in [lo, hi]; a multiple of ``step`` except for the ``ragged`` share."""
    v = _log_uniform(rng, lo, hi)
    if rng.random() >= ragged:
        v = max(step, v // step * step)
    return min(max(v, lo), hi)


def draw(rng):
    op = rng.choice(["linear"] * 4 + ["q4_1"] * 3 + ["matmul", "qdq", "fp_act", "conv", "conv"])
    if op in ("linear", "q4_1", "fp_act"):
        k = _size(rng, 64, 16384, 64)
        n = _size(rng, 64, min(28672, _MOST_WEIGHTS // k), 64)
        m = _size(rng, 1, max(1, min(4096, _MOST_MACS // (n * k))), 1)
        if op == "linear":
            out = rng.choice(["s8", "s8", "f16", "f16", "u8", "s32", "f32"])
            act = rng.choice(["none", "relu"] if out in ("s8", "u8", "s32") else ["none", "relu", "gelu", "silu"])
            return {"op": op, "m": m, "n": n, "k": k, "out": out, "a": rng.choice(["s8", "s8", "u8"]),
                    "zp_a": rng.choice(["none", "none", "tensor", "token"]), "zp_w": rng.random() < 0.2, "act": act,
                    "packed": rng.random() < 0.3}
        if op == "q4_1":
            a = rng.choice(["f16", "f16", "f16", "f32"])
            k = max(32, k // 32 * 32)
            # The packed planes serve one row and prompts, over whole groups of four blocks.
            packed = rng.random() < 0.3 and k % 128 == 0 and (m == 1 or m >= 256)
            return {"op": op, "m": m, "n": n, "k": k, "a": a, "out": a if rng.random() < 0.7 else "f32", "packed": packed,
                    "act": rng.choice(["none", "silu"])}
        return {"op": op, "m": m, "n": n, "k": k, "x": rng.choice(["f16", "f32"]), "per_token": rng.random() < 0.7}
    if op == "matmul":
        m, n, k = (_size(rng, 16, 1024, 16) for _ in range(3))
        batch = _log_uniform(rng, 2, 128)
        return {"op": op, "batch": batch, "m": m, "n": n, "k": k, "out": rng.choice(["s32", "s8", "f32", "f16"]),
                "pose": rng.choice(["nt", "nn", "tn", "tt"]), "shared_w": rng.random() < 0.2}
    if op == "qdq":
        return {"op": op, "rows": _size(rng, 1, 8192, 1), "cols": _size(rng, 64, 16384, 64), "x": rng.choice(["f32", "f16"]),
                "q": rng.choice(["s8", "u8"]), "axis": rng.choice([-1, -1, 0, 1, 2])}
    groups = rng.choice([1, 1, 1, 1, 2, 4])
    ks = rng.choice([1, 3, 3, 3, 5, 7])
    ic = rng.choice([3, 16, 32, 64, 128, 128, 256, 256, 512]) if groups == 1 else 32 * groups * rng.choice([1, 2, 4])
    hw = _log_uniform(rng, 7, 112)
    oc = groups * _size(rng, 16, 1024 // groups, 16, ragged=0.15)
    stride = rng.choice([1, 1, 2])
    batch = _log_uniform(rng, 1, 32)
    # Keep the layer, and its column matrix, within what the listed ones cost.
    while batch > 1 and (hw * hw * batch * ic * ks * ks > 600_000_000 or hw * hw * batch * ic // groups * ks * ks * oc > _MOST_MACS // 8):
        batch //= 2
    return {"op": op, "batch": batch, "h": hw, "w": max(7, hw + rng.choice([0, 0, -1, 3])), "ic": ic, "oc": oc, "ks": ks,
            "stride": stride, "dil": 1, "pad": rng.choice([0, ks // 2, ks // 2]), "groups": groups, "a": rng.choice(["u8", "u8", "s8"]),
            "out": rng.choice(["s8", "s8", "u8", "f16"]), "zp_w": rng.random() < 0.15, "oc2": 0}


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _ints(g, shape, lo, hi, dtype):
    return torch.randint(lo, hi, shape, generator=g, device="cuda", dtype=dtype)


def _s8(g, *shape):
    """Symmetric 8-bit values, uniform in [-127, 127], as in the benchmark's configurations."""
    return _ints(g, shape, -127, 128, torch.int8)


def _act8(g, kind, *shape):
    return _s8(g, *shape) if kind == "s8" else _ints(g, shape, 0, 256, torch.uint8)


def _scales(g, n, lo=0.001, hi=0.02):
    return torch.rand(n, generator=g, device="cuda") * (hi - lo) + lo


def _normal(g, dtype, *shape):
    return torch.randn(shape, generator=g, device="cuda", dtype=dtype)


def _bias(g, n, out):
    if out in ("s32", "s8", "u8"):
        return _ints(g, (n,), -1000, 1001, torch.int32)
    return (torch.rand(n, generator=g, device="cuda") - 0.5).to(_DTYPE[out])


def _q4_1_blocks(g, n, k):
    """Rows of Q4_1 blocks: f16 scale d in [0.005, 0.02], f16 minimum about -8 d, 16 bytes of nibbles."""
    blocks = k // 32
    d = (torch.rand((n, blocks, 1), generator=g, device="cuda") * 0.015 + 0.005).half()
    low = (-8.0 * d.float() * (torch.rand((n, blocks, 1), generator=g, device="cuda") * 0.4 + 0.8)).half()
    nibbles = _ints(g, (n, blocks, 16), 0, 256, torch.uint8)
    return torch.cat([d.view(torch.uint8), low.view(torch.uint8), nibbles], dim=2).reshape(n, blocks * 20)


def _out_scale(k):
    """A destination scale that keeps most results of a K-long sum of uniform products in range."""
    return math.sqrt(k) * 73.0 * 73.0 * 0.02 * 0.0105 / 45.0


def _prepare_linear(c, g):
    m, n, k, out = c["m"], c["n"], c["k"], c["out"]
    w = _s8(g, n, k)
    scale_w = _scales(g, n)
    kw = {"out_kind": out, "bias": _bias(g, n, out), "scale_a": 0.02}
    if out in ("s8", "u8", "s32"):
        kw.update(relu=c["act"] == "relu", out_scale=_out_scale(k), out_zp=100 if out == "u8" else 0)
    else:
        kw["activation"] = c["act"]
    if c["zp_a"] == "tensor":
        kw["zp_a"] = 128 if c["a"] == "u8" else 3
    elif c["zp_a"] == "token":
        kw["scale_a"] = _scales(g, m, 0.01, 0.03)
        kw["zp_a"] = _ints(g, (m,), 118, 139, torch.int32) if c["a"] == "u8" else _ints(g, (m,), -10, 11, torch.int32)
    zp_w = _ints(g, (n,), -3, 4, torch.int32) if c["zp_w"] else 0
    state = {"a": _act8(g, c["a"], m, k), "kw": kw}
    if c["packed"]:
        state["packed"] = ops.prepack_i8(w, scale_w=scale_w, zp_w=zp_w)
    else:
        state["w"] = w
        kw.update(scale_w=scale_w, zp_w=zp_w)
    return state


def _prepare_matmul(c, g):
    b, m, n, k, pose = c["batch"], c["m"], c["n"], c["k"], c["pose"]
    a = _s8(g, b, k, m).transpose(1, 2) if pose[0] == "t" else _s8(g, b, m, k)
    shape = (n, k) if pose[1] == "t" else (k, n)
    w = _s8(g, *shape) if c["shared_w"] else _s8(g, b, *shape)
    if pose[1] == "n":
        w = w.transpose(-1, -2)
    return {"a": a, "w": w, "kw": {"out_kind": c["out"], "scale_a": 0.02, "scale_w": 0.0105, "out_scale": _out_scale(k)}}


def _prepare_conv(c, g):
    def layer(ic, oc, ks, stride, dil, pad, groups, a):
        w = _s8(g, ks, ks, ic // groups, oc)
        out = c["out"]
        kw = {"stride": (stride, stride), "dilation": (dil, dil), "padding": (pad, pad), "groups": groups, "out_kind": out,
              "bias": _bias(g, oc, out), "scale_x": 0.02, "zp_x": 128 if a == "u8" else 0, "scale_w": _scales(g, oc),
              "zp_w": _ints(g, (oc,), -3, 4, torch.int32) if c["zp_w"] else 0,
              "out_scale": _out_scale(ks * ks * ic // groups), "out_zp": 100 if out == "u8" else 0}
        if out in ("s8", "u8"):
            kw["relu"] = True
        else:
            kw["activation"] = "relu"
        return ops.prepack_conv2d_i8(w, groups), kw

    layers = [layer(c["ic"], c["oc"], c["ks"], c["stride"], c["dil"], c["pad"], c["groups"], c["a"])]
    if c["oc2"]:
        layers.append(layer(c["oc"], c["oc2"], 1, 1, 1, 0, 1, c["out"]))
    return {"x": _act8(g, c["a"], c["batch"], c["h"], c["w"], c["ic"]), "layers": layers}


def prepare(case, seed):
    g = _gen(seed)
    op = case["op"]
    if op == "linear":
        state = _prepare_linear(case, g)
    elif op == "matmul":
        state = _prepare_matmul(case, g)
    elif op == "conv":
        state = _prepare_conv(case, g)
    elif op == "q4_1":
        w = _q4_1_blocks(g, case["n"], case["k"])
        if case["packed"]:
            w = ops.prepack_q4_1(w, case["k"])
        state = {"a": _normal(g, _DTYPE[case["a"]], case["m"], case["k"]), "w": w}
    elif op == "qdq":
        rows, cols, axis, unsigned = case["rows"], case["cols"], case["axis"], case["q"] == "u8"
        # axis -1: one parameter per row (token); 0 / 1: per index of that axis; 2: one for the tensor.
        count = {-1: rows, 0: rows, 1: cols, 2: 1}[axis]
        dtype = torch.uint8 if unsigned else torch.int8
        state = {"x": _normal(g, _DTYPE[case["x"]], rows, cols), "scale": _scales(g, count, 0.02, 0.04),
                 "zp": _ints(g, (count,), 118 if unsigned else -10, 139 if unsigned else 11, dtype), "dtype": dtype}
    else:
        m, n, k = case["m"], case["n"], case["k"]
        x = _normal(g, _DTYPE[case["x"]], m, k)
        scale = x.float().abs().amax(dim=1) / 127.0 if case["per_token"] else float(4.0 / 127.0)
        state = {"a": x, "w": _s8(g, n, k), "scale_a": scale, "scale_w": _scales(g, n), "bias": _bias(g, n, case["x"])}
    state["case"] = case
    return state


def run(state):
    c = state["case"]
    op = c["op"]
    if op == "linear":
        if c["packed"]:
            return ops.gemm_i8_packed(state["a"], state["packed"], **state["kw"])
        return ops.gemm_i8(state["a"], state["w"], **state["kw"])
    if op == "matmul":
        return ops.gemm_i8(state["a"], state["w"], **state["kw"])
    if op == "q4_1":
        return ops.linear_q4_1(state["a"], state["w"], c["k"], out_dtype=_DTYPE[c["out"]], activation=c["act"])
    if op == "qdq":
        axis = c["axis"] if c["axis"] < 2 else -1
        q = ops.quantize_linear(state["x"], state["scale"], state["zp"], axis=axis, out_dtype=state["dtype"])
        return q, ops.dequantize_linear(q, state["scale"], state["zp"], axis=axis, out_dtype=_DTYPE[c["x"]])
    if op == "fp_act":
        return ops.linear_fp_act(state["a"], state["w"], scale_a=state["scale_a"], scale_w=state["scale_w"], bias=state["bias"])
    x, made = state["x"], []
    for packed, kw in state["layers"]:
        x = ops.conv2d_i8(x, packed, **kw)
        made.append(x)
    return made


def work(case):
    """Bytes: every input read once, every output written once.  Flops: two per multiply-add."""
    c, op = case, case["op"]
    if op == "linear":
        m, n, k = c["m"], c["n"], c["k"]
        return {"bytes": m * k + n * k + 8 * n + m * n * _BYTES[c["out"]], "flops": 2 * m * n * k}
    if op == "matmul":
        b, m, n, k = c["batch"], c["m"], c["n"], c["k"]
        return {"bytes": b * m * k + (1 if c["shared_w"] else b) * n * k + b * m * n * _BYTES[c["out"]], "flops": 2 * b * m * n * k}
    if op == "q4_1":
        m, n, k = c["m"], c["n"], c["k"]
        return {"bytes": n * (k // 32) * 20 + m * k * _BYTES[c["a"]] + m * n * _BYTES[c["out"]], "flops": 2 * m * n * k}
    if op == "qdq":
        e = c["rows"] * c["cols"]
        return {"bytes": 2 * e * (_BYTES[c["x"]] + 1), "flops": 0}
    if op == "fp_act":
        m, n, k, b = c["m"], c["n"], c["k"], _BYTES[c["x"]]
        return {"bytes": m * k * b + n * k + 8 * n + m * n * b, "flops": 2 * m * n * k}
    oh, ow = ops.conv2d_out_hw(c["h"], c["w"], c["ks"], c["ks"], (c["stride"],) * 2, (c["dil"],) * 2, (c["pad"],) * 2)
    pixels, taps = c["batch"] * oh * ow, c["ks"] * c["ks"] * c["ic"] // c["groups"]
    nbytes = c["batch"] * c["h"] * c["w"] * c["ic"] + taps * c["oc"] + pixels * c["oc"] * _BYTES[c["out"]]
    flops = 2 * pixels * taps * c["oc"]
    if c["oc2"]:
        nbytes += pixels * c["oc"] * _BYTES[c["out"]] + c["oc"] * c["oc2"] + pixels * c["oc2"] * _BYTES[c["out"]]
        flops += 2 * pixels * c["oc"] * c["oc2"]
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    if case["op"] == "q4_1":
        # A weight decoded to f16 carries one rounding of 2^-11: against a 64-bit evaluation that is
        # 1.9e-4 of the result in the 2-norm and 1e-3 at worst, with the f16 result's own rounding
        # 2.8e-4 and 1.1e-3 (measured at K = 4096, 1 to 300 rows).
        return {"rel": 1e-3, "max": 4e-3}
    if case.get("act") in ("gelu", "silu") and case["out"] in _DTYPE:
        # Exponentials in f32: a few units in the last place, or one rounding of an f16 result.
        return {"rel": 1e-5 if case["out"] == "f32" else 2e-4, "max": 2e-3}
    # Integer sums and operations rounded one by one in a fixed order: the bytes are the contract.
    return "exact"


def _activated(x, act):
    if act == "relu":
        return x.clamp_min(0)
    if act == "gelu":
        return 0.5 * x * (1 + torch.tanh(math.sqrt(2.0 / math.pi) * (x + 0.044715 * x ** 3)))
    return x * torch.sigmoid(x) if act == "silu" else x


def exact(case, seed):
    """The floating destinations of the products in 64 bits; whole-number results are compared byte for byte instead."""
    c, op = case, case["op"]
    if op not in ("linear", "matmul", "q4_1") or c["out"] not in _DTYPE:
        return None
    state = prepare(case, seed)
    a = state["a"].double()
    if op == "q4_1":
        if c["packed"]:
            state["w"] = _q4_1_blocks(_gen(seed), c["n"], c["k"])
        blocks = state["w"].view(c["n"], -1, 20)
        d, low = (blocks[:, :, i:i + 2].contiguous().view(torch.float16).double() for i in (0, 2))
        nibbles = torch.cat([blocks[:, :, 4:] & 15, blocks[:, :, 4:] >> 4], dim=2).double()
        w = (d * nibbles + low).reshape(c["n"], c["k"])
        return _activated(a @ w.t(), c["act"])
    kw = state["kw"]
    if op == "matmul":
        return a @ state["w"].double().transpose(-1, -2) * (kw["scale_a"] * kw["scale_w"])

    def column(v):
        return v.double().unsqueeze(1) if isinstance(v, torch.Tensor) else v

    if c["packed"]:
        g = _gen(seed)
        w, scale_w = _s8(g, c["n"], c["k"]), _scales(g, c["n"])
        zp_w = state["packed"].zp_w
    else:
        w, scale_w, zp_w = state["w"], kw["scale_w"], kw["zp_w"]
    x = (a - column(kw.get("zp_a", 0))) @ (w.double() - column(zp_w)).t()
    return _activated(x * column(kw["scale_a"]) * scale_w.double() + kw["bias"].double(), c["act"])
