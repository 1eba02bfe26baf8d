"""The work that performance is judged on: one training step (or inference call) of each kind of layer the library
serves, issued through the C ABI the way the benchmark and a binding issue it.

A case names one layer: a convolution (forward, dInput, dWeight, dBias), the same layer at inference, a network's first
convolution (no dInput: the image needs no gradient), BatchNorm, GroupNorm, attention, or a linear layer (addmm and the
two products of its backward).  A caller keeps its tensors, gradients and workspace between steps, so `prepare` allocates
them and builds the argument lists; `run` only issues the calls.  Everything is FP32, as the operators are.

  listed()        the fixed cases         draw(rng)       one more of the same ranges
  prepare(c, s)   inputs from seed s      run(state)      one pass, its outputs
  work(c)         bytes and operations that one pass cannot do without
  tolerance(c)    how far another correct implementation's results may be
"""
import ctypes
import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.getcwd(), "pytorch-vulkan_b200"))
import b200conv  # noqa: E402

BUDGET = 512 << 20      # scratch that the benchmark grants a convolution call
MAX_FLOPS = 6.5e11      # a drawn case stays below the largest listed one
MAX_BYTES = 7.0e8


def _conv(name, n, cin, cout, hw, k=3, stride=1, dilation=1, groups=1, layout="nchw", kind="conv"):
    return {"name": name, "kind": kind, "n": n, "cin": cin, "cout": cout, "hw": hw, "k": k, "stride": stride,
            "dilation": dilation, "groups": groups, "layout": layout}


def listed():
    return [
        # the smallest call: one image through one residual-block layer with its ReLU; launches and host time count
        _conv("infer_64_28_b1", 1, 64, 64, 28, kind="infer"),
        # configuration 1: the single layer, batch 8
        _conv("conv_64_56_b8", 8, 64, 64, 56),
        # configuration 2, the ResNet-50 sweep at batch 64: its smallest (and odd) image, its strided and its 1x1 layer
        _conv("conv_512_7_b64", 64, 512, 512, 7),
        _conv("conv_128_56_s2_b64_cl", 64, 128, 128, 56, stride=2, layout="channels_last"),
        _conv("conv_256to64_56_1x1_b64", 64, 256, 64, 56, k=1),
        # configuration 4, the U-Net mix on sliced views: its grouped layer
        _conv("conv_256_32_g32_b16_sliced", 16, 256, 256, 32, groups=32, layout="sliced"),
        # configuration 5, one of eight ranks: the largest
        _conv("conv_256_56_b64", 64, 256, 256, 56),
        # a network's first layer: three input channels, 7x7, stride 2
        _conv("stem_3to64_224_b64", 64, 3, 64, 224, k=7, stride=2, kind="stem"),
        # the commonest BatchNorm of that network (256 channels at 14x14)
        {"name": "bn_256_14_b64", "kind": "batch_norm", "n": 64, "c": 256, "hw": 14, "layout": "nchw"},
        # GroupNorm of a diffusion U-Net's middle resolution
        {"name": "gn_512_32_b16", "kind": "group_norm", "n": 16, "c": 512, "hw": 32, "groups": 32},
        # self-attention of the same network
        {"name": "attn_16x1024x64", "kind": "attention", "heads": 16, "tq": 1024, "tk": 1024, "d": 64, "causal": False},
        # the wide linear layer of its transformer block (16 images of 16x16 tokens)
        {"name": "linear_4096x512x2048", "kind": "linear", "m": 4096, "k": 512, "n": 2048},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _channels(rng, lo, hi):
    """Mostly multiples of 16, as networks have them, and some that are not."""
    c = _log(rng, lo, hi)
    return max(16, (c + 8) // 16 * 16) if rng.random() < 0.8 else max(16, c)


def _draw_one(rng):
    kind = rng.choice(["infer", "conv", "conv", "conv", "conv", "conv", "stem", "batch_norm", "group_norm", "attention", "linear"])
    if kind == "infer":
        return _conv("", rng.choice([1, 1, 2, 4]), _channels(rng, 16, 512), _channels(rng, 16, 512), _log(rng, 7, 64), rng.choice([1, 3, 3]),
                     layout=rng.choice(["nchw", "channels_last"]), kind=kind)
    if kind == "conv":
        c = _conv("", _log(rng, 1, 64), _channels(rng, 16, 512), _channels(rng, 16, 512), _log(rng, 7, 112), rng.choice([1, 3, 3, 3]),
                  layout=rng.choice(["nchw", "nchw", "channels_last", "sliced"]))
        variant = rng.choice(["plain", "plain", "plain", "stride", "dilation", "groups"])
        if variant == "stride":
            c["stride"] = 2
        elif variant == "dilation" and c["k"] == 3:
            c["dilation"] = 2
        elif variant == "groups" and c["k"] == 3:
            c["groups"] = 32
            c["cin"] = c["cout"] = 32 * rng.choice([4, 8, 16])
        return c
    if kind == "stem":
        return _conv("", _log(rng, 1, 64), rng.choice([1, 3, 3, 4]), 16 * rng.randint(2, 8), _log(rng, 56, 224), rng.choice([3, 7]), rng.choice([1, 2]),
                     layout=rng.choice(["nchw", "channels_last"]), kind=kind)
    if kind == "batch_norm":
        return {"kind": kind, "n": _log(rng, 4, 64), "c": _channels(rng, 16, 2048), "hw": _log(rng, 7, 112),
                "layout": rng.choice(["nchw", "nchw", "channels_last"])}
    if kind == "group_norm":
        return {"kind": kind, "n": _log(rng, 1, 32), "c": 32 * rng.randint(2, 40), "hw": _log(rng, 8, 128), "groups": 32}
    if kind == "attention":
        tq = _log(rng, 64, 2048)
        tk = rng.choice([tq, tq, 77])      # itself, or a text encoder's 77 tokens
        return {"kind": kind, "heads": _log(rng, 4, 64), "tq": tq, "tk": tk, "d": rng.choice([32, 40, 64, 64, 80, 128]),
                "causal": tk == tq and rng.random() < 0.4}
    return {"kind": kind, "m": _log(rng, 16, 16384), "k": _log(rng, 64, 4096), "n": _log(rng, 64, 4096)}


def draw(rng):
    while True:
        c = _draw_one(rng)
        c.pop("name", None)
        w = work(c)
        limit = 3.0e10 if c["kind"] == "stem" else 1.0e11 if c["kind"] in ("attention", "linear") else MAX_FLOPS
        scores = c["heads"] * c["tq"] * c["tk"] if c["kind"] == "attention" else 0
        if w["flops"] <= limit and w["bytes"] <= MAX_BYTES and scores <= 1 << 26:
            return c


# ---- sizes ---------------------------------------------------------------------------------------------------------
def _conv_dims(c):
    """(padding, output extent) of the layer: "same" padding, as every configuration has it."""
    pad = c["dilation"] * (c["k"] - 1) // 2
    return pad, (c["hw"] + 2 * pad - c["dilation"] * (c["k"] - 1) - 1) // c["stride"] + 1


def work(case):
    c = case
    if c["kind"] in ("conv", "infer", "stem"):
        _, o = _conv_dims(c)
        x, y = c["n"] * c["cin"] * c["hw"] ** 2, c["n"] * c["cout"] * o ** 2
        w = c["cout"] * (c["cin"] // c["groups"]) * c["k"] ** 2
        macs = y * (c["cin"] // c["groups"]) * c["k"] ** 2
        if c["kind"] == "infer":
            return {"bytes": 4 * (x + w + c["cout"] + y), "flops": 2 * macs}
        if c["kind"] == "stem":     # x, w, b, dy read; y, dw, db written
            return {"bytes": 4 * (x + 2 * y + 2 * w + 2 * c["cout"]), "flops": 4 * macs}
        return {"bytes": 4 * (2 * x + 2 * y + 2 * w + 2 * c["cout"]), "flops": 6 * macs}
    if c["kind"] in ("batch_norm", "group_norm"):     # x, dy read; y, dx written
        e = c["n"] * c["c"] * c["hw"] ** 2
        return {"bytes": 4 * (4 * e + 8 * c["c"]), "flops": 20 * e}
    if c["kind"] == "attention":     # q, k, v, grad read; out, dq, dk, dv written; two products forward, five backward
        q, kv = c["heads"] * c["tq"] * c["d"], c["heads"] * c["tk"] * c["d"]
        pairs = c["heads"] * c["tq"] * c["tk"] * (0.5 if c["causal"] else 1.0)
        return {"bytes": 4 * (4 * q + 4 * kv), "flops": 14 * pairs * c["d"]}
    m, k, n = c["m"], c["k"], c["n"]     # x, w, b, dy read; y, dx, dw, db written
    return {"bytes": 4 * (2 * m * k + 2 * m * n + 2 * n * k + 2 * n), "flops": 6 * m * n * k}


def tolerance(case):
    """Matrix products run in split precision with FP32 accumulation, two correct orders of which differ by 2e-5 to 3e-5
    on long sums; normalisation is plain FP32."""
    if case["kind"] in ("batch_norm", "group_norm"):
        return {"rel": 1e-5, "max": 1e-3}
    return {"rel": 4e-5, "max": 2e-3}


# ---- inputs and calls ----------------------------------------------------------------------------------------------
def _randn(gen, *shape):
    return torch.randn(*shape, device="cuda", generator=gen)


def _view(t):
    return b200conv.View4(t.data_ptr(), (ctypes.c_int64 * 4)(*t.stride()))


def _laid_out(t, layout):
    """The tensor as the caller holds it: dense NCHW, channels-last, or the interior of a larger NCHW allocation."""
    if layout == "channels_last":
        return t.contiguous(memory_format=torch.channels_last)
    if layout == "sliced":
        n, ch, h, w = t.shape
        parent = torch.zeros(n, ch + 8, h + 2, w + 2, device=t.device)
        inside = parent[:, 4:4 + ch, 1:1 + h, 1:1 + w]
        inside.copy_(t)
        return inside
    return t


def _prepare_conv(c, gen, stream):
    L, (pad, o) = b200conv.lib(), _conv_dims(c)
    n, cin, cout, hw, k, groups = c["n"], c["cin"], c["cout"], c["hw"], c["k"], c["groups"]
    p = b200conv.geometry((n, cin, hw, hw), cout, (k, k), (c["stride"],) * 2, (pad, pad), (c["dilation"],) * 2, groups)
    x = _laid_out(_randn(gen, n, cin, hw, hw), c["layout"])
    bound = 1.0 / math.sqrt(cin // groups * k * k)     # kaiming-uniform with a = sqrt(5), PyTorch's default
    w = (torch.rand(cout, cin // groups, k, k, device="cuda", generator=gen) * 2 - 1) * bound
    b = (torch.rand(cout, device="cuda", generator=gen) * 2 - 1) * bound
    y = torch.empty(n, cout, o, o, device="cuda")
    infer = c["kind"] == "infer"
    phases = (0,) if infer else (0, 2, 3) if c["kind"] == "stem" else (0, 1, 2, 3)
    ws_n = max(max(b200conv.workspace_bytes(p, ph, budget=BUDGET) for ph in phases), 1)
    ws = torch.empty(ws_n, dtype=torch.uint8, device="cuda")
    P, ref, work_args = ctypes.c_void_p, ctypes.byref(p), (ctypes.c_void_p(ws.data_ptr()), ctypes.c_size_t(ws_n))
    xv, wv = _view(x), _view(w)
    if infer:      # relu(conv + bias), one call
        none = b200conv.View4(None, (ctypes.c_int64 * 4)(0, 0, 0, 0))
        calls = [(L.b200_conv2d_forward_fused, (ref, xv, wv, P(b.data_ptr()), 1, none, 1, P(y.data_ptr()), 0, *work_args, 0, stream))]
        return calls, (y,), (p, x, w, b, ws)
    go = _laid_out(_randn(gen, n, cout, o, o), "channels_last" if c["layout"] == "channels_last" else "nchw")
    dw, db, gv = torch.empty_like(w), torch.empty_like(b), _view(go)
    calls = [(L.b200_conv2d_forward, (ref, xv, wv, P(b.data_ptr()), 1, P(y.data_ptr()), *work_args, 0, stream)),
             (L.b200_conv2d_dweight, (ref, xv, gv, P(dw.data_ptr()), *work_args, 0, stream)),
             (L.b200_conv2d_dbias, (ref, gv, P(db.data_ptr()), *work_args, stream))]
    out = (y, dw, db)
    if 1 in phases:
        dx = torch.empty(n, cin, hw, hw, device="cuda")
        calls.append((L.b200_conv2d_dinput, (ref, gv, wv, P(dx.data_ptr()), *work_args, 0, stream)))
        out += (dx,)
    return calls, out, (p, x, w, b, go, ws)


def _prepare_batch_norm(c, gen, stream):
    L, n, ch, hw = b200conv.lib(), c["n"], c["c"], c["hw"]
    s, cl = hw * hw, c["layout"] == "channels_last"
    layout = b200conv.BN_INTERLEAVED if cl else b200conv.BN_PLANAR
    lay = "channels_last" if cl else "nchw"
    x, g = _laid_out(_randn(gen, n, ch, hw, hw) * 1.5 + 0.25, lay), _laid_out(_randn(gen, n, ch, hw, hw), lay)
    w, b = 1 + 0.1 * _randn(gen, ch), 0.1 * _randn(gen, ch)
    rm, rv = torch.zeros(ch, device="cuda"), torch.ones(ch, device="cuda")
    y, dx = torch.empty_like(x), torch.empty_like(x)
    sm, si, dw, db = (torch.empty(ch, device="cuda") for _ in range(4))
    ws_n = L.b200_batch_norm_workspace(n, ch, s, layout)
    ws = torch.empty(ws_n, dtype=torch.uint8, device="cuda")
    P = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    calls = [(L.b200_batch_norm_forward, (n, ch, s, layout, P(x), P(w), 1, P(b), 1, P(rm), 1, P(rv), 1, 1, 0.1, 1e-5, P(y), P(sm), P(si),
                                          P(ws), ws_n, stream)),
             (L.b200_batch_norm_backward, (n, ch, s, layout, P(g), P(x), P(w), 1, P(sm), 1, P(si), 1, 1, 1e-5, P(dx), P(dw), P(db),
                                           P(ws), ws_n, stream))]
    return calls, (y, sm, si, rm, rv, dx, dw, db), (x, g, w, b, ws)


def _prepare_group_norm(c, gen, stream):
    L, n, ch, hw, groups = b200conv.lib(), c["n"], c["c"], c["hw"], c["groups"]
    s = hw * hw
    x, g = _randn(gen, n, ch, hw, hw) * 1.5 + 0.25, _randn(gen, n, ch, hw, hw)
    w, b = 1 + 0.1 * _randn(gen, ch), 0.1 * _randn(gen, ch)
    y, dx = torch.empty_like(x), torch.empty_like(x)
    mean, rstd = torch.empty(n, groups, device="cuda"), torch.empty(n, groups, device="cuda")
    dw, db = torch.empty(ch, device="cuda"), torch.empty(ch, device="cuda")
    ws_n = L.b200_group_norm_workspace(n, ch, s, groups)
    ws = torch.empty(ws_n, dtype=torch.uint8, device="cuda")
    P = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    calls = [(L.b200_group_norm_forward, (n, ch, s, groups, P(x), P(w), P(b), 1e-5, P(y), P(mean), P(rstd), stream)),
             (L.b200_group_norm_backward, (n, ch, s, groups, P(g), P(x), P(mean), P(rstd), P(w), P(dx), P(dw), P(db), P(ws), ws_n, stream))]
    return calls, (y, mean, rstd, dx, dw, db), (x, g, w, b, ws)


def _prepare_attention(c, gen, stream):
    L, h, tq, tk, d = b200conv.lib(), c["heads"], c["tq"], c["tk"], c["d"]
    q, k, v, g = _randn(gen, h, tq, d), _randn(gen, h, tk, d), _randn(gen, h, tk, d), _randn(gen, h, tq, d)
    out, lse = torch.empty_like(q), torch.empty(h, tq, device="cuda")
    dq, dk, dv = torch.empty_like(q), torch.empty_like(k), torch.empty_like(v)
    n_f, n_b = (L.b200_attention_workspace(h, tq, tk, d, d, back) for back in (0, 1))
    ws = torch.empty(max(n_f, n_b), dtype=torch.uint8, device="cuda")
    causal, scale = int(c["causal"]), 1.0 / math.sqrt(d)
    P = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    calls = [(L.b200_attention_forward, (h, tq, tk, d, d, P(q), P(k), P(v), None, 0, causal, scale, 0.0, None, P(out), P(lse), P(ws), n_f, stream)),
             (L.b200_attention_backward, (h, tq, tk, d, d, P(g), P(q), P(k), P(v), None, 0, P(out), P(lse), causal, scale, 0.0, None, P(dq), P(dk),
                                          P(dv), None, P(ws), n_b, stream))]
    return calls, (out, lse, dq, dk, dv), (q, k, v, g, ws)


def _prepare_linear(c, gen, stream):
    """y = x W^T + b and its gradients dx = g W, dW = g^T x, db = sum of g over rows."""
    L, m, k, n = b200conv.lib(), c["m"], c["k"], c["n"]
    bound = 1.0 / math.sqrt(k)
    x, g = _randn(gen, m, k), _randn(gen, m, n)
    w = (torch.rand(n, k, device="cuda", generator=gen) * 2 - 1) * bound
    b = (torch.rand(n, device="cuda", generator=gen) * 2 - 1) * bound
    y, dx, dw, db = torch.empty_like(g), torch.empty_like(x), torch.empty_like(w), torch.empty_like(b)
    P = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    sizes, strides, reduce = (ctypes.c_int64 * 2)(m, n), (ctypes.c_int64 * 2)(n, 1), ctypes.create_string_buffer(b"\x01\x00", 2)
    calls = [(L.b200_gemm, (m, n, k, P(x), k, 1, P(w), 1, k, P(b), 1.0, 1.0, P(y), 0, stream)),
             (L.b200_gemm, (m, k, n, P(g), n, 1, P(w), k, 1, None, 1.0, 0.0, P(dx), 0, stream)),
             (L.b200_gemm, (n, k, m, P(g), 1, n, P(x), k, 1, None, 1.0, 0.0, P(dw), 0, stream)),
             (L.b200_sum_strided, (P(db), P(g), 2, sizes, strides, reduce, stream))]
    return calls, (y, dx, dw, db), (x, g, w, b)


_PREPARE = {"conv": _prepare_conv, "infer": _prepare_conv, "stem": _prepare_conv, "batch_norm": _prepare_batch_norm,
            "group_norm": _prepare_group_norm, "attention": _prepare_attention, "linear": _prepare_linear}


def prepare(case, seed):
    b200conv.init()
    gen = torch.Generator(device="cuda").manual_seed(seed)
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    calls, outputs, keep = _PREPARE[case["kind"]](case, gen, stream)
    return {"calls": calls, "outputs": outputs, "keep": keep}


def run(state):
    for call, args in state["calls"]:
        b200conv.check(call(*args))
    return state["outputs"]
