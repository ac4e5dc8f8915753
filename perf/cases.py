"""Performance cases of the library: the calls a client makes, at the sizes and options it makes them with.

Every case goes through the public entry points of the package (gemm, conv, conv_fused, attention) on buffers that the
client owns: operands, result and - where the package can be asked for its size - the workspace. The sizes are those of
the benchmark, of the tuning problem list and of the end-to-end test matrices, or plain sizes of the same kind.
"""
from __future__ import annotations

import math

import torch

from rocmlir_b200 import conv as rb_conv
from rocmlir_b200.attention import attention
from rocmlir_b200.gemm import Epilogue, gemm, problem, rb_dtype, workspace_size

TORCH = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16, "i8": torch.int8, "i32": torch.int32,
         "fp8": torch.float8_e4m3fn}
BYTES = {"f32": 4, "f16": 2, "bf16": 2, "i8": 1, "i32": 4, "fp8": 1}
REQUANT_SCALE = 12.0
FP8_ALPHA = 0.25 * 0.5


def gemm_case(name, m, n, k, dtype, out, g=1, trans_a=False, trans_b=False, epilogue="none"):
    c = dict(op="gemm", g=g, m=m, n=n, k=k, dtype=dtype, out=out, trans_a=trans_a, trans_b=trans_b, epilogue=epilogue)
    return dict(c, name=name) if name else c


def conv_case(name, direction, n, c, k, hw, fil, stride, dtype, layout, epilogue="none"):
    d = dict(op="conv", direction=direction, n=n, c=c, k=k, hw=hw, fil=fil, stride=stride, dtype=dtype, layout=layout,
             epilogue=epilogue)
    return dict(d, name=name) if name else d


def attention_case(name, g, sq, sk, d, dtype, causal=False, mask=False):
    c = dict(op="attention", g=g, sq=sq, sk=sk, d=d, dtype=dtype, causal=causal, mask=mask)
    return dict(c, name=name) if name else c


def listed():
    return [
        # one linear layer (weight stored out x in) for a handful of tokens: what a generation step is made of; the
        # smallest call here, bound by reading the weight and by launches
        gemm_case("linear_f16_m8", 8, 4096, 4096, "f16", "f16", trans_b=True, epilogue="bias"),
        # a batch of matrix products with an odd inner extent: the shape of the GEMM test matrices, whose rows cannot
        # be loaded as they lie
        gemm_case("gemm_f16_g3_k769", 1024, 1024, 769, "f16", "f16", g=3),
        # the large square product with its fused bias and rectifier
        gemm_case("gemm_f16_4096_bias_relu", 4096, 4096, 4096, "f16", "f16", epilogue="bias_relu"),
        # quantised linear layer of a language model over a full prompt, requantised to int8
        gemm_case("linear_i8_requant", 2048, 11008, 4096, "i8", "i8", trans_b=True, epilogue="requant"),
        # single-precision product at full accuracy
        gemm_case("gemm_f32_4096", 4096, 4096, 4096, "f32", "f32"),
        # 3x3 layer of a residual network with fused bias and rectifier, channels last
        conv_case("conv_fwd_f16_3x3", "conv", 256, 64, 64, 56, 3, 1, "f16", "nhwc", epilogue="bias_relu"),
        # the down-sampling 3x3 layer in training: gradient of the input and of the filter
        conv_case("conv_bwd_data_f16_3x3s2", "conv_bwd_data", 256, 128, 128, 28, 3, 2, "f16", "nhwc"),
        conv_case("conv_bwd_weight_f16_3x3s2", "conv_bwd_weight", 256, 128, 128, 28, 3, 2, "f16", "nhwc"),
        # first layer of the network: three image channels, 7x7 filter, stride 2
        conv_case("conv_stem_f16_7x7s2", "conv", 64, 3, 64, 224, 7, 2, "f16", "nhwc"),
        # single-precision inference in the channels-first layout
        conv_case("conv_fwd_f32_nchw_3x3", "conv", 64, 128, 128, 28, 3, 1, "f32", "nchw"),
        # prompt of a language model: 16 sequences, 32 heads, causal; the largest call here
        attention_case("attention_prefill_causal", 512, 2048, 2048, 128, "f16", causal=True),
        # one generation step over cached keys and values (stored sequence x head) of a few sequences, with a
        # mask over the padded positions
        attention_case("attention_decode", 64, 1, 4096, 128, "f16", mask=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi, step=64):
    """Half of the time any whole number, otherwise a multiple of `step`."""
    v = _log(rng, lo, hi)
    return v if rng.random() < 0.5 else max(step, v // step * step)


def draw(rng):
    kind = rng.choice(["linear_small", "gemm16", "linear8", "gemm32", "conv16", "conv16", "stem", "conv32", "prefill", "decode"])
    f = rng.choice(["f16", "bf16"])
    if kind == "linear_small":
        return gemm_case(None, _log(rng, 1, 64), _size(rng, 512, 11008), _log(rng, 512, 8192) // 8 * 8, f, f, trans_b=True,
                         epilogue=rng.choice(["none", "bias"]))
    if kind == "gemm16":
        return gemm_case(None, _size(rng, 128, 4096), _size(rng, 128, 4096), _size(rng, 128, 4096), f, f, g=rng.choice([1, 1, 3]),
                         trans_a=rng.random() < 0.25, trans_b=rng.random() < 0.5, epilogue=rng.choice(["none", "bias_relu"]))
    if kind == "linear8":
        m, n, k = _log(rng, 16, 2048), _log(rng, 1024, 11008) // 16 * 16, _log(rng, 1024, 4096) // 64 * 64
        return rng.choice([gemm_case(None, m, n, k, "i8", "i8", trans_b=True, epilogue="requant"),
                           gemm_case(None, m, n, k, "i8", "i32", trans_b=True),
                           gemm_case(None, m, n, k, "fp8", "bf16", trans_b=True, epilogue="alpha")])
    if kind == "gemm32":
        return gemm_case(None, _size(rng, 128, 4096), _size(rng, 128, 4096), _size(rng, 128, 4096), "f32", "f32",
                         trans_a=rng.random() < 0.25, trans_b=rng.random() < 0.5)
    if kind == "conv16":
        while True:
            c = conv_case(None, rng.choice(["conv", "conv_bwd_data", "conv_bwd_weight"]), _log(rng, 1, 256),
                          rng.choice([64, 128, 256, 512]), rng.choice([64, 128, 256, 512]), rng.randint(7, 56),
                          rng.choice([1, 3]), rng.choice([1, 1, 2]), f, "nhwc")
            if c["direction"] == "conv" and rng.random() < 0.5:
                c["epilogue"] = "bias_relu"
            if work(c)["flops"] <= 6e10:
                return c
    if kind == "stem":
        while True:
            c = conv_case(None, "conv", _log(rng, 1, 128), rng.choice([3, 3, 4, 7, 8, 16]), rng.choice([32, 64, 128]),
                          _log(rng, 14, 224), rng.choice([3, 5, 7]), rng.choice([1, 2]), f, rng.choice(["nhwc", "nhwc", "nchw"]))
            if work(c)["flops"] <= 2e10:
                return c
    if kind == "conv32":
        while True:
            c = conv_case(None, "conv", _log(rng, 1, 64), rng.choice([16, 64, 128, 256]), rng.choice([64, 128, 256]),
                          rng.randint(7, 56), rng.choice([1, 3]), rng.choice([1, 1, 2]), "f32", "nchw")
            if work(c)["flops"] <= 1.5e10:
                return c
    if kind == "prefill":
        s, d = _size(rng, 64, 2048), rng.choice([64, 128])
        g = _log(rng, 1, 512)
        return attention_case(None, g, s, s, d, f, causal=rng.random() < 0.6)
    return attention_case(None, _log(rng, 8, 512), _log(rng, 1, 16), _log(rng, 128, 8192), rng.choice([64, 128]), f,
                          mask=rng.random() < 0.5)


def _conv_config(case):
    pad = case["fil"] // 2
    lay = {"nhwc": ("gkyxc", "nhwgc", "nhwgk"), "nchw": ("gkcyx", "ngchw", "ngkhw")}[case["layout"]]
    return rb_conv.ConvConfig(case["n"], case["c"], case["k"], case["hw"], case["hw"], case["fil"], case["fil"],
                              stride_h=case["stride"], stride_w=case["stride"], pad_h=pad, pad_w=pad,
                              fil_layout=lay[0], in_layout=lay[1], out_layout=lay[2])


def _normal(gen, shape, scale, dtype):
    return torch.empty(shape, dtype=torch.float32, device="cuda").normal_(0.0, scale, generator=gen).to(dtype)


def _uniform(gen, shape, lo, hi, dtype=torch.float32):
    return torch.empty(shape, dtype=torch.float32, device="cuda").uniform_(lo, hi, generator=gen).to(dtype)


def _inputs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    dt = TORCH[case["dtype"]]
    if case["op"] == "gemm":
        g, m, n, k = case["g"], case["m"], case["n"], case["k"]
        sa, sb = ((g, k, m) if case["trans_a"] else (g, m, k)), ((g, n, k) if case["trans_b"] else (g, k, n))
        if case["dtype"] == "i8":
            ab = [torch.randint(-127, 128, s, dtype=torch.int8, device="cuda", generator=gen) for s in (sa, sb)]
        elif case["dtype"] == "f32":
            ab = [_normal(gen, s, 1.0, dt) for s in (sa, sb)]
        else:
            ab = [_normal(gen, s, 1.0 if case["dtype"] == "fp8" else 0.1, dt) for s in (sa, sb)]
        vec = None
        if case["epilogue"] in ("bias", "bias_relu"):
            vec = _normal(gen, (n,), 0.1, dt)
        elif case["epilogue"] == "requant":
            vec = _uniform(gen, (n,), 0.001, 0.01)
        return ab + [vec]
    if case["op"] == "conv":
        cfg = _conv_config(case)
        made = []
        for which in ("fil", "in", "out"):
            if case["dtype"] == "f32":
                made.append(_uniform(gen, (cfg.numel(which),), -1.0, 1.0))
            else:
                made.append(_normal(gen, (cfg.numel(which),), 0.05, dt))
        vec = _normal(gen, (case["k"],), 0.1, dt) if case["epilogue"] == "bias_relu" else None
        return made + [vec]
    g, sq, sk, d = case["g"], case["sq"], case["sk"], case["d"]
    q, k, v = (_normal(gen, s, 1.0, dt) for s in ((g, sq, d), (g, sk, d), (g, sk, d)))
    mask = None
    if case["mask"]:   # each group has its own number of valid positions, between a half and all of them
        length = torch.randint((sk + 1) // 2, sk + 1, (g, 1, 1), device="cuda", generator=gen)
        mask = (torch.arange(sk, device="cuda")[None, None, :] < length).to(torch.int8).expand(g, sq, sk).contiguous()
    return [q, k, v, mask]


def prepare(case, seed):
    state = {"case": case, "inputs": _inputs(case, seed)}
    if case["op"] == "gemm":
        a, b, vec = state["inputs"]
        out = TORCH[case["out"]]
        epilogue = None
        if case["epilogue"] == "bias":
            epilogue = Epilogue(bias=vec, mid_type=rb_dtype(out))
        elif case["epilogue"] == "bias_relu":
            epilogue = Epilogue(bias=vec, relu=True, mid_type=rb_dtype(out))
        elif case["epilogue"] == "requant":
            epilogue = Epilogue(col_scale=vec, requant_scale=REQUANT_SCALE)
        elif case["epilogue"] == "alpha":
            epilogue = Epilogue(alpha=FP8_ALPHA)
        state["epilogue"] = epilogue
        state["out"] = torch.empty((case["g"], case["m"], case["n"]), dtype=out, device="cuda")
        size = workspace_size(problem(a, b, case["trans_a"], case["trans_b"], False, out))
        state["workspace"] = torch.empty(max(16, size), dtype=torch.uint8, device="cuda")
    elif case["op"] == "conv":
        fil, inp, out, vec = state["inputs"]
        cfg = state["config"] = _conv_config(case)
        if case["epilogue"] == "bias_relu":
            state["epilogue"] = Epilogue(bias=vec, relu=True, mid_type=rb_dtype(out.dtype))
        else:
            size = rb_conv.workspace_size(cfg, inp.dtype, rb_conv.OPERATIONS[case["direction"]])
            state["workspace"] = torch.empty(max(16, size), dtype=torch.uint8, device="cuda")
    else:
        state["out"] = torch.empty_like(state["inputs"][0])
    return state


def run(state):
    case = state["case"]
    if case["op"] == "gemm":
        a, b, _ = state["inputs"]
        return gemm(a, b, trans_a=case["trans_a"], trans_b=case["trans_b"], out_dtype=TORCH[case["out"]],
                    epilogue=state["epilogue"], out=state["out"], workspace=state["workspace"])
    if case["op"] == "conv":
        fil, inp, out, _ = state["inputs"]
        if case["epilogue"] == "bias_relu":
            return rb_conv.conv_fused(state["config"], fil, inp, out, state["epilogue"])
        return rb_conv.conv(state["config"], rb_conv.OPERATIONS[case["direction"]], fil, inp, out, workspace=state["workspace"])
    q, k, v, mask = state["inputs"]
    return attention(q, k, v, trans_k=True, scale=1.0 / math.sqrt(case["d"]), causal=case["causal"], mask=mask, out=state["out"])


def work(case):
    es = BYTES[case["dtype"]]
    if case["op"] == "gemm":
        g, m, n, k = case["g"], case["m"], case["n"], case["k"]
        extra = {"none": 0, "alpha": 0, "bias": n * es, "bias_relu": n * es, "requant": n * 4}[case["epilogue"]]
        return {"bytes": g * (m * k + k * n) * es + g * m * n * BYTES[case["out"]] + extra, "flops": 2.0 * g * m * n * k}
    if case["op"] == "conv":
        cfg = _conv_config(case)
        return {"bytes": sum(cfg.numel(w) for w in ("fil", "in", "out")) * es, "flops": cfg.flops()}
    g, sq, sk, d = case["g"], case["sq"], case["sk"], case["d"]
    pairs = sq * (sk + 1) / 2 if case["causal"] else sq * sk
    return {"bytes": g * (2 * sq + 2 * sk) * d * es + (g * sq * sk if case["mask"] else 0), "flops": 4.0 * g * pairs * d}


def tolerance(case):
    if case["op"] == "gemm" and case["dtype"] == "i8":
        return "exact"
    if case["op"] == "attention":   # probabilities carry one rounding to the element type before the second product
        return {"rel": 3e-3, "max": 0.1} if case["dtype"] == "f16" else {"rel": 2e-2, "max": 0.5}
    out = case["out"] if case["op"] == "gemm" else case["dtype"]
    return {"f32": {"rel": 1e-5, "max": 1e-3}, "f16": {"rel": 1e-3, "max": 1e-2}, "bf16": {"rel": 8e-3, "max": 8e-2}}[out]


def _exact_gemm(case, a, b, vec):
    a = a.double().transpose(1, 2) if case["trans_a"] else a.double()
    b = b.double().transpose(1, 2) if case["trans_b"] else b.double()
    acc = a @ b
    if case["epilogue"] == "requant":   # int32 sums are exact in 64 bits; the chain after them is defined in f32
        x = acc.float() * vec
        x = x * torch.tensor(1.0 / REQUANT_SCALE, dtype=torch.float32, device=x.device)
        return x.round().clamp(-128, 127).to(torch.int8)
    if case["epilogue"] == "alpha":
        acc = acc * FP8_ALPHA
    if case["epilogue"] in ("bias", "bias_relu"):
        acc = acc + vec.double()
    if case["epilogue"] == "bias_relu":
        acc = acc.relu()
    return acc.to(torch.int32) if case["out"] == "i32" else acc


def _exact_conv(case, fil, inp, out, vec):
    cfg = _conv_config(case)
    n, c, k, hw, f = case["n"], case["c"], case["k"], case["hw"], case["fil"]
    args = dict(stride=case["stride"], padding=f // 2)
    last = case["layout"] == "nhwc"

    def first(t, rows, ch, h, w):   # channels first, in 64 bits
        return (t.view(rows, h, w, ch).permute(0, 3, 1, 2) if last else t.view(rows, ch, h, w)).double().contiguous()

    def back(t):
        return (t.permute(0, 2, 3, 1) if last else t).contiguous().view(-1)

    if case["direction"] == "conv_bwd_data":
        return back(torch.nn.grad.conv2d_input((n, c, hw, hw), first(fil, k, c, f, f), first(out, n, k, cfg.ho, cfg.wo), **args))
    if case["direction"] == "conv_bwd_weight":
        return back(torch.nn.grad.conv2d_weight(first(inp, n, c, hw, hw), (k, c, f, f), first(out, n, k, cfg.ho, cfg.wo), **args))
    y = torch.nn.functional.conv2d(first(inp, n, c, hw, hw), first(fil, k, c, f, f), **args)
    if case["epilogue"] == "bias_relu":
        y = (y + vec.double().view(1, -1, 1, 1)).relu()
    return back(y)


def _exact_attention(case, q, k, v, mask):
    res = torch.empty(q.shape, dtype=torch.float64, device=q.device)
    sq, sk = case["sq"], case["sk"]
    step = max(1, int(2e8 // (sq * sk)))
    above = torch.ones((sq, sk), dtype=torch.bool, device=q.device).triu(1) if case["causal"] else None
    for i in range(0, case["g"], step):
        s = q[i:i + step].double() @ k[i:i + step].double().transpose(1, 2) / math.sqrt(case["d"])
        if above is not None:
            s.masked_fill_(above, -math.inf)
        if mask is not None:
            s.masked_fill_(mask[i:i + step] == 0, -math.inf)
        res[i:i + step] = s.softmax(-1) @ v[i:i + step].double()
    return res


def exact(case, seed):
    made = _inputs(case, seed)
    with torch.backends.cudnn.flags(enabled=False):
        if case["op"] == "gemm":
            return _exact_gemm(case, *made)
        if case["op"] == "conv":
            return _exact_conv(case, *made)
        return _exact_attention(case, *made)
