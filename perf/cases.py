"""The work that is measured: the corrected W4A16 linears of decoder layers, as a user's program calls them.

A case is one pass over the quantised projections of one or more decoder layers (q/k/v, o, gate/up, down), converted with
``CudaW4A16Linear.from_float`` and wrapped by ``patch_svd_correction_wrappers_cumulative``, or the conversion itself:

  linear   one plain ``CudaW4A16Linear`` called from Python
  layer    the patched modules called from Python, one after another (prompts; decode without a graph)
  step     the same calls captured once in a CUDA graph and replayed (decode as it is served)
  convert  ``CudaW4A16Linear.from_float`` of a layer's ``nn.Linear`` modules (what loading a model costs)
"""
from __future__ import annotations

import os
import random

import torch
import torch.nn as nn

from glowq_b200.correction import patch_svd_correction_wrappers_cumulative
from glowq_b200.cuda_w4a16.linear import CudaW4A16Linear

GROUP = 128
# hidden, q outputs, k/v outputs, intermediate, rank, q/k/v bias - the shapes of glowq_b200.stack.SHAPES
OPT, L3B, Q7B, L13B, Q14B = ((2048, 2048, 2048, 8192, 64, False), (3072, 3072, 1024, 8192, 64, False),
                             (3584, 3584, 512, 18944, 128, True), (5120, 5120, 5120, 13824, 128, False),
                             (5120, 5120, 1024, 17408, 256, False))


def _case(call, m, shape, layers=1, out="fp16", alpha=1.0, share=1.0, **kw):
    hidden, q, kv, inter, rank, bias = shape
    return dict(kw, call=call, m=m, hidden=hidden, q=q, kv=kv, inter=inter, rank=rank, bias=bias, layers=layers, out=out,
                alpha=alpha, share=share)


def listed():
    return [
        # one uncorrected projection for one token, default output type: nothing but latency
        _case("linear", 1, OPT, out="fp32", name="linear-2048-m1"),
        # batch-1 decode without a graph: seven module calls, four launches
        _case("layer", 1, L3B, name="layer-3b-m1"),
        # batch-1 decode as it is served; several layers, so that weights come from HBM as in a whole model
        _case("step", 1, L13B, layers=4, name="step-13b-m1"),
        # a handful of sequences (or of speculated tokens), half of the groups corrected, q/k/v bias
        _case("step", 5, Q7B, layers=4, share=0.5, name="step-7b-m5-half"),
        # decode batches above one weight-streaming launch
        _case("step", 16, L13B, layers=4, name="step-13b-m16"),
        _case("step", 32, L3B, layers=4, name="step-3b-m32"),
        _case("step", 64, Q7B, layers=4, share=0.5, name="step-7b-m64-half"),
        # a short prompt of odd length
        _case("layer", 211, Q14B, name="layer-14b-m211"),
        # prompts: default output type; odd length with a correction weight; the longest
        _case("layer", 2048, L3B, out="fp32", name="prefill-3b-m2048"),
        _case("layer", 777, L13B, alpha=0.5, name="prefill-13b-m777-alpha"),
        _case("layer", 4096, Q14B, name="prefill-14b-m4096"),
        # loading: quantising and packing one layer
        _case("convert", 0, L13B, name="convert-13b"),
    ]


def draw(rng):
    def loguni(lo, hi):
        return int(round(lo * (hi / lo) ** rng.random()))

    call = rng.choice(["linear", "layer", "step", "step", "layer", "convert"])
    if rng.random() < 0.5:
        shape = rng.choice([OPT, L3B, Q7B, L13B, Q14B])
    else:   # other widths: odd numbers of quantisation groups, now and then a last group that is not full
        hidden = 128 * rng.randint(12, 40) + (64 if rng.random() < 0.125 else 0)
        q = 128 * rng.randint(12, 40)
        kv = rng.choice([q, 128 * rng.randint(2, 12)])
        inter = 128 * rng.randint(32, 136)
        shape = (hidden, q, kv, inter, rng.choice([16, 40, 64, 128, 256]), rng.random() < 0.3)
    out = rng.choice(["fp16", "fp16", "fp32"])
    alpha = 1.0 if rng.random() < 0.75 else 0.5
    share = 1.0 if rng.random() < 0.75 else 0.5
    if call == "convert":
        return _case(call, 0, shape)
    if call == "linear":
        return _case(call, loguni(1, 512), shape, out=out)
    if call == "step":
        return _case(call, loguni(1, 128), shape, layers=rng.randint(2, 4), out=out, alpha=alpha, share=share)
    return _case(call, loguni(1, 4096), shape, out=out, alpha=alpha, share=share)


class _Attn(nn.Module):
    def __init__(self, c, lin):
        super().__init__()
        self.q_proj = lin(c["hidden"], c["q"], c["bias"])
        self.k_proj = lin(c["hidden"], c["kv"], c["bias"])
        self.v_proj = lin(c["hidden"], c["kv"], c["bias"])
        self.o_proj = lin(c["q"], c["hidden"], False)


class _Mlp(nn.Module):
    def __init__(self, c, lin):
        super().__init__()
        self.gate_proj = lin(c["hidden"], c["inter"], False)
        self.up_proj = lin(c["hidden"], c["inter"], False)
        self.down_proj = lin(c["inter"], c["hidden"], False)


class _Layer(nn.Module):
    def __init__(self, c, lin):
        super().__init__()
        self.self_attn = _Attn(c, lin)
        self.mlp = _Mlp(c, lin)


class _Model(nn.Module):
    def __init__(self, c, lin):
        super().__init__()
        self.model = nn.Module()
        self.model.layers = nn.ModuleList([_Layer(c, lin) for _ in range(c["layers"])])


def _float_linear(gen):
    """An fp16 nn.Linear with N(0, 0.02) weights, drawn on the device."""
    def make(ic, oc, bias):
        lin = nn.Linear(ic, oc, bias=bias, device="meta", dtype=torch.float16)
        lin.weight = nn.Parameter(torch.randn(oc, ic, generator=gen, device="cuda", dtype=torch.float16) * 0.02, requires_grad=False)
        if bias:
            lin.bias = nn.Parameter(torch.randn(oc, generator=gen, device="cuda", dtype=torch.float16) * 0.1, requires_grad=False)
        return lin
    return make


def _factors(c, gen):
    """Correction factors and the map from weights to right factors, in the key scheme that the patchers read."""
    def fac(rows, cols):
        return torch.randn(rows, cols, generator=gen, device="cuda", dtype=torch.float16) * 0.01

    shared, bmap, keys, r = {}, {}, [], c["rank"]
    for li in range(c["layers"]):
        at = f"model.layers.{li}"
        for key, parent, ic, members in (
                (f"layer{li}_qkv", "self_attn", c["hidden"], (("q_proj", c["q"]), ("k_proj", c["kv"]), ("v_proj", c["kv"]))),
                (f"layer{li}_mlp", "mlp", c["hidden"], (("gate_proj", c["inter"]), ("up_proj", c["inter"])))):
            shared[f"{key}.B_shared"] = fac(r, ic)
            keys.append(key)
            for name, oc in members:
                shared[f"{key}.{name}.A"] = fac(oc, r)
                bmap[f"{at}.{parent}.{name}.weight"] = f"{key}.B_shared"
        for mod, ic in ((f"{at}.self_attn.o_proj", c["q"]), (f"{at}.mlp.down_proj", c["inter"])):
            shared[f"{mod}.A"], shared[f"{mod}.B"] = fac(c["hidden"], r), fac(r, ic)
            keys.append(mod)
            bmap[f"{mod}.weight"] = f"{mod}.B"
    return shared, bmap, keys


def _enabled(c):
    """How many of the (layer, group) pairs are corrected: the same number for every seed."""
    return int(round(c["share"] * 4 * c["layers"]))


def _mask(c):
    """Which of them, by position in model order."""
    n = 4 * c["layers"]
    on = set(random.Random(1).sample(range(n), _enabled(c)))
    return [i in on for i in range(n)]


def _forward(layers, x):
    outs = []
    for layer in layers:
        a, f = layer.self_attn, layer.mlp
        outs += [a.q_proj(x["hidden"]), a.k_proj(x["hidden"]), a.v_proj(x["hidden"]), a.o_proj(x["attn"]),
                 f.gate_proj(x["hidden"]), f.up_proj(x["hidden"]), f.down_proj(x["inter"])]
    return outs


def prepare(case, seed):
    c = case
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if c["call"] == "convert":
        model = _Model(c, _float_linear(gen))
        return {"call": "convert", "linears": [m for m in model.modules() if isinstance(m, nn.Linear)]}

    def act(cols):
        return torch.randn(c["m"], cols, generator=gen, device="cuda", dtype=torch.float16)

    before = os.environ.get("W4A16_KERNEL_OUT_DTYPE")   # read when a module is built
    os.environ["W4A16_KERNEL_OUT_DTYPE"] = c["out"]
    try:
        make = _float_linear(gen)

        def quantised(ic, oc, bias):
            return CudaW4A16Linear.from_float(make(ic, oc, bias), GROUP)

        if c["call"] == "linear":
            return {"call": "linear", "lin": quantised(c["hidden"], c["q"], c["bias"]), "x": act(c["hidden"])}
        model = _Model(c, quantised)
    finally:
        if before is None:
            del os.environ["W4A16_KERNEL_OUT_DTYPE"]
        else:
            os.environ["W4A16_KERNEL_OUT_DTYPE"] = before
    shared, bmap, keys = _factors(c, gen)
    order = [k for li in range(c["layers"]) for k in (f"layer{li}_qkv", f"model.layers.{li}.self_attn.o_proj", f"layer{li}_mlp",
                                                      f"model.layers.{li}.mlp.down_proj")]
    on = {k for k, use in zip(order, _mask(c)) if use}
    assert set(order) == set(keys)
    patch_svd_correction_wrappers_cumulative(model, shared, bmap, on, alpha_svd=c["alpha"])
    x = {"hidden": act(c["hidden"]), "attn": act(c["q"]), "inter": act(c["inter"])}
    state = {"call": c["call"], "model": model, "layers": list(model.model.layers), "x": x}
    if c["call"] == "step":
        with torch.no_grad():
            for _ in range(2):     # plans and workspaces, and every launch knows its successor
                _forward(state["layers"], x)
            torch.cuda.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                state["outs"] = _forward(state["layers"], x)
        state["graph"] = graph
    return state


def run(state):
    call = state["call"]
    with torch.no_grad():
        if call == "linear":
            return state["lin"](state["x"])
        if call == "layer":
            return _forward(state["layers"], state["x"])
        if call == "step":
            state["graph"].replay()
            return state["outs"]
        mods = [CudaW4A16Linear.from_float(lin, GROUP) for lin in state["linears"]]
        return [(m.qweight_i32, m.qzeros_i32, m.scales_f16) for m in mods]


def _linears(c):
    """(input columns, output columns of the members, corrected) of every group."""
    if c["call"] == "linear":
        return [(c["hidden"], [c["q"]], False)]
    groups = [(c["hidden"], [c["q"], c["kv"], c["kv"]]), (c["q"], [c["hidden"]]), (c["hidden"], [c["inter"]] * 2),
              (c["inter"], [c["hidden"]])]
    return [(ic, ocs, on) for (ic, ocs), on in zip(groups * c["layers"], _mask(c))]


def work(case):
    c, m, r = case, case["m"], case["rank"]
    osz = 4 if c["out"] == "fp32" else 2
    nbytes = flops = 0
    for ic, ocs, on in _linears(c):
        groups = -(-ic // GROUP)
        packed = groups * (GROUP // 2) + groups * 2 + -(-groups // 8) * 4
        for oc in ocs:
            if c["call"] == "convert":
                nbytes += oc * (ic * 2 + packed)
                continue
            nbytes += oc * packed + m * oc * osz + (oc * r * 2 if on else 0)
            flops += 2 * m * oc * ic + (2 * m * oc * r if on else 0)
        if c["call"] != "convert":
            nbytes += m * ic * 2 + (r * ic * 2 if on else 0)
            flops += 2 * m * r * ic if on else 0
    if c["call"] == "convert":
        flops = 0
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # codes, zero points and scales are the same bits whoever computes them in fp16
    if case["call"] == "convert":
        return "exact"
    # Four times what the outputs are off from the same product in 64 bits (2-norms).  fp16 outputs: 2.1e-4, the rounding
    # of the output, and 2.8e-4 where the weights are rounded to fp16 before the product as well, as the reference rounds
    # them (more than 8 tokens).  fp32 outputs: 1.9e-4 from those weights; 4.7e-6 for up to 8 tokens, where the codes
    # enter the product exactly and only the sums and r, an fp16 value, are rounded.
    if case["m"] <= 8:
        return {"rel": 2e-5 if case["out"] == "fp32" else 8e-4}
    return {"rel": 1.1e-3}
