"""Workloads of the MoE feed-forward path, as a serving program drives it through ``mference_b200.moe``.

Two layer families, with the shapes of this repository's configurations:

  q   hidden 2048, intermediate 512, 256 experts top-8 + 1 shared, 4-bit codes, softmax router
  v   hidden 4096, intermediate 2048, 256 experts top-6 + 1 shared, 2-bit routed and 4-bit shared codes, sqrt-softplus
      router with a selection bias and the SwiGLU clamp; ``gate_group`` 32 is that family's own conversion (gate_proj
      with one scale per 32 elements), 64 the plain one

and three ways to call them:

  layers   ``encode_layer`` once per layer on that layer's own rows: decode steps with attention between the layers
  stack    all layers of a decode step in one call: ``encode_stack`` carries one residual stream through the layers,
           ``encode_stack_rows`` gives every layer the rows of its own micro-batch
  prefill  ``encode_layer_prefill``: a block of prompt rows, or a packed mix of prompt chunks and decode rows

Options met in real model files: activations bf16 or fp16, scales fp16 or bf16, the bf16 gate or the INT8 affine gate
with a sigmoid-gated shared expert (``gate`` = "int8"), routing skewed over the experts (``zipf``).

Weights are zero-mean (bias = minus half the code range times the scale, as min-max quantisation of real weights gives)
and scaled so that hidden activations are of order one and a layer adds about a fifth of the residual's size, as in a
trained model; activations are N(0,1) residual rows.
"""
from __future__ import annotations

import math

import torch

from mference_b200 import _lib as L
from mference_b200.moe import MoE, MoELayerWeights, expert_layout

FAMILIES = {
    "q": dict(d=2048, f=512, experts=256, top_k=8, bits=4, shared_bits=4),
    "v": dict(d=4096, f=2048, experts=256, top_k=6, bits=2, shared_bits=4),
}


def _case(name=None, *, call, family="q", tokens, layers=1, x="bf16", scales="f16", gate="bf16", gate_group=64, chained=False,
          zipf=False):
    case = dict(call=call, family=family, tokens=tokens, layers=layers, x=x, scales=scales, gate=gate, gate_group=gate_group,
                chained=chained, zipf=zipf)
    return case if name is None else dict(case, name=name)


def listed():
    return [
        # one user's decode step, layer by layer with attention in between: the smallest calls there are
        _case("layers q 1 row", call="layers", tokens=1, layers=4),
        # the same for a few users of a model file with the INT8 gate, the gated shared expert and bf16 scales
        _case("layers q int8 gate 5 rows", call="layers", tokens=5, layers=4, x="f16", scales="bf16", gate="int8"),
        # decode of the 2-bit family, one user
        _case("layers v 1 row", call="layers", family="v", tokens=1, layers=2, gate_group=32),
        # ... and a small odd batch of users
        _case("layers v 13 rows", call="layers", family="v", tokens=13, layers=2),
        # fused decode step, one user, the residual stream carried through the layers
        _case("stack q 1 row", call="stack", tokens=1, layers=8, chained=True),
        # fused decode step, small and full batch of users
        _case("stack q 8 rows", call="stack", tokens=8, layers=8),
        _case("stack q 64 rows", call="stack", tokens=64, layers=8),
        # a short prompt of odd length
        _case("prefill q 203 rows", call="prefill", tokens=203, x="f16", scales="bf16"),
        # a full prompt chunk with a skewed router
        _case("prefill q 4096 rows zipf", call="prefill", tokens=4096, zipf=True),
        # prompt chunks of the 2-bit family, in both conversions
        _case("prefill v 2048 rows", call="prefill", family="v", tokens=2048),
        _case("prefill v 640 rows gate32", call="prefill", family="v", tokens=640, gate_group=32),
        # continuous batching: 48 sequences, each one decode row and prompt chunks of 256, 512 and 1024 rows
        _case("prefill q 86064 rows", call="prefill", tokens=48 * (1 + 256 + 512 + 1024)),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    family = rng.choice(("q", "q", "v"))
    call = rng.choice(("layers", "stack", "prefill") if family == "q" else ("layers", "prefill"))
    dtypes = dict(x=rng.choice(("bf16", "f16")), scales=rng.choice(("f16", "bf16")))
    if call == "prefill":
        if family == "v":
            group = rng.choice((32, 64))
            return _case(call=call, family=family, tokens=_log_int(rng, 65, 4096 if group == 64 else 640), gate_group=group, **dtypes)
        return _case(call=call, tokens=_log_int(rng, 65, 60000), zipf=rng.random() < 0.4, **dtypes)
    tokens = _log_int(rng, 1, 64)
    if family == "v":
        return _case(call=call, family=family, tokens=_log_int(rng, 1, 32), layers=rng.randint(1, 2), gate_group=rng.choice((32, 64)), **dtypes)
    if call == "stack":
        return _case(call=call, tokens=tokens, layers=rng.randint(2, 8), chained=tokens == 1, **dtypes)
    return _case(call=call, tokens=tokens, layers=rng.randint(2, 6), gate=rng.choice(("bf16", "int8")), **dtypes)


# ------------------------------------------------------------------------------------------------- inputs

_TORCH = {"bf16": torch.bfloat16, "f16": torch.float16}
_MFB = {"bf16": L.DT_BF16, "f16": L.DT_F16}


def _normal(gen, shape, std, dtype):
    return (torch.randn(shape, generator=gen, device="cuda") * std).to(dtype)


def _expert_slab(gen, n, bits, d, f, scale_dtype, gate_group):
    """`n` expert blobs: uniform codes, positive scales, biases that centre the weights."""
    off, blob = expert_layout(bits, d, f, gate_group)
    stride = (blob + 255) // 256 * 256
    slab = torch.randint(0, 256, (n, stride), generator=gen, device="cuda", dtype=torch.uint8)
    top = 2 ** bits - 1
    code_std = math.sqrt(((top + 1) ** 2 - 1) / 12)
    for m in ("gate", "up", "down"):
        k = f if m == "down" else d
        per = gate_group if m == "gate" else 64
        count = d * f // per
        spread = torch.rand((n, count), generator=gen, device="cuda")
        gain = 0.25 if m == "down" else 1.0
        scale = ((0.5 + spread) * (gain / (code_std * math.sqrt(k)))).to(scale_dtype)
        s0, b0 = getattr(off, m + "_s"), getattr(off, m + "_b")
        slab[:, s0:s0 + 2 * count] = scale.view(torch.uint8)
        slab[:, b0:b0 + 2 * count] = (scale.float() * (-top / 2)).to(scale_dtype).view(torch.uint8)
    return slab, stride, off


def _int8_rows(gen, rows, cols, std):
    """Affine INT8 rows with one bf16 scale and bias per 64 elements, zero-mean, standard deviation `std`."""
    codes = torch.randint(0, 256, (rows, cols), generator=gen, device="cuda", dtype=torch.uint8)
    scale = ((0.5 + torch.rand((rows, cols // 64), generator=gen, device="cuda")) * (std / 73.9)).to(torch.bfloat16)
    return codes, scale, (scale.float() * -127.5).to(torch.bfloat16)


def _layer(gen, case):
    fam = FAMILIES[case["family"]]
    d, f, E = fam["d"], fam["f"], fam["experts"]
    sdt = _TORCH[case["scales"]]
    slab, stride, off = _expert_slab(gen, E, fam["bits"], d, f, sdt, case["gate_group"])
    shared, _, shared_off = _expert_slab(gen, 1, fam["shared_bits"], d, f, sdt, 64)
    w = MoELayerWeights(router_w=None, pool=slab.view(-1), slot_stride=stride, routed_off=off, shared_blob=shared.view(-1),
                        shared_off=shared_off, norm_w=(1.0 + _normal(gen, (d,), 0.1, torch.float32)).to(torch.bfloat16),
                        gate_group_size=case["gate_group"])
    if case["gate"] == "int8":
        w.router_w, w.router_scales, w.router_biases = _int8_rows(gen, E, d, 0.06)
        w.shared_gate_w, w.shared_gate_s, w.shared_gate_b = (t.view(-1) for t in _int8_rows(gen, 1, d, 0.02))
    else:
        w.router_w = _normal(gen, (E, d), 0.02 if case["zipf"] else 0.06, torch.bfloat16)
    if case["zipf"]:
        rank = torch.randperm(E, generator=gen, device="cuda").float() + 1.0
        w.logit_bias = -1.1 * torch.log(rank)
    if case["family"] == "v":
        w.correction_bias = _normal(gen, (E,), 0.05, torch.float32)
    return w


class _State:
    pass


def prepare(case, seed):
    fam = FAMILIES[case["family"]]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    s = _State()
    s.case = case
    T, NL, d = case["tokens"], case["layers"], fam["d"]
    v = case["family"] == "v"
    s.moe = MoE(d, fam["f"], fam["experts"], fam["top_k"], bits=fam["bits"], shared_bits=fam["shared_bits"],
                scale_dtype=_MFB[case["scales"]], x_dtype=_MFB[case["x"]],
                router_mode=L.ROUTER_SQRTSOFTPLUS if v else L.ROUTER_SOFTMAX_TOPK, swiglu_limit=10.0 if v else 0.0,
                route_scale=1.5 if v else 1.0, max_tokens=T, tensor_core_prefill=case["call"] == "prefill", max_layers=NL)
    s.layers = [_layer(gen, case) for _ in range(NL)]
    rows = 1 if case["chained"] else NL
    s.x = _normal(gen, (rows, T, d), 1.0, _TORCH[case["x"]])
    s.out = torch.empty_like(s.x)
    s.stack = s.moe.make_stack(s.layers) if case["call"] == "stack" else None
    return s


def run(s):
    case = s.case
    if case["call"] == "stack":
        s.out.copy_(s.x)          # the call updates its rows in place
        if case["chained"]:
            s.moe.encode_stack(s.stack, s.out[0])
        else:
            s.moe.encode_stack_rows(s.stack, s.out)
    elif case["call"] == "layers":
        for l, w in enumerate(s.layers):
            s.moe.encode_layer(w, s.x[l], s.out[l])
    else:
        for l, w in enumerate(s.layers):
            s.moe.encode_layer_prefill(w, s.x[l], s.out[l])
    return s.out


# ------------------------------------------------------------------------------------------------- what a pass needs

def work(case):
    """Bytes: every distinct expert that the rows are expected to pick, the shared expert and the gate once per layer, the
    rows in and out.  Operations: two per weight and row of the experts and the gate."""
    fam = FAMILIES[case["family"]]
    d, f, E, K, T, NL = fam["d"], fam["f"], fam["experts"], fam["top_k"], case["tokens"], case["layers"]
    _, blob = expert_layout(fam["bits"], d, f, case["gate_group"])
    _, shared = expert_layout(fam["shared_bits"], d, f)
    distinct = E * (1.0 - (1.0 - K / E) ** T)
    if case["zipf"]:
        distinct = min(distinct, E / 2)      # half of the experts draw no row at all under the skewed gate
    gate = E * d * (1 if case["gate"] == "int8" else 2)
    moved = distinct * blob + shared + gate + 2 * T * d * 2
    flops = 2 * 3 * d * f * T * (K + 1) + 2 * T * d * E
    return {"bytes": NL * moved, "flops": NL * flops}


def tolerance(case):
    # fp16 hidden activations, outputs rounded to bf16 (2^-9) or fp16: two correct implementations differ by a rounding
    # step here and there.  Carried through the layers, an element that rounds the other way can also exchange the last of
    # a token's experts for one with nearly the same logit and a small weight.
    if case["chained"]:
        return {"rel": 1.5e-2, "max": 0.1}
    return {"rel": 2e-3, "max": 0.03}
