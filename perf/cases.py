"""Workloads of the MoE layer library: what a user's program calls, over the sizes it is used at.

A case is one pass of a program that keeps its quantised expert weights, a workspace and an output buffer, and is
handed new activations. Kinds of pass:

  layer    route indices given: quantise the bf16 activations dynamically (where the mode wants it), run the layer into
           d [T, k, H] (ops.moe_forward)
  block    the whole MoE block: router, quantisation inside the gather, layer, weighted combine (ops.moe_block)
  nvfp4    the layer on NVFP4 operands: quantise with calibrated global scales, run (ops.moe_forward_nvfp4)
  weights  load time: bf16 expert weights -> e4m3 with 128x128 block scales (ops.per_block_cast_to_fp8)

Shapes: Mixtral-8x7B (H 4096, I 14336, 8 experts, top 2), DeepSeek-V3 routed experts (H 7168, I 2048, 256 experts, top 8)
and one of eight ranks' share of them (32 experts), Qwen-MoE (H 2048, I 768, 128 experts, top 8), the wide bf16 shape of
the reference's driver (H = I = 2880, 64 experts, top 3), and small odd models. Activations and router logits N(0, 1),
weights N(0, 0.02).
"""
import math

import torch

from dqmoe_b200 import ops

MODES = {"bf16": ops.QUANT_NONE, "tensor": ops.QUANT_FP8_TENSOR, "channel": ops.QUANT_FP8_CHANNEL,
         "block": ops.QUANT_FP8_BLOCK, "mx": ops.QUANT_FP8_MX}
MIXTRAL = dict(H=4096, I=14336, E=8, k=2)
DEEPSEEK = dict(H=7168, I=2048, E=256, k=8)
DEEPSEEK_RANK = dict(H=7168, I=2048, E=32, k=8)
QWEN = dict(H=2048, I=768, E=128, k=8)
WIDE = dict(H=2880, I=2880, E=64, k=3)
MAX_FLOPS = 5.7e12  # of FP8 work; the unquantised path counts double


def _case(kind, quant, T, shape, *, scoring="softmax", zipf=False, shared=0, bias=False):
    return dict(kind=kind, quant=quant, T=T, scoring=scoring, zipf=zipf, shared=shared, bias=bias, **shape)


def listed():
    return [
        # one user's next token, unquantised model: the smallest call of the decode path
        dict(name="decode_bf16_1", **_case("layer", "bf16", 1, MIXTRAL)),
        # a small decode batch on per-tensor FP8 weights: memory-bound
        dict(name="decode_tensor_16", **_case("layer", "tensor", 16, MIXTRAL)),
        # a few tokens through a small model's whole block: launches and latency
        dict(name="small_block_5", **_case("block", "block", 5, dict(H=1024, I=2048, E=8, k=2))),
        # serving batch on one rank's share of a 256-expert model, with its shared expert
        dict(name="serve_block_96", **_case("block", "block", 96, DEEPSEEK_RANK, scoring="sigmoid", shared=1)),
        # chunked prefill of odd length, per-tensor FP8 with expert biases
        dict(name="chunk_tensor_777", **_case("layer", "tensor", 777, MIXTRAL, bias=True)),
        # prefill, block-scaled FP8: the library's headline configuration
        dict(name="prefill_block_4096", **_case("layer", "block", 4096, MIXTRAL)),
        # the same model in MXFP8, odd length, whole block
        dict(name="prefill_mx_2049", **_case("block", "mx", 2049, MIXTRAL)),
        # the same model in NVFP4
        dict(name="prefill_nvfp4_4096", **_case("nvfp4", "nvfp4", 4096, MIXTRAL)),
        # many small experts with skewed routing, per-token / per-channel scales: short reductions, ragged experts
        dict(name="prefill_channel_16384", **_case("layer", "channel", 16384, QWEN, zipf=True)),
        # unquantised prefill / training-style forward at the reference driver's own size
        dict(name="prefill_bf16_16384", **_case("layer", "bf16", 16384, WIDE)),
        # the largest: prefill of a 256-expert model on one GPU, whole block
        dict(name="prefill_block_8192", **_case("block", "block", 8192, DEEPSEEK, scoring="sigmoid")),
        # loading a checkpoint: one projection of every expert to block-scaled FP8
        dict(name="load_block_weights", kind="weights", E=8, rows=4096, cols=14336),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["decode", "small", "serve", "prefill", "prefill", "weights"])
    if family == "weights":
        return dict(kind="weights", E=_log_int(rng, 1, 16), rows=8 * rng.randint(64, 600), cols=8 * rng.randint(64, 1000))
    if family == "small":  # odd small models: every mode that takes rows of 64 elements, partial 128-wide blocks among them
        quant = rng.choice(["bf16", "tensor", "channel", "block", "mx"])
        unit = 128 if quant == "mx" else 64
        E = rng.randint(3, 20)
        shape = dict(H=unit * rng.randint(512 // unit, 2048 // unit), I=unit * rng.randint(512 // unit, 3072 // unit), E=E,
                     k=rng.randint(1, min(4, E)))
        return _case(rng.choice(["layer", "block"]), quant, _log_int(rng, 1, 300), shape)
    if family == "decode":
        return _case("layer", rng.choice(["bf16", "tensor"]), _log_int(rng, 1, 256), MIXTRAL)
    if family == "serve":
        return _case("block", rng.choice(["block", "block", "mx"]), _log_int(rng, 16, 512), DEEPSEEK_RANK, scoring="sigmoid",
                     shared=rng.randint(0, 1))
    quant = rng.choice(["block", "block", "tensor", "channel", "mx", "nvfp4", "bf16"])
    shapes = [MIXTRAL, DEEPSEEK_RANK, QWEN] + ([] if quant == "nvfp4" else [DEEPSEEK]) + ([] if quant in ("mx", "nvfp4") else [WIDE])
    shape = rng.choice(shapes)
    if quant == "bf16" and shape is DEEPSEEK:
        shape = DEEPSEEK_RANK
    per_token = 6.0 * shape["k"] * shape["H"] * shape["I"] * (2 if quant == "bf16" else 1)
    T = _log_int(rng, 300, min(16384, MAX_FLOPS / per_token))
    kind = "nvfp4" if quant == "nvfp4" else rng.choice(["layer", "block"])
    return _case(kind, quant, T, shape, scoring=rng.choice(["softmax", "sigmoid"]), zipf=rng.random() < 0.3,
                 bias=kind == "layer" and rng.random() < 0.2)


# ---------------------------------------------------------------------------------------------------- inputs

def _weights(g, E, rows, cols, cast):
    """cast() of E experts' N(0, 0.02) weights, built a few experts at a time; a tuple of tensors over all experts."""
    step = max(1, (1 << 27) // (rows * cols))
    parts = []
    for e in range(0, E, step):
        n = min(step, E - e)
        w = torch.randn(n, rows, cols, generator=g, device="cuda", dtype=torch.bfloat16).mul_(0.02)
        parts.append(cast(w))
    if len(parts) == 1:
        return parts[0]
    return tuple(torch.cat([p[i].view(torch.uint8) if p[i].dtype == ops.FP8 else p[i] for p in parts]).view(parts[0][i].dtype)
                 for i in range(len(parts[0])))


def _cast_channel(w):
    q, s = ops.per_channel_cast_to_fp8(w)
    return q, s.reshape(-1)


_CASTS = {"bf16": lambda w: (w,), "tensor": lambda w: ops.per_tensor_cast_to_fp8(w, per_expert=True), "channel": _cast_channel,
          "block": ops.per_block_cast_to_fp8, "mx": ops.mx_cast_weights_to_fp8, "nvfp4": ops.nvfp4_cast_weights}


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    if case["kind"] == "weights":
        return dict(case=case, w=torch.randn(case["E"], case["rows"], case["cols"], generator=g, device="cuda", dtype=torch.bfloat16).mul_(0.02))
    T, H, I, E, k, quant = case["T"], case["H"], case["I"], case["E"], case["k"], case["quant"]
    E_all = E + case["shared"]
    b = _weights(g, E_all, 2 * I, H, _CASTS[quant])
    b1 = _weights(g, E_all, H, I, _CASTS[quant])
    x = torch.randn(T, H, generator=g, device="cuda", dtype=torch.bfloat16)
    logits = torch.randn(T, E, generator=g, device="cuda")
    if case["zipf"]:  # a few popular experts
        logits -= (1.1 * torch.log(torch.arange(1, E + 1, device="cuda")))[torch.randperm(E, generator=g, device="cuda")]
    st = dict(case=case, x=x, logits=logits, b=b, b1=b1)
    if case["kind"] == "block":
        need = ops._lib.load().dqmoe_moe_block_workspace_bytes(T, H, I, E_all, k + case["shared"], MODES[quant])
        st["workspace"] = torch.empty(need, dtype=torch.uint8, device="cuda")
        return st
    st["m_indices"] = torch.topk(logits, k, dim=1).indices.to(torch.int32)
    st["d"] = torch.empty(T, k, H, dtype=torch.bfloat16, device="cuda")
    mode = 4096 if quant == "nvfp4" else MODES[quant]
    st["workspace"] = torch.empty(ops.moe_workspace_bytes(T, H, I, E, k, mode), dtype=torch.uint8, device="cuda")
    if quant == "nvfp4":  # calibrated global scales of the activations and of the intermediate
        st["x_g"] = torch.full((1,), 6.0 / 2688.0, device="cuda")
        st["act_g"] = torch.full((1,), 16.0 / 2688.0, device="cuda")
    st["bias1"] = st["bias2"] = None
    if case["bias"]:
        st["bias1"] = torch.randn(E, 2 * I, generator=g, device="cuda") * 0.1
        st["bias2"] = torch.randn(E, H, generator=g, device="cuda") * 0.1
    return st


# ---------------------------------------------------------------------------------------------------- one pass

def run(st):
    case = st["case"]
    if case["kind"] == "weights":
        return ops.per_block_cast_to_fp8(st["w"])
    x, b, b1 = st["x"], st["b"], st["b1"]
    quant = case["quant"]
    if case["kind"] == "block":
        bs, b1s = (None, None) if quant == "bf16" else (b[1], b1[1])
        return ops.moe_block(x, st["logits"], b[0], bs, b1[0], b1s, case["k"], scoring=case["scoring"], quant_mode=MODES[quant],
                             workspace=st["workspace"], n_shared=case["shared"])
    if quant == "nvfp4":
        q, s = ops.nvfp4_cast(x, st["x_g"])
        ops.moe_forward_nvfp4(q, s, st["x_g"], *b, *b1, st["act_g"], st["d"], st["m_indices"], st["workspace"])
        return st["d"]
    bs, b1s = (None, None) if quant == "bf16" else (b[1], b1[1])
    if quant == "bf16":
        q, s = x, None
    elif quant == "tensor":
        q, s = ops.per_tensor_cast_to_fp8(x)
    elif quant == "channel":
        q, s = ops.per_token_cast_to_fp8(x)
    elif quant == "block":
        q, s = ops.per_token_block_cast_to_fp8(x)
    else:
        q, s = ops.mx_cast_to_fp8(x)
    ops.moe_forward(q, s, b[0], bs, b1[0], b1s, st["d"], st["m_indices"], st["workspace"], MODES[quant], bias1=st["bias1"], bias2=st["bias2"])
    return st["d"]


def work(case):
    if case["kind"] == "weights":
        n = case["E"] * case["rows"] * case["cols"]
        return {"bytes": 3 * n, "flops": 0}
    T, H, I, E, k = case["T"], case["H"], case["I"], case["E"], case["k"]
    # experts that T tokens with k choices are expected to hit
    hit = E * (1.0 - (1.0 - k / E) ** T) + case["shared"]
    per_weight = {"bf16": 2.0, "nvfp4": 0.5 + 1 / 16, "mx": 1.0 + 1 / 32}.get(case["quant"], 1.0)
    rows_out = T if case["kind"] == "block" else T * k
    routing = 4 * T * (E if case["kind"] == "block" else k)
    return {"bytes": hit * 3 * H * I * per_weight + 2 * T * H + 2 * rows_out * H + routing,
            "flops": 6.0 * T * (k + case["shared"]) * H * I}


def tolerance(case):
    # Four times what was measured against the same rounding points evaluated in 64 bits, and between two orders of the
    # first reduction: 7.9e-4 to 9.6e-4 for bf16 operands (roundings of the intermediate and the output flip), 1.0e-5 to
    # 3.0e-4 for the FP8 modes. NVFP4's sums came out the same in either order, but a bf16 rounding that flips before the
    # re-quantisation moves an e2m1 code by up to a quarter of its value, twice the step of e4m3.
    if case["kind"] == "weights":
        return "exact"
    return {"rel": {"bf16": 4e-3, "nvfp4": 2.4e-3}.get(case["quant"], 1.2e-3)}
