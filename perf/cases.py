"""The work that users of the weight-only GEMM have it do, as cases that can be timed and compared.

A case is one of three kinds:

* ``linear``: one pass through a set of weight-only linear layers (one layer, or the linear layers of
  one transformer block) through ``torch.ops.trtllm``. ``shapes`` names the layers, "KxN" each; the
  layers of a pass are independent calls on activations that are already on the GPU.
* ``experts``: the same GEMM over 3-D weights, ``ops.moe_gemm``, the rows sorted by expert.
* ``quantize``: weights of a layer, on the GPU in the checkpoint's type, to the integers and scales
  that the GEMM takes (``quantize.symmetric_quantize_last_axis_of_batched_matrix_cuda``).

Values are those of the path's own problems: integer weights over their whole range, scales
~U(0.001, 0.02), scale-multiplied zeros ~U(-0.1, 0.1), activations and bias ~N(0, 1), pre-quant scales
~U(0.5, 1.5); float weights ~N(0, 0.02).
"""
import math

import torch

import tensorrt_llm_b200 as pkg
import tensorrt_llm_b200.torch_ops  # noqa: F401  (registers torch.ops.trtllm)
from tensorrt_llm_b200 import ops, quantize

DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16, "fp32": torch.float32}
SIZES = {"fp16": 2, "bf16": 2, "fp32": 4}

# Linear layers of one block: Llama-3-8B (q, k, v, o, gate, up, down) on one GPU, and Llama-3-70B (fused
# qkv, o, fused gate and up, down) on one GPU and as one rank of eight holds it.
BLOCK_8B = "4096x4096,4096x1024,4096x1024,4096x4096,4096x14336,4096x14336,14336x4096"
BLOCK_70B = "8192x10240,8192x8192,8192x57344,28672x8192"
BLOCK_70B_TP8 = "8192x1280,1024x8192,8192x7168,3584x8192"

MOST_FLOPS = 2 * 4096 * 14336 * 4096
MOST_WEIGHT = 4096 * 57344  # elements


def linear(name, shapes, m, bits, group, dtype, zeros=False, bias=False, prequant=False):
    case = {"kind": "linear", "shapes": shapes, "m": m, "bits": bits, "group": group, "dtype": dtype,
            "zeros": zeros, "bias": bias, "prequant": prequant}
    return dict(case, name=name) if name else case


def listed():
    return [
        # the smallest layer there is in one-token decode (a k or v projection): what a call costs
        linear("kv_m1", "4096x1024", 1, 4, 128, "bf16", zeros=True),
        # one token through one block of an AWQ checkpoint: seven calls, 109 MB of weights
        linear("block8b_m1_awq", BLOCK_8B, 1, 4, 128, "bf16", zeros=True, prequant=True),
        # a few sequences through one block of a large model on one GPU: 428 MB of weights
        linear("block70b_m4", BLOCK_70B, 4, 4, 128, "bf16", zeros=True),
        # eight sequences, GPTQ with 64-wide groups: a down projection
        linear("down_m8_g64", "14336x4096", 8, 4, 64, "fp16", zeros=True),
        # sixteen sequences, int8 with one scale per column
        linear("attn_m16_w8", "4096x4096", 16, 8, 0, "fp16"),
        # a batch of 64 through one rank's share of a block
        linear("block70b_tp8_m64", BLOCK_70B_TP8, 64, 4, 128, "bf16", zeros=True),
        # an odd batch on a ragged layer, all options on
        linear("ragged_m37", "4160x3008", 37, 4, 64, "fp16", zeros=True, bias=True, prequant=True),
        # a large batch (or a short prompt), int8
        linear("gate_m256_w8", "4096x14336", 256, 8, 0, "bf16"),
        # a prompt of ordinary length through one block, its length no multiple of any tile
        linear("block8b_m777", BLOCK_8B, 777, 4, 128, "fp16", zeros=True, bias=True),
        # the longest prefill chunk
        linear("down_m4096", "14336x4096", 4096, 4, 128, "bf16", zeros=True),
        # a mixture of experts: 48 tokens, two experts each out of eight
        {"name": "experts8_m96", "kind": "experts", "experts": 8, "m": 96, "k": 4096, "n": 14336, "bits": 4, "group": 128,
         "dtype": "bf16", "zeros": True},
        # loading: a bf16 weight matrix to int4
        {"name": "quantize_gate", "kind": "quantize", "k": 4096, "n": 14336, "bits": 4, "dtype": "bf16"},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _multiple(rng, lo, hi, step):
    return max(step, int(round(_log(rng, lo, hi) / step)) * step)


def draw(rng):
    kind = rng.choices(("linear", "experts", "quantize"), (10, 1, 1))[0]
    bits = rng.choice((4, 4, 8))
    # the layout takes k in steps of 64 and n in steps of 64 (int4) or 32 (int8)
    n_step = 64 if bits == 4 else 32
    if kind == "quantize":
        k, n = _multiple(rng, 1024, 14336, 64), _multiple(rng, 1024, 14336, n_step)
        while k * n > MOST_WEIGHT // 3:
            k, n = _multiple(rng, 1024, 14336, 64), _multiple(rng, 1024, 14336, n_step)
        return {"kind": kind, "k": k, "n": n, "bits": bits, "dtype": rng.choice(("bf16", "fp16", "fp32"))}
    dtype = rng.choice(("bf16", "fp16"))
    group = rng.choice((128, 128, 64, 0)) if bits == 4 else rng.choice((0, 0, 128, 64))
    k_step = max(64, group)
    if kind == "experts":
        return {"kind": kind, "experts": rng.randint(4, 16), "m": int(_log(rng, 4, 512)),
                "k": _multiple(rng, 1024, 4096, k_step), "n": _multiple(rng, 1024, 8192, n_step), "bits": bits,
                "group": group, "dtype": dtype, "zeros": bool(group) and rng.random() < 0.5}
    while True:
        m = int(_log(rng, 1, 4097))
        k, n = _multiple(rng, 1024, 28672, k_step), _multiple(rng, 1024, 57344, n_step)
        if k * n * bits <= MOST_WEIGHT * 4 and 2 * m * k * n <= MOST_FLOPS:
            break
    options = [bool(group) and rng.random() < p for p in (0.6, 0.3, 0.3)]
    return linear(None, "%dx%d" % (k, n), m, bits, group, dtype, *options)


def _shapes(case):
    return [tuple(int(x) for x in s.split("x")) for s in case["shapes"].split(",")]


def _layer(g, lead, k, n, bits, group, dtype, zeros):
    """(weight, scales, zeros) of a layer, or of the experts of one (``lead`` = (experts,))."""
    def uniform(shape, lo, hi):
        return torch.rand(shape, generator=g, device="cuda").mul_(hi - lo).add_(lo).to(dtype)

    packed = torch.randint(-128, 128, lead + (k, n * bits // 8), dtype=torch.int8, generator=g, device="cuda")
    qt = torch.quint4x2 if bits == 4 else torch.int8
    if lead:
        weight = torch.stack([quantize.preprocess_weights_for_mixed_gemm_cuda(p, qt) for p in packed])
    else:
        weight = quantize.preprocess_weights_for_mixed_gemm_cuda(packed, qt)
    shape = lead + ((k // group, n) if group else (n,))
    return weight, uniform(shape, 0.001, 0.02), uniform(shape, -0.1, 0.1) if zeros else None


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    dtype = DTYPES[case["dtype"]]
    if case["kind"] == "quantize":
        w = torch.randn((case["k"], case["n"]), generator=g, device="cuda").mul_(0.02).to(dtype)
        return {"case": case, "weight": w, "type": torch.quint4x2 if case["bits"] == 4 else torch.int8}
    if case["kind"] == "experts":
        e, m = case["experts"], case["m"]
        weight, scales, zeros = _layer(g, (e,), case["k"], case["n"], case["bits"], case["group"], dtype, case["zeros"])
        act = torch.randn((m, case["k"]), generator=g, device="cuda").to(dtype)
        # routing: an uneven share of the rows for each expert, some perhaps without any
        share = torch.rand(e, generator=g, device="cuda").add_(0.1)
        pick = torch.multinomial(share, m, replacement=True, generator=g)
        first = [0] + torch.bincount(pick, minlength=e).cumsum(0).tolist()
        return {"case": case, "weight": weight, "scales": scales, "zeros": zeros, "act": act, "first": first}
    m, group = case["m"], case["group"]
    algo = (pkg.INT8_WEIGHT if case["bits"] == 8 else 0) | (pkg.ZERO if case["zeros"] else 0) \
        | (pkg.BIAS if case["bias"] else 0) | (pkg.PRE_QUANT_SCALE if case["prequant"] else 0)
    calls, acts = [], {}
    for k, n in _shapes(case):
        if k not in acts:
            acts[k] = torch.randn((m, k), generator=g, device="cuda").to(dtype)
        weight, scales, zeros = _layer(g, (), k, n, case["bits"], group, dtype, case["zeros"])
        bias = torch.randn((n,), generator=g, device="cuda").to(dtype) if case["bias"] else None
        ps = (torch.rand((k,), generator=g, device="cuda") + 0.5).to(dtype) if case["prequant"] else None
        if group:
            calls.append((acts[k], ps, weight, scales, zeros, bias, 1.0, algo, group, True))
        else:
            calls.append((acts[k], weight, scales, 1 if case["bits"] == 8 else 2, True))
    op = torch.ops.trtllm.weight_only_groupwise_quant_gemm if group else torch.ops.trtllm.weight_only_quant_gemm
    return {"case": case, "op": op, "calls": calls}


def run(state):
    case = state["case"]
    if case["kind"] == "linear":
        op = state["op"]
        return [op(*args) for args in state["calls"]]
    if case["kind"] == "experts":
        return ops.moe_gemm(state["act"], state["weight"], state["scales"], state["first"], weight_bits=case["bits"],
                            group_size=case["group"], zeros=state["zeros"], weights_static=True)
    return quantize.symmetric_quantize_last_axis_of_batched_matrix_cuda(state["weight"], state["type"])


def _gemm_work(m, k, n, case, weights):
    rows = k // case["group"] if case["group"] else 1
    constants = k * n * case["bits"] // 8 + rows * n * 2 * (2 if case["zeros"] else 1)
    constants += n * 2 * case.get("bias", False) + k * 2 * case.get("prequant", False)
    return constants * weights + m * n * 2, 2 * m * n * k


def work(case):
    if case["kind"] == "quantize":
        k, n = case["k"], case["n"]
        return {"bytes": k * n * (SIZES[case["dtype"]] + case["bits"] / 8) + n * SIZES[case["dtype"]], "flops": 4 * k * n}
    m = case["m"]
    if case["kind"] == "experts":
        # every expert that has rows is read; with few rows some have none
        used = min(case["experts"], m)
        by, fl = _gemm_work(m, case["k"], case["n"], case, used)
        return {"bytes": by + m * case["k"] * 2, "flops": fl}
    each = [_gemm_work(m, k, n, case, 1) for k, n in _shapes(case)]
    acts = sum(m * k * 2 for k in {k for k, _ in _shapes(case)})
    return {"bytes": sum(b for b, _ in each) + acts, "flops": sum(f for _, f in each)}


def tolerance(case):
    if case["kind"] == "quantize":
        return "exact"
    # The outputs are rounded to the activation type, and a weight may or may not be rounded to it before
    # the product; sums are 32-bit.
    return {"rel": 1e-3} if case["dtype"] == "fp16" else {"rel": 5e-3}
