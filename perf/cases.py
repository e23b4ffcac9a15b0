"""The work a user of this library has it do, as cases that can be timed and compared.

Four kinds of call, each through the package's public entry points:

* ``linear``  one product: ``QuantLinear(weight)(x)``, or ``ops.quant_matmul`` where a 16-bit result is asked for;
* ``layer``   the quantized linears of one decoder layer called one after the other: RMSNorm + q/k/v, the output
              projection, the feed-forward block;
* ``step``    a decoding step of a whole model, captured once and replayed with new hidden states (``DecodeGraph``);
* ``dequant`` a packed weight decoded to a dense one.

Weights are random blocks of the distributions in ``boostr_b200.synth``, activations N(0, 1).
"""
import math

import torch

from boostr_b200 import ops, synth
from boostr_b200.decode_graph import DecodeGraph
from boostr_b200.decode_stack import DecodeStack
from boostr_b200.format import QuantFormat
from boostr_b200.linear import QuantLinear

DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
K_QUANTS = ("Q2_K", "Q3_K", "Q4_K", "Q5_K", "Q6_K")
EPS = 1e-5

# The format of most linears of a layer, and of its v and down projections: the mixes that GGUF files come in.
MIXES = (("Q4_K", "Q6_K"), ("Q4_K", "Q6_K"), ("Q5_K", "Q6_K"), ("Q8_0", "Q8_0"), ("Q4_0", "Q4_0"), ("Q6_K", "Q6_K"), ("Q3_K", "Q5_K"),
         ("Q2_K", "Q3_K"), ("Q5_0", "Q5_0"))


def listed():
    return [
        # one token through one projection of the smallest format: latency
        dict(name="linear_q4_0_m1", kind="linear", fmt="Q4_0", m=1, k=4096, n=4096, act="f32", out="f32"),
        # a few sequences decoded together, 8-bit weights
        dict(name="linear_q8_0_m8", kind="linear", fmt="Q8_0", m=8, k=4096, n=11008, act="f32", out="f32"),
        # the logits of one token: the largest single weight of a model
        dict(name="lm_head_q6_k_m1", kind="linear", fmt="Q6_K", m=1, k=4096, n=128256, act="f32", out="f32"),
        # a short prompt (or a batch of odd size), a vocabulary slice of odd size, 16-bit activations
        dict(name="linear_q5_k_m37", kind="linear", fmt="Q5_K", m=37, k=5120, n=13825, act="bf16", out="f32"),
        # a prompt through the widest projection, 16-bit activations and results
        dict(name="prompt_q4_k_m512", kind="linear", fmt="Q4_K", m=512, k=4096, n=14336, act="bf16", out="bf16"),
        # one token through a layer, call by call, as a program without graphs decodes
        dict(name="layer_q4_k_m1", kind="layer", fmt="Q4_K", fmt_vd="Q6_K", m=1, hidden=4096, kv=1024, ffn=14336, act="f32"),
        # four tokens (a draft being verified) through a layer of a low-bit file
        dict(name="layer_q3_k_m4", kind="layer", fmt="Q3_K", fmt_vd="Q5_K", m=4, hidden=4096, kv=1024, ffn=14336, act="f32"),
        # a long prompt of odd length through a layer
        dict(name="layer_q4_k_m1999", kind="layer", fmt="Q4_K", fmt_vd="Q6_K", m=1999, hidden=4096, kv=1024, ffn=14336, act="bf16"),
        # a prompt through a layer of the smallest file there is
        dict(name="layer_q2_k_m512", kind="layer", fmt="Q2_K", fmt_vd="Q3_K", m=512, hidden=4096, kv=1024, ffn=14336, act="f32"),
        # the headline: one token through the whole model, as a graph
        dict(name="step_m1", kind="step", m=1, layers=32, hidden=4096, kv=1024, ffn=14336, vocab=128256),
        # sixteen sequences decoded together
        dict(name="step_m16", kind="step", m=16, layers=32, hidden=4096, kv=1024, ffn=14336, vocab=128256),
        # a layer's widest weight decoded for a dense matmul
        dict(name="dequant_q4_k_bf16", kind="dequant", fmt="Q4_K", n=14336, k=4096, out="bf16"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _rows(rng):
    """Single rows, small batches and prompts, a third each."""
    return rng.choice((1, _log(rng, 2, 63), _log(rng, 64, 2048)))


def _k(rng, fmt, lo, hi):
    """A multiple of 256, or for the formats with blocks of 32 now and then only of 32."""
    step = 32 if fmt not in K_QUANTS and rng.random() < 0.3 else 256
    return max(lo, _log(rng, lo, hi) // step * step)


def draw(rng):
    kind = rng.choice(("linear",) * 5 + ("layer",) * 3 + ("step",) * 2 + ("dequant",))
    if kind == "linear":
        fmt = rng.choice(("Q4_K", "Q4_K", "Q6_K", "Q6_K", "Q8_0", "Q8_0", "Q5_K", "Q4_0", "Q5_0", "Q3_K", "Q2_K"))
        m = _rows(rng)
        k = _k(rng, fmt, 1024, 14336)
        n = _log(rng, 512, 58720256 // k)
        if m <= 16 and rng.random() < 0.2:
            k, n = _k(rng, fmt, 2048, 4096), _log(rng, 32000, 128256)
        if fmt in ("Q2_K", "Q3_K"):
            m = min(m, rng.randint(256, 512))
        act = rng.choice(("f32", "f32", "bf16"))
        return dict(kind=kind, fmt=fmt, m=m, k=k, n=n if rng.random() < 0.4 else n // 64 * 64, act=act, out="bf16" if act == "bf16" and rng.random() < 0.5 else "f32")
    hidden = _log(rng, 1024, 4096) // 256 * 256
    ffn = min(14336, int(hidden * rng.uniform(2.6, 3.5)) // 256 * 256)
    kv = max(256, hidden // rng.choice((1, 4, 8)) // 64 * 64)
    if kind == "layer":
        fmt, fmt_vd = rng.choice(MIXES)
        m = _rows(rng)
        if fmt in ("Q2_K", "Q3_K"):
            m = min(m, rng.randint(256, 512))
        return dict(kind=kind, fmt=fmt, fmt_vd=fmt_vd, m=m, hidden=hidden, kv=kv, ffn=ffn, act=rng.choice(("f32", "f32", "bf16")))
    if kind == "step":
        return dict(kind=kind, m=rng.choice((1, 1, _log(rng, 2, 16))), layers=rng.randint(4, 32), hidden=hidden, kv=kv, ffn=ffn,
                    vocab=_log(rng, 32000, 128256) // 64 * 64)
    fmt = rng.choice([f.name for f in QuantFormat])
    k = _k(rng, fmt, 1024, 14336)
    return dict(kind=kind, fmt=fmt, n=_log(rng, 64, 58720256 // k), k=k, out=rng.choice(("f32", "bf16", "bf16", "f16")))


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    kind = case["kind"]
    if kind == "step":
        stack = DecodeStack(case["m"], layers=case["layers"], hidden=case["hidden"], kv=case["kv"], ffn=case["ffn"], vocab=case["vocab"], seed=seed)
        graph = DecodeGraph(stack.step, {"x": stack.x}, {"logits": stack.logits, "q": stack.q, "k": stack.k, "v": stack.v, "o": stack.o, "h": stack.h,
                                                         "d": stack.d}).capture()
        return dict(kind=kind, stack=stack, graph=graph, x=torch.randn(case["m"], case["hidden"], device="cuda", generator=gen))
    if kind == "dequant":
        return dict(kind=kind, w=synth.device_weight(case["fmt"], case["n"], case["k"], gen), out=DTYPES[case["out"]])
    if kind == "linear":
        w = synth.device_weight(case["fmt"], case["n"], case["k"], gen)
        x = torch.randn(case["m"], case["k"], device="cuda", generator=gen).to(DTYPES[case["act"]])
        return dict(kind=kind, linear=QuantLinear(w), x=x, out=DTYPES[case["out"]])
    hidden, kv, ffn = case["hidden"], case["kv"], case["ffn"]
    main, vd = case["fmt"], case["fmt_vd"]
    weights = {name: synth.device_weight(fmt, n, k, gen) for name, fmt, n, k in (
        ("q", main, hidden, hidden), ("k", main, kv, hidden), ("v", vd, kv, hidden), ("o", main, hidden, hidden),
        ("gate", main, ffn, hidden), ("up", main, ffn, hidden), ("down", vd, hidden, ffn))}
    return dict(kind=kind, w=weights, o=QuantLinear(weights["o"]), norm=1 + 0.1 * torch.randn(hidden, device="cuda", generator=gen),
                x=torch.randn(case["m"], hidden, device="cuda", generator=gen).to(DTYPES[case["act"]]))


def run(state):
    kind = state["kind"]
    if kind == "step":
        return state["graph"].replay(x=state["x"])
    if kind == "dequant":
        return ops.dequantize(state["w"], state["out"])
    if kind == "linear":
        if state["out"] is torch.float32:
            return state["linear"](state["x"])
        return ops.quant_matmul(state["x"], state["linear"].weight, out_dtype=state["out"])
    w = state["w"]
    q, k, v = ops.rmsnorm_quant_matmul_batch(state["x"], state["norm"], EPS, [w["q"], w["k"], w["v"]])
    o = state["o"](q)  # attention lies between the two in a model; here the output projection reads q
    return q, k, v, o, ops.quant_mlp(o, w["gate"], w["up"], w["down"])


def _packed(fmt, n, k):
    return QuantFormat[fmt].storage_bytes(n * k)


def work(case):
    kind = case["kind"]
    size = {"f32": 4, "bf16": 2, "f16": 2}
    if kind == "dequant":
        return {"bytes": _packed(case["fmt"], case["n"], case["k"]) + case["n"] * case["k"] * size[case["out"]], "flops": case["n"] * case["k"]}
    m = case["m"]
    if kind == "linear":
        k, n = case["k"], case["n"]
        return {"bytes": _packed(case["fmt"], n, k) + m * (k * size[case["act"]] + n * size[case["out"]]), "flops": 2 * m * n * k}
    hidden, kv, ffn = case["hidden"], case["kv"], case["ffn"]
    main, vd, act = (case["fmt"], case["fmt_vd"], size[case["act"]]) if kind == "layer" else ("Q4_K", "Q6_K", 4)
    packed = 2 * _packed(main, hidden, hidden) + _packed(main, kv, hidden) + _packed(vd, kv, hidden) + 2 * _packed(main, ffn, hidden) + _packed(vd, hidden, ffn)
    weights = 2 * hidden * hidden + 2 * kv * hidden + 3 * ffn * hidden
    if kind == "layer":
        return {"bytes": packed + hidden * 4 + m * (hidden * act + 4 * (3 * hidden + 2 * kv)), "flops": 2 * m * weights}
    vocab = case["vocab"]
    outputs = case["layers"] * (3 * hidden + 2 * kv) + vocab
    return {"bytes": case["layers"] * packed + _packed("Q6_K", vocab, hidden) + 4 * m * (hidden + outputs), "flops": 2 * m * (case["layers"] * weights + vocab * hidden)}


def tolerance(case):
    kind = case["kind"]
    if kind == "dequant":
        return "exact"
    prompt = case["m"] >= 64
    if kind == "linear":
        if case["fmt"] in ("Q2_K", "Q3_K"):
            rel = 1e-5  # integer products, 32-bit sums, whatever the number of rows
        elif prompt:
            rel = 1e-2  # bf16 operands
        else:
            # 32-bit sums; above eight rows the formats with blocks of 32 take their activations as 16-bit integers
            rel = 1e-5 if case["fmt"] in K_QUANTS or case["m"] <= 8 else 1e-4
        return {"rel": max(rel, 5e-3 if case["out"] == "bf16" else 0.0)}
    # chained products: a last-place difference in one result can move an 8-bit activation code of the next by one
    if prompt and not (kind == "layer" and case["fmt"] in ("Q2_K", "Q3_K") and case["fmt_vd"] in ("Q2_K", "Q3_K")):
        return {"rel": 2e-2}  # and with bf16 operands most of them may
    return {"rel": 1e-3}
