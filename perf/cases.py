"""The work that is timed: what a model runtime asks of this package, through its public entry points.

A case is one call (or the few calls that belong together) of a decode step or of a prefill chunk:

  gemv   one decode linear on 1..16 rows                        VQMV.encode
  head   the decode tail: lm_head logits, then the sampler's    VQMV.encode, TopK64.encode, or
         64 candidates, or arg-max and the next embedding       argmax_rows + DenseQ.encode_embed
  gemm   one prefill linear                                     DenseQ.encode_qmm_f32
  ffn    a dense gated FFN, decode or prefill rows              DenseMLP.encode
  moe    one MoE FFN block on the residual: norm, router,       rmsnorm, MoELayer.encode
         experts, weighted sum added to the residual

Weights, scratch and outputs are made once, as a loaded model has them. Values follow ingot_b200/synth.py.
Weight formats: q4 / q8 / q6 (affine, groups of 64), q4g32 (groups of 32), mxfp4, tern (rotated ternary, groups of 128).
"""
import math

import torch

from ingot_b200 import synth
from ingot_b200.ep import rmsnorm
from ingot_b200.linear import DenseMLP, DenseQ, VQMV
from ingot_b200.moe import MoELayer, RouterSpec
from ingot_b200.sampling import TopK64, argmax_rows

DT = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
SIZE = {"f32": 4, "f16": 2, "bf16": 2}


def listed():
    return [
        # an attention output projection at one row, added to the fp32 residual: the smallest call, latency and host cost
        {"name": "gemv_q4_2048x4096_r1", "kind": "gemv", "rows": 1, "n": 2048, "k": 4096, "fmt": "q4", "x": "f16", "y": "f32", "add": True},
        # a large FFN matrix at one row (the first benchmark configuration)
        {"name": "gemv_q4_14336x4096_r1", "kind": "gemv", "rows": 1, "n": 14336, "k": 4096, "fmt": "q4", "x": "bf16", "y": "bf16", "add": False},
        # a ternary model's projection on a short speculative run of five rows, input rotation included
        {"name": "gemv_tern_9216x5120_r5", "kind": "gemv", "rows": 5, "n": 9216, "k": 5120, "fmt": "tern", "x": "f16", "y": "f32", "add": False},
        # the decode tail of a batch of eight: 6-bit lm_head and the sampler's candidates
        {"name": "head_q6_128000x2048_r8", "kind": "head", "rows": 8, "n": 128000, "k": 2048, "fmt": "q6", "sample": True},
        # prefill linears: a short chunk at 4 bits, a long one through the 8-bit down projection
        {"name": "gemm_q4_512x14336x4096", "kind": "gemm", "rows": 512, "n": 14336, "k": 4096, "fmt": "q4", "x": "bf16", "y": "bf16", "add": False},
        {"name": "gemm_q8_2048x4096x14336", "kind": "gemm", "rows": 2048, "n": 4096, "k": 14336, "fmt": "q8", "x": "f16", "y": "f32", "add": True},
        # a whole dense FFN: 8-bit on a decode batch of three, 4-bit on a ragged prefill chunk
        {"name": "ffn_q8_2048_7680_r3", "kind": "ffn", "rows": 3, "d": 2048, "d_ff": 7680, "fmt": "q8", "act": "silu", "x": "bf16"},
        {"name": "ffn_q4_4096_14336_r1088", "kind": "ffn", "rows": 1088, "d": 4096, "d_ff": 14336, "fmt": "q4", "act": "silu", "x": "bf16"},
        # the 128-expert MoE block: one token, a decode batch, a prefill chunk
        {"name": "moe_q4_t1", "kind": "moe", "rows": 1, "experts": 128, "top_k": 8, "d": 2048, "d_ff": 768, "fmt": "q4", "act": "silu", "score": "softmax", "shared": 0, "bias": False},
        {"name": "moe_q4_t64", "kind": "moe", "rows": 64, "experts": 128, "top_k": 8, "d": 2048, "d_ff": 768, "fmt": "q4", "act": "silu", "score": "softmax", "shared": 0, "bias": False},
        {"name": "moe_q4_t4096", "kind": "moe", "rows": 4096, "experts": 128, "top_k": 8, "d": 2048, "d_ff": 768, "fmt": "q4", "act": "silu", "score": "softmax", "shared": 0, "bias": False},
        # the MXFP4 MoE block (clamped SwiGLU, expert biases, widths that are no power of two) on an odd number of tokens
        {"name": "moe_mxfp4_t257", "kind": "moe", "rows": 257, "experts": 32, "top_k": 4, "d": 2880, "d_ff": 2880, "fmt": "mxfp4", "act": "swiglu_oai", "score": "softmax", "shared": 0, "bias": True},
    ]


def _log(rng, lo, hi, step):
    """A multiple of step between lo and hi, spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return int(min(max(round(v / step) * step, -(-lo // step) * step), hi // step * step))


def draw(rng):
    kind = rng.choice(["gemv", "gemv", "gemv", "head", "gemm", "gemm", "ffn", "ffn", "moe", "moe", "moe", "moe"])
    if kind == "gemv":
        fmt = rng.choice(["q4", "q4", "q8", "q6", "q4g32", "mxfp4", "tern"])
        step = {"q6": 2048, "tern": 1024}.get(fmt, 64)
        # 6-bit matrices are lm_heads: their GEMV takes inputs of 2048 and 4096
        k = _log(rng, 1024, 4096 if fmt == "q6" else 14336, step) if step > 64 or rng.random() < 0.4 else rng.choice([1024, 2048, 2880, 4096, 5120, 7680])
        return {"kind": kind, "rows": rng.choice([1, 1, rng.randint(2, 16)]), "n": _log(rng, 1024, 32768, 16), "k": k, "fmt": fmt,
                "x": "f16" if fmt == "tern" else rng.choice(["f16", "bf16", "f32"]), "y": rng.choice(["f32", "f32", "bf16"]),
                "add": rng.random() < 0.5}
    if kind == "head":
        return {"kind": kind, "rows": rng.choice([1, rng.randint(2, 16)]), "n": _log(rng, 32000, 262144, 16),
                "k": rng.choice([2048, 4096]), "fmt": rng.choice(["q4", "q6", "q8"]), "sample": rng.random() < 0.6}
    if kind == "gemm":
        fmt = rng.choice(["q4", "q4", "q8", "q4g32", "mxfp4", "tern"])
        k = _log(rng, 1024, 14336, 1024 if fmt == "tern" else 64)
        n = _log(rng, 1024, 14336, 64)
        return {"kind": kind, "rows": _log(rng, 64, min(4096, 250e9 / (2 * n * k)), 64), "n": n, "k": k, "fmt": fmt,
                "x": "f16" if fmt == "tern" else rng.choice(["f16", "bf16", "f32"]), "y": rng.choice(["f32", "f16", "bf16"]),
                "add": rng.random() < 0.5}
    if kind == "ffn":
        d, d_ff = _log(rng, 1024, 4096, 64), _log(rng, 2048, 14336, 64)
        if rng.random() < 0.6:
            d, d_ff = rng.choice([(2048, 7680), (4096, 14336), (2048, 8192), (2880, 5760)])
        rows = rng.randint(1, 16) if rng.random() < 0.5 else _log(rng, 64, min(2048, 380e9 / (6 * d * d_ff)), 64)
        return {"kind": kind, "rows": rows, "d": d, "d_ff": d_ff, "fmt": rng.choice(["q4", "q4", "q8", "q4g32", "mxfp4"]),
                "act": rng.choice(["silu", "silu", "gelu", "swiglu_oai"]), "x": rng.choice(["bf16", "f16", "f32"])}
    fmt = rng.choice(["q4", "q4", "q4", "mxfp4"])
    if rng.random() < 0.5:
        experts, top_k, d, d_ff = (128, 8, 2048, 768) if fmt == "q4" else (32, 4, 2880, 2880)
    else:
        experts, top_k = rng.choice([(32, 4), (64, 6), (128, 8), (256, 8), (512, 10)])
        d = _log(rng, 1024, 4096, rng.choice([64, 512]))
        d_ff = _log(rng, 512, 2048 if experts < 256 else 768, rng.choice([64, 256]))
    most = min(4096, 300e9 / (6.0 * top_k * d * d_ff))
    return {"kind": kind, "rows": _log(rng, 1, most, 1), "experts": experts, "top_k": top_k, "d": d, "d_ff": d_ff, "fmt": fmt,
            "act": "swiglu_oai" if fmt == "mxfp4" else "silu", "score": rng.choice(["softmax", "softmax", "sigmoid"]),
            "shared": 0 if fmt == "mxfp4" or rng.random() < 0.7 else 64 * rng.randint(8, 24), "bias": fmt == "mxfp4"}


# ---- what a program holds before the call -----------------------------------------------------------------------------
def _matrix(gen, n, k, fmt, experts=1):
    if fmt == "mxfp4":
        return synth.mxfp4_cuda(gen, n, k, experts)
    if fmt == "tern":
        dev = gen.device
        w = torch.zeros(n, k // 16, dtype=torch.int64, device=dev)
        for j in range(16):
            w |= torch.randint(0, 3, (n, k // 16), dtype=torch.int64, device=dev, generator=gen) << (2 * j)
        w = torch.where(w >= 2**31, w - 2**32, w).to(torch.int32)
        s = (0.01 + 0.03 * torch.rand((n, k // 128), device=dev, generator=gen)).to(torch.float16)
        m = DenseQ(w, s, None, n, k, 2, 128, "affine")
        m.set_hadamard(torch.randint(0, 2, (k,), device=dev, generator=gen).float() * 2 - 1)
        return m
    bits, group = {"q4": (4, 64), "q8": (8, 64), "q6": (6, 64), "q4g32": (4, 32)}[fmt]
    return synth.affine_cuda(gen, n, k, bits, experts, group)


def _residual(gen, rows, d):
    return torch.randn(rows, d, device=gen.device, generator=gen)


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    return _PREPARE[case["kind"]](case, gen)


def _gemv(c, gen):
    m = _matrix(gen, c["n"], c["k"], c["fmt"])
    x = synth.activations_cuda(gen, c["rows"], c["k"], DT[c["x"]])
    y = _residual(gen, c["rows"], c["n"]).to(DT[c["y"]])
    rows, add = c["rows"], c["add"]

    def step():
        VQMV.encode(x, m, y, rows, accumulate=add)
        return y

    return step


def _head(c, gen):
    m = _matrix(gen, c["n"], c["k"], c["fmt"])
    rows = c["rows"]
    x = synth.activations_cuda(gen, rows, c["k"], torch.float16)
    logits = torch.zeros(rows, c["n"], dtype=torch.float32, device="cuda")
    if c["sample"]:
        top = TopK64(rows, c["n"], logits.device)

        def step():
            VQMV.encode(x, m, logits, rows)
            idx, val, z = top.encode(logits, rows, [0.7])
            return logits, idx, val, z
    else:
        emb = torch.zeros(rows, c["k"], dtype=torch.float32, device="cuda")

        def step():
            VQMV.encode(x, m, logits, rows)
            tok = argmax_rows(logits, rows)
            m.encode_embed(tok, rows, out_f=emb)  # tied embedding table
            return logits, tok, emb

    return step


def _gemm(c, gen):
    m = _matrix(gen, c["n"], c["k"], c["fmt"])
    rows, add = c["rows"], c["add"]
    x = synth.activations_cuda(gen, rows, c["k"], DT[c["x"]])
    y = _residual(gen, rows, c["n"]).to(DT[c["y"]])
    ws = torch.empty(max(m.qmm_workspace_bytes(rows, x.dtype), 256), dtype=torch.uint8, device="cuda")

    def step():
        m.encode_qmm_f32(x, y, rows, accumulate=add, workspace=ws)
        return y

    return step


def _ffn(c, gen):
    mlp = DenseMLP(_matrix(gen, 2 * c["d_ff"], c["d"], c["fmt"]), _matrix(gen, c["d"], c["d_ff"], c["fmt"]), c["act"])
    rows = c["rows"]
    x = synth.activations_cuda(gen, rows, c["d"], DT[c["x"]])
    out = _residual(gen, rows, c["d"])

    def step():
        mlp.encode(x, out, rows, accumulate=True)
        return out

    return step


def _moe(c, gen):
    E, D, I, rows = c["experts"], c["d"], c["d_ff"], c["rows"]
    router = synth.router_cuda(gen, E, D)
    mats = [_matrix(gen, n, k, c["fmt"], E) for n, k in ((I, D), (I, D), (D, I))]
    bias = [(0.01 * torch.randn(E, n, device="cuda", generator=gen)).to(torch.bfloat16).float() for n in (I, I, D)] if c["bias"] else [None] * 3
    select = 0.05 * torch.rand(E, device="cuda", generator=gen) if c["score"] == "sigmoid" else None
    spec = RouterSpec(E, c["top_k"], score=c["score"], select_bias=select)
    shared = gate = None
    if c["shared"]:
        shared = tuple(_matrix(gen, n, k, "q4") for n, k in ((c["shared"], D), (c["shared"], D), (D, c["shared"])))
        gate = _matrix(gen, 1, D, "q8")
    layer = MoELayer(spec, router, *mats, act=c["act"], gate_bias=bias[0], up_bias=bias[1], down_bias=bias[2], max_tokens=rows,
                     shared=shared, shared_gate=gate)
    h = _residual(gen, rows, D)  # the residual as it enters; the update goes to a copy of it, so every pass sees the same input
    r = h.clone()
    xn = torch.empty(rows, D, dtype=torch.bfloat16, device="cuda")

    def step():
        rmsnorm(h, xn, rows)
        layer.encode(xn, r, rows, accumulate=True)
        return r

    return step


_PREPARE = {"gemv": _gemv, "head": _head, "gemm": _gemm, "ffn": _ffn, "moe": _moe}


def run(state):
    return state()


# ---- what one pass cannot do without ----------------------------------------------------------------------------------
def _weights(n, k, fmt):
    """Bytes of codes, scales and biases of an n x k matrix."""
    per = {"q4": 0.5 + 4 / 64, "q8": 1 + 4 / 64, "q6": 0.75 + 4 / 64, "q4g32": 0.5 + 4 / 32, "mxfp4": 0.5 + 1 / 32, "tern": 0.25 + 2 / 128}
    return n * k * per[fmt]


def work(case):
    c = case
    rows = c["rows"]
    if c["kind"] in ("gemv", "gemm"):
        n, k = c["n"], c["k"]
        return {"bytes": _weights(n, k, c["fmt"]) + rows * k * SIZE[c["x"]] + rows * n * SIZE[c["y"]] * (2 if c["add"] else 1),
                "flops": 2.0 * rows * n * k}
    if c["kind"] == "head":
        n, k = c["n"], c["k"]
        return {"bytes": _weights(n, k, c["fmt"]) + rows * k * 2 + rows * n * 4 + (rows * 64 * 8 if c["sample"] else rows * k * 4),
                "flops": 2.0 * rows * n * k}
    if c["kind"] == "ffn":
        d, f = c["d"], c["d_ff"]
        return {"bytes": 3 * _weights(d, f, c["fmt"]) + rows * d * (SIZE[c["x"]] + 8), "flops": 6.0 * rows * d * f}
    E, k, d, f = c["experts"], c["top_k"], c["d"], c["d_ff"]
    touched = E * (1 - (1 - k / E) ** rows)
    sh = c["shared"]
    return {"bytes": touched * 3 * _weights(d, f, c["fmt"]) + (3 * _weights(d, sh, "q4") if sh else 0) + E * d * 2 + rows * d * 12,
            "flops": rows * (6.0 * d * (k * f + sh) + 2.0 * d * E)}


def tolerance(case):
    # operands of 16 bits (fp16 weights and activations), sums of 32 bits; bf16 and fp16 outputs are rounded once more
    if case["kind"] == "moe":
        return {"rel": 2e-3}
    if case["kind"] == "head":
        return {"rel": 1e-3, "differ": 0.01}  # near ties among the candidates
    if case.get("y") == "bf16":
        return {"rel": 5e-3}
    return {"rel": 1e-3}
