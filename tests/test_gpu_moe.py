"""MoE layer (iq_moe_* through MoELayer) against the CPU oracle: routing indices bit-exact, weights 1e-5, outputs within
the tolerance. Mirrors the reference's MoE and router kernel cases (Tests/IngotTests/KernelCaseMoE.swift:45-114,
KernelCaseRouter.swift:110-141, KernelCaseGptOss.swift:13-65, KernelCaseMXFP4.swift:49-134)."""
import json
import os

import numpy as np
import pytest
import torch

from ingot_b200 import capi, synth
from ingot_b200.moe import MoELayer, RouterSpec
from oracle import qref
from gpu_util import TOL, x_tensor

pytestmark = pytest.mark.gpu
GOLD = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden")


def build_layer(rng, device, E, K, D, I, fmt="affine", act="silu", biases=False, router_bias=False, max_tokens=16,
                expert_lo=0, expert_count=None):
    host = {}
    if fmt == "affine":
        g, u, d = synth.affine_np(rng, I, D, 4, E), synth.affine_np(rng, I, D, 4, E), synth.affine_np(rng, D, I, 4, E)
        mk = lambda t, lo, hi: synth.dense_q_affine(t[0][lo:hi], t[1][lo:hi], t[2][lo:hi], 4, device)
        host["deq"] = lambda t, e: qref.dequant_affine(t[0][e], t[1][e], t[2][e], 4)
    else:
        g, u, d = synth.mxfp4_np(rng, I, D, E), synth.mxfp4_np(rng, I, D, E), synth.mxfp4_np(rng, D, I, E)
        mk = lambda t, lo, hi: synth.dense_q_mxfp4(t[0][lo:hi], t[1][lo:hi], device)
        host["deq"] = lambda t, e: qref.dequant_mxfp4(t[0][e], t[1][e])
    host["g"], host["u"], host["d"] = g, u, d
    wr = synth.router_np(rng, E, D)
    host["router"] = wr
    lo = expert_lo
    hi = lo + (expert_count if expert_count is not None else E)
    bt = {}
    if biases:
        host["biases"] = tuple(synth.round_bf16(rng.normal(0, 0.01, size=(E, n)).astype(np.float32)) for n in (I, I, D))
        bt = dict(zip(("gate_bias", "up_bias", "down_bias"),
                      (torch.from_numpy(b[lo:hi].copy()).to(device) for b in host["biases"])))
    else:
        host["biases"] = None
    lb = None
    if router_bias:
        host["router_bias"] = rng.uniform(-1, 1, size=E).astype(np.float32)
        lb = torch.from_numpy(host["router_bias"]).to(device)
    else:
        host["router_bias"] = None
    layer = MoELayer(RouterSpec(E, K, logit_bias=lb), synth.bf16_values_tensor(wr, device), mk(g, lo, hi), mk(u, lo, hi),
                     mk(d, lo, hi), act=act, max_tokens=max_tokens, expert_lo=lo, **bt)
    host["weights"] = lambda e: (host["deq"](g, e), host["deq"](u, e), host["deq"](d, e))
    return layer, host


def check_layer(layer, host, x, T, act, tol=TOL, half_gu=False):
    dev = layer.device
    xt = x_tensor(x, dev)
    out = torch.zeros(T, layer.D, dtype=torch.float32, device=dev)
    layer.encode(xt, out, T)
    assert capi.context(0).device_status() == 0
    v = layer.views(T)
    logits = qref.router_logits(x, host["router"])
    inds, wts = qref.route(logits, layer.router.top_k, logit_bias=host["router_bias"])
    # The logits of the chosen experts are the correctly rounded dot products, bit for bit. So are all the others,
    # except with many tokens and a bf16 router, where logits that cannot reach the top k stay at their tensor-core
    # value (within the kernel's error bound, far below 2e-2 here).
    got_logits = v["logits"][:, : layer.router.experts].cpu().numpy()
    pick = inds.astype(np.int64)
    assert np.array_equal(np.take_along_axis(got_logits, pick, axis=1), np.take_along_axis(logits, pick, axis=1)), \
        "router logits of the chosen experts differ"
    if T <= 64 or layer.router.experts % 64 != 0:
        assert np.array_equal(got_logits, logits), "router logits differ"
    else:
        assert np.abs(got_logits - logits).max() <= 2e-2
    assert np.array_equal(v["inds"].cpu().numpy().astype(np.uint32), inds), "routing indices differ"
    assert qref.max_rel(v["wts"].cpu().numpy(), wts) <= 1e-5
    # permutation: a bijection, grouped by expert in ascending pair order
    offsets, row_map, pos = qref.group_pairs(inds, layer.router.experts)
    assert np.array_equal(v["offsets"].cpu().numpy().astype(np.uint32), offsets)
    assert np.array_equal(v["row_map"].cpu().numpy().astype(np.uint32), row_map)
    assert np.array_equal(v["pos"].cpu().numpy().astype(np.uint32), pos)
    ref = qref.moe_ffn(x, inds, wts, host["weights"], act=act, biases=host["biases"], half_gu=half_gu)
    err = qref.max_rel(out.cpu().numpy(), ref)
    assert err <= tol, err
    return out


@pytest.mark.parametrize("T", [1, 2, 5, 16, 64, 300, 1000, 2150, 2500, 3500])
def test_moe_small_affine(cuda_device, T):
    rng = np.random.default_rng(T)
    layer, host = build_layer(rng, cuda_device, 32, 4, 256, 128, max_tokens=T)
    check_layer(layer, host, synth.activations_np(rng, T, 256), T, "silu")


@pytest.mark.parametrize("T", [1, 7, 40, 2100, 2600])
def test_moe_small_mxfp4_gptoss_style(cuda_device, T):
    """gpt-oss style: MXFP4 experts, expert biases, clamped swiglu_oai, router bias, hidden 576 (not a multiple of 128)."""
    rng = np.random.default_rng(50 + T)
    layer, host = build_layer(rng, cuda_device, 32, 4, 576, 192, fmt="mxfp4", act="swiglu_oai", biases=True,
                              router_bias=True, max_tokens=T)
    check_layer(layer, host, synth.activations_np(rng, T, 576), T, "swiglu_oai")


@pytest.mark.parametrize("T", [1, 8, 16, 64, 100, 256, 512])
def test_moe_c2_configuration(cuda_device, T):
    """128 experts, top-8, d_model 2048, d_ff 768, 4-bit g64, bf16 router ~ N(0, 0.02), x ~ N(0, 1), seed 0. The token
    counts walk the three-kernel path, the decode tile kernels (8-row tiles with one and two live row sets) and the grouped GEMM
    (from 100 tokens on)."""
    rng = np.random.default_rng(0)
    layer, host = build_layer(rng, cuda_device, 128, 8, 2048, 768, max_tokens=T)
    check_layer(layer, host, synth.activations_np(rng, T, 2048), T, "silu")


def test_moe_c2_layer_at_the_benchmarked_size(cuda_device):
    """The layer the 48-layer stack is made of, at the benchmark's 4096 prefill tokens (32,768 routed rows: the chunked
    counting sort, tiles of 192 and 64 rows): logits, indices, weights and the whole permutation
    against the oracle in full, the outputs on 32 sampled tokens."""
    rng = np.random.default_rng(4096)
    T, E, K, D, I = 4096, 128, 8, 2048, 768
    layer, host = build_layer(rng, cuda_device, E, K, D, I, max_tokens=T)
    x = synth.activations_np(rng, T, D)
    out = torch.zeros(T, D, dtype=torch.float32, device=cuda_device)
    layer.encode(x_tensor(x, cuda_device), out, T)
    assert capi.context(0).device_status() == 0
    v = layer.views(T)
    logits = qref.router_logits(x, host["router"])
    inds, wts = qref.route(logits, K)
    assert np.array_equal(v["inds"].cpu().numpy().astype(np.uint32), inds), "routing indices differ"
    assert qref.max_rel(v["wts"].cpu().numpy(), wts) <= 1e-5
    offsets, row_map, pos = qref.group_pairs(inds, E)
    assert np.array_equal(v["offsets"].cpu().numpy().astype(np.uint32), offsets)
    assert np.array_equal(v["row_map"].cpu().numpy().astype(np.uint32), row_map)
    assert np.array_equal(v["pos"].cpu().numpy().astype(np.uint32), pos)
    sel = np.sort(rng.choice(T, size=32, replace=False))
    ref = qref.moe_ffn(x[sel], inds[sel], wts[sel], host["weights"])
    got = out.cpu().numpy()
    assert np.isfinite(got).all()
    err = qref.max_rel(got[sel], ref)
    assert err <= TOL, err


@pytest.mark.parametrize("T", [1, 256])
def test_moe_c3_configuration(cuda_device, T):
    """32 experts, top-4, d_model = d_ff = 2880, MXFP4, expert biases, clamped SwiGLU."""
    rng = np.random.default_rng(0)
    layer, host = build_layer(rng, cuda_device, 32, 4, 2880, 2880, fmt="mxfp4", act="swiglu_oai", biases=True,
                              max_tokens=T)
    check_layer(layer, host, synth.activations_np(rng, T, 2880), T, "swiglu_oai")


def router_cases():
    with open(os.path.join(GOLD, "router_vectors.json")) as f:
        return json.load(f)["cases"]


@pytest.mark.parametrize("case", router_cases(), ids=lambda c: c["name"])
def test_route_kernel_against_mlx_lm_vectors(cuda_device, case):
    """The route kernel on the reference's router vectors (logits at the stride padded to 64): indices bit-exact against
    the CPU rule, weights 1e-5, chosen sets and weights against mlx-lm on rows 2.. (KernelCaseRouter.swift:110-141)."""
    rng = np.random.default_rng(1)
    E, K, B = case["experts"], case["topK"], case["rows"]
    lb = case.get("logitBias")
    pes = case.get("perExpertScale")
    sig = case["score"] == "sigmoid"
    sb = case.get("bias") if sig else None  # sigmoid families: the bias only steers the selection
    dev_f32 = lambda v: None if v is None else torch.tensor(v, dtype=torch.float32, device=cuda_device)
    g, u, d = synth.affine_np(rng, 64, 128, 4, E), synth.affine_np(rng, 64, 128, 4, E), synth.affine_np(rng, 128, 64, 4, E)
    mk = lambda t: synth.dense_q_affine(t[0], t[1], t[2], 4, cuda_device)
    spec = RouterSpec(E, K, scale=case["scale"], logit_bias=dev_f32(lb), per_expert_scale=dev_f32(pes),
                      score=case["score"], select_bias=dev_f32(sb), eps=case["eps"] if sig else 0.0)
    layer = MoELayer(spec, synth.bf16_values_tensor(synth.router_np(rng, E, 128), cuda_device), mk(g), mk(u), mk(d))
    ld = (E + 63) // 64 * 64
    lg = np.array(case["logits"], dtype=np.float32).reshape(B, E)
    padded = np.zeros((B, ld), dtype=np.float32)
    padded[:, :E] = lg
    inds, wts = layer.route(torch.from_numpy(padded).to(cuda_device), B)
    torch.cuda.synchronize()
    ri, rw = qref.route(lg, K, logit_bias=lb, scale=case["scale"], per_expert_scale=pes, sigmoid=sig, select_bias=sb,
                        eps=case["eps"] if sig else 0.0)
    assert np.array_equal(inds.cpu().numpy().astype(np.uint32), ri)
    assert qref.max_rel(wts.cpu().numpy(), rw) <= 1e-5
    dense = np.zeros((B, E), dtype=np.float32)
    gi, gw = inds.cpu().numpy(), wts.cpu().numpy()
    for r in range(B):
        for k in range(K):
            dense[r, gi[r, k]] += gw[r, k]
    mlx = np.array(case["weights"], dtype=np.float32).reshape(B, E)
    assert ((dense[2:] != 0) == (mlx[2:] != 0)).all()
    assert qref.max_rel(dense[2:], mlx[2:]) <= 1e-5


def test_route_kernel_ties_e512_k10_and_edge_rows(cuda_device):
    rng = np.random.default_rng(2)
    E, K = 512, 10
    g, u, d = synth.affine_np(rng, 64, 128, 4, E), synth.affine_np(rng, 64, 128, 4, E), synth.affine_np(rng, 128, 64, 4, E)
    mk = lambda t: synth.dense_q_affine(t[0], t[1], t[2], 4, cuda_device)
    layer = MoELayer(RouterSpec(E, K), synth.bf16_values_tensor(synth.router_np(rng, E, 128), cuda_device), mk(g), mk(u), mk(d))
    lg = rng.uniform(-4, 4, size=(12, E)).astype(np.float32)
    lg[0, :] = -3
    for e in [5, 17, 33, 64, 100, 200, 255, 256, 511]:
        lg[0, e] = 5
    lg[0, 301] = lg[0, 450] = 2          # exact tie for the 10th place: 301 wins
    lg[1, :] = -np.inf                   # nothing to choose from: indices 0..9
    lg[2, 7] = np.nan                    # NaN counts as -inf
    inds, wts = layer.route(torch.from_numpy(lg).to(cuda_device), 12)
    torch.cuda.synchronize()
    ri, rw = qref.route(lg, K)
    got = inds.cpu().numpy().astype(np.uint32)
    assert np.array_equal(got, ri)
    assert got[0].tolist() == [5, 17, 33, 64, 100, 200, 255, 256, 511, 301]
    assert got[1].tolist() == list(range(10))
    ok = np.ones(12, dtype=bool)
    ok[1] = False  # weights of the all -inf row are NaN on both sides
    assert qref.max_rel(wts.cpu().numpy()[ok], rw[ok]) <= 1e-5


def tensor_router_layer(rng, device, wr, K, T):
    E, D = wr.shape
    I = 64
    g, u, d = synth.affine_np(rng, I, D, 4, E), synth.affine_np(rng, I, D, 4, E), synth.affine_np(rng, D, I, 4, E)
    mk = lambda t: synth.dense_q_affine(t[0], t[1], t[2], 4, device)
    return MoELayer(RouterSpec(E, K), synth.bf16_values_tensor(wr, device), mk(g), mk(u), mk(d), max_tokens=T)


def test_tensor_router_error_bound_and_exact_selection(cuda_device):
    """Many tokens, bf16 router, bf16 activations: the logits come from the tensor cores, then the route kernel recomputes
    exactly every logit within twice the error bound of the k-th largest. The approximate logits must sit far inside the
    bound the kernel assumes (K * 2^-21 * ||x|| * max||w||); indices, the chosen logits and the weights must be what
    float64 logits give."""
    rng = np.random.default_rng(77)
    E, K, D, T = 128, 8, 2048, 1024
    wr = synth.router_np(rng, E, D)
    layer = tensor_router_layer(rng, cuda_device, wr, K, T)
    x = synth.activations_np(rng, T, D)
    xt = x_tensor(x, cuda_device)
    out = torch.zeros(T, D, dtype=torch.float32, device=cuda_device)
    layer.encode(xt, out, T, only="router")
    torch.cuda.synchronize()
    approx = layer.views(T)["logits"][:, :E].cpu().numpy().copy()
    exact = qref.router_logits(x, wr)
    bound = D * 2.0 ** -21 * np.linalg.norm(wr, axis=1).max() * np.linalg.norm(x, axis=1)  # per token
    worst = (np.abs(approx - exact).max(axis=1) / bound).max()
    assert worst <= 1 / 8, f"tensor-core logits use {worst:.3f} of the assumed error bound"
    assert not np.array_equal(approx, exact)  # (they really are the approximate ones)
    layer.encode(xt, out, T, only="route")
    assert capi.context(0).device_status() == 0
    v = layer.views(T)
    inds, wts = qref.route(exact, K)
    assert np.array_equal(v["inds"].cpu().numpy().astype(np.uint32), inds)
    assert qref.max_rel(v["wts"].cpu().numpy(), wts) <= 1e-5
    pick = inds.astype(np.int64)
    refined = v["logits"][:, :E].cpu().numpy()
    assert np.array_equal(np.take_along_axis(refined, pick, axis=1), np.take_along_axis(exact, pick, axis=1))


def test_tensor_router_near_ties_at_the_boundary(cuda_device):
    """Adversarial margins: the 128 experts are 64 pairs whose rows differ by one bf16 ulp in one weight, and x is tiny at
    that position, so the two logits of a pair differ by a few fp32 ulps at most (or tie). With top-7 the boundary between
    the 7th and the 8th place falls inside a pair for every token: only the exact recomputation (and the lower-index
    rule on ties) can give the oracle's indices."""
    rng = np.random.default_rng(78)
    E, K, D, T = 128, 7, 2048, 512
    base = synth.router_np(rng, E // 2, D)
    wr = np.repeat(base, 2, axis=0)
    k0 = 1000
    bits = synth.to_bf16_bits(wr[1::2, k0])
    wr[1::2, k0] = synth.bf16_bits_to_f32((bits + 1).astype(np.uint16))  # one ulp up in the odd rows
    x = synth.activations_np(rng, T, D)
    x[:, k0] = synth.round_bf16((2.0 ** -rng.integers(8, 13, size=T)).astype(np.float32) * rng.choice([-1.0, 1.0], size=T).astype(np.float32))
    exact = qref.router_logits(x, wr)
    gap = np.abs(exact[:, 0::2] - exact[:, 1::2])
    ulp = np.spacing(np.abs(exact[:, 0::2]).astype(np.float32))
    assert (gap <= 8 * ulp).mean() > 0.8 and (gap == 0).any() and (gap > 0).any()  # a few ulps apart, some exact ties
    layer = tensor_router_layer(rng, cuda_device, wr, K, T)
    out = torch.zeros(T, D, dtype=torch.float32, device=cuda_device)
    layer.encode(x_tensor(x, cuda_device), out, T, only=("router", "route"))
    assert capi.context(0).device_status() == 0
    inds, wts = qref.route(exact, K)
    got = layer.views(T)["inds"].cpu().numpy().astype(np.uint32)
    assert np.array_equal(got, inds)
    # the boundary really splits a pair: the 7th choice's partner is the runner-up that was left out
    assert ((inds[:, -1] ^ 1)[:, None] != inds).all(axis=1).mean() > 0.9


@pytest.mark.parametrize("T", [3, 200])
def test_router_8bit_affine(cuda_device, T):
    """A router stored as 8-bit affine codes (MoE.swift:258-273 keeps the router quantized when the checkpoint does): the
    logits are the float64 dot products with the fp32 weights s*q + b, bit for bit, in the cluster that routes a few tokens
    and in the kernel for more (the tiled GEMM for many: test_router_tiled_float64_gemm)."""
    rng = np.random.default_rng(70 + T)
    E, K, D, I = 64, 4, 256, 128
    g, u, d = synth.affine_np(rng, I, D, 4, E), synth.affine_np(rng, I, D, 4, E), synth.affine_np(rng, D, I, 4, E)
    mk = lambda t: synth.dense_q_affine(t[0], t[1], t[2], 4, cuda_device)
    rw, rs, rb = synth.affine_np(rng, E, D, 8)
    dev_t = lambda a, dt: torch.from_numpy(a[0].view(dt).copy()).to(cuda_device)
    layer = MoELayer(RouterSpec(E, K), dev_t(rw, np.int32), mk(g), mk(u), mk(d), max_tokens=T,
                     router_scales=dev_t(rs, np.int16).view(torch.bfloat16), router_biases=dev_t(rb, np.int16).view(torch.bfloat16))
    x = synth.activations_np(rng, T, D)
    xt = x_tensor(x, cuda_device)
    out = torch.zeros(T, D, dtype=torch.float32, device=cuda_device)
    layer.encode(xt, out, T, only=("router", "route"))
    torch.cuda.synchronize()
    v = layer.views(T)
    wr = qref.dequant_affine(rw[0], rs[0], rb[0], 8)
    logits = qref.router_logits(x, wr)
    assert np.array_equal(v["logits"][:, :E].cpu().numpy(), logits)
    inds, _ = qref.route(logits, K)
    assert np.array_equal(v["inds"].cpu().numpy().astype(np.uint32), inds)


@pytest.mark.parametrize("act", ["gelu", "relu2"])
@pytest.mark.parametrize("T", [3, 40, 700])
def test_moe_other_activations(cuda_device, act, T):
    """GELU (tanh form) gate and relu^2 without gate (qmm.metal:9-31 ACT 1 and 3) through the three-kernel path, the decode tiles and
    the tcgen05 grouped GEMM."""
    rng = np.random.default_rng(90 + T)
    layer, host = build_layer(rng, cuda_device, 32, 2, 2048, 128, act=act, max_tokens=T)
    check_layer(layer, host, synth.activations_np(rng, T, 2048), T, act)


@pytest.mark.parametrize("E,K,D,I,T", [
    (32, 4, 192, 64, 1), (32, 4, 192, 64, 3), (96, 16, 320, 192, 2), (512, 10, 1024, 64, 3),  # the three-kernel path: odd
    (32, 4, 192, 64, 4),             # group counts, one slice per expert, experts beyond a warp's four; and past its end
    (32, 4, 832, 128, 5),            # few rows, a width the int8 kernels do not take
    (32, 4, 256, 128, 48), (32, 4, 256, 128, 49),     # six rows per expert: the last on the int8 kernels, the first beyond
    (32, 4, 256, 128, 65), (32, 4, 256, 128, 385), (32, 4, 256, 128, 767), (32, 4, 256, 128, 768)])  # GEMM tile heights
def test_moe_edges_of_the_paths(cuda_device, E, K, D, I, T):
    rng = np.random.default_rng(800 + E + D + T)
    layer, host = build_layer(rng, cuda_device, E, K, D, I, max_tokens=T)
    check_layer(layer, host, synth.activations_np(rng, T, D), T, "silu")


@pytest.mark.parametrize("T", [3, 33, 257])
def test_moe_mxfp4_low_tiles(cuda_device, T):
    """MXFP4 experts on tiles of 32 and 64 rows, two CTAs per SM: an odd number of K steps (9), a last tile of features that is
    not full in the down projection (576 = 4.5 x 128)."""
    rng = np.random.default_rng(900 + T)
    layer, host = build_layer(rng, cuda_device, 32, 4, 576, 192, fmt="mxfp4", act="swiglu_oai", biases=True, max_tokens=T)
    check_layer(layer, host, synth.activations_np(rng, T, 576), T, "swiglu_oai")


def test_router_tensor_logits_of_96_experts(cuda_device):
    """The tensor-core logits with exact refinement where the experts do not fill the tile (96 of 128 columns)."""
    rng = np.random.default_rng(950)
    E, K, D, T = 96, 6, 1024, 600
    layer, host = build_layer(rng, cuda_device, E, K, D, 64, max_tokens=T)
    x = synth.activations_np(rng, T, D)
    out = torch.zeros(T, D, dtype=torch.float32, device=cuda_device)
    layer.encode(x_tensor(x, cuda_device), out, T)
    v = layer.views(T)
    logits = qref.router_logits(x, host["router"])
    inds, wts = qref.route(logits, K)
    got = v["logits"].cpu().numpy()
    pick = inds.astype(np.int64)
    assert np.array_equal(np.take_along_axis(got, pick, axis=1), np.take_along_axis(logits, pick, axis=1))
    assert np.array_equal(v["inds"].cpu().numpy().astype(np.uint32), inds)
    assert not got[:, E:].any()  # the columns past the experts
    assert qref.max_rel(out.cpu().numpy(), qref.moe_ffn(x, inds, wts, host["weights"])) <= TOL


@pytest.mark.parametrize("gated", [True, False])
@pytest.mark.parametrize("T,D,IS", [(1, 256, 192), (19, 256, 192), (300, 256, 192), (50, 2048, 256), (100, 2048, 320)])
def test_moe_shared_expert(cuda_device, T, D, IS, gated):
    """A shared expert of its own width beside the routed experts, with its 8-bit sigmoid gate or weight 1
    (MoE.swift:140-154; KernelCaseMoE.swift:45-114): GEMV tiles for few tokens, the tcgen05 path for many; at 2048 inputs its gate/up
    tiles, of token rows that are no multiple of 16, are divided along K."""
    rng = np.random.default_rng(300 + T)
    E, K, I = 32, 4, 128
    assert D == 256 or capi.qmm_plan(2 * IS, D, 4, 64, T, gate_up=True).split_tiles > 0
    sg, su, sd = synth.affine_np(rng, IS, D, 4), synth.affine_np(rng, IS, D, 4), synth.affine_np(rng, D, IS, 4)
    gw = synth.affine_np(rng, 1, D, 8)
    mk = lambda t, bits: synth.dense_q_affine(t[0], t[1], t[2], bits, cuda_device)
    g, u, d = synth.affine_np(rng, I, D, 4, E), synth.affine_np(rng, I, D, 4, E), synth.affine_np(rng, D, I, 4, E)
    wr = synth.router_np(rng, E, D)
    layer = MoELayer(RouterSpec(E, K), synth.bf16_values_tensor(wr, cuda_device), mk(g, 4), mk(u, 4), mk(d, 4), max_tokens=T,
                     shared=(mk(sg, 4), mk(su, 4), mk(sd, 4)), shared_gate=mk(gw, 8) if gated else None)
    x = synth.activations_np(rng, T, D)
    out = torch.zeros(T, D, dtype=torch.float32, device=cuda_device)
    layer.encode(x_tensor(x, cuda_device), out, T)
    torch.cuda.synchronize()
    assert capi.context(0).device_status() == 0
    deq = lambda t, e=0, bits=4: qref.dequant_affine(t[0][e], t[1][e], t[2][e], bits)
    inds, wts = qref.route(qref.router_logits(x, wr), K)
    ref = qref.moe_ffn(x, inds, wts, lambda e: (deq(g, e), deq(u, e), deq(d, e)))
    ref = ref + qref.shared_expert(x, deq(sg), deq(su), deq(sd), deq(gw, 0, 8)[0] if gated else None)
    assert qref.max_rel(out.cpu().numpy(), ref) <= TOL


def test_moe_load_guards(cuda_device):
    """Shapes the reference refuses at load (MoE.swift:186-219) come back as named errors."""
    rng = np.random.default_rng(3)
    with pytest.raises(capi.IngotError) as e:
        build_layer(rng, cuda_device, 48, 4, 256, 128)  # experts not a multiple of 32
    assert e.value.status == -2
    with pytest.raises(capi.IngotError):
        build_layer(rng, cuda_device, 32, 4, 256, 96)  # d_ff not a multiple of 64


def test_moe_pieces_and_external_routing(cuda_device):
    """`only:` runs single pieces on what earlier pieces left in the scratch; routing set by the caller is honoured."""
    rng = np.random.default_rng(4)
    T = 24
    layer, host = build_layer(rng, cuda_device, 32, 4, 256, 128, max_tokens=T)
    x = synth.activations_np(rng, T, 256)
    xt = x_tensor(x, cuda_device)
    full = torch.zeros(T, 256, dtype=torch.float32, device=cuda_device)
    layer.encode(xt, full, T)
    torch.cuda.synchronize()
    out = torch.zeros_like(full)
    for piece in ("router", "route", "group", "gateup", "down", "combine"):
        layer.encode(xt, out, T, only=piece)
    torch.cuda.synchronize()
    assert torch.equal(out, full)
    # accumulate into a residual
    res = torch.ones_like(full)
    layer.encode(xt, res, T, accumulate=True)
    torch.cuda.synchronize()
    assert torch.allclose(res - 1, full, atol=1e-5)
    # routing chosen by hand
    inds = torch.from_numpy(np.stack([rng.permutation(32)[:4] for _ in range(T)]).astype(np.int32)).to(cuda_device)
    wts = torch.from_numpy(rng.uniform(0.1, 1, size=(T, 4)).astype(np.float32)).to(cuda_device)
    layer.set_external_routing(inds, wts)
    layer.encode(xt, out, T)
    torch.cuda.synchronize()
    layer.set_external_routing(None, None)
    ref = qref.moe_ffn(x, inds.cpu().numpy().astype(np.uint32), wts.cpu().numpy(), host["weights"])
    assert qref.max_rel(out.cpu().numpy(), ref) <= TOL


@pytest.mark.parametrize("D,I,T", [(2880, 192, 1), (1600, 320, 2), (2880, 768, 3), (128, 64, 3)])
def test_moe_few_tokens_keep_activations_whole(cuda_device, D, I, T):
    """Up to three tokens, input channels 100 times the rest: h is the fp16 rounding of the 64-bit gated product but for the values
    that lie within the fp32 sums' error of a rounding boundary: some 3e-6 of a value either way, of 2^-11: about 1 %. (16-bit
    digits: a third to a half of all h.)"""
    rng = np.random.default_rng(960 + D + I + T)
    E, K = 32, 4
    layer, host = build_layer(rng, cuda_device, E, K, D, I, max_tokens=T)
    x = rng.normal(0, 0.2, size=(T, D)).astype(np.float32)
    x[:, rng.choice(D, 3, replace=False)] *= 100
    xt = torch.from_numpy(x).to(cuda_device).to(torch.bfloat16)
    out = torch.zeros(T, D, dtype=torch.float32, device=cuda_device)
    layer.encode(xt, out, T)
    assert capi.context(0).device_status() == 0
    v = layer.views(T)
    x64 = xt.double().cpu().numpy()
    inds, row_map, h = (v[k].cpu().numpy() for k in ("inds", "row_map", "h"))
    off = total = 0
    for r, pair in enumerate(row_map.astype(np.int64)):
        g, u, _ = (w.astype(np.float64) for w in host["weights"](int(inds.reshape(-1)[pair])))
        xg, xu = g @ x64[pair // K], u @ x64[pair // K]
        want = (xg / (1 + np.exp(-xg)) * xu).astype(np.float16)
        off += int((want.view(np.uint16) != h[r].view(np.uint16)).sum())
        total += I
    assert off <= 0.03 * total, (off, total)


@pytest.mark.parametrize("T", [2, 70])
def test_moe_mxfp4_scales_at_odd_addresses(cuda_device, T):
    """Expert scales one byte into a larger tensor: the same bits as from an aligned one."""
    rng = np.random.default_rng(970 + T)
    E, K, D, I = 32, 4, 576, 192
    w = [synth.mxfp4_np(rng, n, k, E) for n, k in ((I, D), (I, D), (D, I))]
    wr = synth.bf16_values_tensor(synth.router_np(rng, E, D), cuda_device)
    xt = x_tensor(synth.activations_np(rng, T, D), cuda_device)
    outs = []
    for by in (0, 1):
        mats = []
        for codes, scales in w:
            m = synth.dense_q_mxfp4(codes, scales, cuda_device)
            buf = torch.full((m.s.numel() + 16,), 255, dtype=torch.uint8, device=cuda_device)
            m.s = buf[by: by + m.s.numel()].view_as(m.s).copy_(m.s)
            assert m.s.data_ptr() % 2 == by
            mats.append(m)
        layer = MoELayer(RouterSpec(E, K), wr, *mats, max_tokens=T)
        out = torch.zeros(T, D, dtype=torch.float32, device=cuda_device)
        layer.encode(xt, out, T)
        assert capi.context(0).device_status() == 0
        outs.append(out)
    assert torch.equal(outs[0], outs[1])


@pytest.mark.parametrize("D,I", [(1536, 128), (3072, 64), (5120, 64), (768, 1536)])
@pytest.mark.parametrize("T", [4, 40])
def test_moe_decode_widths_that_are_no_power_of_two(cuda_device, D, I, T):
    """Inputs that are no power of two: the decode tiles take them as three digits, and h as two (1536 features) or three."""
    rng = np.random.default_rng(980 + D + T)
    layer, host = build_layer(rng, cuda_device, 32, 4, D, I, max_tokens=T)
    check_layer(layer, host, synth.activations_np(rng, T, D), T, "silu")


@pytest.mark.parametrize("kind,E,D,T", [("q8", 512, 2048, 100), ("q8", 64, 1408, 1030), ("sigmoid", 256, 4096, 101), ("f16", 96, 2880, 333),
                                       ("f32", 32, 4096, 1025)])
def test_router_tiled_float64_gemm(cuda_device, kind, E, D, T):
    """More than 90 million products and no tensor-core route (an 8-bit router, sigmoid scores, activations that are not bf16): the
    register-tiled float64 GEMM, both tile heights, token and expert tiles that are not full, the K range over a cluster or not.
    The logits are the correctly rounded float64 dot products."""
    assert T * E * D > 90_000_000 and T > 64
    rng = np.random.default_rng(990 + E + T)
    K, I = 4, 64
    g, u, d = synth.affine_np(rng, I, D, 4, E), synth.affine_np(rng, I, D, 4, E), synth.affine_np(rng, D, I, 4, E)
    mk = lambda t: synth.dense_q_affine(t[0], t[1], t[2], 4, cuda_device)
    extra, spec = {}, RouterSpec(E, K)
    if kind == "q8":
        rw, rs, rb = synth.affine_np(rng, E, D, 8)
        dev_t = lambda a, dt: torch.from_numpy(a[0].view(dt).copy()).to(cuda_device)
        w, wr = dev_t(rw, np.int32), qref.dequant_affine(rw[0], rs[0], rb[0], 8)
        extra = {"router_scales": dev_t(rs, np.int16).view(torch.bfloat16), "router_biases": dev_t(rb, np.int16).view(torch.bfloat16)}
    else:
        wr = synth.router_np(rng, E, D)
        w = synth.bf16_values_tensor(wr, cuda_device)
        if kind == "sigmoid":
            spec = RouterSpec(E, K, score="sigmoid")
    layer = MoELayer(spec, w, mk(g), mk(u), mk(d), max_tokens=T, **extra)
    dt = {"f16": torch.float16, "f32": torch.float32}.get(kind, torch.bfloat16)
    xt = torch.from_numpy(rng.normal(0, 1, size=(T, D)).astype(np.float32)).to(cuda_device).to(dt)
    out = torch.zeros(T, D, dtype=torch.float32, device=cuda_device)
    layer.encode(xt, out, T, only=("router", "route"))
    assert capi.context(0).device_status() == 0
    v = layer.views(T)
    logits = qref.router_logits(xt.float().cpu().numpy(), wr)
    got = v["logits"].cpu().numpy()
    assert np.array_equal(got[:, :E], logits) and not got[:, E:].any()
    inds, _ = qref.route(logits, K, sigmoid=kind == "sigmoid")
    assert np.array_equal(v["inds"].cpu().numpy().astype(np.uint32), inds)


@pytest.mark.parametrize("fmt,act", [("affine", "silu"), ("mxfp4", "swiglu_oai")])
@pytest.mark.parametrize("D,I,T", [(448, 576, 900), (192, 64, 3000)])
def test_moe_tall_tiles_on_pairs(cuda_device, fmt, act, D, I, T):
    """Tiles of up to 192 rows run on pairs of CTAs: widths that fill a pair's features in part, or only its first CTA's, tiles of a
    few rows among full ones, odd numbers of K steps."""
    rng = np.random.default_rng(91 + D + T)
    layer, host = build_layer(rng, cuda_device, 32, 4, D, I, fmt=fmt, act=act, biases=fmt == "mxfp4", max_tokens=T)
    check_layer(layer, host, synth.activations_np(rng, T, D), T, act)


@pytest.mark.parametrize("D,I", [(1024, 320), (2048, 1408), (4096, 256)])
@pytest.mark.parametrize("T", [5, 40])
def test_moe_int8_experts_by_width(cuda_device, D, I, T):
    """The decode tiles with inputs as two digits, h as two (256 features) or three: up to four rows per expert and more."""
    rng = np.random.default_rng(95 + D + T)
    layer, host = build_layer(rng, cuda_device, 32, 4, D, I, max_tokens=T)
    check_layer(layer, host, synth.activations_np(rng, T, D), T, "silu")


@pytest.mark.parametrize("T", [4, 30, 34])
@pytest.mark.parametrize("D,I", [(448, 192), (2880, 64), (320, 832), (1088, 320), (512, 448)])
def test_moe_decode_tiles_edges(cuda_device, D, I, T):
    """The decode tiles' kernel where a step of 256 inputs or a tile of weight rows is not full: seven, forty-five, five and seventeen groups
    of inputs (scales of rows that are no multiple of eight bytes) as three digits and eight as two, output tiles of 64 of 128 rows, one group
    of h; experts without rows, with one, with eight and with more (second tiles), biases; both sides of four rows per expert, where three
    digits end."""
    rng = np.random.default_rng(D + I + T)
    E, K = 32, 4
    layer, host = build_layer(rng, cuda_device, E, K, D, I, biases=True, max_tokens=T)
    out = check_layer(layer, host, synth.activations_np(rng, T, D), T, "silu")
    assert np.isfinite(out.cpu().numpy()).all()


def test_moe_decode_tiles_pieces_and_bits(cuda_device):
    """Gate/up and down alone give the bits of the whole call (h as fixed point then comes from its halves), and a token's bits do not
    depend on which row of its tiles it is."""
    rng = np.random.default_rng(77)
    T, D, I = 40, 512, 320
    layer, _ = build_layer(rng, cuda_device, 32, 4, D, I, max_tokens=T)
    x = x_tensor(synth.activations_np(rng, T, D), cuda_device)
    full, part, back = (torch.zeros(T, D, dtype=torch.float32, device=cuda_device) for _ in range(3))
    layer.encode(x, full, T)
    for piece in ("router", "route", "group", "gateup", "down", "combine"):
        layer.encode(x, part, T, only=piece)
    assert torch.equal(full, part)
    layer.encode(x.flip(0).contiguous(), back, T)
    assert torch.equal(back.flip(0), full)
    assert capi.context(0).device_status() == 0


@pytest.mark.parametrize("T", [1, 2, 3])
@pytest.mark.parametrize("D,I,K", [(2048, 1472, 4), (2880, 704, 4)])
def test_moe_two_and_three_tokens_by_size(cuda_device, D, I, K, T):
    """One, two and three tokens on both sides of 24 million weights (two tokens 24.1 and 16.2, three 36 and 24.3), where the
    decode tiles take over from the kernels for few tokens."""
    rng = np.random.default_rng(D + I + T)
    layer, host = build_layer(rng, cuda_device, 32, K, D, I, max_tokens=T)
    check_layer(layer, host, synth.activations_np(rng, T, D), T, "silu")


@pytest.mark.parametrize("T", [1, 5, 24, 300])
def test_moe_layers_of_one_shape_share_a_workspace(cuda_device, T):
    """Layers of one shape share their scratch: an affine layer, whose decode tiles need more than the rest, runs in the workspace of
    an MXFP4 layer, and in that of one that owns a quarter of the experts, as in its own."""
    rng = np.random.default_rng(61 + T)
    E, K, D, I = 32, 4, 576, 1152
    mx, _ = build_layer(rng, cuda_device, E, K, D, I, fmt="mxfp4", act="swiglu_oai", max_tokens=T)
    part, _ = build_layer(rng, cuda_device, E, K, D, I, max_tokens=T, expert_lo=8, expert_count=8)
    layer, _ = build_layer(rng, cuda_device, E, K, D, I, max_tokens=T)
    x = x_tensor(synth.activations_np(rng, T, D), cuda_device)
    own, shared = (torch.zeros(T, D, dtype=torch.float32, device=cuda_device) for _ in range(2))
    layer.encode(x, own, T)
    for other in (mx, part):
        layer.share_scratch(other)
        layer.encode(x, shared, T)
        assert torch.equal(own, shared)


def block_in_pieces(layer, x, T):
    """The block of one token batch as the expert-parallel pieces run it: rows out, the experts on them, rows back."""
    dev, P = layer.device, T * layer.router.top_k
    out = torch.zeros(T, layer.D, dtype=torch.float32, device=dev)
    layer.encode(x, out, T, only=("router", "route", "group"))
    off = layer.views(T)["offsets"]
    counts = (off[1:] - off[:-1]).to(torch.int32).contiguous()
    rows, yd = (torch.zeros(P, layer.D, dtype=torch.float16, device=dev) for _ in range(2))
    layer.pack_rows(x, rows, T)
    layer.experts(rows, P, counts, 1, yd, torch.empty(layer.experts_workspace_bytes(P, 1), dtype=torch.uint8, device=dev))
    layer.combine_rows(yd, out, T)
    return out


@pytest.mark.parametrize("T", [4, 13, 44])
@pytest.mark.parametrize("D,I", [(256, 4096), (512, 512), (512, 6144), (1024, 2048), (1024, 1280), (2048, 768), (2048, 1536), (2048, 256)])
def test_moe_whole_layer_has_the_bits_of_its_pieces(cuda_device, D, I, T):
    """Where the decode tiles and the expert-parallel pieces' kernel take the same rows as two digits (activations in half, h rounded to halves),
    they give the same bits: one, two, four and eight K slices of h, tiles of one to eight rows and second tiles, expert biases."""
    rng = np.random.default_rng(D + I + T)
    layer, host = build_layer(rng, cuda_device, 32, 4, D, I, biases=True, max_tokens=T)
    x = synth.activations_np(rng, T, D)
    whole = check_layer(layer, host, x, T, "silu")
    xt = x_tensor(x, cuda_device, torch.float16)
    layer.encode(xt, whole, T)
    assert torch.equal(block_in_pieces(layer, xt, T), whole)
    assert capi.context(0).device_status() == 0


@pytest.mark.parametrize("T", [1, 2, 3, 24, 120])
@pytest.mark.parametrize("D,I", [(512, 256), (576, 192)])
def test_moe_down_alone_takes_the_h_of_the_workspace(cuda_device, D, I, T):
    """After a whole call on any of the paths (three kernels, decode tiles, GEMM) down and combine alone give its result again, and of an h that the
    caller doubled twice that: every rounding scales with h, except of expert outputs below 2^-14, where halves lie 2^-24 apart (two such roundings, the
    weights add up to one: 2^-23)."""
    rng = np.random.default_rng(D + T)
    layer, host = build_layer(rng, cuda_device, 32, 4, D, I, max_tokens=T)
    x = synth.activations_np(rng, T, D)
    whole = check_layer(layer, host, x, T, "silu")
    out = torch.zeros_like(whole)
    layer.encode(x_tensor(x, cuda_device), out, T, only=("down", "combine"))
    assert qref.max_rel(out.cpu().numpy(), whole.cpu().numpy()) <= TOL
    layer.views(T)["h"].mul_(2)
    twice = torch.zeros_like(whole)
    layer.encode(x_tensor(x, cuda_device), twice, T, only=("down", "combine"))
    assert (twice - 2 * out).abs().max().item() <= 2.0**-23 and twice.abs().max().item() > 0.1


def outlier_layer(rng, device, E, K, D, I, max_tokens):
    """Experts whose h has one feature of every 64 some 256 times the rest, which the down projection multiplies by zero: what counts are the others."""
    g, u, d = synth.affine_np(rng, I, D, 4, E), synth.affine_np(rng, I, D, 4, E), synth.affine_np(rng, D, I, 4, E)
    for t in u[1:]:
        t[:, 5::64, :] += 8 << 7  # scales and biases of these rows times 2^8
    sd = synth.bf16_bits_to_f32(d[1])
    d = (d[0], d[1], synth.to_bf16_bits(-8 * sd))
    d[0][:, :, 0::8] = (d[0][:, :, 0::8] & np.uint32(~(0xF << 20) & 0xFFFFFFFF)) | np.uint32(8 << 20)  # input 5 of a group: code 8, weight 0
    mk = lambda t: synth.dense_q_affine(t[0], t[1], t[2], 4, device)
    wr = synth.router_np(rng, E, D)
    layer = MoELayer(RouterSpec(E, K), synth.bf16_values_tensor(wr, device), mk(g), mk(u), mk(d), max_tokens=max_tokens)
    return layer, lambda e: tuple(qref.dequant_affine(t[0][e], t[1][e], t[2][e], 4).astype(np.float64) for t in (g, u, d))


@pytest.mark.parametrize("D,I,T", [(512, 320, 24), (576, 192, 24), (1024, 1792, 12), (2048, 1536, 3)])
def test_moe_decode_tiles_keep_h_beside_large_features(cuda_device, D, I, T):
    """h beside features 256 times as large is as good as its halves are: widths that the tiles take as three digits, and three tokens of experts too
    large for the kernels of few tokens. Against 64 bits; the bound is the error of h and the expert outputs rounded to halves, which both sides
    have, and a tenth of it."""
    rng = np.random.default_rng(D + I + T)
    E, K = 32, 4
    layer, weights = outlier_layer(rng, cuda_device, E, K, D, I, T)
    x = synth.activations_np(rng, T, D)
    out = torch.zeros(T, D, dtype=torch.float32, device=cuda_device)
    layer.encode(x_tensor(x, cuda_device), out, T)
    v = layer.views(T)
    inds, wts = v["inds"].cpu().numpy(), v["wts"].cpu().numpy().astype(np.float64)
    exact, halves, large, rest = np.zeros((T, D)), np.zeros((T, D)), 0.0, 0.0
    for e in np.unique(inds):
        gate, up, down = weights(int(e))
        for t, k in zip(*np.nonzero(inds == e)):
            a = gate @ x[t].astype(np.float64)
            h = a / (1 + np.exp(-a)) * (up @ x[t].astype(np.float64))
            large, rest = large + np.abs(h[5::64]).mean(), rest + np.abs(np.delete(h, np.s_[5::64])).mean()
            exact[t] += wts[t, k] * (down @ h)
            halves[t] += wts[t, k] * (down @ h.astype(np.float16).astype(np.float64)).astype(np.float16).astype(np.float64)
    assert large > 100 * rest
    rel = lambda y: np.linalg.norm(y - exact) / np.linalg.norm(exact)
    assert rel(out.cpu().numpy()) <= 1.1 * rel(halves), (rel(out.cpu().numpy()), rel(halves))


@pytest.mark.parametrize("D,I", [(512, 256), (512, 320), (576, 192)])
def test_moe_decode_tiles_non_finite_and_overflowing_rows(cuda_device, D, I):
    """A token with a NaN or an infinity comes out NaN, one whose h passes the range of halves non-finite where an expert's h does, and the other
    tokens keep their bits: two and three digits of inputs and of h."""
    rng = np.random.default_rng(D + I)
    T = 24
    layer, _ = build_layer(rng, cuda_device, 32, 4, D, I, max_tokens=T)
    x = x_tensor(synth.activations_np(rng, T, D), cuda_device)
    clean, got = (torch.zeros(T, D, dtype=torch.float32, device=cuda_device) for _ in range(2))
    layer.encode(x, clean, T)
    inds, wts = layer.views(T)["inds"].clone(), layer.views(T)["wts"].clone()
    layer.set_external_routing(inds, wts)  # (the router's logits of such a token are not the point)
    layer.encode(x, got, T)
    assert torch.equal(got, clean)
    bad = x.clone()
    bad[3, 70] = float("nan")
    bad[9, 5] = float("inf")
    bad[17] *= 2.0**13  # h is a product of two: 2^26 times as large
    layer.encode(bad, got, T)
    assert torch.isnan(got[3]).all() and torch.isnan(got[9]).all()
    assert not torch.isfinite(got[17]).any()
    keep = [t for t in range(T) if t not in (3, 9, 17)]
    assert torch.equal(got[keep], clean[keep])
    layer.set_external_routing(None, None)
