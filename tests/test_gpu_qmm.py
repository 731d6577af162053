"""Prefill GEMM on the tcgen05 tensor cores (iq_qmm through DenseQ.encode_qmm_f32) against the CPU oracle. Mirrors the
reference's qmm kernel cases (Tests/IngotTests/KernelCaseG32.swift:44-78, KernelCaseMixedBits.swift:98-121)."""
import numpy as np
import pytest
import torch

from ingot_b200 import capi, synth
from ingot_b200.linear import DenseMLP, DenseQ, VQMV
from oracle import qref
from gpu_util import TOL, affine_case, deq, mxfp4_case, x_tensor

pytestmark = pytest.mark.gpu


def run_qmm(m, x, rows, y_dtype=torch.float32, accumulate=False, y=None):
    ws = torch.empty(max(m.qmm_workspace_bytes(rows, x.dtype), 256), dtype=torch.uint8, device=x.device)
    if y is None:
        y = torch.zeros(rows, m.N, dtype=y_dtype, device=x.device)
    m.encode_qmm_f32(x, y, rows, accumulate=accumulate, workspace=ws)
    assert capi.context(0).device_status() == 0  # synchronises; no bounded wait gave up
    return y


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("M,N,K", [(64, 128, 64), (64, 64, 128), (128, 256, 512), (192, 192, 256), (256, 128, 2048),
                                   (320, 384, 1024), (512, 512, 4096)])
def test_qmm_affine_matches_oracle(cuda_device, bits, M, N, K):
    rng = np.random.default_rng(100 * bits + M + N + K)
    m, host = affine_case(rng, N, K, bits, cuda_device)
    x = synth.activations_np(rng, M, K)
    y = run_qmm(m, x_tensor(x, cuda_device), M)
    ref = qref.matmul_t(x, deq(host, bits))
    err = qref.max_rel(y.cpu().numpy(), ref)
    assert err <= TOL, err


def test_qmm_outputs_and_accumulate(cuda_device):
    rng = np.random.default_rng(21)
    M, N, K = 128, 256, 512
    m, host = affine_case(rng, N, K, 4, cuda_device)
    xh = synth.activations_np(rng, M, K)
    ref = qref.matmul_t(xh, deq(host, 4))
    x = x_tensor(xh, cuda_device)
    y32 = run_qmm(m, x, M)
    # half / bf16 outputs are the rounding of the kernel's own fp32 result (the reference loosens half outputs to 2e-3,
    # KernelCaseG32.swift:77)
    assert torch.equal(run_qmm(m, x, M, torch.float16), y32.to(torch.float16))
    assert torch.equal(run_qmm(m, x, M, torch.bfloat16), y32.to(torch.bfloat16))
    y0 = torch.from_numpy(rng.normal(size=(M, N)).astype(np.float32)).to(cuda_device)
    y = run_qmm(m, x, M, accumulate=True, y=y0.clone())
    assert qref.max_rel((y - y0).cpu().numpy(), ref) <= TOL
    # fp16 activations are used in place (no conversion pass), fp32 activations are converted
    for dt in (torch.float16, torch.float32):
        assert qref.max_rel(run_qmm(m, x_tensor(xh, cuda_device, dt), M).cpu().numpy(), ref) <= TOL


def test_qmm_mxfp4(cuda_device):
    rng = np.random.default_rng(22)
    M, N, K = 128, 192, 576
    m, host = mxfp4_case(rng, N, K, cuda_device)
    x = synth.activations_np(rng, M, K)
    y = run_qmm(m, x_tensor(x, cuda_device), M)
    assert qref.max_rel(y.cpu().numpy(), qref.matmul_t(x, deq(host))) <= TOL


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("M,N,K", [(512, 14336, 4096), (2048, 14336, 4096), (512, 4096, 14336), (2048, 4096, 14336)])
def test_qmm_prefill_configuration(cuda_device, bits, M, N, K):
    """The prefill configuration at full size: the oracle on 192 sampled output features, and agreement with the decode
    GEMV kernel (itself checked against the oracle) on 16 sampled token rows over every output feature."""
    rng = np.random.default_rng(bits + M + N)
    m, host = affine_case(rng, N, K, bits, cuda_device)
    x = synth.activations_np(rng, M, K)
    xt = x_tensor(x, cuda_device)
    y = run_qmm(m, xt, M)
    sel = np.sort(rng.choice(N, size=192, replace=False))
    wf = qref.dequant_affine(host[0][0][sel], host[1][0][sel], host[2][0][sel], bits)
    ref = qref.matmul_t(x, wf)
    err = qref.max_rel(y[:, torch.from_numpy(sel).to(cuda_device)].cpu().numpy(), ref)
    assert err <= TOL, err
    rows = torch.from_numpy(np.sort(rng.choice(M, size=16, replace=False))).to(cuda_device)
    yv = torch.zeros(16, N, dtype=torch.float32, device=cuda_device)
    VQMV.encode(xt[rows].contiguous(), m, yv, 16)
    torch.cuda.synchronize()
    scale = float(yv.abs().max())
    assert float((y[rows] - yv).abs().max()) / scale <= TOL


def test_qmm_rejects_what_the_reference_rejects(cuda_device):
    rng = np.random.default_rng(23)
    m, _ = affine_case(rng, 128, 128, 4, cuda_device)
    x = torch.zeros(96, 128, dtype=torch.float16, device=cuda_device)
    y = torch.zeros(96, 128, dtype=torch.float32, device=cuda_device)
    with pytest.raises(capi.IngotError) as e:
        m.encode_qmm_f32(x, y, 96)  # rows % 64 (Linear.swift:695)
    assert e.value.status == -1
    xb = torch.zeros(64, 128, dtype=torch.bfloat16, device=cuda_device)
    with pytest.raises(capi.IngotError) as e:
        m.encode_qmm_f32(xb, y, 64)  # bf16 activations need the conversion workspace
    assert e.value.status == -4


@pytest.mark.parametrize("fmt", ["q4", "q8", "mxfp4"])
@pytest.mark.parametrize("M,N,K", [(64, 64, 64), (192, 64, 192), (448, 192, 832), (1088, 2112, 320), (2048, 128, 1088), (64, 19008, 192)])
def test_qmm_tile_edges(cuda_device, fmt, M, N, K):
    """Odd numbers of K steps (1, 3, 5, 13, 17: stages of codes that end early, scales whose row pitch allows no vector copy),
    half tiles of output features, token tiles of other heights, more low tiles than SMs; accumulation onto an existing result."""
    rng = np.random.default_rng(M + N + K)
    m, host = mxfp4_case(rng, N, K, cuda_device) if fmt == "mxfp4" else affine_case(rng, N, K, int(fmt[1]), cuda_device)
    x = synth.activations_np(rng, M, K)
    ref = qref.matmul_t(x, deq(host, 4 if fmt == "mxfp4" else int(fmt[1])))
    xt = x_tensor(x, cuda_device)
    y = run_qmm(m, xt, M)
    assert qref.max_rel(y.cpu().numpy(), ref) <= TOL
    y2 = run_qmm(m, xt, M, accumulate=True, y=y.clone())
    assert torch.equal(y2, 2 * y)


def test_qmm_8bit_stages_of_odd_number(cuda_device):
    """64 rows at 8 bits: three stages of codes, each converted by two of the four groups; launches with the weights out of
    L2 give the same bits every time."""
    rng = np.random.default_rng(65)
    M, N, K = 64, 2048, 4096
    m, host = affine_case(rng, N, K, 8, cuda_device)
    x = synth.activations_np(rng, M, K)
    xt = x_tensor(x, cuda_device)
    y = run_qmm(m, xt, M)
    assert qref.max_rel(y.cpu().numpy(), qref.matmul_t(x, deq(host, 8))) <= TOL
    flush = torch.empty(160 << 20, dtype=torch.uint8, device=cuda_device)
    for _ in range(20):
        flush.zero_()
        assert torch.equal(run_qmm(m, xt, M), y)


@pytest.mark.parametrize("fmt,group", [("q4", 64), ("q8", 64), ("q4", 32), ("mxfp4", 32)])
@pytest.mark.parametrize("M", [64, 320])
def test_qmm_scales_by_plain_loads(cuda_device, fmt, group, M):
    """2880 inputs: the rows of scales are no multiple of the pieces that asynchronous copies take, so they go through plain loads
    and stores. Launches with everything out of L2, and with it in L2, give the same bits every time."""
    rng = np.random.default_rng(66 + M + group)
    N, K = 1152, 2880
    bits = 8 if fmt == "q8" else 4
    m, host = mxfp4_case(rng, N, K, cuda_device) if fmt == "mxfp4" else affine_case(rng, N, K, bits, cuda_device, group=group)
    x = synth.activations_np(rng, M, K)
    xt = x_tensor(x, cuda_device)
    y = run_qmm(m, xt, M)
    assert qref.max_rel(y.cpu().numpy(), qref.matmul_t(x, deq(host, bits, group=group))) <= TOL
    flush = torch.empty(160 << 20, dtype=torch.uint8, device=cuda_device)
    for i in range(20):
        if i % 2 == 0:
            flush.zero_()
        assert torch.equal(run_qmm(m, xt, M), y)


def shifted_scales(m, by):
    """The matrix with its MXFP4 scales `by` bytes into a larger tensor, as views of a mapped file have them."""
    buf = torch.full((m.s.numel() + 16,), 255, dtype=torch.uint8, device=m.s.device)  # (255 is NaN: a scale read beside its place shows)
    s = buf[by: by + m.s.numel()].view_as(m.s)
    s.copy_(m.s)
    assert s.data_ptr() % 16 == by
    return DenseQ(m.w, s, None, m.N, m.K, 4, 32, "mxfp4", m.experts)


@pytest.mark.parametrize("by", [1, 2, 4, 8, 9])
@pytest.mark.parametrize("K", [64, 576, 1024])
def test_mxfp4_scales_at_any_address(cuda_device, K, by):
    """MXFP4 scales are bytes: any address will do, in the GEMM, the GEMV and the dense FFN of few and of many rows."""
    rng = np.random.default_rng(67 + K + by)
    N = 192
    m, host = mxfp4_case(rng, N, K, cuda_device)
    o = shifted_scales(m, by)
    for M in (64, 320):
        x = synth.activations_np(rng, M, K)
        assert qref.max_rel(run_qmm(o, x_tensor(x, cuda_device), M).cpu().numpy(), qref.matmul_t(x, deq(host))) <= TOL
    dn, _ = mxfp4_case(rng, K, 64, cuda_device)
    gu, _ = mxfp4_case(rng, 128, K, cuda_device)
    for rows in (1, 7, 64):
        xt = x_tensor(synth.activations_np(rng, rows, K), cuda_device)
        a, b = (torch.zeros(rows, K, dtype=torch.float32, device=cuda_device) for _ in range(2))
        DenseMLP(gu, dn).encode(xt, a, rows)
        DenseMLP(shifted_scales(gu, by), shifted_scales(dn, by)).encode(xt, b, rows)
        assert qref.max_rel(b.cpu().numpy(), a.cpu().numpy()) <= TOL  # (other kernels where the address rules the first out)
        if rows <= 16:
            y = torch.zeros(rows, N, dtype=torch.float32, device=cuda_device)
            VQMV.encode(xt, o, y, rows)
            assert qref.max_rel(y.cpu().numpy(), qref.matmul_t(xt.float().cpu().numpy(), deq(host))) <= TOL
    assert capi.context(0).device_status() == 0


def path_of(fmt, group, rows, n, k, gate_up=False):
    """Which way the library takes: "pair" or "one" CTA per tile, "+split" where all tiles are divided along K, "+split+whole" where the
    first ones are."""
    p = capi.qmm_plan(2 * n if gate_up else n, k, 8 if fmt == "q8" else 4, group, rows, capi.IQ_MODE_MXFP4 if fmt == "mxfp4" else capi.IQ_MODE_AFFINE,
                      gate_up, torch.cuda.get_device_properties(0).multi_processor_count)
    return ("pair" if p.pair else "one") + ("" if p.split_tiles == 0 else "+split" if p.split_tiles == p.tiles else "+split+whole")


@pytest.mark.parametrize("fmt,group", [("q4", 64), ("q8", 64), ("q4", 32), ("mxfp4", 32)])
@pytest.mark.parametrize("M,N,K,path", [
    (64, 192, 14336, "one+split"), (64, 2112, 5824, "one+split"), (192, 128, 9216, "one+split"), (256, 9600, 1664, "one+split+whole"),
    (320, 9600, 2112, "one+split+whole"), (704, 1216, 8256, "pair+split"), (704, 5056, 4160, "pair+split+whole"),
    (64, 19456, 2112, "pair+split+whole"), (128, 7744, 2880, "one"), (320, 4096, 4160, "one"), (2048, 4096, 5120, "pair")])
def test_qmm_split_along_k(cuda_device, fmt, group, M, N, K, path):
    """Tiles that fill no whole round are divided along K: one tile in eight pieces and more, runs that end inside a tile, an odd number
    of stages, pieces before whole tiles, on one CTA and on pairs (a second CTA without features, a last token tile of another height,
    odd numbers of K steps). Against the oracle, against the call whose workspace has no room for the sums (every tile in one
    piece), the same bits every time, and added onto a result."""
    assert path_of(fmt, group, M, N, K) == path
    rng = np.random.default_rng(71 + M + N + K + group)
    bits = 8 if fmt == "q8" else 4
    m, host = mxfp4_case(rng, N, K, cuda_device) if fmt == "mxfp4" else affine_case(rng, N, K, bits, cuda_device, group=group)
    x = synth.activations_np(rng, M, K)
    xt = x_tensor(x, cuda_device)
    y = run_qmm(m, xt, M)
    sel = np.sort(rng.choice(N, size=min(N, 96), replace=False))
    some = tuple(h[:, sel] for h in host)
    ref = qref.matmul_t(x, deq(some, bits, group=group))
    got = y[:, torch.from_numpy(sel).to(cuda_device)].cpu().numpy()
    assert qref.max_rel(got, ref) <= TOL
    assert bool(torch.isfinite(y).all())
    whole = torch.zeros_like(y)
    m.encode_qmm_f32(xt, whole, M, workspace=torch.empty(M * K * 2, dtype=torch.uint8, device=cuda_device))
    # the same products in another order of sums: 14336 roundings of 2^-24, as a random walk, are 7e-6 of a sum's size
    assert float((y - whole).abs().max() / whole.abs().max()) <= 2e-5
    assert ("split" in path) or torch.equal(y, whole)
    assert torch.equal(run_qmm(m, xt, M), y)
    y0 = torch.randn(M, N, device=cuda_device)
    assert torch.equal(run_qmm(m, xt, M, accumulate=True, y=y0.clone()), y0 + y)
    assert torch.equal(run_qmm(m, x_tensor(x, cuda_device, torch.float16), M, torch.float16), y.to(torch.float16))


@pytest.mark.parametrize("fmt,group,act", [("q4", 64, "silu"), ("q4", 64, "swiglu_oai"), ("q8", 64, "silu"), ("q4", 32, "gelu"),
                                           ("mxfp4", 32, "swiglu_oai")])
@pytest.mark.parametrize("rows,d,d_ff,gate_up,down", [
    (64, 1216, 8768, "one", "one+split"), (256, 2048, 7680, "one", "one+split"), (320, 4160, 1088, "one", "one"),
    (64, 2112, 64, "one+split", "one"), (192, 2048, 256, "one+split", "one"), (704, 5120, 2880, "pair+split+whole", "one")])
def test_dense_ffn_split_along_k(cuda_device, fmt, group, act, rows, d, d_ff, gate_up, down):
    """The gated epilogue on the sums of pieces (on one CTA and on pairs, the last one with features for one of its CTAs), and the down
    projection's split, against a float64 product."""
    assert path_of(fmt, group, rows, d_ff, d, gate_up=True) == gate_up and path_of(fmt, group, rows, d, d_ff) == down
    rng = np.random.default_rng(72 + rows)
    bits = 8 if fmt == "q8" else 4
    mk = (lambda n, k: mxfp4_case(rng, n, k, cuda_device)) if fmt == "mxfp4" else (lambda n, k: affine_case(rng, n, k, bits, cuda_device, group=group))
    gu, hg = mk(2 * d_ff, d)
    dn, hd = mk(d, d_ff)
    x = x_tensor(synth.activations_np(rng, rows, d), cuda_device)
    out = torch.zeros(rows, d, dtype=torch.float32, device=cuda_device)
    DenseMLP(gu, dn, act).encode(x, out, rows)
    assert capi.context(0).device_status() == 0
    w = [torch.from_numpy(deq(h, bits, group=group)).to(cuda_device).double() for h in (hg, hd)]
    g, u = (x.double() @ w[0].T).split(d_ff, dim=1)
    if act == "silu":
        h = g / (1 + torch.exp(-g)) * u
    elif act == "gelu":
        h = torch.nn.functional.gelu(g, approximate="tanh") * u
    else:
        g, u = g.clamp(max=7.0), u.clamp(-7.0, 7.0)
        h = (u + 1) * g / (1 + torch.exp(-1.702 * g))
    ref = h.to(torch.float16).double() @ w[1].T
    assert float((out - ref).abs().max() / ref.abs().max()) <= TOL


@pytest.mark.parametrize("fmt,group", [("q4", 64), ("q8", 64), ("q4", 32), ("mxfp4", 32)])
@pytest.mark.parametrize("M,N,K,path", [
    (1472, 2112, 2112, "pair"), (576, 5056, 2112, "pair"), (1024, 2880, 2944, "pair"), (4096, 2880, 576, "pair"), (192, 9600, 2112, "pair"),
    (4096, 2112, 832, "one"), (2048, 192, 1088, "one"), (1088, 14400, 320, "one"), (4096, 64, 64, "one")])
def test_qmm_pairs_of_ctas(cuda_device, fmt, group, M, N, K, path):
    """Tall calls run on pairs of CTAs with twice the features per tile: a last pair with features for half of its first CTA, for half of
    its second one, token tiles whose halves differ and a last one of another height, odd numbers of K steps (and the same calls'
    neighbours that run on single CTAs); the same bits every time, and added onto a result."""
    assert path_of(fmt, group, M, N, K) == path
    rng = np.random.default_rng(81 + M + N + K + group)
    bits = 8 if fmt == "q8" else 4
    m, host = mxfp4_case(rng, N, K, cuda_device) if fmt == "mxfp4" else affine_case(rng, N, K, bits, cuda_device, group=group)
    x = synth.activations_np(rng, M, K)
    xt = x_tensor(x, cuda_device)
    y = run_qmm(m, xt, M)
    sel = np.unique(np.concatenate([np.sort(rng.choice(N, size=min(N, 64), replace=False)), np.arange(max(0, N - 16), N)]))
    rows = np.unique(np.concatenate([np.sort(rng.choice(M, size=64, replace=False)), np.arange(M - 16, M)]))
    ref = qref.matmul_t(x[rows], deq(tuple(h[:, sel] for h in host), bits, group=group))
    got = y[torch.from_numpy(rows).to(cuda_device)][:, torch.from_numpy(sel).to(cuda_device)].cpu().numpy()
    assert qref.max_rel(got, ref) <= TOL
    assert bool(torch.isfinite(y).all())
    for _ in range(3):
        assert torch.equal(run_qmm(m, xt, M), y)
    assert torch.equal(run_qmm(m, xt, M, accumulate=True, y=y.clone()), 2 * y)


def test_dense_ffn_scratch_outlives_fewer_rows(cuda_device):
    """Scratch sized by the largest call serves all smaller ones: a captured graph's addresses stay the module's own when fewer rows,
    whose GEMMs divide along K in more pieces, follow."""
    d, d_ff = 2048, 7680
    rng = np.random.default_rng(73)
    gu, _ = affine_case(rng, 2 * d_ff, d, 8, cuda_device)
    dn, _ = affine_case(rng, d, d_ff, 8, cuda_device)
    assert capi.qmm_plan(d, d_ff, 8, 64, 640).split_bytes < capi.qmm_plan(d, d_ff, 8, 64, 512).split_bytes
    mlp = DenseMLP(gu, dn)
    x = x_tensor(synth.activations_np(rng, 640, d), cuda_device)
    want = torch.zeros(640, d, dtype=torch.float32, device=cuda_device)
    mlp.encode(x, want, 640)
    at = mlp._ws.data_ptr()
    got = torch.zeros_like(want)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        mlp.encode(x, got, 640)
    for rows in (512, 320, 256, 64, 16, 3):
        out = torch.zeros(rows, d, dtype=torch.float32, device=cuda_device)
        mlp.encode(x[:rows], out, rows)
        assert mlp._ws.data_ptr() == at
        assert qref.max_rel(out.cpu().numpy(), want[:rows].cpu().numpy()) <= TOL
    g.replay()
    assert torch.equal(got, want)
    for fmt in (torch.bfloat16, torch.float16):
        assert dn.qmm_workspace_bytes(4096, fmt) >= max(dn.qmm_workspace_bytes(r, fmt) for r in range(64, 4096, 64))


@pytest.mark.parametrize("group", [64, 32])
def test_qmm_affine4_weights_are_one_rounding_at_any_scale(cuda_device, group):
    """Unit rows of x read the fp16 weights back: fma(q, s, b) rounded once, for scales just below and at 2^-4 (from where on the codes are
    converted another way, for all 32 rows of a warp as soon as one of their scales is that large), tiny, large and negative ones."""
    rng = np.random.default_rng(30 + group)
    N, K, M = 256, 512, 64
    w, _, _ = synth.affine_np(rng, N, K, 4, 1, group)
    s = rng.uniform(0.001, 0.0624, size=(1, N, K // group)).astype(np.float32) * rng.choice([-1, 1], size=(1, N, K // group))
    s[0, 32:64] = 2.0 ** rng.integers(-30, -5, size=(32, K // group))
    s[0, 70, ::2] = 0.0625           # one row of a warp, every other group
    s[0, 100:128] = rng.uniform(0.05, 300, size=(28, K // group))
    s[0, 130, 1] = -0.0625
    s[0, 131] = 0.06225586           # the largest below
    s = synth.bf16_bits_to_f32(synth.to_bf16_bits(s.astype(np.float32)))
    b = synth.bf16_bits_to_f32(synth.to_bf16_bits((-8 * s + rng.normal(0, 0.001, size=s.shape)).astype(np.float32)))
    m = synth.dense_q_affine(w, synth.to_bf16_bits(s), synth.to_bf16_bits(b), 4, cuda_device, group)
    q = np.stack([(w[0] >> (4 * j)) & 15 for j in range(8)], axis=-1).reshape(N, K).astype(np.float64)
    want = (q * np.repeat(s[0], group, axis=1).astype(np.float64) + np.repeat(b[0], group, axis=1)).astype(np.float16)
    for k0 in range(0, K, M):
        x = torch.zeros(M, K, dtype=torch.float16, device=cuda_device)
        x[torch.arange(M), k0 + torch.arange(M)] = 1
        got = run_qmm(m, x, M).cpu().numpy()
        assert np.array_equal(got.T, want[:, k0:k0 + M].astype(np.float32)), k0
