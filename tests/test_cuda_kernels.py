"""Numerics of the sm_100a kernels against plain PyTorch fp32 references of the same op."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from openvino_b200.ops import cuda as k
    k.lib()
    return k


def _rel_err(a, b):
    a, b = a.float(), b.float()
    return ((a - b).norm() / b.norm().clamp_min(1e-12)).item()


@pytest.mark.parametrize("T,N,K", [(1, 128, 64), (16, 256, 256), (64, 4096, 4096), (100, 384, 1024), (300, 512, 448),
                                   (2048, 1024, 512)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_gemm_dense(ops, T, N, K, dtype):
    torch.manual_seed(0)
    x = torch.randn(T, K, device="cuda", dtype=dtype)
    w = (torch.randn(N, K, device="cuda") * 0.05).to(dtype)
    bias = torch.randn(N, device="cuda").to(dtype)
    res = torch.randn(T, N, device="cuda").to(dtype)
    pw = ops.PackedWeight.from_dense(w, bias)
    y = ops.gemm(x, pw, residual=res)
    ops.check_status("gemm")
    ref = x.float() @ w.float().t() + bias.float() + res.float()
    assert _rel_err(y, ref) < 1e-2
    # activation epilogue, fp32 output
    y2 = ops.gemm(x, ops.PackedWeight.from_dense(w), act=ops.ACT_GELU_ERF, out_f32=True)
    ref2 = torch.nn.functional.gelu(x.float() @ w.float().t())
    assert _rel_err(y2, ref2) < 1e-2
    ops.check_status("gemm")


@pytest.mark.parametrize("T,N,K,splits", [(4, 256, 512, 1), (64, 512, 4096, 4), (64, 4096, 14336, 0), (33, 384, 1024, 8),
                                          (512, 1024, 1024, 1), (1000, 256, 2048, 1)])
def test_gemm_u4(ops, T, N, K, splits):
    from openvino_b200.utils import quant
    torch.manual_seed(1)
    gs = 128
    w = torch.randn(N, K, device="cuda") * 0.05
    q, s, z = quant.quantize_u4_asym(w, gs)
    wdq = quant.dequantize_u4(q, s, z, gs)
    pw = ops.PackedWeight.from_ir_u4(quant.pack_u4(q), s, quant.pack_u4(z), N, K, gs)
    x = torch.randn(T, K, device="cuda", dtype=torch.bfloat16)
    y = ops.gemm(x, pw, splits=splits)
    ops.check_status("gemm_u4")
    ref = x.float() @ wdq.t()
    assert _rel_err(y, ref) < 1.5e-2
    # run twice: identical bits (split-K reduction order is fixed)
    y2 = ops.gemm(x, pw, splits=splits)
    assert torch.equal(y, y2)


@pytest.mark.parametrize("fmt", ["bf16", "u4"])
@pytest.mark.parametrize("counts,block_t", [([40, 0, 300, 17], 0), ([5, 9, 1, 3, 0, 0, 7, 2], 16), ([256, 256], 128)])
def test_gemm_grouped_moe(ops, fmt, counts, block_t):
    """One launch runs every group (expert) on its own rows of stacked weights; the row offsets live on the device.
    Mode 1 (stacked along N: gate/up projections) and mode 2 (stacked along K: down projections), empty groups and
    partial row tiles included; the sorted gather / weighted combine kernels around it against plain indexing."""
    from openvino_b200.utils import quant
    torch.manual_seed(11)
    G, H, F = len(counts), 256, 384
    rows = sum(counts)
    cap = rows + 19                                      # rows past the last group hold garbage and stay untouched
    w1 = torch.randn(G, F, H, device="cuda") * 0.05      # [G, N = F, K = H]
    w2 = torch.randn(G, H, F, device="cuda") * 0.05      # [G, N = H, K = F]
    w1s = w1.reshape(G * F, H)                           # stacked along N
    w2s = w2.permute(1, 0, 2).reshape(H, G * F)          # stacked along K
    if fmt == "bf16":
        pw1 = ops.PackedWeight.from_dense(w1s.to(torch.bfloat16))
        pw2 = ops.PackedWeight.from_dense(w2s.to(torch.bfloat16))
        d1, d2 = w1s.to(torch.bfloat16).float(), w2s.to(torch.bfloat16).float()
    else:
        gs = 128
        q1, s1, z1 = quant.quantize_u4_asym(w1s, gs)
        q2, s2, z2 = quant.quantize_u4_asym(w2s, gs)
        pw1 = ops.PackedWeight.from_ir_u4(quant.pack_u4(q1), s1, quant.pack_u4(z1), G * F, H, gs)
        pw2 = ops.PackedWeight.from_ir_u4(quant.pack_u4(q2), s2, quant.pack_u4(z2), H, G * F, gs)
        d1, d2 = quant.dequantize_u4(q1, s1, z1, gs), quant.dequantize_u4(q2, s2, z2, gs)
    d1 = d1.reshape(G, F, H)
    d2 = d2.reshape(H, G, F).permute(1, 0, 2)
    offs = torch.tensor([0] + list(torch.tensor(counts).cumsum(0)), dtype=torch.int32, device="cuda")
    x = torch.randn(cap, H, device="cuda", dtype=torch.bfloat16)
    y1 = torch.full((cap, F), 7.0, device="cuda", dtype=torch.bfloat16)
    ops.gemm_grouped(x, pw1, offs, G, 1, out=y1, block_t=block_t)
    ops.check_status("grouped gemm, stacked along N")
    y2 = torch.full((cap, H), 7.0, device="cuda", dtype=torch.bfloat16)
    ops.gemm_grouped(y1, pw2, offs, G, 2, out=y2, block_t=block_t)
    ops.check_status("grouped gemm, stacked along K")
    o = 0
    for g, c in enumerate(counts):
        if c:
            ref1 = x[o:o + c].float() @ d1[g].t()
            assert _rel_err(y1[o:o + c], ref1) < 1.5e-2, (g, c)
            ref2 = y1[o:o + c].float() @ d2[g].t()
            assert _rel_err(y2[o:o + c], ref2) < 1.5e-2, (g, c)
        o += c
    assert torch.all(y1[rows:] == 7.0) and torch.all(y2[rows:] == 7.0)


def test_moe_sorted_gather_combine(ops):
    torch.manual_seed(12)
    T, E, k, H, e0, nloc = 300, 8, 2, 128, 2, 4
    logits = torch.randn(T, E, device="cuda")
    route = ops.moe_route_topk(logits, k)
    pos = torch.zeros(T, nloc, dtype=torch.int32, device="cuda")
    counts = torch.zeros(nloc, dtype=torch.int32, device="cuda")
    offsets = torch.zeros(nloc + 1, dtype=torch.int32, device="cuda")
    x = torch.randn(T, H, device="cuda", dtype=torch.bfloat16)
    xg = torch.zeros(T * k, H, device="cuda", dtype=torch.bfloat16)
    ops.moe_positions(route, e0, nloc, pos, counts)
    ops.moe_gather_sorted(x, pos, counts, offsets, xg)
    hit = route[:, e0:e0 + nloc] != 0
    assert counts.tolist() == hit.sum(0).tolist()
    assert offsets.tolist() == [0] + hit.sum(0).cumsum(0).tolist()
    for e in range(nloc):
        toks = hit[:, e].nonzero().flatten()
        assert torch.equal(pos[toks, e].long(), torch.arange(len(toks), device="cuda"))
        assert torch.equal(xg[offsets[e]:offsets[e + 1]], x[toks])
    assert torch.all(pos[~hit] == -1)
    # the experts' "results": row r of expert e becomes (e + 1) * row
    y = xg.clone()
    for e in range(nloc):
        y[offsets[e]:offsets[e + 1]] *= (e + 1)
    base = torch.randn(T, H, device="cuda", dtype=torch.bfloat16)
    dst = base.clone()
    ops.moe_combine_sorted(y, route, pos, offsets, dst, e0, accumulate=True)
    w = (route[:, e0:e0 + nloc] * torch.arange(1, nloc + 1, device="cuda")).sum(1, keepdim=True)
    ref = base.float() + w * x.float()
    assert _rel_err(dst, ref) < 1e-2
    dst2 = torch.full_like(base, 3.0)
    ops.moe_combine_sorted(y, route, pos, offsets, dst2, e0, accumulate=False)
    assert _rel_err(dst2, w * x.float()) < 1e-2
    # silu(gate) * up over the valid rows only (the count is read on the device)
    gu = torch.randn(T * k, 2 * H, device="cuda", dtype=torch.bfloat16)
    act = torch.full((T * k, H), 5.0, device="cuda", dtype=torch.bfloat16)
    ops.silu_mul(gu, out=act, nrows=offsets[nloc:])
    n = int(offsets[nloc])
    ref = torch.nn.functional.silu(gu[:n, :H].float()) * gu[:n, H:].float()
    assert _rel_err(act[:n], ref) < 1e-2 and torch.all(act[n:] == 5.0)
    ops.check_status("moe sorted")


def test_gemm_u8(ops):
    from openvino_b200.utils import quant
    torch.manual_seed(2)
    T, N, K, gs = 48, 256, 1024, 128
    w = torch.randn(N, K, device="cuda") * 0.05
    q, s, z = quant.quantize_u8_asym(w, gs)
    wdq = ((q.float().reshape(N, K // gs, gs) - z.float().unsqueeze(-1)) * s.float().unsqueeze(-1)).reshape(N, K)
    pw = ops.PackedWeight.from_ir_u8(q, s, z, N, K, gs)
    x = torch.randn(T, K, device="cuda", dtype=torch.bfloat16)
    y = ops.gemm(x, pw)
    ops.check_status("gemm_u8")
    assert _rel_err(y, x.float() @ wdq.t()) < 1.5e-2


@pytest.mark.parametrize("T,N,K", [(48, 256, 1024), (300, 384, 512), (7, 1000, 256)])
def test_gemm_f8_block_scaled(ops, T, N, K):
    """fp8 e4m3 weights with one fp32 scale per 128 x 128 tile (weight-only: activations stay bf16)."""
    from openvino_b200.utils import quant
    torch.manual_seed(4)
    w = torch.randn(N, K, device="cuda") * 0.05
    w[0, :16] = 1e-5          # lands in the fp8 sub-normal range of its tile
    q, s = quant.quantize_f8_block(w, 128)
    wdq = quant.dequantize_f8_block(q, s, 128)
    assert _rel_err(wdq, w) < 5e-2
    pw = ops.PackedWeight.from_f8_block(q, s, N, K, 128)
    x = torch.randn(T, K, device="cuda", dtype=torch.bfloat16)
    y = ops.gemm(x, pw)
    ops.check_status("gemm_f8")
    assert _rel_err(y, x.float() @ wdq.t()) < 1e-2


@pytest.mark.parametrize("B,C,H,W,O,k,stride,pad,dil", [(2, 3, 32, 32, 64, 7, 2, 3, 1), (1, 64, 14, 14, 128, 3, 1, 1, 1),
                                                        (3, 32, 9, 11, 48, 3, 2, 1, 1), (2, 16, 8, 8, 32, 1, 1, 0, 1), (1, 8, 12, 12, 16, 3, 1, 2, 2)])
def test_conv2d_im2col_gemm(ops, B, C, H, W, O, k, stride, pad, dil):
    torch.manual_seed(5)
    x = torch.randn(B, C, H, W, device="cuda", dtype=torch.bfloat16)
    w = (torch.randn(O, C, k, k, device="cuda") * 0.1).to(torch.bfloat16)
    pw = ops.pack_conv_weight(w)
    y = ops.conv2d(x, pw, [k, k], [stride, stride], [pad, pad], [pad, pad], [dil, dil])
    ops.check_status("conv2d")
    ref = torch.nn.functional.conv2d(x.float(), w.float(), None, stride, pad, dil)
    assert list(y.shape) == list(ref.shape)
    assert _rel_err(y, ref) < 1e-2


@pytest.mark.parametrize("T,wmode", [(48, "bf16"), (300, "bf16"), (64, "u4"), (1000, "u4")])
def test_gemm_fused_swiglu(ops, T, wmode):
    from openvino_b200.utils import quant
    torch.manual_seed(9)
    F, K = 384, 512
    gate = torch.randn(F, K, device="cuda") * 0.05
    up = torch.randn(F, K, device="cuda") * 0.05
    w = ops.interleave_gate_up(gate, up)
    x = torch.randn(T, K, device="cuda", dtype=torch.bfloat16)
    if wmode == "bf16":
        pw = ops.PackedWeight.from_dense(w.to(torch.bfloat16))
        gq, uq = gate.to(torch.bfloat16).float(), up.to(torch.bfloat16).float()
    else:
        q, s, z = quant.quantize_u4_asym(w, 128)
        pw = ops.PackedWeight.from_ir_u4(quant.pack_u4(q), s, quant.pack_u4(z), 2 * F, K, 128)
        wd = quant.dequantize_u4(q, s, z, 128).float().reshape(F // 64, 2, 64, K)
        gq, uq = wd[:, 0].reshape(F, K), wd[:, 1].reshape(F, K)
    y = ops.gemm(x, pw, act=ops.ACT_SWIGLU)
    ops.check_status("gemm swiglu")
    assert list(y.shape) == [T, F]
    ref = torch.nn.functional.silu(x.float() @ gq.t()) * (x.float() @ uq.t())
    assert _rel_err(y, ref) < 2e-2


def test_gumbel_sampling_matches_softmax_and_shards_agree(ops):
    torch.manual_seed(8)
    V = 512
    logits = (torch.randn(1, V, device="cuda") * 2.0).to(torch.bfloat16)
    step = torch.zeros(1, dtype=torch.int32, device="cuda")
    rows = logits.expand(4096, V).contiguous()
    counts = torch.zeros(V, device="cuda")
    for it in range(8):
        step.fill_(it)
        ids = ops.sample_gumbel(rows, 0.8, seed=11, step=step)
        counts += torch.bincount(ids.long(), minlength=V).float()
    ops.check_status("sample_gumbel")
    p = torch.softmax(logits.float()[0] / 0.8, -1)
    freq = counts / counts.sum()
    top = torch.topk(p, 20).indices
    assert (freq[top] - p[top]).abs().max() < 0.01 and (freq - p).abs().sum() < 0.12
    # two vocabulary shards with global indices give the full-vocabulary draw
    x = (torch.randn(32, V, device="cuda") * 3.0).to(torch.bfloat16)
    full_max = torch.empty(32, device="cuda")
    full = ops.sample_gumbel(x, 1.3, seed=5, step=step, out_max=full_max)
    m0, m1 = torch.empty(32, device="cuda"), torch.empty(32, device="cuda")
    i0 = ops.sample_gumbel(x[:, :256].contiguous(), 1.3, seed=5, step=step, vocab_offset=0, out_max=m0)
    i1 = ops.sample_gumbel(x[:, 256:].contiguous(), 1.3, seed=5, step=step, vocab_offset=256, out_max=m1)
    merged = torch.where(m0 >= m1, i0, i1 + 256)
    assert torch.equal(merged, full) and torch.equal(torch.maximum(m0, m1), full_max)


def test_gumbel_noise_stays_finite_on_a_large_flat_vocabulary(ops):
    # 64 rows x 128256 tokens x 4 steps = 33M uniforms: with a 24-bit mapping about two of them would round to exactly 1
    V = 128256
    logits = torch.zeros(64, V, device="cuda", dtype=torch.bfloat16)
    step = torch.zeros(1, dtype=torch.int32, device="cuda")
    out_max = torch.empty(64, device="cuda")
    for it in range(4):
        step.fill_(it)
        ids = ops.sample_gumbel(logits, 1.0, seed=3, step=step, out_max=out_max)
        assert torch.isfinite(out_max).all() and int(ids.min()) >= 0 and int(ids.max()) < V
    ops.check_status("sample_gumbel")


def test_act_quant_fp8_groups_of_128(ops):
    torch.manual_seed(6)
    x = (torch.randn(37, 512, device="cuda") * torch.logspace(-2, 1, 512, device="cuda")).to(torch.bfloat16)
    q, s = ops.act_quant_fp8(x)
    ops.check_status("act_quant_fp8")
    xf = x.float().reshape(37, 4, 128)
    want_s = xf.abs().amax(-1) / 448.0
    assert torch.allclose(s, want_s, rtol=1e-5), (s - want_s).abs().max()
    deq = q.view(torch.float8_e4m3fn).float().reshape(37, 4, 128) * s.unsqueeze(-1)
    assert _rel_err(deq, xf) < 4e-2                       # e4m3: 3 mantissa bits
    ref_q = (xf / want_s.unsqueeze(-1)).to(torch.float8_e4m3fn).view(torch.uint8).reshape(37, 512)
    assert (q == ref_q).float().mean() > 0.98          # x * (1 / scale) against x / scale: the last bit may differ on ties


def test_kv_block_copy_and_lora(ops):
    torch.manual_seed(7)
    k = torch.randn(12, 8, 16, 128, device="cuda", dtype=torch.bfloat16)
    v = torch.randn(12, 8, 16, 128, device="cuda", dtype=torch.bfloat16)
    k0, v0 = k.clone(), v.clone()
    src = torch.tensor([1, 5, 7], dtype=torch.int32, device="cuda")
    dst = torch.tensor([2, 9, 7], dtype=torch.int32, device="cuda")
    ops.kv_block_copy(k, v, src, dst)
    ops.check_status("kv_block_copy")
    want_k, want_v = k0.clone(), v0.clone()
    want_k[dst.long()], want_v[dst.long()] = k0[src.long()], v0[src.long()]
    assert torch.equal(k, want_k) and torch.equal(v, want_v)
    x = torch.randn(40, 256, device="cuda", dtype=torch.bfloat16)
    a = (torch.randn(64, 256, device="cuda") * 0.05).to(torch.bfloat16)
    b = (torch.randn(384, 64, device="cuda") * 0.05).to(torch.bfloat16)
    y = torch.randn(40, 384, device="cuda", dtype=torch.bfloat16)
    out = ops.lora_apply(x, ops.PackedWeight.from_dense(a), ops.PackedWeight.from_dense(b), y, alpha=0.5)
    ref = y.float() + 0.5 * (x.float() @ a.float().t()) @ b.float().t()
    assert _rel_err(out, ref) < 1e-2


@pytest.mark.parametrize("rows,cols", [(3, 128), (64, 4096), (17, 8192), (5, 14336)])
def test_rmsnorm(ops, rows, cols):
    torch.manual_seed(3)
    x = torch.randn(rows, cols, device="cuda", dtype=torch.bfloat16)
    r = torch.randn(rows, cols, device="cuda", dtype=torch.bfloat16)
    g = torch.randn(cols, device="cuda", dtype=torch.bfloat16)
    y = ops.rmsnorm(x, g, 1e-5)
    xf = x.float()
    ref = xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + 1e-5) * g.float()
    assert _rel_err(y, ref) < 5e-3
    ro = torch.empty_like(x)
    y2 = ops.rmsnorm(x, g, 1e-5, residual=r, residual_out=ro)
    h = (x.float() + r.float()).to(torch.bfloat16).float()
    ref2 = h * torch.rsqrt(h.pow(2).mean(-1, keepdim=True) + 1e-5) * g.float()
    assert _rel_err(y2, ref2) < 5e-3
    assert _rel_err(ro, h) < 1e-6


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_layernorm(ops, dtype):
    torch.manual_seed(4)
    x = torch.randn(33, 1024, device="cuda", dtype=dtype)
    r = torch.randn(33, 1024, device="cuda", dtype=dtype)
    g = torch.randn(1024, device="cuda", dtype=dtype)
    b = torch.randn(1024, device="cuda", dtype=dtype)
    y = ops.layernorm(x, g, b, 1e-12, residual=r)
    ref = torch.nn.functional.layer_norm(x.float() + r.float(), (1024,), g.float(), b.float(), 1e-12)
    assert _rel_err(y, ref) < 5e-3


def test_silu_mul_embedding_argmax_add(ops):
    torch.manual_seed(5)
    gu = torch.randn(37, 2 * 1024, device="cuda", dtype=torch.bfloat16)
    y = ops.silu_mul(gu)
    ref = torch.nn.functional.silu(gu[:, :1024].float()) * gu[:, 1024:].float()
    assert _rel_err(y, ref) < 5e-3
    table = torch.randn(1000, 256, device="cuda", dtype=torch.bfloat16)
    ids = torch.randint(0, 1000, (77,), device="cuda")
    assert torch.equal(ops.embedding(ids, table), table[ids])
    logits = torch.randn(9, 128256, device="cuda", dtype=torch.bfloat16)
    am = ops.argmax(logits)
    ref_max = logits.float().max(dim=-1).values
    assert torch.equal(logits.float().gather(1, am[:, None])[:, 0], ref_max)
    # first index on ties
    logits[:, 5] = 100.0
    logits[:, 77] = 100.0
    assert torch.equal(ops.argmax(logits), torch.full((9,), 5, device="cuda"))
    a = torch.randn(64, 512, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(64, 512, device="cuda", dtype=torch.bfloat16)
    assert _rel_err(ops.add(a, b), a.float() + b.float()) < 5e-3


def _rope_ref(x, pos, theta):
    # x [T, H, D] float; half-rotate (LLaMA) convention
    T, H, D = x.shape
    inv = theta ** (-torch.arange(0, D, 2, device=x.device, dtype=torch.float32) / D)
    ang = pos.float()[:, None] * inv[None, :]
    cos, sin = ang.cos()[:, None, :], ang.sin()[:, None, :]
    x1, x2 = x[..., : D // 2], x[..., D // 2:]
    return torch.cat([x1 * cos - x2 * sin, x2 * cos + x1 * sin], dim=-1)


def _make_paged_batch(q_lens, past_lens, block_size, device, shuffle=True):
    """Block tables for a ragged batch; returns descriptors and total block count."""
    B = len(q_lens)
    nblocks = [(p + q + block_size - 1) // block_size for p, q in zip(past_lens, q_lens)]
    total = sum(nblocks)
    perm = torch.randperm(total) if shuffle else torch.arange(total)
    block_indices = perm.to(torch.int32)
    bib = [0]
    for n in nblocks:
        bib.append(bib[-1] + n)
    sb = [0]
    for q in q_lens:
        sb.append(sb[-1] + q)
    to = lambda v: torch.tensor(v, dtype=torch.int32, device=device)
    return to(past_lens), to(sb), block_indices.to(device), to(bib), total


def _attn_ref(q, k_all, v_all, q_lens, past_lens, Hq, Hkv, D, scale, window=0):
    """q [T, Hq, D] fp32; k_all/v_all: list per sequence of [ctx, Hkv, D] fp32."""
    outs = []
    t = 0
    G = Hq // Hkv
    for b, (ql, pl) in enumerate(zip(q_lens, past_lens)):
        qb = q[t:t + ql]                                  # [ql, Hq, D]
        kb = k_all[b].repeat_interleave(G, dim=1)         # [ctx, Hq, D]
        vb = v_all[b].repeat_interleave(G, dim=1)
        s = torch.einsum("qhd,khd->hqk", qb, kb) * scale
        ctx = pl + ql
        qpos = pl + torch.arange(ql, device=q.device)
        kpos = torch.arange(ctx, device=q.device)
        mask = kpos[None, :] <= qpos[:, None]
        if window > 0:
            mask &= kpos[None, :] > (qpos[:, None] - window)
        s = s.masked_fill(~mask[None], float("-inf"))
        p = torch.softmax(s, dim=-1)
        outs.append(torch.einsum("hqk,khd->qhd", p, vb))
        t += ql
    return torch.cat(outs, dim=0)


@pytest.mark.parametrize("q_lens,past_lens,Hq,Hkv", [
    ([5], [0], 4, 1),
    ([40, 17, 128], [0, 3, 70], 8, 2),
    ([1, 1, 1, 1], [0, 15, 16, 300], 8, 2),            # decode
    ([1] * 7, [5, 1000, 77, 256, 31, 32, 511], 32, 8),  # decode, GQA 4
    ([200, 1], [56, 9], 32, 8),                         # mixed
    ([700, 130, 33], [330, 900, 0], 32, 8),             # long contexts: many key tiles per query tile, both stages reused
    ([300, 520], [0, 64], 8, 8),                        # one query head per KV head
    ([260], [100], 16, 2),                              # eight query heads per KV head
])
def test_rope_kv_write_and_paged_attention(ops, q_lens, past_lens, Hq, Hkv):
    torch.manual_seed(6)
    D, bs, theta = 128, 16, 500000.0
    dev = "cuda"
    pl_t, sb_t, bi_t, bib_t, total_blocks = _make_paged_batch(q_lens, past_lens, bs, dev)
    T = sum(q_lens)
    k_cache = torch.zeros(total_blocks, Hkv, bs, D, device=dev, dtype=torch.bfloat16)
    v_cache = torch.zeros_like(k_cache)
    # history: fill the cache with past tokens through the same write kernel
    k_hist, v_hist = [], []
    for b, pl in enumerate(past_lens):
        kh = torch.randn(pl, Hkv, D, device=dev).to(torch.bfloat16)
        vh = torch.randn(pl, Hkv, D, device=dev).to(torch.bfloat16)
        k_hist.append(kh)
        v_hist.append(vh)
        blocks = bi_t[bib_t[b]:bib_t[b + 1]].long()
        for j in range(pl):
            k_cache[blocks[j // bs], :, j % bs] = kh[j]
            v_cache[blocks[j // bs], :, j % bs] = vh[j]
    qkv = torch.randn(T, (Hq + 2 * Hkv) * D, device=dev).to(torch.bfloat16)
    positions, slots = [], []
    for b, (ql, pl) in enumerate(zip(q_lens, past_lens)):
        blocks = bi_t[bib_t[b]:bib_t[b + 1]].long().tolist()
        for j in range(pl, pl + ql):
            positions.append(j)
            slots.append(blocks[j // bs] * bs + j % bs)
    positions = torch.tensor(positions, dtype=torch.int32, device=dev)
    slots = torch.tensor(slots, dtype=torch.int32, device=dev)
    qkv0 = qkv.clone()
    ops.rope_kv_write(qkv, positions, slots, k_cache, v_cache, Hq, Hkv, D, theta, bs)
    q_ref = _rope_ref(qkv0[:, : Hq * D].float().reshape(T, Hq, D), positions, theta)
    k_new = _rope_ref(qkv0[:, Hq * D:(Hq + Hkv) * D].float().reshape(T, Hkv, D), positions, theta)
    v_new = qkv0[:, (Hq + Hkv) * D:].float().reshape(T, Hkv, D)
    assert _rel_err(qkv[:, : Hq * D].reshape(T, Hq, D), q_ref) < 5e-3
    # gather cache rows of the new tokens
    kc = k_cache.permute(0, 2, 1, 3).reshape(-1, Hkv, D)[slots.long()]
    vc = v_cache.permute(0, 2, 1, 3).reshape(-1, Hkv, D)[slots.long()]
    assert _rel_err(kc, k_new) < 5e-3
    assert torch.equal(vc.float(), v_new)

    scale = 1.0 / math.sqrt(D)
    out = ops.paged_attention(qkv, k_cache, v_cache, pl_t, sb_t, bi_t, bib_t, Hq, Hkv, D, scale=scale,
                              max_context_len=max(p + q for p, q in zip(past_lens, q_lens)), max_q_len=max(q_lens))
    ops.check_status("paged_attention")
    k_all, v_all = [], []
    t = 0
    for b, ql in enumerate(q_lens):
        k_all.append(torch.cat([k_hist[b].float(), kc[t:t + ql].float()], dim=0))
        v_all.append(torch.cat([v_hist[b].float(), vc[t:t + ql].float()], dim=0))
        t += ql
    ref = _attn_ref(qkv[:, : Hq * D].float().reshape(T, Hq, D), k_all, v_all, q_lens, past_lens, Hq, Hkv, D, scale)
    assert _rel_err(out.reshape(T, Hq, D), ref) < 1e-2


@pytest.mark.parametrize("q_lens,past_lens,Hq,Hkv", [
    ([1, 1, 1, 1], [0, 15, 16, 300], 8, 2),             # decode
    ([1] * 5, [5, 1000, 77, 256, 511], 32, 8),          # decode, split over the keys
    ([40, 17, 128], [0, 3, 70], 8, 2),                  # prefill with history
    ([200, 1], [56, 9], 32, 8),                         # mixed
    ([90], [300], 4, 4),
])
def test_u8_kv_cache_write_and_attention(ops, q_lens, past_lens, Hq, Hkv):
    """KV_CACHE_PRECISION = u8: rows are quantised per (token, head) by the write kernel; decode and prefill attention read
    the bytes. Reference: fp32 attention over the dequantised cache ((byte - zero point) * scale)."""
    torch.manual_seed(16)
    D, bs, theta, dev = 128, 16, 10000.0, "cuda"
    pl_t, sb_t, bi_t, bib_t, total_blocks = _make_paged_batch(q_lens, past_lens, bs, dev)
    B = len(q_lens)
    k_cache = torch.zeros(total_blocks, Hkv, bs, D, device=dev, dtype=torch.uint8)
    v_cache = torch.zeros_like(k_cache)
    k_meta = torch.zeros(total_blocks, Hkv, bs, 2, device=dev, dtype=torch.float16)
    v_meta = torch.zeros_like(k_meta)

    def write(n_tok_per_seq, start_per_seq):
        """Runs the write kernel for tokens [start, start + n) of every sequence; returns (qkv after RoPE, raw qkv, positions)."""
        pos, slots = [], []
        for b in range(B):
            blocks = bi_t[bib_t[b]:bib_t[b + 1]].long().tolist()
            for j in range(start_per_seq[b], start_per_seq[b] + n_tok_per_seq[b]):
                pos.append(j)
                slots.append(blocks[j // bs] * bs + j % bs)
        T = len(pos)
        if T == 0:
            return None, None, None, None
        qkv = torch.randn(T, (Hq + 2 * Hkv) * D, device=dev).to(torch.bfloat16)
        raw = qkv.clone()
        pos_t = torch.tensor(pos, dtype=torch.int32, device=dev)
        slots_t = torch.tensor(slots, dtype=torch.int32, device=dev)
        ops.rope_kv_write_u8(qkv, pos_t, slots_t, k_cache, v_cache, k_meta, v_meta, Hq, Hkv, D, theta, bs)
        return qkv, raw, pos_t, slots_t

    write(past_lens, [0] * B)                                        # history
    qkv, raw, pos_t, slots_t = write(q_lens, past_lens)              # the step's tokens
    T = sum(q_lens)
    # the write: queries rotated in place, rows quantised within half a step of the fp32 value
    q_ref = _rope_ref(raw[:, : Hq * D].float().reshape(T, Hq, D), pos_t, theta)
    assert _rel_err(qkv[:, : Hq * D].reshape(T, Hq, D), q_ref) < 5e-3
    k_new = _rope_ref(raw[:, Hq * D:(Hq + Hkv) * D].float().reshape(T, Hkv, D), pos_t, theta)
    v_new = raw[:, (Hq + Hkv) * D:].float().reshape(T, Hkv, D)

    def deq(cache, meta):
        return (cache.float() - meta[..., 1:2].float()) * meta[..., 0:1].float()
    kd, vd = deq(k_cache, k_meta), deq(v_cache, v_meta)
    kc = kd.permute(0, 2, 1, 3).reshape(-1, Hkv, D)[slots_t.long()]
    vc = vd.permute(0, 2, 1, 3).reshape(-1, Hkv, D)[slots_t.long()]
    for got, want in ((kc, k_new), (vc, v_new)):
        step = (want.amax(-1) - want.amin(-1)) / 255.0
        assert ((got - want).abs() <= 0.75 * step.unsqueeze(-1) + 1e-3).all()

    out = ops.paged_attention(qkv, k_cache, v_cache, pl_t, sb_t, bi_t, bib_t, Hq, Hkv, D, scale=1.0 / math.sqrt(D),
                              max_context_len=max(p + q for p, q in zip(past_lens, q_lens)), max_q_len=max(q_lens), k_meta=k_meta, v_meta=v_meta)
    ops.check_status("paged_attention u8")
    k_all, v_all = [], []
    for b in range(B):
        blocks = bi_t[bib_t[b]:bib_t[b + 1]].long()
        ctx = past_lens[b] + q_lens[b]
        k_all.append(kd[blocks].permute(0, 2, 1, 3).reshape(-1, Hkv, D)[:ctx])
        v_all.append(vd[blocks].permute(0, 2, 1, 3).reshape(-1, Hkv, D)[:ctx])
    ref = _attn_ref(qkv[:, : Hq * D].float().reshape(T, Hq, D), k_all, v_all, q_lens, past_lens, Hq, Hkv, D, 1 / math.sqrt(D))
    assert _rel_err(out.reshape(T, Hq, D), ref) < 1e-2


@pytest.mark.parametrize("Hq,Hkv,window", [(32, 8, 0), (8, 8, 0), (16, 8, 0), (64, 8, 0), (32, 8, 300), (64, 8, 77)])
def test_u8_kv_cache_decode_shares_keys_per_sequence(ops, Hq, Hkv, window):
    """A captured length (2048) above the real ones: the keys of every sequence are shared out by its own length, some splits stay
    empty. Zero points far from 128, and rows that are not visible (behind the last key, before the window) hold pairs of NaN and inf."""
    g = torch.Generator(device="cuda").manual_seed(Hq + window)
    D, bs, dev, top = 128, 16, "cuda", 2048
    ctx = ([1, 2, 15, 255, 256, 257, 300, 900, 1023, 1500, 1999, 2048] * 2)
    B = len(ctx)
    past, sub, bi, bib, blocks = _make_paged_batch([1] * B, [c - 1 for c in ctx], bs, dev)
    caches, metas, wide = [], [], []
    seen = torch.zeros(blocks, bs, dtype=torch.bool, device=dev)
    for b in range(B):
        pos = torch.arange(max(0, ctx[b] - window) if window else 0, ctx[b], device=dev)
        seen[bi[bib[b]:bib[b + 1]].long()[pos // bs], pos % bs] = True
    for _ in range(2):
        q = torch.randint(0, 256, (blocks, Hkv, bs, D), dtype=torch.uint8, device=dev, generator=g)
        scale = torch.rand(blocks, Hkv, bs, device=dev, generator=g) * 0.02 + 0.004
        zero = torch.tensor([128.0, 0.0, 255.0, -300.0, 700.0, 131.5], device=dev)[torch.randint(0, 6, (blocks, Hkv, bs), device=dev, generator=g)]
        meta = torch.stack([scale, zero], -1).half()
        wide.append((q.double() - meta[..., 1:].double()) * meta[..., :1].double())
        meta = torch.where(seen[:, None, :, None], meta, torch.tensor([float("nan"), float("inf")], device=dev, dtype=torch.float16))
        caches.append(q)
        metas.append(meta.contiguous())
    qkv = (torch.randn(B, (Hq + 2 * Hkv) * D, device=dev, generator=g) * 0.3).bfloat16()
    out = ops.paged_attention(qkv, *caches, past, sub, bi, bib, Hq, Hkv, D, scale=1.0 / math.sqrt(D), sliding_window=window, max_context_len=top, max_q_len=1,
                              k_meta=metas[0], v_meta=metas[1])
    ops.check_status("paged_attention u8")
    rows = [[c[bi[bib[b]:bib[b + 1]].long()].permute(0, 2, 1, 3).reshape(-1, Hkv, D)[:ctx[b]] for b in range(B)] for c in wide]
    ref = _attn_ref(qkv[:, :Hq * D].double().reshape(B, Hq, D), *rows, [1] * B, [c - 1 for c in ctx], Hq, Hkv, D, 1 / math.sqrt(D), window)
    # the bytes, scales and sums are exact to fp32 and the weights of the values to 2^-17: what is left is the rounding of the result to
    # bf16, uniform up to 2^-8 of a value and less towards the upper end of a binade: 1.7e-3 in the 2-norm of many values
    off = (out.reshape(B, Hq, D).double() - ref).norm(dim=(1, 2)) / ref.norm(dim=(1, 2))
    assert off.max() < 2.2e-3, off


def test_paged_attention_sliding_window(ops):
    torch.manual_seed(7)
    Hq, Hkv, D, bs = 8, 2, 128, 16
    for q_lens, past_lens in ([[90], [40]], [[1, 1], [200, 37]]):
        pl_t, sb_t, bi_t, bib_t, total_blocks = _make_paged_batch(q_lens, past_lens, bs, "cuda")
        T = sum(q_lens)
        k_cache = torch.randn(total_blocks, Hkv, bs, D, device="cuda").to(torch.bfloat16)
        v_cache = torch.randn(total_blocks, Hkv, bs, D, device="cuda").to(torch.bfloat16)
        q = torch.randn(T, Hq * D, device="cuda").to(torch.bfloat16)
        out = ops.paged_attention(q, k_cache, v_cache, pl_t, sb_t, bi_t, bib_t, Hq, Hkv, D,
                                  max_context_len=max(p + q_ for p, q_ in zip(past_lens, q_lens)),
                                  max_q_len=max(q_lens), sliding_window=32)
        k_all, v_all = [], []
        for b in range(len(q_lens)):
            blocks = bi_t[bib_t[b]:bib_t[b + 1]].long()
            ctx = past_lens[b] + q_lens[b]
            k_all.append(k_cache[blocks].permute(0, 2, 1, 3).reshape(-1, Hkv, D)[:ctx].float())
            v_all.append(v_cache[blocks].permute(0, 2, 1, 3).reshape(-1, Hkv, D)[:ctx].float())
        ref = _attn_ref(q.float().reshape(T, Hq, D), k_all, v_all, q_lens, past_lens, Hq, Hkv, D, 1 / math.sqrt(D), 32)
        assert _rel_err(out.reshape(T, Hq, D), ref) < 1e-2


@pytest.mark.parametrize("S", [200, 384, 1000])
@pytest.mark.parametrize("dtype,D", [(torch.float16, 64), (torch.bfloat16, 128), (torch.bfloat16, 64), (torch.float16, 128)])
def test_sdpa_dense(ops, dtype, D, S):
    torch.manual_seed(8)
    B, H = 3, 4
    qkv = torch.randn(B * S, 3 * H * D, device="cuda").to(dtype)
    q, k, v = qkv[:, : H * D], qkv[:, H * D: 2 * H * D], qkv[:, 2 * H * D:]
    out = ops.sdpa_dense(q, k, v, B, S, H, D, ld=3 * H * D)
    qf, kf, vf = [t.float().reshape(B, S, H, D).transpose(1, 2) for t in (q, k, v)]
    ref = torch.nn.functional.scaled_dot_product_attention(qf, kf, vf).transpose(1, 2).reshape(B * S, H * D)
    assert _rel_err(out, ref) < 1e-2


def _expected_draw(row: np.ndarray, temp: float, top_k: int, top_p: float, seed: int, step: int, index: int):
    """The kept set in 64 bits and, for the random number of (seed, step, row), the tokens around the target: a target within 1e-5
    of the total mass of a boundary between two tokens (fp32 sums of up to 128k terms) may fall on either side."""
    def mix(z):
        z = (z + 0x9E3779B97F4A7C15) & M
        z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & M
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & M
        return z ^ (z >> 31)
    M = (1 << 64) - 1
    u = ((mix(seed ^ mix((step << 20) ^ index)) >> 40) + 0.5) / 16777216.0
    p = np.exp((row.astype(np.float64) - row.max()) / temp)
    order = np.argsort(-row, kind="stable")
    thr = []
    if 0 < top_k < len(row):
        thr.append(row[order[top_k - 1]])
    if top_p < 1.0:
        thr.append(row[order[np.searchsorted(np.cumsum(p[order]), top_p * p.sum())]])
    kept = np.nonzero(row >= max(thr))[0] if thr else np.arange(len(row))
    cum = np.cumsum(p[kept]) / p[kept].sum()
    at = [min(np.searchsorted(cum, u + d), len(kept) - 1) for d in (-1e-5, 1e-5)]
    return {int(t) for t in kept[at[0]:at[1] + 1]}


@pytest.mark.parametrize("V,ld,dtype", [(128256, 128256, torch.bfloat16), (32007, 32011, torch.bfloat16), (1, 8, torch.bfloat16), (9, 9, torch.float32),
                                        (8191, 8192, torch.float32), (70001, 70001, torch.bfloat16)])
@pytest.mark.parametrize("top_k,top_p", [(50, 0.95), (0, 1.0), (0, 0.6), (9000, 1.0), (1, 1.0)])
def test_sampling_kernel_draws(ops, V, ld, dtype, top_k, top_p):
    """Rows of aligned, odd and tiny lengths; kept sets that fit the per-warp lists and sets that do not (top_k 9000; equal logits)."""
    g = torch.Generator(device="cuda").manual_seed(V + top_k)
    rows = (torch.randn(5, ld, device="cuda", generator=g) * 2).to(dtype)
    rows[3, :V] = 0.25                                       # all equal
    rows[4, :V] = torch.arange(V, device="cuda").flip(0).to(dtype) * -1e-4   # large entries side by side: one warp's piece holds them all
    rows[4, V // 2] = 3.0
    step = torch.tensor([17], dtype=torch.int32, device="cuda")
    got = ops.sample(rows[:, :V], 0.8, top_k=top_k, top_p=top_p, seed=21, step=step).cpu()
    again = ops.sample(rows[:, :V], 0.8, top_k=top_k, top_p=top_p, seed=21, step=step).cpu()
    ops.check_status("sample")
    assert torch.equal(got, again)
    for i in range(5):
        want = _expected_draw(rows[i, :V].float().cpu().numpy(), 0.8, top_k, top_p, 21, 17, i)
        assert int(got[i]) in want, (i, int(got[i]), want)


@pytest.mark.parametrize("V", [130, 50257])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_sampling_kernel_masked_logits(ops, V, dtype):
    """Masked entries (-inf, the type's lowest value) and entries far below the rest leave top-k and top-p as they are."""
    g = torch.Generator(device="cuda").manual_seed(V)
    for fill in (float("-inf"), torch.finfo(dtype).min, -1e30, -3000.0):
        row = (torch.randn(1, V, device="cuda", generator=g) * 2).to(dtype)
        row[0, torch.randperm(V, device="cuda", generator=g)[:V // 2]] = fill
        for top_k, top_p in ((5, 1.0), (0, 0.3), (5, 0.5)):
            for step in range(24):
                got = int(ops.sample(row, 0.8, top_k=top_k, top_p=top_p, seed=9, step=torch.tensor([step], dtype=torch.int32, device="cuda"))[0])
                assert got in _expected_draw(np.nan_to_num(row[0].float().cpu().numpy(), neginf=-1e30), 0.8, top_k, top_p, 9, step, 0), (fill, top_k, top_p, step)
    few = torch.full((1, V), float("-inf"), device="cuda", dtype=dtype)      # fewer entries than top-k
    few[0, 3], few[0, V - 1] = 1.0, 0.5
    assert {int(ops.sample(few, 1.0, top_k=40, top_p=1.0, seed=s)[0]) for s in range(64)} == {3, V - 1}
    ops.check_status("sample")


def _seed_for(u_bits: int, step: int, index: int = 0) -> int:
    """The seed with which row ``index`` of a step draws u = (u_bits + 0.5) / 2^24 (the mixing function is a bijection)."""
    M = (1 << 64) - 1
    def mix(z):
        z = (z + 0x9E3779B97F4A7C15) & M
        z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & M
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & M
        return z ^ (z >> 31)
    def unshift(z, s):
        x = z
        for _ in range(64 // s + 1):
            x = z ^ (x >> s)
        return x
    z = unshift(u_bits << 40, 31)
    z = unshift(z * pow(0x94D049BB133111EB, -1, 1 << 64) & M, 27)
    z = unshift(z * pow(0xBF58476D1CE4E5B9, -1, 1 << 64) & M, 30)
    seed = ((z - 0x9E3779B97F4A7C15) & M) ^ mix((step << 20) ^ index)
    assert mix(seed ^ mix((step << 20) ^ index)) == u_bits << 40
    return seed


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_sampling_kernel_always_draws(ops, dtype):
    """The largest random number (1 after rounding) and others, with a handful of kept entries spread over the row: the fp32 prefixes of
    the 32 pieces and their total are rounded in different orders, so the target may lie above the last kept piece's prefix. A kept token
    comes out all the same, and a row without a distribution gives its largest entry."""
    V, step = 32000, torch.tensor([3], dtype=torch.int32, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(4)
    for i in range(150):
        kept = 3 + i % 17
        row = torch.full((1, V), -50.0, device="cuda", dtype=dtype)
        at = torch.randperm(V, device="cuda", generator=g)[:kept]
        row[0, at] = torch.randn(kept, device="cuda", generator=g).to(dtype)
        for bits in ((1 << 24) - 1, (1 << 24) - 3, 0):
            out = torch.full((1,), -7, dtype=torch.int32, device="cuda")
            ops.sample(row, 0.8, top_k=kept, top_p=1.0, seed=_seed_for(bits, 3), step=step, out=out)
            got = int(out[0])
            assert got in set(at.tolist()), (i, bits, got)
            if bits != 0:       # within 2^-22 of the whole mass: the last kept entry, whatever the rounding
                assert got == int(at.max()), (i, bits, got)
    for bad, want in ((float("nan"), 4), (float("inf"), 9000)):
        row = torch.zeros((1, V), device="cuda", dtype=dtype)
        row[0, 4], row[0, 9000] = 5.0, bad
        out = torch.full((1,), -7, dtype=torch.int32, device="cuda")
        ops.sample(row, 0.8, top_k=50, top_p=0.9, seed=1, step=step, out=out)
        assert 0 <= int(out[0]) < V and (bad != bad or int(out[0]) == want), int(out[0])
    ops.check_status("sample")


def test_sampling_kernel(ops):
    torch.manual_seed(11)
    V = 1000
    logits = (torch.randn(6, V, device="cuda") * 2).to(torch.bfloat16)
    step = torch.zeros(1, dtype=torch.int32, device="cuda")
    greedy = logits.float().argmax(-1).int()
    # top_k = 1 and a tiny nucleus both reduce to the argmax
    assert torch.equal(ops.sample(logits, 1.0, top_k=1, seed=3, step=step), greedy)
    assert torch.equal(ops.sample(logits, 1.0, top_p=1e-4, seed=4, step=step), greedy)
    assert torch.equal(ops.sample(logits, 0.01, seed=5, step=step), greedy)
    # the same (seed, step) repeats, another step differs somewhere
    a = ops.sample(logits, 1.0, seed=7, step=step)
    b = ops.sample(logits, 1.0, seed=7, step=step)
    assert torch.equal(a, b)
    draws = []
    for _ in range(40):
        ops.bump(step)
        draws.append(ops.sample(logits, 1.0, top_k=5, seed=7, step=step))
    draws = torch.stack(draws)
    fifth = logits.float().topk(5, -1).values[:, -1]           # ties with the 5th value stay in the kept set
    picked = torch.gather(logits.float(), 1, draws.t().long())  # [rows, draws]
    assert (picked >= fifth[:, None]).all()
    assert len({tuple(d.tolist()) for d in draws}) > 5
    # frequencies follow the softmax: small vocabulary, many draws
    small = torch.tensor([[2.0, 1.0, 0.0, -1.0, -30.0, 0.5, 0.5, 1.5]], device="cuda").to(torch.bfloat16).repeat(512, 1)
    counts = torch.zeros(8)
    for _ in range(8):
        ops.bump(step)
        counts += torch.bincount(ops.sample(small, 1.0, seed=9, step=step).cpu().long(), minlength=8).float()
    want = torch.softmax(small[0].float().cpu(), -1)
    assert (counts / counts.sum() - want).abs().max() < 0.03
    # nucleus: with top_p = 0.5 only the most likely tokens whose mass reaches 0.5 can appear
    ops.bump(step)
    nuc = ops.sample(small, 1.0, top_p=0.5, seed=10, step=step).cpu()
    order = want.argsort(descending=True)
    keep = order[: int((want[order].cumsum(0) < 0.5).sum()) + 1].tolist()
    assert set(nuc.tolist()) <= set(keep)


def test_bounded_wait_reports_a_timeout_and_the_context_survives(ops):
    """Failure detection on the device: a wait on a flag that nobody sets runs out of polls, the status word says so,
    and the next kernels run normally."""
    flag = torch.zeros(1, dtype=torch.int32, device="cuda")
    res = torch.full((1,), -1, dtype=torch.int32, device="cuda")
    ops.wait_flag(flag, 1, max_polls=20000, result=res)          # a few milliseconds
    assert ops.read_status() == 2 and int(res.item()) == 0        # STATUS_PEER_TIMEOUT
    assert ops.read_status() == 0                                 # reading clears the word
    flag.fill_(3)
    ops.wait_flag(flag, 3, max_polls=20000, result=res)
    assert ops.read_status() == 0 and int(res.item()) == 1
    x = torch.randn(4, 256, device="cuda", dtype=torch.bfloat16)
    y = ops.rmsnorm(x, torch.ones(256, device="cuda", dtype=torch.bfloat16), 1e-5)
    assert torch.isfinite(y.float()).all()


# Two correct kernels round the same fp32 sums (taken in another order) to bf16: each is off by 2^-9 / sqrt(3) of a value on average,
# 1.6e-3 between the two in the 2-norm.
PAIR_REL = 4e-3


def _pair_weight(ops, fmt, N, K, dtype=torch.bfloat16):
    g = torch.Generator(device="cuda").manual_seed(N + K)
    if fmt == "dense":
        return ops.PackedWeight.from_dense((torch.randn(N, K, device="cuda", generator=g) * 0.05).to(dtype))
    if fmt == "u4":
        q = torch.randint(0, 256, (N * K // 2,), dtype=torch.uint8, device="cuda", generator=g)
        z = torch.randint(0, 256, (N * (K // 64) // 2,), dtype=torch.uint8, device="cuda", generator=g)
        return ops.PackedWeight.from_ir_u4(q, (torch.rand(N, K // 64, device="cuda", generator=g) * 0.01 + 0.005).half(), z, N, K, 64)
    if fmt == "u8":
        q = torch.randint(0, 256, (N, K), dtype=torch.uint8, device="cuda", generator=g)
        z = torch.randint(100, 156, (N, K // 128), dtype=torch.uint8, device="cuda", generator=g)
        return ops.PackedWeight.from_ir_u8(q, (torch.rand(N, K // 128, device="cuda", generator=g) * 0.001 + 0.0005).half(), z, N, K, 128)
    q = torch.randn(N, K, device="cuda", generator=g).to(torch.float8_e4m3fn)
    return ops.PackedWeight.from_f8_block(q, torch.rand((N + 127) // 128, K // 128, device="cuda", generator=g) * 0.05 + 0.02, N, K)


def _is_expanded(ops, T, w):
    """Does a plain product of T tokens expand these weights first?"""
    import ctypes as C
    a = ops.GemmArgs()
    a.x, a.w, a.out, a.T, a.N, a.K, a.ldx, a.group_size, a.wmode = 16, 16, 16, T, w.N, w.K, w.K, w.group_size, w.mode
    return ops.lib().ovb_gemm_scratch_bytes(C.byref(a)) > 0


@pytest.mark.parametrize("fmt,T,N,K", [("dense", 129, 3328, 64), ("dense", 999, 6144, 448), ("dense", 257, 4224, 1024), ("dense", 2049, 384, 128), ("dense", 8191, 256, 512),
                                       ("u4", 1024, 1280, 256), ("u4", 1031, 640, 4096), ("u8", 1025, 896, 256), ("f8", 1100, 768, 384), ("u4", 1024, 36864, 2048)])
def test_gemm_pair(ops, fmt, T, N, K):
    """Edges of the token tile, an odd number of 128-row tiles, one k-block, weights expanded in one piece and in several: against the
    single-CTA kernel (an explicit token tile selects it), in every epilogue."""
    torch.manual_seed(1)
    x = torch.randn(T, K + 64, device="cuda", dtype=torch.bfloat16)[:, :K]
    w = _pair_weight(ops, fmt, N, K)
    out, ref = (torch.full((T, N + 2), 7.0, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    ops.gemm(x, w, out=out[:, :N])
    ops.gemm(x, w, out=ref[:, :N], block_t=256)
    ops.check_status("gemm_pair")
    assert _rel_err(out, ref) < PAIR_REL and (out[:, N:] == 7.0).all()
    w.bias = torch.randn(N, device="cuda").to(torch.bfloat16)
    res = torch.randn(T, N, device="cuda").to(torch.bfloat16)
    for kw in (dict(residual=res), dict(residual=res, act=ops.ACT_GELU_ERF), dict(act=ops.ACT_RELU2), dict(out_f32=True), dict(out_f32=True, act=ops.ACT_SILU)):
        a, b = ops.gemm(x, w, **kw), ops.gemm(x, w, block_t=256, **kw)
        assert _rel_err(a, b) < (1e-5 if kw.get("out_f32") else PAIR_REL), kw
    w.bias = None
    for kw in (dict(act=ops.ACT_SWIGLU), dict(act=ops.ACT_GLU_LIMITED, glu=(7.0, 1.702, 1.0))):
        assert _rel_err(ops.gemm(x, w, **kw), ops.gemm(x, w, block_t=256, **kw)) < PAIR_REL, kw
    h = res.clone()
    ops.gemm(x, w, out=h, residual=h)                       # in place, as the residual stream
    assert _rel_err(h, ops.gemm(x, w, residual=res, block_t=256)) < PAIR_REL
    ops.check_status("gemm_pair")


@pytest.mark.parametrize("fmt,T,N,K", [("u8", 1024, 36864, 2048), ("u8", 1025, 4992, 2048), ("f8", 1100, 4224, 4096), ("u4", 2560, 28800, 4096), ("u4", 2049, 33024, 4096)])
def test_gemm_expanded_weights(ops, fmt, T, N, K):
    """Problems whose weights are expanded, in one piece and in several, odd numbers of 128-row tiles among them."""
    x = torch.randn(T, K, device="cuda", dtype=torch.bfloat16, generator=torch.Generator(device="cuda").manual_seed(T))
    w = _pair_weight(ops, fmt, N, K)
    assert _is_expanded(ops, T, w)
    assert _rel_err(ops.gemm(x, w), ops.gemm(x, w, block_t=256)) < PAIR_REL
    assert _rel_err(ops.gemm(x, w, act=ops.ACT_SWIGLU), ops.gemm(x, w, block_t=256, act=ops.ACT_SWIGLU)) < PAIR_REL
    ops.check_status("gemm_pair")


def test_gemm_runs_without_scratch_memory(ops, monkeypatch):
    """A device without room for expanded weights still runs the product."""
    x = torch.randn(1025, 2048, device="cuda", dtype=torch.bfloat16)
    w = _pair_weight(ops, "u8", 4992, 2048)
    assert _is_expanded(ops, 1025, w)
    want = ops.gemm(x, w)
    out = torch.empty_like(want)

    def full(*size, **kw):
        raise torch.OutOfMemoryError("no room")
    with monkeypatch.context() as m:
        m.setattr(ops.torch, "empty", full)
        ops.gemm(x, w, out=out)
    assert _rel_err(out, want) < PAIR_REL
    ops.check_status("gemm")


@pytest.mark.parametrize("T,N,dtype", [(256, 19200, torch.bfloat16), (225, 19200, torch.float16), (999, 28672, torch.bfloat16), (512, 28544, torch.bfloat16), (4033, 4096, torch.float16)])
def test_gemm_pair_cut_wave(ops, T, N, dtype):
    """Products whose last wave is cut along the tokens (one tile in eight parts, parts behind the last token, an odd number of 128-row tiles):
    the same sums in the same order as in whole tiles, up to the order of the single-CTA kernel."""
    K = 2048
    x = torch.randn(T, K, device="cuda", generator=torch.Generator(device="cuda").manual_seed(T)).to(dtype)
    w = _pair_weight(ops, "dense", N, K, dtype)
    res = torch.randn(T, N, device="cuda").to(dtype)
    for kw in (dict(), dict(residual=res), dict(act=ops.ACT_SWIGLU), dict(out_f32=True)):
        a, b = ops.gemm(x, w, **kw), ops.gemm(x, w, block_t=256, **kw)
        assert a.shape == b.shape and _rel_err(a, b) < (1e-5 if kw.get("out_f32") else PAIR_REL), kw
    ops.check_status("gemm_pair")


@pytest.mark.parametrize("sizes", [[31, 0, 257, 33, 512, 1], [513, 224, 225, 65], [770, 0, 0, 0], [96] * 9])
@pytest.mark.parametrize("mode", [1, 2])
def test_gemm_groups_of_even_tiles(ops, sizes, mode):
    """Rows of a group shared out evenly among its tiles: one row, one more than a tile holds, empty groups, rows behind the last group."""
    G, N, K, total = len(sizes), 640, 320, sum(sizes)
    off = torch.tensor(np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32), device="cuda")
    w = _pair_weight(ops, "dense", N * (G if mode == 1 else 1), K * (G if mode == 2 else 1))
    x = torch.randn(total + 70, K, device="cuda", dtype=torch.bfloat16, generator=torch.Generator(device="cuda").manual_seed(G))
    for act, n in ((ops.ACT_NONE, N), (ops.ACT_SWIGLU, N // 2)):
        out, ref = (torch.full((total + 70, n), 3.0, device="cuda", dtype=torch.bfloat16) for _ in range(2))
        ops.gemm_grouped(x, w, off, G, mode, out, act=act, block_t=256)
        ops.gemm_grouped(x, w, off, G, mode, ref, act=act, block_t=64)
        assert _rel_err(out, ref) < PAIR_REL and (out[total:] == 3.0).all()
    ops.check_status("gemm_groups")


def test_gemm_pair_fp16_window_and_groups(ops):
    torch.manual_seed(2)
    x = torch.randn(700, 512, device="cuda", dtype=torch.float16)
    w = _pair_weight(ops, "dense", 2560, 1024, torch.float16)
    win = w.window(128, 2304, 256, 512)
    assert _rel_err(ops.gemm(x, win), ops.gemm(x, win, block_t=256)) < PAIR_REL
    for mode, N in ((1, 384), (2, 512)):
        sizes = [0, 130, 1, 517, 0, 256]
        off = torch.tensor(np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32), device="cuda")
        cap, K = 1000, 256
        w = _pair_weight(ops, "dense", N * (6 if mode == 1 else 1), K * (6 if mode == 2 else 1))
        xg = torch.randn(cap, K, device="cuda", dtype=torch.bfloat16)
        out, ref = (torch.full((cap, N), 3.0, device="cuda", dtype=torch.bfloat16) for _ in range(2))
        ops.gemm_grouped(xg, w, off, 6, mode, out, block_t=256)
        ops.gemm_grouped(xg, w, off, 6, mode, ref, block_t=64)
        ops.check_status("gemm_pair")
        assert _rel_err(out, ref) < PAIR_REL and (out[sum(sizes):] == 3.0).all()



@pytest.mark.parametrize("q_lens,past_lens,Hq,Hkv,window", [
    ([1300, 1, 77, 640], [3, 500, 0, 129], 32, 8, 0),   # two query tiles of one CTA, the second of them empty, one row, whole
    ([1, 2500, 2600], [700, 0, 17], 8, 8, 0),           # one query head per KV head
    ([2049, 511], [0, 1000], 16, 8, 300),               # two query heads; tiles that the window hides from one of the two
    ([700, 33], [100, 0], 64, 8, 0),                    # eight query heads
    ([1] * 12 + [32, 33, 1500, 64], [40 * i for i in range(12)] + [5, 0, 130, 64], 32, 8, 0),     # CTAs with one tile: decoding rows, a whole tile; one row more
    ([1] * 5 + [129, 2000, 128], [300 * i for i in range(5)] + [77, 0, 1], 8, 8, 200),            # the same with one query head and a window
    ([1] * 40 + [64], [17 * i for i in range(40)] + [300], 32, 8, 0),                             # mostly decoding rows: one tile per CTA
])
def test_paged_attention_long_prompts(ops, q_lens, past_lens, Hq, Hkv, window):
    torch.manual_seed(5)
    D, bs, dev, T = 128, 16, "cuda", sum(q_lens)
    pl_t, sb_t, bi_t, bib_t, total_blocks = _make_paged_batch(q_lens, past_lens, bs, dev)
    k_cache = torch.randn(total_blocks, Hkv, bs, D, device=dev).to(torch.bfloat16)
    v_cache = torch.randn(total_blocks, Hkv, bs, D, device=dev).to(torch.bfloat16)
    qkv = (torch.randn(T, (Hq + 2 * Hkv) * D, device=dev) * 1.5).to(torch.bfloat16)     # some scores stand out: the running maximum is raised
    scale = 1.0 / math.sqrt(D)
    out = ops.paged_attention(qkv, k_cache, v_cache, pl_t, sb_t, bi_t, bib_t, Hq, Hkv, D, scale=scale, sliding_window=window,
                              max_context_len=max(p + q for p, q in zip(past_lens, q_lens)), max_q_len=max(q_lens))
    ops.check_status("paged_attention")
    rows = [[c[bi_t[bib_t[b]:bib_t[b + 1]].long()].permute(0, 2, 1, 3).reshape(-1, Hkv, D)[:p + q].float() for b, (q, p) in enumerate(zip(q_lens, past_lens))]
            for c in (k_cache, v_cache)]
    ref = _attn_ref(qkv[:, :Hq * D].float().reshape(T, Hq, D), rows[0], rows[1], q_lens, past_lens, Hq, Hkv, D, scale, window)
    assert _rel_err(out.reshape(T, Hq, D), ref) < 1e-2


def test_gelu_epilogue_range(ops):
    """The erf form of GELU over its range, infinities and NaN, against 64 bits: absolutely, and relative to the result where that is
    of the size of an activation: erff is good to two units in the last place, its argument and 1 + erf to half a unit each."""
    v = torch.cat([torch.linspace(-12, 12, 4093), torch.tensor([float("inf"), float("-inf"), float("nan")])]).cuda().to(torch.bfloat16)
    for T, kw in ((300, {}), (300, {"block_t": 64}), (5, {})):
        x = torch.zeros(T, 128, device="cuda", dtype=torch.bfloat16)
        x[:, 0] = 1.0
        w = torch.zeros(4096, 128, device="cuda", dtype=torch.bfloat16)
        w[:, 0] = v
        got = ops.gemm(x, ops.PackedWeight.from_dense(w), act=ops.ACT_GELU_ERF, out_f32=True, **kw)[3].double()
        want = 0.5 * v.double() * torch.special.erfc(-v.double() * math.sqrt(0.5))
        assert (got[:4093] - want[:4093]).abs().max() < 1e-6
        z = v[:4093].double() * math.sqrt(0.5)
        erf = torch.special.erf(z)
        bound = (2.0 ** -22 * erf.abs() + z.abs() * torch.exp(-z * z) * 2 / math.sqrt(math.pi) * 2.0 ** -23 + 2.0 ** -24) / (1 + erf) + 2.0 ** -23
        off = ((got[:4093] - want[:4093]).abs() / want[:4093].abs().clamp_min(1e-30))[z > -2]
        assert (off <= bound[z > -2]).all(), (off / bound[z > -2]).max()
        assert got[4093] == float("inf") and got[4094] == 0 and got[4095].isnan()


@pytest.mark.parametrize("T,kw", [(300, {}), (300, {"block_t": 64}), (5, {})])
def test_gelu_epilogue_is_no_further_off_than_the_library_function(ops, T, kw):
    """Per range of arguments, largest and mean error relative to the result: at most that of 0.5 v (1 + erf(v / sqrt 2)) in fp32."""
    g = torch.Generator(device="cuda").manual_seed(6)
    x = torch.zeros(T, 128, device="cuda", dtype=torch.bfloat16)
    x[:, 0], x[:, 1] = 1.0, 2.0 ** -8
    w = torch.zeros(65536, 128, device="cuda", dtype=torch.bfloat16)
    w[:, 0] = (torch.randn(65536, device="cuda", generator=g) * 1.5).bfloat16()
    w[:, 1] = torch.randn(65536, device="cuda", generator=g).bfloat16()
    pw = ops.PackedWeight.from_dense(w)
    v = ops.gemm(x, pw, out_f32=True, **kw)[3]                   # two exact products: the argument as the epilogue has it
    got = ops.gemm(x, pw, act=ops.ACT_GELU_ERF, out_f32=True, **kw)[3]
    plain = 0.5 * v * (1 + torch.erf(v * math.sqrt(0.5)))
    want = 0.5 * v.double() * torch.special.erfc(-v.double() * math.sqrt(0.5))
    for lo, hi in ((0.01, 1), (1, 3), (3, 9), (-1, -0.01), (-2, -1), (-3, -2), (-4, -3)):
        at = (v > lo) & (v < hi)
        here, lib = (((y.double() - want).abs() / want.abs())[at] for y in (got, plain))
        assert at.sum() > 50 and here.max() <= lib.max() and here.square().mean() <= lib.square().mean(), (lo, hi, here.max(), lib.max(), here.mean(), lib.mean())


@pytest.mark.parametrize("fmt", ["u4", "u8", "f8"])
def test_expanded_weights_exact(ops, fmt):
    """Every byte and zero point, with scales from the smallest to the largest fp16: one weight at a time through the product is
    (q - z) * scale rounded once to bf16, bit for bit."""
    K, N = 256, 2048
    k = torch.arange(K, device="cuda")
    n = torch.arange(N, device="cuda")
    scale = torch.tensor([6e-8, 6.1e-5, 0.0137, 1.0, 333.25, 65504.0], device="cuda")[n % 6].half()
    s = scale.bfloat16()
    if fmt == "u4":
        q = ((k[None] + n[:, None]) % 16).to(torch.uint8)
        z = (n // 6 % 16).to(torch.uint8)
        w = ops.PackedWeight.from_ir_u4((q[:, 0::2] | (q[:, 1::2] << 4)).reshape(-1), scale[:, None].repeat(1, 2).contiguous(), z[:, None].repeat(1, 2).contiguous(), N, K, 128,
                                        zp_is_u8=True)
    elif fmt == "f8":
        q = ((k[None] * 5 + n[:, None]) % 256).to(torch.uint8)
        q = torch.where((q & 0x7F) == 0x7F, 0, q).to(torch.uint8)                  # no NaN
        blocks = torch.tensor([3e-5, 0.0137, 1.0, 117.25], device="cuda")[torch.arange(N // 128 * 2, device="cuda") % 4].reshape(N // 128, 2)
        w = ops.PackedWeight.from_f8_block(q, blocks, N, K)
    else:
        q = k[None].repeat(N, 1).to(torch.uint8)
        z = (n // 6 % 256).to(torch.uint8)
        w = ops.PackedWeight.from_ir_u8(q, scale[:, None].repeat(1, 2).contiguous(), z[:, None].repeat(1, 2).contiguous(), N, K, 128)
    if fmt == "f8":
        want = (q.view(torch.float8_e4m3fn).double() * blocks.bfloat16().double().repeat_interleave(128, 0).repeat_interleave(128, 1)).to(torch.bfloat16)
    else:
        want = ((q.double() - z.double()[:, None]) * s.double()[:, None]).to(torch.bfloat16)
    x = torch.eye(K, device="cuda", dtype=torch.bfloat16)
    for kw in ({"block_t": 64}, {"block_t": 256}):
        assert torch.equal(ops.gemm(x, w, out_f32=True, **kw).t().contiguous(), want.float()), kw
    many = ops.gemm(x.repeat(32, 1), w, out_f32=True)        # expanded in a pass of its own
    assert _is_expanded(ops, 32 * K, w)
    assert torch.equal(many[:K].t().contiguous(), want.float()) and torch.equal(many[31 * K:].t().contiguous(), want.float())
    ops.check_status("gemm")


@pytest.mark.parametrize("rows,cols", [(1, 8), (3, 1016), (5, 1024), (6, 1032), (9, 256)])
def test_layernorm_row_widths(ops, rows, cols):
    """Rows of a warp and of a block, whole and ragged, with and without a residual."""
    torch.manual_seed(rows)
    x, r = (torch.randn(rows, cols, device="cuda", dtype=torch.float16) * 3 + 1 for _ in range(2))
    g, b = (torch.randn(cols, device="cuda", dtype=torch.float16) for _ in range(2))
    for res in (None, r):
        y = ops.layernorm(x, g, b, 1e-5, residual=res)
        h = x.double() + (res.double() if res is not None else 0)
        ref = torch.nn.functional.layer_norm(h, (cols,), g.double(), b.double(), 1e-5)
        assert _rel_err(y, ref) < 1e-3          # one rounding to fp16: 2^-11 of a value at most


def _weight_and_values(ops, fmt, N, K):
    """A packed weight and its values in 64 bits (scales as the kernels' tables hold them)."""
    g = torch.Generator(device="cuda").manual_seed(N)
    if fmt == "dense":
        d = (torch.randn(N, K, device="cuda", generator=g) * 0.05).bfloat16()
        return ops.PackedWeight.from_dense(d), d.double()
    if fmt == "f8":
        q = torch.randn(N, K, device="cuda", generator=g).to(torch.float8_e4m3fn)
        s = torch.rand((N + 127) // 128, K // 128, device="cuda", generator=g) * 0.05 + 0.02
        return ops.PackedWeight.from_f8_block(q, s, N, K), q.double() * s.bfloat16().double().repeat_interleave(128, 0)[:N].repeat_interleave(128, 1)
    top = 16 if fmt == "u4" else 256
    q = torch.randint(0, top, (N, K), dtype=torch.uint8, device="cuda", generator=g)
    z = torch.randint(0, top, (N, K // 128), dtype=torch.uint8, device="cuda", generator=g)
    s = ((torch.rand(N, K // 128, device="cuda", generator=g) + 0.5) * (0.16 / top)).half()
    wide = ((q.reshape(N, -1, 128).double() - z.double()[..., None]) * s.bfloat16().double()[..., None]).reshape(N, K)
    if fmt == "u8":
        return ops.PackedWeight.from_ir_u8(q, s, z, N, K, 128), wide
    return ops.PackedWeight.from_ir_u4((q[:, 0::2] | (q[:, 1::2] << 4)).reshape(-1), s, z, N, K, 128, zp_is_u8=True), wide


@pytest.mark.parametrize("fmt,N,K", [("dense", 96, 64), ("dense", 4096, 1088), ("u4", 128, 128), ("u4", 6240, 4096), ("u4", 1024, 14336), ("u8", 32, 256), ("u8", 2080, 4096),
                                     ("f8", 160, 128), ("f8", 4096, 7168)])
@pytest.mark.parametrize("T", [1, 3, 4, 5, 8, 9])
def test_gemm_stream(ops, fmt, N, K, T):
    """Edges of the token fragment, one unit of K, K shared by a cluster, tiles that are no multiple of 128 rows, token counts on both sides
    of the kernel's limit (8 with 16-bit weights, 4 with quantised ones): element by element against the product in 64 bits."""
    torch.manual_seed(T)
    x = torch.randn(T, K + 8, device="cuda", dtype=torch.bfloat16)[:, :K]
    w, wide = _weight_and_values(ops, fmt, N, K)
    exact, size = x.double() @ wide.t(), x.double().abs() @ wide.abs().t()
    # fp32 sums of exact products: K roundings of at most 2^-24 of the sum of magnitudes, in practice their root; behind the limit the weights are
    # rounded to bf16 first (half a unit in the last place of 8 bits: up to 2^-8 of the value each), and a bf16 result once more
    streamed = T <= (8 if fmt == "dense" else 4)
    sums = 2.0 ** -18 * size if streamed or fmt == "dense" else 2.0 ** -8 * size
    for f32 in (True, False):
        y = ops.gemm(x, w, out_f32=f32)
        assert ((y.double() - exact).abs() <= sums + (0.0 if f32 else 2.0 ** -8) * exact.abs()).all(), (f32, ((y.double() - exact).abs() / size).max())
    if streamed or fmt == "dense":
        assert _rel_err(ops.gemm(x, w, out_f32=True), exact) <= 1.5 * _rel_err(ops.gemm(x, w, out_f32=True, block_t=16), exact) + 2.0 ** -22
    act = ops.gemm(x, w, out_f32=True, act=ops.ACT_SILU)
    assert ((act.double() - torch.nn.functional.silu(exact)).abs() <= 1.2 * sums + 2.0 ** -20 * exact.abs()).all()       # |silu'| < 1.1
    w.bias = torch.randn(N, device="cuda").to(torch.bfloat16)
    h = torch.randn(T + 1, N, device="cuda").to(torch.bfloat16)
    keep, want = h[T].clone(), exact + w.bias.double() + h[:T].double()
    ops.gemm(x, w, out=h[:T], residual=h[:T])
    assert ((h[:T].double() - want).abs() <= sums + 2.0 ** -8 * want.abs() + 2.0 ** -20).all() and torch.equal(h[T], keep)
    w.bias = None
    if N % 128 == 0:
        for kw in (dict(act=ops.ACT_SWIGLU), dict(act=ops.ACT_GLU_LIMITED, glu=(7.0, 1.702, 1.0))):
            assert _rel_err(ops.gemm(x, w, **kw), ops.gemm(x, w, block_t=16, **kw)) < 2 * PAIR_REL, kw      # a product of two such values
    ops.check_status("gemm_stream")


def test_gemm_stream_fp16_and_window(ops):
    torch.manual_seed(3)
    x = torch.randn(5, 256, device="cuda", dtype=torch.float16)
    w = _pair_weight(ops, "dense", 512, 1024, torch.float16).window(128, 256, 320, 256)
    assert _rel_err(ops.gemm(x, w), ops.gemm(x, w, block_t=16)) < PAIR_REL


@pytest.mark.parametrize("T", [1, 5, 300, 1024])
def test_gemm_refuses_what_it_cannot_read(ops, T):
    """Misaligned operands, unknown weight formats and unknown token tiles are errors of the call at every size, whichever kernel the
    size belongs to; scratch memory that cannot be used is not."""
    import ctypes as C
    N, K = 1280, 256
    x = torch.randn(T, K, device="cuda", dtype=torch.bfloat16)
    w = _pair_weight(ops, "u8", N, K)
    room = torch.empty(N * K + 16, dtype=torch.uint8, device="cuda")
    room[1:N * K + 1] = w.w.reshape(-1)
    off = ops.PackedWeight(ops.W_U8, room[1:N * K + 1].reshape(N, K), N, K, w.scales, None, 128)
    dense = _pair_weight(ops, "dense", N, K)
    xoff = torch.empty(T * K + 1, device="cuda", dtype=torch.bfloat16)[1:].reshape(T, K)
    for bad in (lambda: ops.gemm(x, off), lambda: ops.gemm(xoff, w), lambda: ops.gemm(xoff, dense), lambda: ops.gemm(x, dense, block_t=200),
                lambda: ops.gemm(x, ops.PackedWeight(7, dense.w, N, K, tiled=True))):
        with pytest.raises(ops.KernelLibraryError):
            bad()
    with pytest.raises(ops.KernelLibraryError):
        ops.gemm_grouped(x, dense, torch.tensor([0, T], dtype=torch.int32, device="cuda"), 1, 1, torch.empty(T, N, device="cuda", dtype=torch.bfloat16), block_t=200)
    a = ops.GemmArgs()
    out = torch.empty(T, N, device="cuda", dtype=torch.bfloat16)
    scratch = torch.empty((16 << 20) + 16, dtype=torch.uint8, device="cuda")
    a.x, a.w, a.out, a.scales = x.data_ptr(), w.w.data_ptr(), out.data_ptr(), w.scales.data_ptr()
    a.T, a.N, a.K, a.ldx, a.ldo, a.group_size, a.wmode = T, N, K, K, N, 128, ops.W_U8
    a.scratch, a.scratch_bytes = scratch.data_ptr() + 8, 16 << 20
    assert ops.lib().ovb_gemm(C.byref(a), C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    assert _rel_err(out, ops.gemm(x, w, block_t=64)) < PAIR_REL
    ops.check_status("gemm")


@pytest.mark.parametrize("T", [1, 64, 200, 700])
def test_rotation_rounds_the_same_at_every_size(ops, T):
    """Bit for bit the rounding that the fused multiply-adds of the kernel name, however many heads a block takes."""
    D, Hq, Hkv, theta, dev = 128, 32, 8, 500000.0, "cuda"
    g = torch.Generator(device=dev).manual_seed(T)
    qkv = torch.randn(T, (Hq + 2 * Hkv) * D, device=dev, generator=g).bfloat16()
    pos = torch.arange(T, device=dev, dtype=torch.int32) + 500
    kc, vc = (torch.zeros(64, Hkv, 16, D, device=dev, dtype=torch.bfloat16) for _ in range(2))
    x = qkv.reshape(T, -1, D)[:, :Hq + Hkv].clone()
    ops.rope_kv_write(qkv, pos, torch.arange(T, device=dev, dtype=torch.int32), kc, vc, Hq, Hkv, D, theta, 16)
    ops.check_status("rope")
    d = torch.arange(D // 2, device=dev, dtype=torch.float32)
    log2_theta = torch.tensor(theta, dtype=torch.float32).log2().to(dev)
    ang = pos.float()[:, None] * torch.exp2(-log2_theta * (2.0 * d / D))
    a, b, c, s = x[..., :D // 2].double(), x[..., D // 2:].double(), ang.cos().double()[:, None], ang.sin().double()[:, None]
    r = lambda v: v.float().double()                         # a product rounded to fp32; a fused sum is exact in 64 bits up to a last rounding
    lo = (a * c - r(b * s)).float().bfloat16()
    hi = torch.where((d % 2 == 0)[None, None], a * s + r(b * c), b * c + r(a * s)).float().bfloat16()
    got = torch.cat([qkv.reshape(T, -1, D)[:, :Hq], kc.permute(0, 2, 1, 3).reshape(-1, Hkv, D)[:T]], 1)
    assert torch.equal(got, torch.cat([lo, hi], -1))


@pytest.mark.parametrize("fmt", ["u4", "u8", "f8"])
@pytest.mark.parametrize("T", [5, 16, 17, 32, 33, 48, 49, 64])
def test_gemm_few(ops, fmt, T):
    """Up to 64 tokens with quantised weights: every token tile's edge, one stage of K, shares of K that are no equal parts, tiles that clusters work
    off in several rounds, every number of splits, against the product in 64 bits and bit for bit against a second run."""
    torch.manual_seed(T)
    for N, K, splits in ((128, 256, (0, 1)), (256, 1280, (0, 2, 3, 5)), (512, 2048, (4, 6, 7, 8)), (128 * 150, 256, (1,)), (128 * 76, 512, (2,)), (128 * 19, 2048, (8,))):
        x = torch.randn(T, K + 8, device="cuda", dtype=torch.bfloat16)[:, :K]
        w, wide = _weight_and_values(ops, fmt, N, K)
        exact, size = x.double() @ wide.t(), x.double().abs() @ wide.abs().t()
        sums = 2.0 ** -8 * size                            # weights rounded to bf16 (fp32 sums are far closer)
        res = torch.randn(T, N, device="cuda").to(torch.bfloat16)
        bias = torch.randn(N, device="cuda").to(torch.bfloat16)
        for s in splits:
            y = ops.gemm(x, w, out_f32=True, splits=s)
            assert ((y.double() - exact).abs() <= sums).all(), (N, K, s, ((y.double() - exact).abs() / size).max())
            assert _rel_err(y, exact) < PAIR_REL and torch.equal(y, ops.gemm(x, w, out_f32=True, splits=s))
            w.bias = bias
            h = torch.randn(T + 1, N, device="cuda").to(torch.bfloat16)
            keep, want = h[T].clone(), exact + bias.double() + res.double()
            ops.gemm(x, w, out=h[:T], residual=res, splits=s)
            assert ((h[:T].double() - want).abs() <= sums + 2.0 ** -8 * want.abs() + 2.0 ** -20).all() and torch.equal(h[T], keep)
            w.bias = None
            for kw in (dict(act=ops.ACT_SWIGLU), dict(act=ops.ACT_GLU_LIMITED, glu=(7.0, 1.702, 1.0)), dict(act=ops.ACT_SILU)):
                assert _rel_err(ops.gemm(x, w, splits=s, **kw), ops.gemm(x, w, block_t=64, **kw)) < 2 * PAIR_REL, kw
    ops.check_status("gemm_few")


@pytest.mark.parametrize("Hq,Hkv", [(4, 4), (4, 2), (32, 8), (16, 2)])
@pytest.mark.parametrize("ctxs,bucket,window", [((1,), 256, 0), ((16, 17, 64, 65), 256, 0), ((256, 257, 512, 1000, 3, 700), 1024, 0), ((2049, 4000, 1), 4096, 0),
                                                ((300, 900), 1024, 100)])
def test_decode_attention_with_its_rotation(ops, Hq, Hkv, ctxs, bucket, window):
    """One launch against rotation, attention and sum of the splits as launches of their own: the last key on every place of a page and of a split,
    splits without keys, a sequence without a slot."""
    B, D, dev, theta = len(ctxs), 128, "cuda", 500000.0
    g = torch.Generator(device=dev).manual_seed(B + Hq)
    nb = [(c + 15) // 16 for c in ctxs]
    tables = torch.randperm(sum(nb) + 3, device=dev, generator=g)[:sum(nb)].int()
    begins = torch.tensor([sum(nb[:i]) for i in range(B + 1)], dtype=torch.int32, device=dev)
    caches = [torch.randn(sum(nb) + 3, Hkv, 16, D, device=dev, generator=g).bfloat16() for _ in range(2)]
    past = torch.tensor([c - 1 for c in ctxs], dtype=torch.int32, device=dev)
    slots = torch.tensor([int(tables[int(begins[i]) + (c - 1) // 16]) * 16 + (c - 1) % 16 for i, c in enumerate(ctxs)], dtype=torch.int32, device=dev)
    if B > 2:
        slots[1] = -1
    sub = torch.arange(B + 1, dtype=torch.int32, device=dev)
    qkv = torch.randn(B, (Hq + 2 * Hkv) * D, device=dev, generator=g).bfloat16()
    want_kv, qkv2 = [c.clone() for c in caches], qkv.clone()
    ops.rope_kv_write(qkv2, past, slots, *want_kv, Hq, Hkv, D, theta, 16)
    want = ops.paged_attention(qkv2, *want_kv, past, sub, tables, begins, Hq, Hkv, D, max_context_len=bucket, max_q_len=1, sliding_window=window)
    for at in (past, None):
        kv = [t.clone() for t in (caches if at is not None else want_kv)]
        got = ops.decode_attention(qkv if at is not None else qkv2, *kv, past, sub, tables, begins, Hq, Hkv, D, at, slots, theta, max_context_len=bucket, sliding_window=window)
        # the same rows in the cache to the bit; the same products, the splits' sums in another order
        assert torch.equal(kv[0], want_kv[0]) and torch.equal(kv[1], want_kv[1])
        assert _rel_err(got, want.double()) < 1e-3
    ops.check_status("decode attention")


@pytest.mark.parametrize("rows,vocab", [(1, 16384), (3, 32000), (64, 128256), (147, 16392), (148, 16384), (2, 16387)])
def test_argmax_in_pieces(ops, rows, vocab):
    """Ties across the pieces, rows of -inf and NaN, odd tails, both sides of the limits; the token is handed on where it has a place."""
    g = torch.Generator(device="cuda").manual_seed(rows)
    l = torch.randn(rows, vocab, device="cuda", generator=g).bfloat16()
    l[0, 5000 % vocab] = l[0, vocab - 1] = 50.0
    if rows > 2:
        l[1], l[2] = float("-inf"), float("nan")
        l[2, vocab // 2] = 1.0
    want = torch.where(l.isnan(), torch.full_like(l, float("-inf")), l).float().argmax(-1)
    out, top = torch.empty(rows, dtype=torch.int32, device="cuda"), torch.empty(rows, dtype=torch.float32, device="cuda")
    ops.argmax(l, out=out, out_max=top)
    assert torch.equal(out.long(), want) and (rows <= 2 or float(top[2]) == 1.0)
    dst = torch.arange(rows, dtype=torch.int32, device="cuda") * 2 - 2
    last = torch.full((2 * rows + 1,), -7, dtype=torch.int32, device="cuda")
    tok = torch.empty(rows, dtype=torch.int32, device="cuda")
    ops.argmax_scatter(l, tok, dst, last)
    assert torch.equal(tok, out)
    keep = torch.full_like(last, -7)
    keep[dst[1:].long()] = out[1:]
    assert torch.equal(last, keep)
    ops.check_status("argmax")


def test_step_edges_in_one_launch(ops):
    """Embedding of resolved ids, and the norm of gathered rows, as the launches that they replace."""
    g = torch.Generator(device="cuda").manual_seed(1)
    for T, H in ((1, 256), (5, 4096), (700, 8192)):
        table, gamma = torch.randn(90, H, device="cuda", generator=g).bfloat16(), torch.randn(H, device="cuda", generator=g).bfloat16()
        ids = torch.randint(-2, 95, (T,), dtype=torch.int32, device="cuda", generator=g)
        src = torch.randint(-1, 8, (T,), dtype=torch.int32, device="cuda", generator=g)
        last = torch.randint(0, 90, (8,), dtype=torch.int32, device="cuda", generator=g)
        ids2 = ids.clone()
        ops.resolve_ids(ids2, src, last)
        want = ops.embedding(ids2, table)
        h = torch.empty(T, H, dtype=torch.bfloat16, device="cuda")
        ops.embed_tokens(ids, src, last, table, h)
        assert torch.equal(h, want) and torch.equal(ids, ids2)
        rows = torch.randint(-1, T + 1, (6,), dtype=torch.int32, device="cuda", generator=g)
        assert torch.equal(ops.rmsnorm_rows(h, rows, gamma, 1e-5, torch.empty(6, H, dtype=torch.bfloat16, device="cuda")), ops.rmsnorm(ops.embedding(rows, h), gamma, 1e-5))


@pytest.mark.parametrize("fmt,N,K", [("u4", 128, 128), ("u4", 1024, 2048), ("u4", 6144, 4096), ("u4", 1280, 8192), ("u4", 4096, 14336), ("u8", 512, 2048), ("f8", 512, 1024),
                                     ("dense", 512, 2048)])
@pytest.mark.parametrize("T", [1, 3, 4, 5])
def test_norm_inside_the_product(ops, fmt, N, K, T):
    """Products that normalise their rows themselves, at the limits of what a thread holds and with K shared by clusters, against norm and product as
    two launches: the sums of squares differ in order only, so a normalised value is at most a neighbour away."""
    import ctypes as C
    g = torch.Generator(device="cuda").manual_seed(T)
    w, _ = _weight_and_values(ops, fmt, N, K)
    h, gamma = torch.randn(T + 3, K, device="cuda", generator=g).bfloat16() * 3, torch.randn(K, device="cuda", generator=g).bfloat16()
    rows = torch.randint(-1, T + 4, (T,), dtype=torch.int32, device="cuda", generator=g)
    for norm, x in (((gamma, 1e-5), h[:T]), ((gamma, 1e-5, rows), h)):
        y = ops.rmsnorm(h[:T], gamma, 1e-5) if len(norm) < 3 else ops.rmsnorm_rows(h, rows, gamma, 1e-5, torch.empty(T, K, dtype=torch.bfloat16, device="cuda"))
        assert _rel_err(ops.gemm(x, w, out_f32=True, norm=norm), ops.gemm(y, w, out_f32=True).double()) < 2.0 ** -9
    a = ops.GemmArgs()
    a.x, a.w, a.out, a.scales = h.data_ptr(), w.w.data_ptr(), h.data_ptr(), w.w.data_ptr()
    a.T, a.N, a.K, a.ldx, a.group_size, a.wmode, a.w_tiled = T, N, K, K, 128, w.mode, 1 if fmt == "dense" else 0
    takes = T <= 4 and K <= (8192 if fmt == "u4" and N * K >= 8 << 20 else 2048)
    assert bool(ops.lib().ovb_gemm_norms(C.byref(a))) == takes
    if not takes:
        a.x_norm = gamma.data_ptr()
        assert ops.lib().ovb_gemm(C.byref(a), C.c_void_p(torch.cuda.current_stream().cuda_stream)) != 0
    ops.check_status("norm in a product")


@pytest.mark.parametrize("V", [16384, 32000, 65537, 128256, 131072])
@pytest.mark.parametrize("kind", ["spread", "peaked", "masked", "equal", "nan", "inf"])
def test_sampling_by_a_cluster(ops, V, kind):
    """A row shared by eight CTAs draws the token that one CTA draws (enough rows go to that kernel): kept sets in one CTA's piece and in all, ties,
    masked entries, rows without a distribution, a vocabulary that fills the registers and one that is no multiple of eight."""
    many, few = 131072 // 2700 + 1, 2
    g = torch.Generator(device="cuda").manual_seed(V)
    l = torch.randn(1, (V + 7) // 8 * 8, device="cuda", generator=g).bfloat16()[:, :V] * (0.01 if kind == "equal" else 3)
    if kind == "peaked":
        l[0, V - 1], l[0, 3] = 60.0, 59.5
    elif kind == "masked":
        l[0, 40:] = float("-inf")
        l[0, V // 2] = torch.finfo(torch.bfloat16).min
    elif kind == "equal":
        l[0] = 1.0
    elif kind == "nan":
        l[0, 5] = float("nan")
    elif kind == "inf":
        l[0, V // 3] = float("inf")
    rows = torch.empty(many, (V + 7) // 8 * 8, device="cuda", dtype=torch.bfloat16)[:, :V].copy_(l.expand(many, V))
    for top_k, top_p, t in ((50, 0.95, 0.8), (1, 1.0, 1.0), (3000, 1.0, 2.0), (5, 0.5, 1.0)):
        for seed in range(8):
            one, shared = ops.sample(rows, t, top_k=top_k, top_p=top_p, seed=seed), ops.sample(rows[:few], t, top_k=top_k, top_p=top_p, seed=seed)
            assert torch.equal(one[:few], shared), (top_k, top_p, seed, one[:few], shared)
    ops.check_status("sample")


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D,S", [(64, 1), (64, 100), (64, 128), (64, 129), (64, 384), (128, 257), (64, 1500)])
def test_sdpa_with_a_value_per_key(ops, dtype, D, S):
    """Padding masks of every kind (-10000, the type's lowest value, -inf, small biases; one row for all sequences), against softmax in 64 bits. A
    sequence without any visible key gives zeros."""
    B, H = 3, 2
    g = torch.Generator(device="cuda").manual_seed(S)
    qkv = torch.randn(B * S, 3 * H * D, device="cuda", generator=g).to(dtype)
    q, k, v = (qkv[:, i * H * D:] for i in range(3))
    lens = torch.tensor([max(1, S // 3), S, max(1, S - 1)], device="cuda")
    far = torch.arange(S, device="cuda")[None] >= lens[:, None]
    for kind in ("-10000", "lowest", "-inf", "soft", "shared", "none visible"):
        bias = torch.zeros(B, S, device="cuda", dtype=dtype)
        if kind == "soft":
            bias = torch.randn(B, S, device="cuda", generator=g).to(dtype) * 3
        elif kind == "shared":
            bias = torch.randn(1, S, device="cuda", generator=g).to(dtype) * 3
        else:
            bias[far] = {"-10000": -10000.0, "lowest": torch.finfo(dtype).min}.get(kind, float("-inf"))
        if kind == "none visible":
            bias[1] = float("-inf")
        out = ops.sdpa_masked(q, k, v, bias, B, S, H, D, 3 * H * D)
        qd, kd, vd = (t[:, :H * D].reshape(B, S, H, D).transpose(1, 2).double() for t in (q, k, v))
        want = torch.softmax(qd @ kd.transpose(-1, -2) / D ** 0.5 + bias.double()[:, None, None], -1).nan_to_num(0.0) @ vd
        # probabilities rounded to 16 bits, and the result once more
        assert _rel_err(out, want.transpose(1, 2).reshape(B * S, H * D)) < (2.0 ** -9 if dtype == torch.float16 else 2.0 ** -7), kind
    with pytest.raises(ops.KernelLibraryError):
        ops.sdpa_masked(torch.zeros(9000, 64, device="cuda", dtype=dtype), *(torch.zeros(9000, 64, device="cuda", dtype=dtype),) * 2,
                        torch.zeros(1, 9000, device="cuda", dtype=dtype), 1, 9000, 1, 64, 64)
    ops.check_status("sdpa_masked")


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D,S", [(64, 1), (64, 100), (64, 129), (64, 384), (128, 257)])
def test_sdpa_of_a_sequence_that_is_all_padding(ops, dtype, D, S):
    """Every key of a sequence at the type's lowest (or largest) finite value: softmax sees equal biases. The 16-bit value times log2(e) does not fit 32
    bits in bf16. NaN in a mask stays NaN."""
    B, H = 4, 16 if S == 384 else 2                       # (more CTAs than SMs: the form with two CTAs on an SM)
    g = torch.Generator(device="cuda").manual_seed(S)
    q, k, v = (torch.randn(B * S, H * D, device="cuda", generator=g).to(dtype) for _ in range(3))
    bias = torch.zeros(B, S, device="cuda", dtype=dtype)
    bias[1], bias[2] = torch.finfo(dtype).min, torch.finfo(dtype).max
    bias[3, : S // 2] = float("-inf")                     # some keys not there, the others at the lowest value
    bias[3, S // 2:] = torch.finfo(dtype).min
    qd, kd, vd = (t.reshape(B, S, H, D).transpose(1, 2).double() for t in (q, k, v))
    want = (torch.softmax(qd @ kd.transpose(-1, -2) / D ** 0.5 + bias.double()[:, None, None], -1) @ vd).transpose(1, 2).reshape(B, S, H * D)
    out = ops.sdpa_masked(q, k, v, bias, B, S, H, D, H * D).reshape(B, S, H * D)
    # probabilities and the result in 16 bits; a score beside 65504 log2(e) is rounded to 2^-7, so a probability of fp16 is off by 2^-8 ln 2 at most
    rel = 2.0 ** -9 + 2.0 ** -8 if dtype == torch.float16 else 2.0 ** -7
    for b in range(B):
        assert _rel_err(out[b], want[b]) < rel, b
    bias[0, S - 1] = float("nan")
    assert ops.sdpa_masked(q, k, v, bias, B, S, H, D, H * D).reshape(B, -1)[0].isnan().all()
    ops.check_status("sdpa_masked")


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("D,S", [(64, 1), (64, 100), (64, 128), (64, 129), (64, 640), (128, 1), (128, 127), (128, 257), (128, 384)])
def test_sdpa_dense_causal_and_not(ops, dtype, causal, D, S):
    """Dense attention without a mask, one CTA per query tile, both head sizes, edges of the tiles of 128 keys, more CTAs than SMs (two to an SM for heads of
    64) and fewer, against softmax in 64 bits."""
    B, H = 3, 2 if S < 600 and (D, S) != (64, 129) else 30
    qkv = torch.randn(B * S, 3 * H * D, device="cuda", generator=torch.Generator(device="cuda").manual_seed(S)).to(dtype)
    q, k, v = (qkv[:, i * H * D:] for i in range(3))
    out = ops.sdpa_dense(q, k, v, B, S, H, D, 3 * H * D, causal=causal)
    qd, kd, vd = (t[:, :H * D].reshape(B, S, H, D).transpose(1, 2).double() for t in (q, k, v))
    s = qd @ kd.transpose(-1, -2) / D ** 0.5
    if causal:
        s = s.masked_fill(torch.ones(S, S, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    want = (torch.softmax(s, -1) @ vd).transpose(1, 2).reshape(B * S, H * D)
    # probabilities rounded to 16 bits, and the result once more
    assert _rel_err(out, want) < (2.0 ** -9 if dtype == torch.float16 else 2.0 ** -7)
    ops.check_status("sdpa_dense")


@pytest.mark.parametrize("Hq,Hkv,B,ctx,u8,clusters", [
    (32, 8, 1, 1000, False, 1), (32, 8, 8, 1000, False, 1), (32, 8, 10, 1000, False, 0), (32, 8, 1, 2000, False, 1), (32, 8, 2, 2000, False, 0), (32, 8, 4, 2000, False, 0),
    (32, 8, 18, 500, False, 1), (32, 8, 20, 500, False, 0), (32, 8, 1, 250, False, 0), (32, 8, 1, 4000, False, 0), (64, 8, 1, 1000, False, 0), (16, 8, 4, 2000, False, 1),
    (16, 8, 4, 2000, True, 0), (32, 8, 24, 500, True, 1), (32, 8, 28, 500, True, 0), (64, 8, 4, 500, True, 0), (64, 8, 8, 1000, True, 1)])
def test_splits_are_clusters_where_all_are_resident(ops, Hq, Hkv, B, ctx, u8, clusters):
    """Both sides of the rule at sizes that were measured (one more wave of clusters costs up to twice the attention), and the result of either form."""
    import ctypes as C
    D, dev = 128, "cuda"
    a = ops.PaArgs()
    a.scratch = a.q = a.out = a.k_cache = a.v_cache = 16
    a.B = a.T = B
    a.Hq, a.Hkv, a.D, a.block_size, a.max_q_len, a.max_context_len, a.kv_u8 = Hq, Hkv, D, 16, 1, 1 << (ctx - 1).bit_length(), 1 if u8 else 0
    assert ops.lib().ovb_decode_attention_clusters(C.byref(a), 0 if u8 else 1) == clusters
    g = torch.Generator(device=dev).manual_seed(B)
    blocks = (ctx + 15) // 16
    tables, begins = torch.randperm(B * blocks, device=dev, generator=g).int(), torch.arange(B + 1, dtype=torch.int32, device=dev) * blocks
    past, sub = torch.full((B,), ctx - 1, dtype=torch.int32, device=dev), torch.arange(B + 1, dtype=torch.int32, device=dev)
    q = torch.randn(B, (Hq + 2 * Hkv) * D, device=dev, generator=g).bfloat16()
    if u8:
        kv = [torch.randint(0, 256, (B * blocks, Hkv, 16, D), device=dev, dtype=torch.uint8, generator=g) for _ in range(2)]
        meta = dict(k_meta=torch.full((B * blocks, Hkv, 16, 2), 0.01, device=dev).half(), v_meta=torch.full((B * blocks, Hkv, 16, 2), 0.01, device=dev).half())
    else:
        kv, meta = [torch.randn(B * blocks, Hkv, 16, D, device=dev, generator=g).bfloat16() for _ in range(2)], {}
    args = (q, *kv, past, sub, tables, begins, Hq, Hkv, D)
    got = ops.decode_attention(*args, max_context_len=a.max_context_len, **meta)
    want = ops.paged_attention(*args, max_context_len=a.max_context_len, max_q_len=1, **meta)
    assert _rel_err(got, want.double()) < 1e-3         # the same products, the splits' sums in another order
    ops.check_status("decode attention")


@pytest.mark.parametrize("rows,vocab", [(1, 32000), (5, 32003), (16, 32000), (17, 32000), (74, 148000), (75, 152000)])
def test_argmax_on_both_sides_of_its_rule(ops, rows, vocab):
    """Rows shared by eight CTAs and rows of one CTA, an odd tail, the largest entry in the first and in the last piece, ties to the lowest index."""
    l = torch.randn(rows, (vocab + 7) // 8 * 8, device="cuda", generator=torch.Generator(device="cuda").manual_seed(rows)).bfloat16()[:, :vocab]
    l[0, vocab - 1] = 60.0
    l[rows - 1, 2] = l[rows - 1, vocab - 2] = 61.0
    out = torch.empty(rows, dtype=torch.int32, device="cuda")
    ops.argmax(l, out=out)
    assert torch.equal(out.long(), l.float().argmax(-1)) and int(out[rows - 1]) == 2
    ops.check_status("argmax")


@pytest.mark.parametrize("rows", [1, 148, 149, 300, 301])
@pytest.mark.parametrize("cols", [256, 2048, 2056, 4096, 8192, 8200, 16384])
def test_rmsnorm_forms(ops, rows, cols):
    """Both forms of the norm (weights ahead of the sum or behind it) at the limits of the rule, with a residual and without, against 64 bits."""
    g = torch.Generator(device="cuda").manual_seed(cols)
    x, r, gamma = (torch.randn(n, cols, device="cuda", generator=g).bfloat16() for n in (rows, rows, 1))
    for res in (None, r):
        y = ops.rmsnorm(x, gamma[0], 1e-5, residual=res)
        y = y[0] if isinstance(y, tuple) else y
        h = x.double() if res is None else (x.float() + res.float()).bfloat16().double()
        want = h * torch.rsqrt(h.square().mean(-1, keepdim=True) + 1e-5) * gamma.double()
        assert ((y.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-6).all()        # one rounding to 16 bits
