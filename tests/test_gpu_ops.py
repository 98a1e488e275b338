"""GPU numerics of the single-GPU kernels against plain PyTorch fp32 references."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref_mm(a, b):
    return a.float() @ b.float().t()


@pytest.mark.parametrize("M,N,K", [(128, 256, 64), (256, 512, 256), (1000, 776, 520), (4096, 1024, 2048), (64, 8, 128)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_gemm_matches_fp32_reference(M, N, K, dtype):
    from triton_distributed_b200 import ops
    torch.manual_seed(0)
    a = torch.randn(M, K, device="cuda", dtype=dtype)
    b = torch.randn(N, K, device="cuda", dtype=dtype) * 0.05
    c = ops.gemm(a, b)
    torch.cuda.synchronize()
    ref = _ref_mm(a, b)
    torch.testing.assert_close(c.float(), ref, rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("M,N,K", [(1, 128, 64), (8, 1280, 5120), (8, 5120, 1024), (16, 384, 4096), (5, 700, 1032), (33, 1000, 520),
                                   (24, 1280, 5120), (128, 512, 1024), (256, 256, 512)])
def test_gemm_skinny(M, N, K):
    from triton_distributed_b200 import ops
    torch.manual_seed(1)
    x = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    w = torch.randn(N, K, device="cuda", dtype=torch.bfloat16) * 0.05
    for splits in (0, 1, 3):
        y = ops.gemm_skinny(x, w, splits=splits)
        torch.cuda.synchronize()
        torch.testing.assert_close(y.float(), _ref_mm(x, w), rtol=2e-2, atol=2e-2)
    # the scratch must be left clean: another call (of at most 16 tokens without `splits` often runs on a kernel that has none) gives
    # the same answer
    for splits in (0, 3):
        y2 = ops.gemm_skinny(x, w, splits=splits)
        torch.testing.assert_close(y2.float(), _ref_mm(x, w), rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("M,I,K", [(8, 3200, 5120), (4, 256, 128), (40, 1000, 520)])
def test_gemm_skinny_swiglu(M, I, K):
    from triton_distributed_b200 import ops
    torch.manual_seed(2)
    x = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    w = torch.randn(2 * I, K, device="cuda", dtype=torch.bfloat16) * 0.03
    y = ops.gemm_skinny(x, w, swiglu=True)
    gu = _ref_mm(x, w)
    ref = torch.nn.functional.silu(gu[:, :I]) * gu[:, I:]
    torch.testing.assert_close(y.float(), ref, rtol=3e-2, atol=3e-2)


@pytest.mark.parametrize("rows,hidden", [(8, 5120), (3, 128), (1000, 8192), (17, 16384)])
def test_rmsnorm(rows, hidden):
    from triton_distributed_b200 import ops
    torch.manual_seed(3)
    x = torch.randn(rows, hidden, device="cuda", dtype=torch.bfloat16)
    g = torch.randn(hidden, device="cuda", dtype=torch.bfloat16)
    y = ops.rmsnorm(x, g, 1e-6)
    xf = x.float()
    ref = xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + 1e-6) * g.float()
    torch.testing.assert_close(y.float(), ref, rtol=2e-2, atol=2e-2)
    res = torch.randn_like(x)
    res0 = res.clone()
    y2 = ops.rmsnorm(x, g, 1e-6, residual=res)
    h = (x.float() + res0.float()).to(torch.bfloat16)
    torch.testing.assert_close(res, h)
    hf = h.float()
    ref2 = hf * torch.rsqrt(hf.pow(2).mean(-1, keepdim=True) + 1e-6) * g.float()
    torch.testing.assert_close(y2.float(), ref2, rtol=2e-2, atol=2e-2)


def _rope_ref(x, pos, theta=1e6):
    # x [T, H, 128] fp32, neox style
    D = x.shape[-1]
    inv = 1.0 / (theta ** (torch.arange(0, D, 2, device=x.device, dtype=torch.float32) / D))
    ang = pos.float()[:, None] * inv[None, :]
    cos, sin = ang.cos()[:, None, :], ang.sin()[:, None, :]
    x1, x2 = x[..., : D // 2], x[..., D // 2:]
    return torch.cat([x1 * cos - x2 * sin, x2 * cos + x1 * sin], -1)


def test_qk_norm_rope_and_cache_write():
    from triton_distributed_b200 import ops
    torch.manual_seed(4)
    T, Hq, Hkv, D = 37, 8, 2, 128
    qkv = torch.randn(T, (Hq + 2 * Hkv) * D, device="cuda", dtype=torch.bfloat16)
    pos = torch.randint(0, 4000, (T,), device="cuda", dtype=torch.int32)
    inv = 1.0 / (1e6 ** (torch.arange(0, D, 2, device="cuda", dtype=torch.float32) / D))
    ang = torch.arange(4096, device="cuda", dtype=torch.float32)[:, None] * inv[None, :]
    cos_sin = torch.cat([ang.cos(), ang.sin()], -1).contiguous()
    qg = torch.randn(D, device="cuda", dtype=torch.bfloat16)
    kg = torch.randn(D, device="cuda", dtype=torch.bfloat16)
    slots = torch.randperm(64, device="cuda")[:T].to(torch.int64)
    kc = torch.zeros(64, Hkv, D, device="cuda", dtype=torch.bfloat16)
    vc = torch.zeros_like(kc)
    q = ops.qk_norm_rope(qkv, pos, cos_sin, Hq, Hkv, kc, vc, slots, qg, kg, 1e-6)
    x = qkv.float().view(T, Hq + 2 * Hkv, D)

    def norm(v, g):
        return (v * torch.rsqrt(v.pow(2).mean(-1, keepdim=True) + 1e-6) * g.float()).to(torch.bfloat16).float()

    q_ref = _rope_ref(norm(x[:, :Hq], qg), pos)
    k_ref = _rope_ref(norm(x[:, Hq:Hq + Hkv], kg), pos)
    torch.testing.assert_close(q.float(), q_ref, rtol=2e-2, atol=2e-2)
    torch.testing.assert_close(kc[slots].float(), k_ref, rtol=2e-2, atol=2e-2)
    torch.testing.assert_close(vc[slots], qkv.view(T, -1, D)[:, Hq + Hkv:])


@pytest.mark.parametrize("T,Hq,Hkv", [(1, 1, 1), (3, 8, 1), (1184, 4, 2), (1185, 4, 2), (2367, 4, 2), (2368, 4, 2), (1200, 8, 1), (800, 16, 8)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_qk_norm_rope_groups_of_heads(T, Hq, Hkv, dtype):
    """One and eight heads a warp (eight above 64 heads an SM), with groups that q, k and v share and that no head fills."""
    from triton_distributed_b200 import ops
    torch.manual_seed(14)
    D, n = 128, Hq + 2 * Hkv
    qkv = torch.randn(T, n * D, device="cuda").to(dtype)
    pos = torch.randint(0, 4000, (T,), device="cuda", dtype=torch.int32)
    inv = 1.0 / (1e6 ** (torch.arange(0, D, 2, device="cuda", dtype=torch.float32) / D))
    ang = torch.arange(4096, device="cuda", dtype=torch.float32)[:, None] * inv[None, :]
    cos_sin = torch.cat([ang.cos(), ang.sin()], -1).contiguous()
    kg = torch.randn(D, device="cuda").to(dtype)
    slots = torch.randperm(T + 5, device="cuda")[:T].to(torch.int64)
    slots[T // 2] = -1   # not cached
    kc = torch.zeros(T + 5, Hkv, D, device="cuda", dtype=dtype)
    vc = torch.zeros_like(kc)
    q = ops.qk_norm_rope(qkv, pos, cos_sin, Hq, Hkv, kc, vc, slots, None, kg, 1e-6)
    x = qkv.float().view(T, n, D)

    def turned(v):
        c, s = cos_sin[pos.long()][:, None].chunk(2, -1)
        v1, v2 = v.chunk(2, -1)
        return torch.cat([v1 * c - v2 * s, v2 * c + v1 * s], -1)

    eps = torch.finfo(dtype).eps
    kx = x[:, Hq:Hq + Hkv]
    k = (kx * torch.rsqrt(kx.pow(2).mean(-1, keepdim=True) + 1e-6) * kg.float()).to(dtype).float()
    torch.testing.assert_close(q.float(), turned(x[:, :Hq]), rtol=eps, atol=1e-5)   # one rounding of an fp32 value
    keep = slots >= 0
    # the norm's rounding may fall to the other side: a place of it on either partner, and one of the result
    torch.testing.assert_close(kc[slots[keep]].float(), turned(k)[keep], rtol=2 * eps, atol=2 * eps * float(k.abs().max()))
    assert torch.equal(vc[slots[keep]], qkv.view(T, n, D)[keep, Hq + Hkv:])
    free = torch.ones(T + 5, dtype=torch.bool, device="cuda")
    free[slots[keep]] = False
    assert not kc[free].any() and not vc[free].any()


def test_silu_mul_and_topk():
    from triton_distributed_b200 import ops
    torch.manual_seed(5)
    x = torch.randn(19, 2 * 1536, device="cuda", dtype=torch.bfloat16)
    y = ops.silu_mul(x)
    ref = torch.nn.functional.silu(x[:, :1536].float()) * x[:, 1536:].float()
    torch.testing.assert_close(y.float(), ref, rtol=2e-2, atol=2e-2)
    logits = torch.randn(77, 256, device="cuda", dtype=torch.float32)
    ids, w = ops.topk_softmax(logits, 8)
    pw, pi = torch.topk(torch.softmax(logits, -1), 8, dim=-1)
    assert torch.equal(ids.long(), pi)
    torch.testing.assert_close(w, pw, rtol=1e-4, atol=1e-6)


def _paged_attn_ref(q, kc, vc, kv_lens, bt, scale, soft_cap=0.0):
    B, Hq, D = q.shape
    page, Hkv = kc.shape[1], kc.shape[2]
    G = Hq // Hkv
    out = torch.zeros(B, Hq, D, device=q.device)
    lse = torch.full((B, Hq), -float("inf"), device=q.device)
    for b in range(B):
        L = int(kv_lens[b])
        if L == 0:
            continue
        nb = (L + page - 1) // page
        k = kc[bt[b, :nb].long()].reshape(-1, Hkv, D)[:L].float()
        v = vc[bt[b, :nb].long()].reshape(-1, Hkv, D)[:L].float()
        k = k.repeat_interleave(G, dim=1)
        v = v.repeat_interleave(G, dim=1)
        s = torch.einsum("hd,lhd->hl", q[b].float(), k) * scale
        if soft_cap > 0:
            s = soft_cap * torch.tanh(s / soft_cap)
        lse[b] = torch.logsumexp(s, -1)
        out[b] = torch.einsum("hl,lhd->hd", torch.softmax(s, -1), v)
    return out, lse


@pytest.mark.parametrize("B,Hq,Hkv,page,max_len,splits,soft_cap", [
    (2, 8, 1, 16, 300, 1, 0.0), (3, 64, 8, 1, 777, 4, 0.0), (1, 32, 4, 64, 4096, 8, 30.0), (4, 16, 16, 32, 130, 3, 0.0),
    (2, 40, 2, 16, 500, 2, 0.0)])
def test_paged_decode_attention(B, Hq, Hkv, page, max_len, splits, soft_cap):
    from triton_distributed_b200 import ops
    torch.manual_seed(6)
    D = 128
    nblk_per = (max_len + page - 1) // page
    nblocks = B * nblk_per + 3
    kc = torch.randn(nblocks, page, Hkv, D, device="cuda", dtype=torch.bfloat16)
    vc = torch.randn_like(kc)
    perm = torch.randperm(nblocks, device="cuda")[: B * nblk_per].to(torch.int32).view(B, nblk_per)
    kv_lens = torch.randint(1, max_len + 1, (B,), device="cuda", dtype=torch.int32)
    kv_lens[0] = max_len
    q = torch.randn(B, Hq, D, device="cuda", dtype=torch.bfloat16)
    scale = 1.0 / math.sqrt(D)
    out, lse = ops.decode_attention(q, kc, vc, kv_lens, perm, scale, soft_cap, splits, return_lse=True)
    ref, ref_lse = _paged_attn_ref(q, kc, vc, kv_lens, perm, scale, soft_cap)
    torch.testing.assert_close(out.float(), ref, rtol=2e-2, atol=2e-2)
    torch.testing.assert_close(lse, ref_lse, rtol=1e-2, atol=1e-2)


def test_top_p_sampling_matches_sorted_reference():
    from triton_distributed_b200 import ops
    torch.manual_seed(7)
    B, V = 6, 151936
    logits = torch.randn(B, V, device="cuda") * 3
    temperature, top_p = 0.6, 0.95
    probs = torch.softmax(logits / temperature, -1)
    sp, si = torch.sort(probs, -1, descending=True)
    keep = (torch.cumsum(sp, -1) - sp) < top_p
    nucleus = torch.zeros_like(probs, dtype=torch.bool).scatter(1, si, keep)
    counts = torch.zeros(B, V, device="cuda")
    n_draws = 400
    for _ in range(n_draws):
        ids = ops.top_p_sample(logits, temperature, top_p)
        assert ids.shape == (B, 1) and ids.dtype == torch.int64
        assert bool(nucleus.gather(1, ids).all()), "sampled a token outside the nucleus"
        counts.scatter_add_(1, ids, torch.ones(B, 1, device="cuda"))
    # the most likely token must be drawn about as often as its renormalised probability says
    pn = probs * nucleus
    pn = pn / pn.sum(-1, keepdim=True)
    top = pn.argmax(-1, keepdim=True)
    want = pn.gather(1, top).squeeze(1)
    got = counts.gather(1, top).squeeze(1) / n_draws
    assert torch.all((got - want).abs() < 4 * torch.sqrt(want * (1 - want) / n_draws) + 0.02)
    # u = 0 picks the first kept index, and peaked logits are deterministic
    peaked = torch.full((2, 1000), -30.0, device="cuda")
    peaked[0, 123] = 10.0
    peaked[1, 999] = 10.0
    ids = ops.top_p_sample(peaked, 1.0, 0.9)
    assert ids.flatten().tolist() == [123, 999]
    # odd vocabulary: rows that are not 16-byte aligned take the scalar path; tiny rows leave some CTAs without work
    odd = torch.full((3, 1001), -30.0, device="cuda")
    odd[0, 1000] = 10.0
    odd[1, 5] = 10.0
    odd[2, 500] = 10.0
    assert ops.top_p_sample(odd, 1.0, 0.9).flatten().tolist() == [1000, 5, 500]
    tiny = torch.full((2, 10), -30.0, device="cuda")
    tiny[0, 9] = 5.0
    tiny[1, 0] = 5.0
    assert ops.top_p_sample(tiny, 0.7, 0.5).flatten().tolist() == [9, 0]


@pytest.mark.parametrize("M,K,Hq,Hkv,with_norm,with_scale", [(8, 5120, 8, 1, True, True), (3, 512, 2, 2, False, False),
                                                             (16, 1024, 64, 8, True, False)])
def test_gemm_skinny_qkv_heads_epilogue(M, K, Hq, Hkv, with_norm, with_scale):
    """The qkv projection that finishes every head in its epilogue (per-head RMSNorm, RoPE, q buffer, cache write),
    optionally with the input's RMSNorm folded in as a per-row scale, against the fp32 statement of the same chain."""
    from triton_distributed_b200 import ops
    torch.manual_seed(11)
    D, eps = 128, 1e-6
    N = (Hq + 2 * Hkv) * D
    h = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    w = torch.randn(N, K, device="cuda", dtype=torch.bfloat16) * K ** -0.5
    pos = torch.randint(0, 4000, (M,), device="cuda", dtype=torch.int32)
    inv = 1.0 / (1e6 ** (torch.arange(0, D, 2, device="cuda", dtype=torch.float32) / D))
    ang = torch.arange(4096, device="cuda", dtype=torch.float32)[:, None] * inv[None, :]
    cos_sin = torch.cat([ang.cos(), ang.sin()], -1).contiguous()
    qg = torch.randn(D, device="cuda", dtype=torch.bfloat16) if with_norm else None
    kg = torch.randn(D, device="cuda", dtype=torch.bfloat16) if with_norm else None
    slots = torch.randperm(64, device="cuda")[:M].to(torch.int64)
    kc = torch.zeros(64, Hkv, D, device="cuda", dtype=torch.bfloat16)
    vc = torch.zeros_like(kc)
    q = torch.zeros(M, Hq, D, device="cuda", dtype=torch.bfloat16)
    ep = ops.skinny_qkv_heads(pos, slots, cos_sin, Hq, Hkv, q, kc, vc, qg, kg, eps)
    x_in = h
    scale = torch.ones(M, 1, device="cuda")
    if with_scale:  # input = h * gain, rows scaled by 1 / rms(h) in the epilogue
        gain = torch.randn(K, device="cuda", dtype=torch.bfloat16)
        x_in = (h.float() * gain.float()).to(torch.bfloat16)
        sumsq = torch.zeros(16, device="cuda")
        sumsq[:M] = h.float().pow(2).sum(-1)
        ops.skinny_row_scale(sumsq, K, eps, base=ep)
        scale = torch.rsqrt(sumsq[:M] / K + eps)[:, None]
    for _ in range(2):
        ops.gemm_skinny(x_in, w, epilogue=ep)
    y = (x_in.float() @ w.float().t() * scale).view(M, Hq + 2 * Hkv, D)

    def norm(v, g):
        return v if g is None else v * torch.rsqrt(v.pow(2).mean(-1, keepdim=True) + eps) * g.float()

    q_ref = _rope_ref(norm(y[:, :Hq], qg), pos)
    k_ref = _rope_ref(norm(y[:, Hq:Hq + Hkv], kg), pos)
    torch.testing.assert_close(q.float(), q_ref, rtol=3e-2, atol=3e-2)
    torch.testing.assert_close(kc[slots].float(), k_ref, rtol=3e-2, atol=3e-2)
    torch.testing.assert_close(vc[slots].float(), y[:, Hq + Hkv:], rtol=3e-2, atol=3e-2)


@pytest.mark.parametrize("M,N,K", [(8, 5120, 1024), (5, 384, 4096), (16, 1000, 520)])
def test_gemm_skinny_residual_and_row_scale_epilogues(M, N, K):
    """Producer side: h = x W^T + residual, h * gain and sum(h^2). Consumer side: (h * gain) W2^T scaled by 1 / rms(h),
    plain and with SwiGLU, i.e. an RMSNorm between two projections without a normalisation kernel."""
    from triton_distributed_b200 import ops
    torch.manual_seed(12)
    eps = 1e-6
    x = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    w = torch.randn(N, K, device="cuda", dtype=torch.bfloat16) * K ** -0.5
    res = torch.randn(M, N, device="cuda", dtype=torch.bfloat16)
    res0 = res.clone()
    gain = torch.randn(N, device="cuda", dtype=torch.bfloat16)
    xg = torch.zeros(M, N, device="cuda", dtype=torch.bfloat16)
    sumsq = torch.zeros(16, device="cuda")
    ops.gemm_skinny(x, w, epilogue=ops.skinny_residual(res, sumsq, gain, xg))
    h = (x.float() @ w.float().t() + res0.float())
    torch.testing.assert_close(res.float(), h, rtol=2e-2, atol=2e-2)
    torch.testing.assert_close(xg.float(), res.float() * gain.float(), rtol=2e-2, atol=2e-2)
    torch.testing.assert_close(sumsq[:M], res.float().pow(2).sum(-1), rtol=1e-3, atol=1e-2)
    assert float(sumsq[M:].abs().sum()) == 0.0
    if N % 8 == 0:
        I = 256
        w2 = torch.randn(2 * I, N, device="cuda", dtype=torch.bfloat16) * N ** -0.5
        normed = (res.float() * torch.rsqrt(res.float().pow(2).mean(-1, keepdim=True) + eps) * gain.float())
        y = ops.gemm_skinny(xg, w2, epilogue=ops.skinny_row_scale(sumsq, N, eps))
        torch.testing.assert_close(y.float(), normed @ w2.float().t(), rtol=3e-2, atol=3e-2)
        act = ops.gemm_skinny(xg, w2, swiglu=True, epilogue=ops.skinny_row_scale(sumsq, N, eps))
        gu = normed @ w2.float().t()
        torch.testing.assert_close(act.float(), torch.nn.functional.silu(gu[:, :I]) * gu[:, I:], rtol=3e-2, atol=3e-2)


def test_embedding_with_norm_outputs():
    from triton_distributed_b200 import ops
    torch.manual_seed(13)
    V, H = 1000, 640
    table = torch.randn(V, H, device="cuda", dtype=torch.bfloat16)
    ids = torch.tensor([[3, 999], [0, 17]], device="cuda")
    gain = torch.randn(H, device="cuda", dtype=torch.bfloat16)
    assert torch.equal(ops.embedding(ids, table), table[ids])
    xg = torch.empty(4, H, device="cuda", dtype=torch.bfloat16)
    ss = torch.zeros(16, device="cuda")
    out = ops.embedding(ids.reshape(-1), table, gamma=gain, scaled_out=xg, sumsq_out=ss)
    assert torch.equal(out, table[ids.reshape(-1)])
    torch.testing.assert_close(xg.float(), out.float() * gain.float(), rtol=1e-2, atol=1e-2)
    torch.testing.assert_close(ss[:4], out.float().pow(2).sum(-1), rtol=1e-4, atol=1e-3)


@pytest.mark.parametrize("M,N,K", [(300, 8, 64), (1167, 4096, 72), (1167, 6144, 64), (129, 25000, 136), (260, 16392, 64), (520, 7560, 328), (2000, 2056, 64)])
@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_gemm_tile_widths(M, N, K, gated, dtype):
    """Sizes for which the pairs' tiles are 128 to 256 columns wide, none of them a multiple of the tile, into rows with a pitch, and
    the gated form. An fp32 sum of K products of norm one is off by less than K * 2^-20, then one rounding to 16 bits."""
    from triton_distributed_b200 import ops
    torch.manual_seed(19)
    a = torch.randn(M, K, device="cuda", dtype=dtype)
    b = torch.randn(2 * N if gated else N, K, device="cuda", dtype=dtype) * K ** -0.5
    out = torch.full((M, N + 8), 7.0, device="cuda", dtype=dtype)
    (ops.gemm_gated if gated else ops.gemm)(a, b, out[:, :N])
    want = a.double() @ b.double().t()
    if gated:
        gate, up = want.chunk(2, dim=1)
        want = gate * torch.sigmoid(gate) * up
    assert (out[:, N:] == 7).all()
    torch.testing.assert_close(out[:, :N].double(), want, rtol=2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -10, atol=K * 2.0 ** -20)


@pytest.mark.parametrize("lens,Hq,Hkv,page,splits", [((1, 15, 16, 17), 8, 1, 64, 1), ((63, 64, 65, 300), 6, 2, 16, 2), ((129, 1000, 2, 777), 32, 4, 48, 5),
                                                     ((500, 31, 64, 4000), 3, 3, 10, 4)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rising", [False, True])
def test_decode_attention_small_groups(lens, Hq, Hkv, page, splits, dtype, rising):
    """Up to eight heads per KV head: lengths around the 16-token slices, pages that slices cross, groups that fill a part of the tile, and
    scores that rise along the keys, so that the reference maximum moves again and again. Error against 64 bits: probabilities and
    the result are rounded to 16 bits, half a unit (2^-9, 2^-12) of the largest value each, doubled for the sums."""
    from triton_distributed_b200 import ops
    torch.manual_seed(21)
    B, D, blocks = len(lens), 128, -(-max(lens) // page)
    table = torch.randperm(B * blocks, device="cuda").to(torch.int32).view(B, blocks)
    q = torch.randn(B, Hq, D, device="cuda", dtype=dtype)
    k, v = (torch.randn(B * blocks, page, Hkv, D, device="cuda", dtype=dtype) for _ in range(2))
    if rising:  # scores climb by up to 60 along the sequence
        for b, n in enumerate(lens):
            at = torch.arange(blocks * page, device="cuda").clamp(max=n - 1) / n
            lift = (q[b].view(Hkv, -1, D)[:, 0].float() / q[b].view(Hkv, -1, D)[:, 0].float().norm(dim=-1, keepdim=True) * 60)
            k[table[b].long()] += (at.view(blocks, page, 1, 1) * lift).to(dtype)
    kv = torch.tensor(lens, dtype=torch.int32, device="cuda")
    out, lse = ops.decode_attention(q, k, v, kv, table, D ** -0.5, 0.0, splits, return_lse=True)
    for b, n in enumerate(lens):
        kb, vb = (c[table[b].long()].flatten(0, 1)[:n].double().repeat_interleave(Hq // Hkv, 1) for c in (k, v))
        s = torch.einsum("hd,nhd->hn", q[b].double(), kb) * D ** -0.5
        want = torch.einsum("hn,nhd->hd", torch.softmax(s, -1), vb)
        half = 2.0 ** -9 if dtype == torch.bfloat16 else 2.0 ** -12
        assert ((out[b].double() - want).abs() <= 2 * half * (want.abs() + vb.abs().amax())).all()
        torch.testing.assert_close(lse[b].double(), torch.logsumexp(s, -1), rtol=1e-5, atol=1e-4)


@pytest.mark.parametrize("E,k", [(1, 1), (8, 8), (33, 4), (128, 8), (129, 8), (256, 32), (257, 3), (512, 8)])
def test_topk_softmax_widths_and_ties(E, k):
    """Every number of values per lane and its edges, equal logits (the lower expert goes first) and -inf logits, against a stable sort
    in fp64; a probability is off by a few units of fp32."""
    from triton_distributed_b200 import ops
    torch.manual_seed(22)
    T = 300
    logits = (torch.randn(T, E, device="cuda") * 4).round() / 2   # many ties
    logits[0] = 0.0
    if E > k:
        logits[1, : E - k] = -torch.inf
    for renorm in (False, True):
        ids, w = ops.topk_softmax(logits, k, renorm)
        p = torch.softmax(logits.double(), -1)
        want_p, want = torch.sort(p, dim=-1, descending=True, stable=True)
        want_p = want_p[:, :k] / (want_p[:, :k].sum(-1, keepdim=True) if renorm else 1.0)
        assert torch.equal(ids.long(), want[:, :k])
        torch.testing.assert_close(w.double(), want_p, rtol=1e-5, atol=1e-9)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_prefill_attention_largest_weight_is_exact(dtype):
    """A key of a later step outweighs the ones before it by a power of two that is no whole number: its weight is held as one, so the
    columns of a row share no rounding error of their own."""
    from triton_distributed_b200 import ops
    torch.manual_seed(8)
    S, n, D = 128, 300, 128
    q, k, v = torch.zeros(S, 1, D), torch.zeros(n, 1, D), torch.zeros(n, 1, D)
    q[:, 0, 0], k[200, 0, 0] = torch.linspace(0.1, 5.5, S), 1.0
    v[200] = torch.rand(1, D) + 1.0
    q, k, v = q.to(dtype), k.to(dtype), v.to(dtype)
    ends = [torch.tensor([0, m], dtype=torch.int32, device="cuda") for m in (S, n)]
    out = ops.prefill_attention(q.cuda(), k.cuda(), v.cuda(), *ends, S, n, 1.0, False).double().cpu()
    w = torch.exp(q[:, 0].double() @ k[:, 0].double().t())
    want = w @ v[:, 0].double() / w.sum(1, keepdim=True)
    # fp32 sums (2^-21 of the result with the exponentials) move the rounding of hardly any of the outputs: up to four of a row's 128,
    # by a unit in the last place each, which is 2^-7 of a value just above a power of two in bf16
    unit = 2.0 ** -7 if dtype == torch.bfloat16 else 2.0 ** -10
    assert ((out[:, 0] - want.to(dtype).double()) / want).mean(1).abs().max() <= 4 * unit / D


@pytest.mark.parametrize("form", ["tiled", "grouped", "wide grouped"])
def test_gated_epilogues_of_very_negative_gates(form):
    """Gates down to the end of the exponential's range: small numbers, not zero, and of full precision times a large up value."""
    from triton_distributed_b200 import ops
    from triton_distributed_b200.kernels.nvidia import create_sort_plan, moe_sort
    from triton_distributed_b200.kernels.nvidia.allgather_group_gemm import grouped_gemm_planned
    M, N, K = {"tiled": 200, "grouped": 8, "wide grouped": 600}[form], 256, 64
    a = torch.zeros(M, K, device="cuda", dtype=torch.bfloat16)
    a[:, 0] = 1.0
    b = torch.zeros(2 * N, K, device="cuda", dtype=torch.bfloat16)
    b[:N, 0] = -torch.linspace(80.0, 90.0, N).to(torch.bfloat16)
    b[N:, 0] = 2.0 ** 20
    if form == "tiled":
        out = ops.gemm_gated(a, b)
    else:
        plan = moe_sort(torch.zeros(M, 1, dtype=torch.int32, device="cuda"), create_sort_plan(M, 1, 4, 128, 1))
        out = grouped_gemm_planned(a, torch.stack([b] * 4), plan, 1, gated=True)
    z = b[:N, 0].double()
    want = (z * torch.exp(z) * 2.0 ** 20).expand(M, N)
    # exp(-z) itself overflows behind 88.7: zero there, as an IEEE division of z by infinity gives. 2^-9 of the rounding to 16 bits and
    # 2 + |z| units of 2^-23 of the exponential, twice
    near = z > -88.7
    assert ((out.double() - want).abs() <= 2.0 ** -8 * want.abs())[:, near].all()
    assert (out[:, z < -88.8] == 0).all()


@pytest.mark.parametrize("B,S", [(1, 1), (3, 1), (1, 257), (3, 300), (70, 5)])
@pytest.mark.parametrize("dtype", [torch.int64, torch.int32])
def test_step_tables(B, S, dtype):
    """Positions from an offset of each sequence, also as rows of a wider matrix and as columns of a transposed one."""
    from triton_distributed_b200 import ops
    from triton_distributed_b200.models import KV_Cache
    torch.manual_seed(9)
    kv = KV_Cache(1, B, 1024, 1, 128, torch.bfloat16, 1)
    pos = (torch.randint(0, 500, (B, 1)) + torch.arange(S)[None]).to(dtype).cuda()
    wide = torch.full((B, S + 3), -1, dtype=dtype, device="cuda")
    wide[:, 2:2 + S] = pos
    for ids in (pos, wide[:, 2:2 + S], pos.t().contiguous().t()):
        step = ops.step_tables(ids, kv.blocks_per_seq * kv.page_size)
        assert step["pos"].dtype == step["kv_lens"].dtype == torch.int32 and step["slots"].dtype == torch.int64
        assert torch.equal(step["pos"], pos.reshape(-1).to(torch.int32))
        assert torch.equal(step["slots"], kv.slots(pos))
        assert torch.equal(step["kv_lens"], (pos[:, -1] + 1).to(torch.int32))
