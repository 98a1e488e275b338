"""Every selectable variant of the attention kernels against fp32 PyTorch references: the three K/V pipelines of the
decode kernel with and without the in-kernel merge of the splits, and the tcgen05 prefill kernel on packed sequences
and on keys read in place from a cache-like slot array."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _paged_ref(q, kc, vc, kv_lens, bt, scale):
    B, Hq, D = q.shape
    page, Hkv = kc.shape[1], kc.shape[2]
    G = Hq // Hkv
    out = torch.zeros(B, Hq, D, device=q.device)
    lse = torch.zeros(B, Hq, device=q.device)
    for b in range(B):
        L = int(kv_lens[b])
        slots = (bt[b].long()[:, None] * page + torch.arange(page, device=q.device)[None, :]).reshape(-1)[:L]
        k = kc.view(-1, Hkv, D)[slots].float().repeat_interleave(G, dim=1)
        v = vc.view(-1, Hkv, D)[slots].float().repeat_interleave(G, dim=1)
        s = torch.einsum("hd,lhd->hl", q[b].float(), k) * scale
        lse[b] = torch.logsumexp(s, -1)
        out[b] = torch.einsum("hl,lhd->hd", torch.softmax(s, -1), v)
    return out, lse


@pytest.mark.parametrize("ring", [0, 3, 6])
@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("B,Hq,Hkv,page,max_len,splits", [(3, 64, 8, 1, 777, 4), (1, 32, 4, 64, 4096, 8), (2, 40, 2, 16, 500, 2),
                                                          (8, 8, 1, 64, 2100, 9), (2, 16, 16, 32, 130, 1)])
def test_decode_attention_pipelines_and_fused_merge(ring, fused, B, Hq, Hkv, page, max_len, splits):
    from triton_distributed_b200 import ops
    torch.manual_seed(6)
    D = 128
    nblk_per = (max_len + page - 1) // page
    nblocks = B * nblk_per + 3
    kc = torch.randn(nblocks, page, Hkv, D, device="cuda", dtype=torch.bfloat16)
    vc = torch.randn_like(kc)
    bt = torch.randperm(nblocks, device="cuda")[: B * nblk_per].to(torch.int32).view(B, nblk_per)
    kv_lens = torch.randint(1, max_len + 1, (B,), device="cuda", dtype=torch.int32)
    kv_lens[0] = max_len
    q = torch.randn(B, Hq, D, device="cuda", dtype=torch.bfloat16)
    scale = 1.0 / math.sqrt(D)
    ws: dict = {}
    for _ in range(2):  # the second call reuses the workspace and finds the tickets zeroed by the first
        out, lse = ops.decode_attention(q, kc, vc, kv_lens, bt, scale, 0.0, splits, return_lse=True, workspace=ws,
                                        fused_combine=fused, ring=ring)
        ref, ref_lse = _paged_ref(q, kc, vc, kv_lens, bt, scale)
        torch.testing.assert_close(out.float(), ref, rtol=2e-2, atol=2e-2)
        torch.testing.assert_close(lse, ref_lse, rtol=1e-2, atol=1e-2)
    if fused and splits > 1:
        assert int(ws["tickets"].abs().sum()) == 0


def _attn_ref(q, k, v, scale, causal):
    """q [lq, Hq, D], k / v [lk, Hkv, D] -> [lq, Hq, D] in fp32 (64 bits for 64-bit inputs) with the bottom-right aligned causal mask."""
    lq, lk, G = q.shape[0], k.shape[0], q.shape[1] // k.shape[1]
    wide = torch.promote_types(q.dtype, torch.float32)
    kk, vv = k.to(wide).repeat_interleave(G, dim=1), v.to(wide).repeat_interleave(G, dim=1)
    s = torch.einsum("qhd,khd->hqk", q.to(wide), kk) * scale
    if causal:
        qi = torch.arange(lq, device=q.device)[:, None] + (lk - lq)
        ki = torch.arange(lk, device=q.device)[None, :]
        s = s.masked_fill(ki > qi, float("-inf"))
    return torch.einsum("hqk,khd->qhd", torch.softmax(s, -1).nan_to_num(0.0), vv)


@pytest.mark.parametrize("lens_q,lens_k,Hq,Hkv,causal", [
    ([128], [128], 2, 1, True), ([300, 77], [300, 77], 8, 2, True), ([64, 200], [256, 333], 4, 4, True),
    ([130], [513], 4, 1, False), ([1024, 1], [1024, 700], 8, 8, True)])
def test_prefill_attention_matches_reference(lens_q, lens_k, Hq, Hkv, causal):
    """Packed variable-length sequences, GQA, and the bottom-right alignment of the causal mask when a sequence has
    more keys than queries."""
    from triton_distributed_b200 import ops
    torch.manual_seed(5)
    D = 128
    cu_q = torch.tensor([0] + list(torch.tensor(lens_q).cumsum(0)), dtype=torch.int32, device="cuda")
    cu_k = torch.tensor([0] + list(torch.tensor(lens_k).cumsum(0)), dtype=torch.int32, device="cuda")
    q = torch.randn(sum(lens_q), Hq, D, device="cuda", dtype=torch.bfloat16)
    k = torch.randn(sum(lens_k), Hkv, D, device="cuda", dtype=torch.bfloat16)
    v = torch.randn(sum(lens_k), Hkv, D, device="cuda", dtype=torch.bfloat16)
    scale = 1 / math.sqrt(D)
    out = ops.prefill_attention(q, k, v, cu_q, cu_k, max(lens_q), max(lens_k), scale, causal)
    ops.check_pipeline_status()
    for b, (lq, lk) in enumerate(zip(lens_q, lens_k)):
        qs, ks = int(cu_q[b]), int(cu_k[b])
        want = _attn_ref(q[qs:qs + lq], k[ks:ks + lk], v[ks:ks + lk], scale, causal)
        torch.testing.assert_close(out[qs:qs + lq].float(), want, rtol=3e-2, atol=3e-2)


@pytest.mark.parametrize("lens_q,lens_k,Hq,Hkv,dk,dv", [
    ([1, 16, 128], [1, 16, 128], 8, 2, 128, 128),              # one step
    ([129, 389, 40], [129, 389, 40], 8, 2, 128, 128), ([300, 5], [300, 700], 8, 8, 128, 136),   # two row blocks of a head; a cached prefix
    ([100, 1, 500], [100, 300, 500], 4, 4, 72, 72), ([700, 260], [1200, 260], 8, 1, 64, 64), ([40], [1000], 6, 2, 40, 200)])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_prefill_attention_forms_agree(lens_q, lens_k, Hq, Hkv, dk, dv, causal, dtype):
    """Small calls have the softmax warps rescale and store, larger ones warps of their own: the same bits, and those of the formula."""
    from itertools import accumulate
    from triton_distributed_b200 import ops
    torch.manual_seed(31)
    cu_q, cu_k = (torch.tensor([0, *accumulate(n)], dtype=torch.int32, device="cuda") for n in (lens_q, lens_k))
    q, k, v = (torch.randn(sum(n), h, d, device="cuda").to(dtype) for n, h, d in ((lens_q, Hq, dk), (lens_k, Hkv, dk), (lens_k, Hkv, dv)))
    gate = torch.randn(sum(lens_q), Hq, device="cuda").to(dtype)
    small = ops.prefill_attention(q, k, v, cu_q, cu_k, max(lens_q), max(lens_k), dk ** -0.5, causal, gate=gate)
    assert torch.equal(small, ops.prefill_attention(q, k, v, cu_q, cu_k, max(lens_q), 1 << 20, dk ** -0.5, causal, gate=gate))
    ops.check_pipeline_status()
    for b, (n, m) in enumerate(zip(lens_q, lens_k)):
        qs, ks, vs = q[cu_q[b]:cu_q[b] + n].double(), k[cu_k[b]:cu_k[b] + m].double(), v[cu_k[b]:cu_k[b] + m].double()
        s = torch.einsum("qhd,khd->hqk", qs, ks.repeat_interleave(Hq // Hkv, 1)) * dk ** -0.5
        if causal:
            s.masked_fill_(torch.ones(n, m, dtype=torch.bool, device="cuda").triu(m - n + 1), -torch.inf)
        want = torch.einsum("hqk,khd->qhd", s.softmax(-1), vs.repeat_interleave(Hq // Hkv, 1)) * torch.sigmoid(gate[cu_q[b]:cu_q[b] + n].double())[..., None]
        # probabilities and result are rounded once each: half a unit in the last place of both
        assert (small[cu_q[b]:cu_q[b] + n].double() - want).norm() <= torch.finfo(dtype).eps * want.norm()


def test_prefill_attention_reads_keys_in_place():
    """Keys of every sequence start at a fixed stride in a larger slot array (a cache whose sequences own contiguous
    runs of slots); rows beyond a sequence's length hold garbage that must not be read into the result."""
    from triton_distributed_b200 import ops
    torch.manual_seed(8)
    D, Hq, Hkv, stride = 128, 8, 2, 640
    lens_q, lens_k = [200, 64, 333], [200, 500, 333]
    B = len(lens_q)
    k = torch.randn(B * stride, Hkv, D, device="cuda", dtype=torch.bfloat16) * 30
    v = torch.randn(B * stride, Hkv, D, device="cuda", dtype=torch.bfloat16) * 30
    cu_q = torch.tensor([0] + list(torch.tensor(lens_q).cumsum(0)), dtype=torch.int32, device="cuda")
    cu_k = torch.arange(0, (B + 1) * stride, stride, dtype=torch.int32, device="cuda")
    q = torch.randn(sum(lens_q), Hq, D, device="cuda", dtype=torch.bfloat16)
    scale = 1 / math.sqrt(D)
    for b, lk in enumerate(lens_k):  # valid rows are well-scaled; everything else stays large
        k[b * stride:b * stride + lk].normal_()
        v[b * stride:b * stride + lk].normal_()
    out = ops.prefill_attention(q, k, v, cu_q, cu_k, max(lens_q), stride, scale, True,
                                seqlens_k=torch.tensor(lens_k, dtype=torch.int32, device="cuda"))
    ops.check_pipeline_status()
    for b, (lq, lk) in enumerate(zip(lens_q, lens_k)):
        qs, ks = int(cu_q[b]), b * stride
        want = _attn_ref(q[qs:qs + lq], k[ks:ks + lk], v[ks:ks + lk], scale, True)
        torch.testing.assert_close(out[qs:qs + lq].float(), want, rtol=3e-2, atol=3e-2)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("lens_q,lens_k,Hq,Hkv,causal,rising", [
    ([1, 129, 300], [1, 129, 300], 6, 2, True, 0),      # odd group: two row blocks of a head, the last one without a partner
    ([257, 3], [640, 131], 5, 5, True, 0),              # behind a cached prefix
    ([128, 2, 255], [127, 0, 384], 4, 1, True, 0),      # a query without keys; the last tile ends with the last key
    ([70, 260], [1000, 5], 8, 2, False, 0),
    ([513], [513], 4, 2, True, 40)])                    # scores that grow with the key: every step moves the reference
def test_prefill_attention_tiles_and_foreign_rows(dtype, lens_q, lens_k, Hq, Hkv, causal, rising):
    """Edges of the row blocks and key tiles, both ways to pair tiles, values that start between two 16-byte boundaries, and NaN
    in every key and value row that belongs to no sequence."""
    from triton_distributed_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(11)
    D, stride, B = 128, 1024, len(lens_q)
    q = torch.randn(sum(lens_q), Hq, D, device="cuda", generator=g).to(dtype)
    k = torch.full((B * stride, Hkv, D), float("nan"), device="cuda", dtype=dtype)
    v = torch.full((B * stride * Hkv * D + 1,), float("nan"), device="cuda", dtype=dtype)[1:].view(B * stride, Hkv, D)
    for b, n in enumerate(lens_k):
        k[b * stride:b * stride + n] = torch.randn(n, Hkv, D, device="cuda", generator=g).to(dtype)
        v[b * stride:b * stride + n] = torch.randn(n, Hkv, D, device="cuda", generator=g).to(dtype)
        if rising:  # one channel adds up to `rising` to the scaled scores
            q[..., 0] = D ** 0.5
            k[b * stride:b * stride + n, :, 0] = torch.linspace(0, rising, n, device="cuda")[:, None].to(dtype)
    cu_q = torch.tensor([0] + lens_q, device="cuda").cumsum(0).int()
    cu_k = torch.arange(0, (B + 1) * stride, stride, dtype=torch.int32, device="cuda")
    out = ops.prefill_attention(q, k, v, cu_q, cu_k, max(lens_q), stride, D ** -0.5, causal,
                                seqlens_k=torch.tensor(lens_k, dtype=torch.int32, device="cuda"))
    ops.check_pipeline_status()
    for b, (lq, lk) in enumerate(zip(lens_q, lens_k)):
        qs, ks = int(cu_q[b]), b * stride
        want = _attn_ref(q[qs:qs + lq].double(), k[ks:ks + lk].double(), v[ks:ks + lk].double(), D ** -0.5, causal)
        # weights and output are each rounded to the storage type: two half units in the last place of the largest value, and as
        # much again for the fp32 scores (2^-24 times the sum of 128 products' magnitudes, in the exponent)
        unit = 2.0 ** (-9 if dtype == torch.bfloat16 else -12)
        top = float(v[ks:ks + lk].abs().max()) if lk else 0.0
        torch.testing.assert_close(out[qs:qs + lq].double(), want, rtol=0, atol=4 * unit * top)


def test_entry_points_of_native_callers():
    """The forms that programs without the Python layer call keep their arguments: GEMM, grouped GEMM, prefill attention with a scratch
    for transposed values (here also with values between two 16-byte boundaries)."""
    import ctypes
    from triton_distributed_b200 import _lib, ops
    from triton_distributed_b200._lib import ptr, stream_ptr
    from triton_distributed_b200.kernels.nvidia import create_sort_plan, grouped_gemm, moe_sort
    torch.manual_seed(5)
    bf, null, one = torch.bfloat16, None, ctypes.c_float(0.1)
    a, b = torch.randn(200, 64, device="cuda").to(bf), torch.randn(72, 64, device="cuda").to(bf)
    out = torch.empty(200, 72, dtype=bf, device="cuda")
    _lib.call("b200_gemm", ptr(a), ptr(b), ptr(out), 200, 72, 64, 64, 64, 72, 0, 0, stream_ptr())
    assert torch.equal(out, ops.gemm(a, b))
    w, ids = torch.randn(4, 72, 64, device="cuda").to(bf), torch.randint(0, 4, (200, 1), dtype=torch.int32, device="cuda")
    plan, scale = moe_sort(ids, create_sort_plan(200, 1, 4, 128, 1)), torch.rand(200, device="cuda")
    _lib.call("b200_grouped_gemm", ptr(a), 64, 1, ptr(w), 4, 72, 64, 200, ptr(plan.sorted_ids), ptr(plan.tile_expert), null, ptr(plan.totals),
              plan.max_tiles, ptr(out), 72, ptr(scale), 0, stream_ptr())
    assert torch.equal(out, grouped_gemm(a, w, ids, row_scale=scale))
    lib = _lib.load()
    lib.b200_prefill_attention_scratch_bytes.restype = ctypes.c_longlong
    n = lib.b200_prefill_attention_scratch_bytes(2, 2, 64, 130)
    assert n == 2 * 2 * 64 * 256 * 2
    q, k = torch.randn(200, 4, 64, device="cuda").to(bf), torch.randn(200, 2, 64, device="cuda").to(bf)
    ends, scratch = torch.tensor([0, 70, 200], dtype=torch.int32, device="cuda"), torch.empty(n, dtype=torch.uint8, device="cuda")
    for shift in (0, 1):
        v = torch.randn(200 * 2 * 64 + shift, device="cuda").to(bf)[shift:].view(200, 2, 64)
        got = torch.empty(200, 4, 64, dtype=bf, device="cuda")
        args = (ptr(q), ptr(k), ptr(v), ptr(ends), ptr(ends), null, 2, 200, 200, 130, 130, 4, 2, 64, 64, one, 1, null, 0)
        _lib.call("b200_prefill_attention", *args, ptr(scratch), ptr(got), 0, null, stream_ptr())
        assert torch.equal(got, ops.prefill_attention(q, k, v, ends, ends, 130, 130, 0.1, True))
        with pytest.raises(_lib.NativeError):
            _lib.call("b200_prefill_attention", *args, null, ptr(got), 0, null, stream_ptr())
