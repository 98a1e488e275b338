"""MoE kernels on one GPU: routing metadata against the CPU references, grouped GEMM against per-expert matmuls,
and the fused AG / RS forms with this GPU as the only rank."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,topk,E,bm,segments", [(37, 3, 8, 16, 1), (512, 8, 128, 128, 1), (64, 2, 4, 8, 4), (1024, 8, 256, 128, 8)])
def test_moe_sort_matches_reference(T, topk, E, bm, segments):
    from triton_distributed_b200 import ref
    from triton_distributed_b200.kernels.nvidia import create_sort_plan, moe_sort, order_tiles
    torch.manual_seed(0)
    ids = torch.stack([torch.randperm(E)[:topk] for _ in range(T)]).to(torch.int32).cuda()
    plan = create_sort_plan(T * topk, topk, E, bm, segments)
    for _ in range(2):  # epochs
        moe_sort(ids, plan, tokens_per_rank=max(1, T // 4))
    torch.cuda.synchronize()
    m_pad, tiles = int(plan.totals[0]), int(plan.totals[1])
    if segments == 1:
        counts, _, gather, expert_index, want_pad = ref.calc_gather_scatter_index_ref(ids.cpu(), E, bm)
        assert m_pad == want_pad and tiles == want_pad // bm
        assert torch.equal(plan.sorted_ids[:m_pad].cpu(), gather)
        assert torch.equal(plan.tile_expert[:tiles].cpu(), expert_index)
        assert torch.equal(plan.group_count.cpu(), counts)
        world = 4
        _, _, s0, s1, order = ref.ag_moe_tile_schedule_ref(ids.cpu(), E, bm, 1, world) if T % world == 0 else (0, 0, None, None, None)
        if s0 is not None:
            assert torch.equal(plan.tile_seg_start[:tiles].cpu(), s0) and torch.equal(plan.tile_seg_end[:tiles].cpu(), s1)
            got = order_tiles(plan, 1, world)
            torch.cuda.synchronize()
            assert torch.equal(got[:tiles].cpu(), order)
    else:
        sorted_ids, expert_ids, barrier_ids, rank_blocks, npad = ref.moe_align_block_size_ref(ids.cpu(), E, bm, segments)
        assert m_pad == npad
        assert torch.equal(plan.sorted_ids[:m_pad].cpu(), sorted_ids)
        assert torch.equal(plan.tile_expert[:tiles].cpu(), expert_ids)
        assert torch.equal(plan.tile_seg_end[:tiles].cpu(), barrier_ids)
        assert torch.equal(plan.totals[2:].cpu(), torch.cumsum(rank_blocks, 0).to(torch.int32))
    assert int(plan.status[0]) == 0


@pytest.mark.parametrize("T,topk,E,N,K", [(64, 2, 4, 128, 64), (300, 4, 16, 384, 512), (1024, 8, 32, 200, 1032),
                                             (256, 4, 8, 512, 256), (200, 2, 4, 1000, 192)])  # the last two: 256-wide tiles
def test_grouped_gemm_matches_per_expert_matmul(T, topk, E, N, K):
    from triton_distributed_b200 import ref
    from triton_distributed_b200.kernels.nvidia import grouped_gemm
    torch.manual_seed(1)
    a = torch.randn(T, K, device="cuda", dtype=torch.bfloat16)
    w = torch.randn(E, N, K, device="cuda", dtype=torch.bfloat16) * 0.05
    ids = torch.stack([torch.randperm(E)[:topk] for _ in range(T)]).to(torch.int32).cuda()
    out = grouped_gemm(a, w, ids)
    torch.cuda.synchronize()
    want = ref.grouped_gemm_ref(a.repeat_interleave(topk, 0), w, ids.reshape(-1).long())
    torch.testing.assert_close(out.float(), want, rtol=2e-2, atol=2e-2)
    # per-pair input and routing weights (the down-projection form)
    x = torch.randn(T * topk, K, device="cuda", dtype=torch.bfloat16)
    sc = torch.rand(T, topk, device="cuda")
    out2 = grouped_gemm(x, w, ids, a_per_pair=True, row_scale=sc)
    want2 = ref.grouped_gemm_ref(x, w, ids.reshape(-1).long()) * sc.reshape(-1, 1)
    torch.testing.assert_close(out2.float(), want2, rtol=2e-2, atol=2e-2)


def test_ag_group_gemm_and_moe_reduce_rs_world1(dist1):
    from triton_distributed_b200 import ref
    from triton_distributed_b200.kernels.nvidia import (ag_group_gemm, create_ag_group_gemm_context, create_moe_rs_context,
                                                        moe_reduce_rs)
    from triton_distributed_b200.runtime.heap import get_heap
    torch.manual_seed(2)
    T, topk, E, K, N = 256, 4, 16, 512, 384
    a = torch.randn(T, K, device="cuda", dtype=torch.bfloat16)
    w1 = torch.randn(E, N, K, device="cuda", dtype=torch.bfloat16) * 0.05
    logits = torch.randn(T, E, device="cuda")
    wt, ids = torch.topk(torch.softmax(logits, -1), topk, -1)
    ids = ids.to(torch.int32)
    ctx = create_ag_group_gemm_context(T, N, K, E, topk, torch.bfloat16, 0, 1)
    for _ in range(3):
        up = ag_group_gemm(a, w1, ctx, ids)
        torch.cuda.synchronize()
        get_heap().check_status("ag_group_gemm")
        torch.testing.assert_close(up.float(), ref.ag_group_gemm_ref(a, w1, ids).float(), rtol=2e-2, atol=2e-2)
    # the reference's [E, K, N] weight layout is accepted too
    up_t = ag_group_gemm(a, w1.transpose(1, 2).contiguous(), ctx, ids)
    torch.testing.assert_close(up_t, up)
    ctx.finalize()
    w2 = torch.randn(E, 640, N, device="cuda", dtype=torch.bfloat16) * 0.05
    rctx = create_moe_rs_context(dist1, 1, T, 640, E, topk, torch.bfloat16, torch.bfloat16)
    for _ in range(3):
        down = moe_reduce_rs(up, w2, ids, wt, rctx)
        torch.cuda.synchronize()
        get_heap().check_status("moe_reduce_rs")
        torch.testing.assert_close(down.float(), ref.moe_reduce_rs_ref(up, w2, ids, wt).float(), rtol=3e-2, atol=3e-2)
    rctx.finalize()


def _dequant_weight_blocks(w8, sw):
    E, N, K = w8.shape
    scale = sw.repeat_interleave(128, 1)[:, :N].repeat_interleave(128, 2)
    return w8.float() * scale


def test_fp8_ag_group_gemm_and_moe_reduce_rs_world1(dist1):
    """The block-scaled fp8 forms of both tensor-parallel MoE fusions against the dequantised fp32 products."""
    from triton_distributed_b200 import ref
    from triton_distributed_b200.kernels.nvidia import (ag_group_gemm_fp8, create_ag_group_gemm_fp8_context,
                                                        create_moe_rs_context, moe_reduce_rs_fp8, quantize_fp8_rows,
                                                        quantize_fp8_weight_blocks)
    from triton_distributed_b200.runtime.heap import get_heap
    torch.manual_seed(12)
    T, topk, E, K, N, H = 256, 4, 16, 512, 384, 640
    a8, sa = quantize_fp8_rows(torch.randn(T, K, device="cuda") * torch.rand(T, 1, device="cuda") * 3)
    w8, sw = quantize_fp8_weight_blocks(torch.randn(E, N, K, device="cuda") * 0.05)
    wt, ids = torch.topk(torch.softmax(torch.randn(T, E, device="cuda"), -1), topk, -1)
    ids = ids.to(torch.int32)
    a_deq = ref.fp8_dequant_ref(a8, sa, dtype=torch.float32)
    want_up = ref.grouped_gemm_ref(a_deq.repeat_interleave(topk, 0), _dequant_weight_blocks(w8, sw), ids.reshape(-1).long())
    ctx = create_ag_group_gemm_fp8_context(T, N, K, E, topk, torch.bfloat16, 0, 1)
    for _ in range(3):
        up = ag_group_gemm_fp8(a8, sa, w8, sw, ctx, ids)
        torch.cuda.synchronize()
        get_heap().check_status("ag_group_gemm_fp8")
        torch.testing.assert_close(up.float(), want_up.float(), rtol=2e-2, atol=2e-2)
    ctx.finalize()
    x8, sx = quantize_fp8_rows(up.float())
    w28, sw2 = quantize_fp8_weight_blocks(torch.randn(E, H, N, device="cuda") * 0.05)
    x_deq = ref.fp8_dequant_ref(x8, sx, dtype=torch.float32)
    pairs = ref.grouped_gemm_ref(x_deq, _dequant_weight_blocks(w28, sw2), ids.reshape(-1).long()) * wt.reshape(-1, 1)
    want_down = pairs.view(T, topk, H).sum(1)
    rctx = create_moe_rs_context(dist1, 1, T, H, E, topk, torch.bfloat16, torch.bfloat16)
    for _ in range(3):
        down = moe_reduce_rs_fp8(x8, sx, w28, sw2, ids, wt, rctx)
        torch.cuda.synchronize()
        get_heap().check_status("moe_reduce_rs_fp8")
        torch.testing.assert_close(down.float(), want_down.float(), rtol=3e-2, atol=3e-2)
    rctx.finalize()


def test_ep_dispatch_combine_world1(dist1):
    from triton_distributed_b200 import ref
    from triton_distributed_b200.layers.nvidia import EPAll2AllLayer
    from triton_distributed_b200.runtime.heap import get_heap
    torch.manual_seed(3)
    T, H, E, topk = 96, 512, 16, 4
    x = torch.randn(T, H, device="cuda", dtype=torch.bfloat16)
    wt, ids = torch.topk(torch.softmax(torch.randn(T, E, device="cuda"), -1), topk, -1)
    ids = ids.to(torch.int32)
    for fp8 in (False, True):
        layer = EPAll2AllLayer(dist1, T, H, topk, 0, E, 1, 1, torch.bfloat16, fp8=fp8)
        for _ in range(3):
            res = layer.dispatch(x, ids)
            torch.cuda.synchronize()
            get_heap().check_status("ep dispatch")
            sorted_ids, tile_expert, totals, rows_per_expert = layer.recv_plan()
            assert int(rows_per_expert.sum()) == T * topk
            assert torch.equal(rows_per_expert.cpu(), torch.bincount(ids.reshape(-1).long().cpu(), minlength=E).to(torch.int32))
            if fp8:
                q, sc = res
                rows = ref.fp8_dequant_ref(q[: T * topk], sc[: T * topk], dtype=torch.bfloat16)
                expert_out = torch.zeros(layer.max_m, H, device="cuda", dtype=torch.bfloat16)
                expert_out[: T * topk] = rows
            else:
                expert_out = res
            out = layer.combine(expert_out, wt)
            torch.cuda.synchronize()
            get_heap().check_status("ep combine")
            torch.testing.assert_close(out.float(), x.float() * wt.sum(-1, keepdim=True), rtol=0.1 if fp8 else 2e-2,
                                       atol=0.1 if fp8 else 2e-2)
        layer.finalize()


@pytest.mark.parametrize("T,topk,E,N,K", [(64, 2, 4, 128, 128), (300, 4, 16, 384, 512), (1024, 8, 32, 200, 1024)])
def test_grouped_gemm_fp8_block_scaled(T, topk, E, N, K):
    """e4m3 operands, 1x128 activation scales and 128x128 weight scales, against the dequantised fp32 product."""
    from triton_distributed_b200 import ref
    from triton_distributed_b200.kernels.nvidia import grouped_gemm_fp8, quantize_fp8_rows, quantize_fp8_weight_blocks
    torch.manual_seed(3)
    a = torch.randn(T, K, device="cuda") * torch.rand(T, 1, device="cuda") * 4   # rows of very different magnitude
    w = torch.randn(E, N, K, device="cuda") * 0.05
    a8, sa = quantize_fp8_rows(a)
    w8, sw = quantize_fp8_weight_blocks(w)
    ids = torch.stack([torch.randperm(E)[:topk] for _ in range(T)]).to(torch.int32).cuda()
    out = grouped_gemm_fp8(a8, sa, w8, sw, ids)
    torch.cuda.synchronize()
    want = ref.grouped_gemm_fp8_ref(a8.repeat_interleave(topk, 0), sa.repeat_interleave(topk, 0), w8, sw, ids.reshape(-1).long())
    torch.testing.assert_close(out.float(), want, rtol=2e-2, atol=2e-2)
    # and it is close to the unquantised product (fp8 has 3 mantissa bits: a few percent of the row norm)
    exact = ref.grouped_gemm_ref(a.repeat_interleave(topk, 0), w, ids.reshape(-1).long())
    err = (out.float() - exact).norm() / exact.norm()
    assert err < 0.06, f"relative error {err:.3f} against the bf16 product"
    # per-pair rows with routing weights (the down-projection form)
    x = torch.randn(T * topk, K, device="cuda")
    x8, sx = quantize_fp8_rows(x)
    sc = torch.rand(T, topk, device="cuda")
    out2 = grouped_gemm_fp8(x8, sx, w8, sw, ids, a_per_pair=True, row_scale=sc)
    want2 = ref.grouped_gemm_fp8_ref(x8, sx, w8, sw, ids.reshape(-1).long()) * sc.reshape(-1, 1)
    torch.testing.assert_close(out2.float(), want2, rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("fp8,fp8_experts", [(False, False), (True, False), (True, True)])
def test_ep_moe_layer_world1(dist1, fp8, fp8_experts):
    """Expert-parallel MoE layer with the GPU as its own only peer: dispatch -> grouped GEMMs -> weighted combine,
    in bf16, with fp8 dispatch, and with the block-scaled fp8 up-projection on the dispatched bytes."""
    from triton_distributed_b200.layers.nvidia import EP_MoE
    from triton_distributed_b200.runtime.heap import get_heap
    E, topk, H, I, T = 8, 2, 256, 384, 64
    torch.manual_seed(11)
    gate = torch.randn(E, H, device="cuda", dtype=torch.bfloat16)  # wide logits: no near-ties between experts
    wgu = torch.randn(E, 2 * I, H, device="cuda", dtype=torch.bfloat16) * 0.05
    wdn = torch.randn(E, H, I, device="cuda", dtype=torch.bfloat16) * 0.05
    x = torch.randn(T, H, device="cuda", dtype=torch.bfloat16)
    ep = EP_MoE(0, 1, dist1, E, topk, H, T, torch.bfloat16, True, fp8_dispatch=fp8, fp8_experts=fp8_experts)
    ep._init_parameters(gate, wgu, wdn)
    want = ep.torch_fwd(x, wgu, wdn)
    for _ in range(2):
        got = ep.dist_triton_fwd(x)
        torch.cuda.synchronize()
        get_heap().check_status("ep_moe")
        torch.testing.assert_close(got.float(), want.float(), rtol=0.12 if fp8 else 5e-2, atol=0.3 if fp8 else 0.1)
    ep.finalize()


@pytest.mark.parametrize("T,I", [(5, 128), (300, 384), (4096, 1536)])
def test_silu_mul_fp8_matches_gate_then_block_quant(T, I):
    """The fused SwiGLU + e4m3 block quantisation against silu_mul followed by the PyTorch quantiser: scales agree to
    rounding, and the dequantised values agree within one e4m3 step."""
    from triton_distributed_b200 import ops
    from triton_distributed_b200.kernels.nvidia import quantize_fp8_rows
    torch.manual_seed(14)
    x = torch.randn(T, 2 * I, device="cuda", dtype=torch.bfloat16)
    q, s = ops.silu_mul_fp8(x)
    xf = x.float()
    act = torch.nn.functional.silu(xf[:, :I]) * xf[:, I:]
    q_ref, s_ref = quantize_fp8_rows(act)
    torch.testing.assert_close(s, s_ref, rtol=1e-4, atol=1e-8)
    deq = (q.float().view(T, I // 128, 128) * s[:, :, None]).view(T, I)
    torch.testing.assert_close(deq, act, rtol=0.07, atol=1e-3)
    deq_ref = (q_ref.float().view(T, I // 128, 128) * s_ref[:, :, None]).view(T, I)
    assert (deq - deq_ref).abs().max() <= 0.07 * act.abs().max()


@pytest.mark.parametrize("T,topk,N", [(1, 1, 8), (3, 8, 2048), (257, 3, 1032), (5, 9, 20), (40000, 2, 64)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("weighted", [False, True])
def test_reduce_topk_against_64_bits(T, topk, N, dtype, weighted):
    """Widths with and without whole 16-byte vectors, odd k, more rows than one wave. Error: one rounding to 16 bits of the result and
    topk + 1 fp32 roundings of the absolute sum. Recording autograd and views keep the torch operators' behaviour."""
    from triton_distributed_b200.kernels.nvidia import reduce_topk
    torch.manual_seed(15)
    x = torch.randn(T * topk, N, device="cuda", dtype=dtype)
    w = torch.rand(T, topk, device="cuda") if weighted else None
    wide = x.double().view(T, topk, N) * (w.double().view(T, topk, 1) if weighted else 1.0)
    want, bound = wide.sum(1), wide.abs().sum(1) * (topk + 1) * 2.0 ** -24
    half_ulp = 2.0 ** -9 if dtype == torch.bfloat16 else 2.0 ** -12
    bound = bound + (want.abs() + bound) * 2 * half_ulp + 1e-7
    assert ((reduce_topk(x, topk, w).double() - want).abs() <= bound).all()
    leaf = x.clone().requires_grad_()
    out = reduce_topk(leaf, topk, w)
    assert out.requires_grad and ((out.detach().double() - want).abs() <= bound).all()
    shifted = torch.empty(x.numel() + 1, device="cuda", dtype=dtype)[1:].view_as(x).copy_(x)  # no 16-byte alignment
    assert ((reduce_topk(shifted, topk, w).double() - want).abs() <= bound).all()


@pytest.mark.parametrize("T,topk,E,bm,segments,ranks", [(1, 1, 1, 128, 1, 1), (128, 8, 128, 128, 1, 1), (1025, 1, 7, 16, 1, 3), (2050, 2, 300, 1, 2, 1),
                                                        (8192, 8, 1024, 128, 1, 8), (8192, 8, 8, 128, 128, 1), (65537, 1, 128, 128, 1, 1)])
def test_moe_sort_all_outputs(T, topk, E, bm, segments, ranks):
    """One to eight CTAs, the edges between them and to the four-launch form, the largest number of groups, ids that are skipped,
    tiles with rows of several ranks: every output against a stable sort on the CPU."""
    import numpy as np
    from triton_distributed_b200.kernels.nvidia import create_sort_plan, moe_sort
    rng = np.random.default_rng(16)
    n = T * topk
    ids = rng.integers(-1, E + 1, (T, topk)).astype(np.int32)   # -1 and E count for nothing
    plan = create_sort_plan(n, topk, E, bm, segments, with_positions=True)
    per_rank = (T + ranks - 1) // ranks
    for _ in range(2):
        moe_sort(torch.from_numpy(ids).cuda(), plan, tokens_per_rank=per_rank)
    flat, seg = ids.reshape(-1), np.arange(n) // (n // segments)
    keep = (flat >= 0) & (flat < E)
    group = np.where(keep, seg * E + flat, -1)
    count = np.bincount(group[keep], minlength=segments * E)
    padded = -(-count // bm) * bm
    first = np.concatenate([[0], np.cumsum(padded)])
    order = np.argsort(group, kind="stable")[n - keep.sum():]
    pos = first[group[order]] + np.arange(len(order)) - (np.cumsum(count) - count)[group[order]]
    rows = np.full(first[-1], n)
    rows[pos] = order
    got = {k: getattr(plan, k).cpu().numpy() for k in ("sorted_ids", "tile_expert", "tile_seg_start", "tile_seg_end", "group_count", "totals", "pair_pos")}
    tiles = first[-1] // bm
    assert np.array_equal(got["group_count"], count) and list(got["totals"][:2]) == [first[-1], tiles]
    assert np.array_equal(got["totals"][2:], first[E::E] // bm)
    assert np.array_equal(got["sorted_ids"][:first[-1]], rows) and np.array_equal(got["pair_pos"][order], pos)
    tile_group = np.repeat(np.arange(segments * E), padded // bm)
    assert np.array_equal(got["tile_expert"][:tiles], tile_group % E)
    source = rows.reshape(tiles, bm) // topk // per_rank
    real = rows.reshape(tiles, bm) < n
    low, high = np.where(real, source, 1 << 30).min(1), np.where(real, source, -1).max(1)
    if segments > 1:
        low = high = tile_group // E
    assert np.array_equal(got["tile_seg_start"][:tiles], low) and np.array_equal(got["tile_seg_end"][:tiles], high)
    assert int(plan.status[0]) == 0


@pytest.mark.parametrize("T,topk,E,N,K", [(1030, 8, 6, 1320, 128), (500, 4, 9, 1536, 640), (2, 3, 5, 520, 384), (700, 1, 1, 136, 1152)])
def test_grouped_gemm_fp8_tile_widths(T, topk, E, N, K):
    """Wide tiles whose second half lies behind N or holds eight columns, one and several k-blocks, more tiles than SMs, and the few
    pairs that stay on narrow tiles. Error of the oracle's fp32 sum in another order plus one rounding to bf16."""
    from triton_distributed_b200 import ref
    from triton_distributed_b200.kernels.nvidia import grouped_gemm_fp8, quantize_fp8_rows, quantize_fp8_weight_blocks
    torch.manual_seed(17)
    a8, sa = quantize_fp8_rows(torch.randn(T, K, device="cuda") * torch.rand(T, 1, device="cuda") * 4)
    w8, sw = quantize_fp8_weight_blocks(torch.randn(E, N, K, device="cuda") * K ** -0.5)
    ids = torch.stack([torch.randperm(E)[:topk] if topk <= E else torch.randint(0, E, (topk,)) for _ in range(T)]).to(torch.int32).cuda()
    out = grouped_gemm_fp8(a8, sa, w8, sw, ids)
    want = ref.grouped_gemm_fp8_ref(a8.repeat_interleave(topk, 0), sa.repeat_interleave(topk, 0), w8, sw, ids.reshape(-1).long())
    torch.testing.assert_close(out.float(), want, rtol=2.0 ** -8, atol=K * 2.0 ** -22)


@pytest.mark.parametrize("T,topk,E,inter,K", [(1, 2, 4, 64, 128), (300, 4, 16, 768, 512), (1024, 8, 32, 200, 1032), (96, 2, 3, 1000, 64)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_gated_grouped_gemm(T, topk, E, inter, K, dtype):
    """Gate, up and product in one kernel against the per-expert products in fp32: widths that are no multiple of a tile's half, few
    pairs and many. Error: fp32 sums in another order, then one rounding to 16 bits."""
    from triton_distributed_b200 import ref
    from triton_distributed_b200.kernels.nvidia import create_sort_plan, moe_sort
    from triton_distributed_b200.kernels.nvidia.allgather_group_gemm import grouped_gemm_planned
    torch.manual_seed(18)
    a = torch.randn(T, K, device="cuda", dtype=dtype)
    w = torch.randn(E, 2 * inter, K, device="cuda", dtype=dtype) * K ** -0.5
    ids = torch.stack([torch.randperm(E)[:topk] for _ in range(T)]).to(torch.int32).cuda()
    plan = moe_sort(ids, create_sort_plan(T * topk, topk, E, 128, 1))
    out = grouped_gemm_planned(a, w, plan, topk, gated=True)
    gate, up = ref.grouped_gemm_ref(a.repeat_interleave(topk, 0), w, ids.reshape(-1).long()).double().chunk(2, dim=1)
    want = gate * torch.sigmoid(gate) * up
    # an fp32 sum of K products is off by about sqrt(K) * 2^-24 of their norm (one here); gate and up each carry that error
    torch.testing.assert_close(out.double(), want, rtol=2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -10, atol=K * 2.0 ** -20)


def test_plan_before_its_first_sort():
    """A new plan holds no pairs and no tiles, whatever the memory held before."""
    from triton_distributed_b200.kernels.nvidia import create_sort_plan
    shapes = [(24, 3, 8, 128, 1), (4096, 8, 64, 128, 4)]
    for args in shapes:
        plan = create_sort_plan(*args)
        whole = plan.sorted_ids._base if plan.sorted_ids._base is not None else plan.sorted_ids
        junk = [torch.full_like(whole, 77) for _ in range(4)]
        del plan, whole, junk
        plan = create_sort_plan(*args)
        assert int(plan.totals.abs().sum()) == 0 and int(plan.group_count.abs().sum()) == 0 and int(plan.status.abs().sum()) == 0


def test_expired_waits_are_reported(monkeypatch):
    """The fp8 grouped GEMM and the 32-bit GEMM get the status word that ``check_pipeline_status`` reads and clears."""
    from triton_distributed_b200 import _lib, ops
    from triton_distributed_b200.kernels.nvidia import quantize_fp8_rows, quantize_fp8_weight_blocks
    from triton_distributed_b200.kernels.nvidia.grouped_gemm_fp8 import grouped_gemm_fp8
    seen, call = {}, _lib.call
    monkeypatch.setattr(_lib, "call", lambda name, *args: (seen.update({name: args}), call(name, *args)))
    x = torch.randn(9, 256, device="cuda")
    ops.gemm_f32(x, x)
    ids = torch.zeros(9, 1, dtype=torch.int32, device="cuda")
    grouped_gemm_fp8(*quantize_fp8_rows(x), *quantize_fp8_weight_blocks(torch.randn(2, 128, 256, device="cuda")), ids)
    word = ops._pipeline_status(x.device)
    for name in ("b200_gemm_f32_checked", "b200_grouped_gemm_fp8"):
        assert seen[name][-2].value == word.data_ptr()
    ops.check_pipeline_status()
    word.fill_(3)
    with pytest.raises(RuntimeError):
        ops.check_pipeline_status()
    ops.check_pipeline_status()


@pytest.mark.parametrize("T,I", [(3, 128), (30, 256), (700, 2176), (500, 4224), (9, 1920)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_silu_mul_fp8_bytes(T, I, dtype):
    """Gates of 32, whose silu is 32, make the products exact: scales and bytes are those of IEEE divisions, ties included. Rows in
    more than one block of CTAs, more rows than CTAs, and scales from 2^-30 on."""
    from triton_distributed_b200 import ops
    g = torch.Generator().manual_seed(21)
    u = torch.randn(T, I // 128, 128, generator=g)
    # a block's largest value is 448 s and others are s times values halfway between two bytes
    s = torch.tensor([1.0, 3.0, 5.0, 7.0])[torch.randint(0, 4, (T, I // 128, 1), generator=g)] / 32
    odd = torch.randint(0, 8, (T, I // 128, 64), generator=g) * 2 + 17
    u[:, :, :64] = s * odd / 16 * 2.0 ** torch.randint(-4, 8, odd.shape, generator=g)
    u[:, :, 64:127] = u[:, :, 64:127].to(dtype).float().clamp(-10, 10) * s
    u[:, :, 127:] = 448 * s
    u[T // 2] *= 2.0 ** (-30 if dtype == torch.bfloat16 else -5)
    u = u.view(T, I).to(dtype)
    q, scale = ops.silu_mul_fp8(torch.cat([torch.full_like(u, 32.0), u], dim=1).cuda())
    blocks = (32 * u.float()).view(T, I // 128, 128)
    want = blocks.abs().amax(2) / 448
    assert torch.equal(scale.cpu(), want)
    assert torch.equal(q.cpu().view(torch.uint8), (blocks / want[:, :, None]).view(T, I).to(torch.float8_e4m3fn).view(torch.uint8))
