"""Model-level GPU checks on one device: native forward modes against the torch-mode model on the same
weights, the engine with and without CUDA graph, and the safetensors round trip."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _mk(dist1, name="tiny-qwen3-gqa", **kw):
    from triton_distributed_b200.models import ModelConfig, Qwen3
    cfg = ModelConfig(model_name=name, max_length=256, rank=0, world_size=1, **kw)
    return cfg, Qwen3(cfg, dist1)


def test_native_forward_matches_torch_mode(dist1):
    from triton_distributed_b200.models import KV_Cache
    cfg, model = _mk(dist1)
    a = model.arch
    ids = torch.randint(0, a.vocab_size, (3, 40), device="cuda")
    pos = torch.arange(40, device="cuda")[None, :].expand(3, 40).contiguous()
    outs = {}
    for mode in ("torch", "triton_dist_AR", "triton_dist"):
        kv = KV_Cache(a.num_hidden_layers, 3, 256, a.num_key_value_heads, a.head_dim, torch.bfloat16, 1)
        if mode == "triton_dist":
            model.init_triton_dist_ctx(3 * 40)
        if mode == "triton_dist_AR":
            model.init_triton_dist_AR_ctx(3 * 40)
        model.set_fwd(mode)
        logits = model.inference(ids, pos, kv)
        # one decode step on top of the prefilled cache
        nxt = logits.argmax(-1)
        pos1 = torch.full((3, 1), 40, device="cuda", dtype=torch.int64)
        logits1 = model.inference(nxt, pos1, kv)
        torch.cuda.synchronize()
        outs[mode] = (torch.softmax(logits, -1), torch.softmax(logits1, -1), nxt)
    for mode in ("triton_dist_AR", "triton_dist"):
        torch.testing.assert_close(outs[mode][0], outs["torch"][0], rtol=2e-2, atol=2e-2)
        if torch.equal(outs[mode][2], outs["torch"][2]):
            torch.testing.assert_close(outs[mode][1], outs["torch"][1], rtol=2e-2, atol=2e-2)
    model.finalize()


@pytest.mark.parametrize("bsz,seqlen", [(9, 1), (16, 1), (1, 5), (2, 8), (1, 16)])
def test_steps_of_few_tokens_match_separate_norms(dist1, bsz, seqlen):
    """Up to 16 tokens of a bf16 model on one GPU have norms and residual adds inside the projections; the path with separate
    kernels is the other side, behind a cached prompt."""
    cfg, model = _mk(dist1)
    model.set_fwd("triton_dist_AR")
    model.init_triton_dist_AR_ctx(64)
    torch.manual_seed(12)
    ids = torch.randint(0, model.arch.vocab_size, (bsz, 20 + seqlen), device="cuda")
    pos = torch.arange(20 + seqlen, device="cuda")[None].repeat(bsz, 1)
    outs, paths = {}, []
    rows = model._step_rows
    for few in (True, False):
        model._step_rows = lambda *a: (paths.append(few), rows(*a))[1]
        if not few:
            model._few_tokens = lambda tokens: False
        for only_hidden in (False, True):
            kv = model.make_cache(bsz)
            model.inference(ids[:, :20], pos[:, :20], kv)
            outs[few, only_hidden] = model.inference(ids[:, 20:].contiguous(), pos[:, 20:].contiguous(), kv, wo_lm_head=only_hidden).double()
    assert paths == [True, True]
    for only_hidden in (False, True):
        got, want = outs[True, only_hidden], outs[False, only_hidden]
        assert got.shape == want.shape
        # three layers of four bf16 roundings each in other places: a few times 2^-9 of the norm
        assert (got - want).norm() <= 0.02 * want.norm()
    model.finalize()


def test_which_steps_have_norms_inside_the_projections(dist1):
    _, model = _mk(dist1)
    assert model._few_tokens(1) and model._few_tokens(16) and not model._few_tokens(17)
    model.dtype = torch.float16     # may not hold the product of the residual stream and a gain
    assert not model._few_tokens(1)
    _, moe = _mk(dist1, "tiny-qwen3-moe")
    assert not moe._few_tokens(1)


def test_engine_graph_equals_eager_and_torch(dist1):
    from triton_distributed_b200.models import Engine
    cfg, model = _mk(dist1)
    ids = torch.randint(0, model.arch.vocab_size, (2, 24), device="cuda")
    res = {}
    for name, backend, no_graph in (("graph", "triton_dist_AR", False), ("eager", "triton_dist_AR", True), ("torch", "torch", True)):
        eng = Engine(cfg, temperature=0.0, group=dist1, model=model)
        eng.backend, eng.no_graph = backend, no_graph
        res[name] = eng.serve(ids, gen_len=6)
    assert torch.equal(res["graph"], res["eager"])
    # greedy decoding of a random-init model can flip on near-ties; the first tokens must agree
    assert torch.equal(res["graph"][:, :26], res["torch"][:, :26])
    model.finalize()


def test_safetensors_roundtrip_matches_random_source(dist1, tmp_path):
    from triton_distributed_b200.models import ARCHS, KV_Cache, ModelConfig, Qwen3
    from triton_distributed_b200.models.weights import write_random_checkpoint
    arch = ARCHS["tiny-qwen3"]
    write_random_checkpoint(str(tmp_path), arch, torch.bfloat16, seed=0, max_shard_bytes=4 << 20)
    assert len([f for f in tmp_path.iterdir() if f.suffix == ".safetensors"]) > 1
    m_ckpt = Qwen3(ModelConfig(model_name="from-disk", checkpoint_dir=str(tmp_path), max_length=128, rank=0, world_size=1), dist1)
    m_rand = Qwen3(ModelConfig(model_name="tiny-qwen3", max_length=128, rank=0, world_size=1, seed=0), dist1)
    assert torch.equal(m_ckpt.layers[1].attn.wqkv, m_rand.layers[1].attn.wqkv)
    assert torch.equal(m_ckpt.lm_head, m_rand.lm_head)
    ids = torch.randint(0, arch.vocab_size, (1, 8), device="cuda")
    pos = torch.arange(8, device="cuda")[None, :]
    outs = []
    for m in (m_ckpt, m_rand):
        kv = KV_Cache(arch.num_hidden_layers, 1, 128, arch.num_key_value_heads, arch.head_dim, torch.bfloat16, 1)
        outs.append(m.inference(ids, pos, kv))
    assert torch.equal(outs[0], outs[1])


def test_moe_model_native_modes_match_torch(dist1):
    from triton_distributed_b200.models import AutoLLM, KV_Cache, ModelConfig
    cfg = ModelConfig(model_name="tiny-qwen3-moe", max_length=128, rank=0, world_size=1)
    model = AutoLLM.from_pretrained(cfg, dist1)
    a = model.arch
    ids = torch.randint(0, a.vocab_size, (2, 24), device="cuda")
    pos = torch.arange(24, device="cuda")[None, :].expand(2, 24).contiguous()
    outs = {}
    for mode in ("torch", "triton_dist_AR", "triton_dist"):
        kv = KV_Cache(a.num_hidden_layers, 2, 128, a.num_key_value_heads, a.head_dim, torch.bfloat16, 1)
        if mode == "triton_dist":
            model.init_triton_dist_ctx(2 * 24)
        if mode == "triton_dist_AR":
            model.init_triton_dist_AR_ctx(2 * 24)
        model.set_fwd(mode)
        outs[mode] = torch.softmax(model.inference(ids, pos, kv), -1)
        torch.cuda.synchronize()
    for mode in ("triton_dist_AR", "triton_dist"):
        torch.testing.assert_close(outs[mode], outs["torch"], rtol=3e-2, atol=3e-2)
    model.finalize()


def test_attention_only_reads_the_step_tables(dist1):
    """One dictionary of step tables, refilled by its owner for prompts of another length: nothing of the first call is left in it."""
    from triton_distributed_b200 import ops
    from triton_distributed_b200.layers.nvidia import TP_Attn, _set_cos_sin_cache
    from triton_distributed_b200.models import KV_Cache
    torch.manual_seed(6)
    att = TP_Attn(0, 1)
    rnd = lambda *shape: torch.randn(shape, device="cuda", dtype=torch.bfloat16)
    att._init_parameters(q=rnd(512, 256), k=rnd(256, 256), v=rnd(256, 256), o=rnd(256, 512), q_norm=rnd(128), k_norm=rnd(128), num_heads=4, num_kv_heads=2)
    cos = _set_cos_sin_cache(10000.0 ** (-torch.arange(64, device="cuda") / 64), 256)
    step = {}
    for seqlen in (40, 70, 9):
        kv, own = (KV_Cache(1, 2, 128, 2, 128, torch.bfloat16, 1) for _ in range(2))
        pos, qkv = torch.arange(seqlen, device="cuda")[None].repeat(2, 1), rnd(2 * seqlen, 1024)
        step.update(ops.step_tables(pos, kv.blocks_per_seq * kv.page_size))
        got = att._attn_native(qkv, pos, cos, kv, 0, 2, seqlen, step)
        assert torch.equal(got, att._attn_native(qkv, pos, cos, own, 0, 2, seqlen))
