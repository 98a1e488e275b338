"""Kernels that start under one another (programmatic dependent launch): what a launch in front computes is complete before it is
read, whichever operand it is and however many launches lie in between."""
import pytest
import torch

pytestmark = pytest.mark.gpu

BF, F32 = torch.bfloat16, torch.float32
LONG = 32768   # k of the producing GEMMs: a few tiles that take a hundred microseconds while the other SMs are free


def _rnd(*shape, dtype=BF):
    return torch.randn(shape, device="cuda").to(dtype)


def _linear(rows):   # at most 16 rows and more run on kernels of their own
    def make(p):
        from triton_distributed_b200 import ops
        x = _rnd(rows, 256)
        return lambda: ops.linear(x, p)
    return make


def _swiglu(rows):
    def make(p):
        from triton_distributed_b200 import ops
        x = _rnd(rows, 256)
        return lambda: ops.gemm_skinny(x, p, swiglu=True)
    return make


def _normed(p):
    from triton_distributed_b200 import ops
    x, w = _rnd(5, 2048), _rnd(512, 2048)
    return lambda: ops.gemm_rows(x, w, gamma=p.view(-1), eps=1e-6)


def _groups(p):
    from triton_distributed_b200 import ops
    x = _rnd(5, 2, 256)
    return lambda: ops.linear_groups(x, p, [128, 384])


def _heads(p):
    from triton_distributed_b200 import ops
    x = _rnd(5, 4, 256)
    return lambda: ops.head_linear(x, p.view(4, 128, 256))


def _tanh(p):
    from triton_distributed_b200 import ops
    x = _rnd(5, 256)
    return lambda: ops.tanh_linear(x, p)


def _rmsnorm(p):
    from triton_distributed_b200 import ops
    x = _rnd(300, 2048)
    return lambda: ops.rmsnorm(x, p.view(-1), 1e-6)


def _rope(p):
    from triton_distributed_b200 import ops
    qkv, pos, cs = _rnd(9, 6 * 128), torch.arange(9, device="cuda", dtype=torch.int32), _rnd(16, 128, dtype=F32)
    k, v = _rnd(9, 2, 128), _rnd(9, 2, 128)
    return lambda: (ops.qk_norm_rope(qkv, pos, cs, 2, 2, k, v, None, p[0, :128], p[0, 128:]), k)


def _embed(p):
    from triton_distributed_b200 import ops
    ids, table = torch.arange(7, device="cuda"), _rnd(10, 2048)
    return lambda: ops.embed_norm(ids, table, 1.0, 2048, p.view(-1), None, 1e-6, True)[1]


def _residual(p):
    from triton_distributed_b200 import ops
    x, a = _rnd(300, 2048, dtype=F32), _rnd(300, 2048)
    return lambda: ops.residual_norm(x, 2048, 1.0, a, gain=p.view(-1), bias=p.view(-1), eps=1e-6)


def _post(p):
    from triton_distributed_b200 import ops
    x, a, g = _rnd(3, 2048, dtype=F32), _rnd(3, 2048), _rnd(2048)
    return lambda: ops.residual_post(x, 2048, 1.0, a, g, post_eps=1e-6, gain=p.view(-1), eps=1e-6)


def _mix(p):
    from triton_distributed_b200 import ops
    h, last = _rnd(40, 512), _rnd(2, 512)
    return lambda: ops.token_mix(h, p, last)


def _conv(p):
    from triton_distributed_b200 import ops
    x, last = _rnd(40, 512), _rnd(2, 3, 512)
    return lambda: ops.short_conv(x, p, last)


def _wkv(tokens):
    def make(p):
        from triton_distributed_b200 import ops
        rows, c, state = [_rnd(2 * tokens, 256) for _ in range(5)], torch.ones(256, device="cuda"), torch.zeros(2, 4, 64, 64, device="cuda")
        return lambda: ops.wkv(*rows, p[0], c, p[1], state, 64, 64, 1e-6)
    return make


def _delta(p):
    from triton_distributed_b200 import ops
    rows, ab, c, state = [_rnd(40, 256) for _ in range(4)], _rnd(40, 8), torch.ones(64, device="cuda"), torch.zeros(2, 4, 64, 64, device="cuda")
    return lambda: ops.gated_delta(*rows[:3], ab[:, :4], ab[:, 4:], rows[3], p[0], p[1], c, state, 64, 64, 1e-6)


def _sink(p):
    from triton_distributed_b200 import ops
    q, cache = _rnd(2, 8, 128), _rnd(8, 64, 128)
    lens, table = torch.tensor([200, 70], dtype=torch.int32, device="cuda"), torch.arange(8, dtype=torch.int32, device="cuda").view(2, 4)
    return lambda: ops.latent_attention(q, cache, lens, table, 1, 0.05, p.view(-1), 3, 16)


CONSUMERS = {"linear": (_linear(5), (512, 256), BF), "swiglu": (_swiglu(5), (512, 256), BF), "linear, 24 rows": (_linear(24), (512, 256), BF),
             "swiglu, 24 rows": (_swiglu(24), (512, 256), BF), "normed": (_normed, (1, 2048), BF), "groups": (_groups, (512, 256), BF),
             "head_linear": (_heads, (512, 256), BF), "tanh_linear": (_tanh, (512, 256), BF), "rmsnorm": (_rmsnorm, (1, 2048), BF),
             "qk_norm_rope": (_rope, (1, 256), BF), "embed_norm": (_embed, (1, 2048), BF), "residual_norm": (_residual, (1, 2048), BF),
             "residual_post": (_post, (1, 2048), BF), "token_mix": (_mix, (3, 512), BF), "short_conv": (_conv, (4, 512), F32),
             "wkv": (_wkv(20), (2, 256), F32), "wkv, one token": (_wkv(1), (2, 256), F32), "gated_delta": (_delta, (2, 4), F32),
             "sink": (_sink, (1, 8), F32)}


@pytest.mark.parametrize("between", [0, 2])
@pytest.mark.parametrize("name", CONSUMERS)
def test_parameters_computed_by_launches_in_front(name, between):
    """The parameter is a GEMM's result; `between` small kernels that let their successors start early lie between the two. A read
    in front of the wait would see the 1000 that stood there."""
    from triton_distributed_b200 import ops
    make, shape, dtype = CONSUMERS[name]
    torch.manual_seed(3)
    a, b = _rnd(shape[0], LONG, dtype=dtype), _rnd(shape[1], LONG, dtype=dtype) * LONG ** -0.5
    gemm = ops.gemm if dtype == BF else ops.gemm_f32
    param, small = torch.empty(shape, dtype=dtype, device="cuda"), _rnd(4, 512)
    exact = a.double() @ b.double().t()
    for i in range(4):
        torch.manual_seed(5 + i)
        late = make(param)
        torch.manual_seed(5 + i)
        done = make(exact.to(dtype))
        want = done()
        param.fill_(1000.0)
        torch.cuda.synchronize()
        gemm(a, b, out=param)
        for _ in range(between):
            ops.silu_mul(small)
        got = late()
        torch.cuda.synchronize()
        # both sides round the same sums to 16 bits, in another order: a unit in the last place of the parameter and of the result
        for g, w in zip(got if isinstance(got, tuple) else (got,), want if isinstance(want, tuple) else (want,)):
            assert (g.double() - w.double()).norm() <= 0.01 * w.double().norm(), (i, name)


def test_expanded_latents_read_rows_just_written():
    """Rows of the latent cache are the second operand of the values' expansion; between their writer and that GEMM lies the tiled
    GEMM of the keys, which lets its successor start early."""
    from triton_distributed_b200 import ops
    from triton_distributed_b200.layers.nvidia.latent_attn import LatentAttention
    from triton_distributed_b200.models.kv_cache import LatentCache
    torch.manual_seed(4)
    H, d, r, S = 2, 64, 128, 520
    att = LatentAttention()
    att._init_parameters(uk=_rnd(H * d, r) * r ** -0.5, uv=_rnd(H * d, r) * r ** -0.5, o=_rnd(256, H * d), latent_norm=_rnd(r), sink=torch.zeros(H, device="cuda"),
                         heads=H, dim=d, vdim=d, kv_rank=r, scale=d ** -0.5, eps=1e-6, width_pad=256)
    cache = LatentCache([r], 1, 576)
    pos = torch.arange(S, device="cuda")[None]
    slots, lens = cache.slots(pos), torch.tensor([S], dtype=torch.int32, device="cuda")
    q, a, b = _rnd(S, H * d), _rnd(S, LONG // 2), _rnd(r, LONG // 2) * (LONG // 2) ** -0.5
    cu = {"cu_q": torch.tensor([0, S], dtype=torch.int32, device="cuda"), "cu_k": torch.tensor([0, S], dtype=torch.int32, device="cuda")}
    latent = torch.empty(S, r, dtype=BF, device="cuda")

    def attend(sync):
        cache.c_cache[0].fill_(100.0)
        torch.cuda.synchronize()
        ops.gemm(a, b, out=latent)
        ops.latent_prep(latent, att.latent_norm, cache.layer(0), slots, r, 1e-6)
        if sync:
            torch.cuda.synchronize()
        return att.attend(q, cache, 0, {"bsz": 1, "seqlen": S, "kv_len": S, "kv_lens": lens, **cu})

    want = attend(True).double()
    for _ in range(5):
        got = attend(False).double()
        torch.cuda.synchronize()
        assert (got - want).norm() <= 1e-3 * want.norm()
