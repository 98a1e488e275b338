"""What is timed: the work that programs on top of this framework have it do on one GPU, through its public entry points.

Every kind of case is a class below: what a serving program holds (``prepare``), one call (``run``), the call's value in 64 bits
(``exact``), the bytes and operations that it cannot do without (``work``) and the range its sizes come from (``draw``). Sizes are
those of the configurations in ``triton_distributed_b200/models/config.py``, of the benchmarks and of the tests.
"""
import functools
import math

import torch
import torch.nn.functional as F

from triton_distributed_b200 import ops
from triton_distributed_b200.kernels.nvidia import gqa_fwd_batch_decode
from triton_distributed_b200.kernels.nvidia.grouped_gemm_fp8 import grouped_gemm_fp8, quantize_fp8_rows, quantize_fp8_weight_blocks
from triton_distributed_b200.kernels.nvidia.moe_utils import reduce_topk
from triton_distributed_b200.layers.nvidia import TP_MLP, TP_MoE
from triton_distributed_b200.models import Engine, ModelConfig
from triton_distributed_b200.models.config import ARCHS
from triton_distributed_b200.models.qwen import Qwen3

DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}
HEAD = 128  # head size of the grouped-query attention kernels


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _normal(g, shape, std=1.0, dtype=torch.bfloat16, mean=0.0):
    """Drawn piece by piece: a large tensor needs no fp32 copy of itself."""
    out = torch.empty(shape, dtype=dtype, device="cuda")
    return out.normal_(mean, std, generator=g)


def _log_int(rng, low, high):
    """A whole number from low to high, even over the logarithm."""
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high))))))


def _silu(x):
    return x / (1 + torch.exp(-x))


def _rms(x, gain, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * gain


def _attend(q, k, v, scale, first):
    """q [S, H, D] at positions first.., k and v [N, G, D] in 64 bits: causal attention, in portions of the queries."""
    S, H, _ = q.shape
    N, G, _ = k.shape
    out = torch.empty(S, H, v.shape[2], dtype=q.dtype, device=q.device)
    key = torch.arange(N, device=q.device)
    for g in range(G):
        heads = slice(g * (H // G), (g + 1) * (H // G))
        for a in range(0, S, 1024):
            rows = torch.arange(a, min(S, a + 1024), device=q.device)
            last = min(N, first + int(rows[-1]) + 1)
            s = torch.einsum("shd,nd->hsn", q[rows, heads], k[:last, g]) * scale
            s.masked_fill_(key[None, None, :last] > (first + rows)[None, :, None], -math.inf)
            out[rows, heads] = torch.einsum("hsn,nd->shd", torch.softmax(s, -1), v[:last, g])
    return out


# ---- whole decoder steps ----------------------------------------------------------------------
class _Weights:
    """Random weights under the checkpoint's names, drawn once; every projection keeps the scale of its input."""

    def __init__(self, arch):
        self.arch, self.g, self.held = arch, _generator(1), {}

    def has(self, name):
        return True

    def get(self, name, rows=None, cols=None):
        if name not in self.held:
            a = self.arch
            q, kv = a.num_attention_heads * a.head_dim, a.num_key_value_heads * a.head_dim
            shape = {"embed_tokens": (a.vocab_size, a.hidden_size), "lm_head": (a.vocab_size, a.hidden_size), "q_proj": (q, a.hidden_size),
                     "k_proj": (kv, a.hidden_size), "v_proj": (kv, a.hidden_size), "o_proj": (a.hidden_size, q),
                     "gate_proj": (a.intermediate_size, a.hidden_size), "up_proj": (a.intermediate_size, a.hidden_size),
                     "down_proj": (a.hidden_size, a.intermediate_size), "q_norm": (a.head_dim,), "k_norm": (a.head_dim,)}.get(
                         name.split(".")[-2], (a.hidden_size,))
            if len(shape) == 1:
                self.held[name] = _normal(self.g, shape, 0.1, mean=1.0)
            else:
                self.held[name] = _normal(self.g, shape, 1.0 if "embed" in name else shape[1] ** -0.5)
        t = self.held[name]
        t = t[rows] if rows is not None else t
        return t[:, cols] if cols is not None else t


class Decoder:
    """``Engine.extend``: the next tokens of every sequence in, logits out. One token per sequence replays the captured decode
    step, several are a prompt (or a portion of one, behind a cached prefix)."""

    # layers of the model that are built: enough for the layers to outweigh the head
    MODELS = {"Qwen/Qwen3-8B": 4, "Qwen3-32B-tp8-shard": 8}
    MAX_LENGTH = 16384 + 256

    @staticmethod
    @functools.lru_cache(maxsize=1)  # a server loads its model once
    def model(name):
        cfg = ModelConfig(name, max_length=Decoder.MAX_LENGTH, rank=0, world_size=1, num_layers_override=Decoder.MODELS[name])
        weights = _Weights(cfg.arch())
        return Qwen3(cfg, source=weights), weights

    @staticmethod
    def inputs(case, seed):
        model, weights = Decoder.model(case["model"])
        g = _generator(seed)
        ids = torch.randint(0, model.arch.vocab_size, (case["batch"], case["tokens"]), device="cuda", generator=g)
        return model, weights, ids, g

    @staticmethod
    def prepare(case, seed):
        model, _, ids, g = Decoder.inputs(case, seed)
        length = (case["cached"] + case["tokens"] + 255) // 256 * 256
        cfg = ModelConfig(case["model"], max_length=length, rank=0, world_size=1, num_layers_override=Decoder.MODELS[case["model"]])
        engine = Engine(cfg, temperature=0.0, model=model)
        engine.start(case["batch"])
        if case["cached"]:  # what earlier steps left: normed keys, values of the projections' scale
            engine.kv_cache.k_cache.normal_(0.0, 1.0, generator=g)
            engine.kv_cache.v_cache.normal_(0.0, 1.0, generator=g)
            engine.kv_cache.inc_offset(case["cached"])
            engine.length = case["cached"]
        if case["tokens"] == 1:
            engine.prepare_decode(ids)
        return {"engine": engine, "ids": ids}

    @staticmethod
    def run(state):
        engine, ids = state["engine"], state["ids"]
        first, n = engine.length, ids.shape[1]
        logits = engine.extend(ids)
        cache = engine.kv_cache
        cache.inc_offset(-n)  # the tokens are taken back, as after a rejected draft: the next pass starts from the same state
        engine.length = first
        layers, _, _, heads, dim = cache.k_cache.shape
        rows = (layers, cache.batch_size, -1, heads, dim)
        return {"logits": logits, "k": cache.k_cache.view(rows)[:, :, first:first + n], "v": cache.v_cache.view(rows)[:, :, first:first + n]}

    @staticmethod
    def exact(case, seed):
        engine = Decoder.prepare(case, seed)["engine"] if case["cached"] else None
        model, weights, ids, _ = Decoder.inputs(case, seed)
        a, B, S, first, D = model.arch, case["batch"], case["tokens"], case["cached"], HEAD
        inv = 1.0 / a.rope_theta ** (torch.arange(0, D, 2, dtype=torch.float64, device="cuda") / D)
        angle = torch.arange(first, first + S, dtype=torch.float64, device="cuda")[:, None] * inv
        cos, sin = angle.cos()[None, :, None], angle.sin()[None, :, None]

        def rope(x):
            x1, x2 = x[..., :D // 2], x[..., D // 2:]
            return torch.cat([x1 * cos - x2 * sin, x2 * cos + x1 * sin], -1)

        x, eps = weights.get("model.embed_tokens.weight")[ids].double(), a.rms_norm_eps
        keys, values = [], []
        for i in range(Decoder.MODELS[case["model"]]):
            def w(name):
                return weights.get(f"model.layers.{i}.{name}.weight").double()
            h = _rms(x, w("input_layernorm"), eps)
            q = rope(_rms((h @ w("self_attn.q_proj").T).view(B, S, -1, D), w("self_attn.q_norm"), eps))
            k = rope(_rms((h @ w("self_attn.k_proj").T).view(B, S, -1, D), w("self_attn.k_norm"), eps))
            v = (h @ w("self_attn.v_proj").T).view(B, S, -1, D)
            o = torch.empty_like(q)
            for b in range(B):
                kb, vb = k[b], v[b]
                if engine is not None:
                    old = [c[i].view(B, -1, *c.shape[-2:])[b, :first].double() for c in (engine.kv_cache.k_cache, engine.kv_cache.v_cache)]
                    kb, vb = torch.cat([old[0], kb]), torch.cat([old[1], vb])
                o[b] = _attend(q[b], kb, vb, D ** -0.5, first)
            x = x + o.reshape(B, S, -1) @ w("self_attn.o_proj").T
            h = _rms(x, w("post_attention_layernorm"), eps)
            x = x + (_silu(h @ w("mlp.gate_proj").T) * (h @ w("mlp.up_proj").T)) @ w("mlp.down_proj").T
            keys.append(k), values.append(v)
        last = _rms(x[:, -1:], weights.get("model.norm.weight").double(), eps)
        return {"logits": last @ weights.get("lm_head.weight").double().T, "k": torch.stack(keys), "v": torch.stack(values)}

    @staticmethod
    def work(case):
        a, n = ARCHS[case["model"]], Decoder.MODELS[case["model"]]
        B, S, first = case["batch"], case["tokens"], case["cached"]
        q, kv, H = a.num_attention_heads * HEAD, a.num_key_value_heads * HEAD, a.hidden_size
        layer = H * (2 * q + 2 * kv) + 3 * H * a.intermediate_size
        pairs = B * (S * first + S * (S + 1) // 2)
        return {"bytes": 2 * (n * layer + a.vocab_size * H + B * S * H + n * B * 2 * kv * (first + S)) + 4 * B * a.vocab_size,
                "flops": 2 * n * layer * B * S + 2 * a.vocab_size * H * B + n * 4 * q * pairs}

    @staticmethod
    def tolerance(case):
        return {"rel": 0.02, "max": 0.3}

    @staticmethod
    def draw(rng):
        name = rng.choice(sorted(Decoder.MODELS))
        if rng.random() < 0.5:  # a step of a running batch
            batch = _log_int(rng, 1, 64)
            return {"model": name, "batch": batch, "tokens": 1, "cached": _log_int(rng, 64, min(8192, 65536 // batch))}
        total = _log_int(rng, 48, 12288)
        batch = _log_int(rng, 1, min(16, total // 16))
        tokens = total // batch
        cached = _log_int(rng, 64, 2048) if rng.random() < 0.3 else 0
        return {"model": name, "batch": batch, "tokens": tokens, "cached": cached}


# ---- attention --------------------------------------------------------------------------------
class PrefillAttention:
    """``ops.prefill_attention`` over a pack of sequences of different lengths (causal, keys and queries from one pass)."""

    HEADS = ((64, 8), (32, 8), (40, 8), (32, 4), (8, 1))

    @staticmethod
    def lengths(case):
        """The pack's lengths, between a half and one and a half of the mean."""
        n, mean = case["sequences"], case["mean"]
        return [max(1, mean // 2 + mean * i // max(1, n - 1)) if n > 1 else mean for i in range(n)]

    @staticmethod
    def prepare(case, seed):
        g, dtype, lens = _generator(seed), DTYPES[case["dtype"]], PrefillAttention.lengths(case)
        total, Hq, Hkv = sum(lens), case["heads"], case["kv_heads"]
        ends = torch.tensor([0] + lens).cumsum(0).to(device="cuda", dtype=torch.int32)
        gate = _normal(g, (total, Hq), 1.0, dtype) if case["gated"] else None
        return {"q": _normal(g, (total, Hq, HEAD), 1.0, dtype), "k": _normal(g, (total, Hkv, HEAD), 1.0, dtype),
                "v": _normal(g, (total, Hkv, HEAD), 1.0, dtype), "gate": gate, "ends": ends, "longest": max(lens)}

    @staticmethod
    def run(s):
        return ops.prefill_attention(s["q"], s["k"], s["v"], s["ends"], s["ends"], s["longest"], s["longest"], HEAD ** -0.5, True, gate=s["gate"])

    @staticmethod
    def exact(case, seed):
        s, at, parts = PrefillAttention.prepare(case, seed), 0, []
        for n in PrefillAttention.lengths(case):
            parts.append(_attend(*(s[t][at:at + n].double() for t in "qkv"), HEAD ** -0.5, 0))
            at += n
        out = torch.cat(parts)
        return out if s["gate"] is None else out * torch.sigmoid(s["gate"].double())[:, :, None]

    @staticmethod
    def work(case):
        lens = PrefillAttention.lengths(case)
        return {"bytes": 4 * HEAD * sum(lens) * (case["heads"] + case["kv_heads"]),
                "flops": 4 * HEAD * case["heads"] * sum(n * (n + 1) // 2 for n in lens)}

    @staticmethod
    def tolerance(case):
        return {"rel": 0.01, "max": 0.15}

    @staticmethod
    def draw(rng):
        heads, kv_heads = rng.choice(PrefillAttention.HEADS)
        total = _log_int(rng, 128, 16384)
        sequences = _log_int(rng, 1, min(16, total // 16))
        return {"sequences": sequences, "mean": total // sequences, "heads": heads, "kv_heads": kv_heads,
                "dtype": rng.choice(("bf16", "bf16", "f16")), "gated": rng.random() < 0.25}


class DecodeAttention:
    """``gqa_fwd_batch_decode``: one query token per sequence over a paged cache whose pages lie in no order."""

    @staticmethod
    def lengths(case):
        """Between three quarters of the longest sequence and all of it."""
        return [case["kv"] - case["kv"] * ((5 * i) % 8) // 32 for i in range(case["batch"])]

    @staticmethod
    def prepare(case, seed):
        g, dtype, page = _generator(seed), DTYPES[case["dtype"]], case["page"]
        B, Hq, Hkv, blocks = case["batch"], case["heads"], case["kv_heads"], -(-case["kv"] // page)
        table = torch.randperm(B * blocks, device="cuda", generator=g).to(torch.int32).view(B, blocks)
        return {"q": _normal(g, (B, Hq, HEAD), 1.0, dtype), "k": _normal(g, (B * blocks, page, Hkv, HEAD), 1.0, dtype),
                "v": _normal(g, (B * blocks, page, Hkv, HEAD), 1.0, dtype), "table": table, "longest": case["kv"], "workspace": {},
                "lens": torch.tensor(DecodeAttention.lengths(case), dtype=torch.int32, device="cuda")}

    @staticmethod
    def run(s):
        return gqa_fwd_batch_decode(s["q"], s["k"], s["v"], s["workspace"], None, s["lens"], s["table"], HEAD ** -0.5, max_kv_len=s["longest"])

    @staticmethod
    def exact(case, seed):
        s = DecodeAttention.prepare(case, seed)
        rows = []
        for b, n in enumerate(DecodeAttention.lengths(case)):
            k, v = (s[t][s["table"][b].long()].flatten(0, 1)[:n].double() for t in "kv")
            rows.append(_attend(s["q"][b:b + 1].double(), k, v, HEAD ** -0.5, n - 1))
        return torch.cat(rows)

    @staticmethod
    def work(case):
        tokens = sum(DecodeAttention.lengths(case))
        return {"bytes": 4 * HEAD * (tokens * case["kv_heads"] + case["batch"] * case["heads"]), "flops": 4 * HEAD * case["heads"] * tokens}

    @staticmethod
    def tolerance(case):
        return {"rel": 0.01, "max": 0.15}

    @staticmethod
    def draw(rng):
        heads, kv_heads = rng.choice(PrefillAttention.HEADS)
        batch = _log_int(rng, 1, 64)
        return {"batch": batch, "kv": _log_int(rng, 256, min(131072, 524288 // batch)), "heads": heads, "kv_heads": kv_heads,
                "page": rng.choice((64, 64, 16)), "dtype": rng.choice(("bf16", "bf16", "f16"))}


class LatentAttention:
    """``ops.latent_attention``: absorbed queries of one token per sequence over paged latents, with a sink logit per head."""

    RANK, PAGE, SCALE = 512, 64, 128 ** -0.5

    @staticmethod
    def lengths(case):
        return DecodeAttention.lengths(case)

    @staticmethod
    def prepare(case, seed):
        g, dtype, L = _generator(seed), DTYPES[case["dtype"]], LatentAttention
        B, H, blocks = case["batch"], case["heads"], -(-case["kv"] // L.PAGE)
        return {"q": _normal(g, (B, H, L.RANK), 0.5, dtype), "cache": _normal(g, (B * blocks, L.PAGE, L.RANK), 1.0, dtype),
                "table": torch.arange(B * blocks, dtype=torch.int32, device="cuda").view(B, blocks),
                "lens": torch.tensor(L.lengths(case), dtype=torch.int32, device="cuda"), "longest": case["kv"],
                "sink": _normal(g, (H,), 1.0, torch.float32)}

    @staticmethod
    def run(s):
        B, H = s["q"].shape[:2]
        splits, rows = ops.choose_latent_splits(B, H, s["longest"])
        return ops.latent_attention(s["q"], s["cache"], s["lens"], s["table"], 1, LatentAttention.SCALE, s["sink"], splits, rows)

    @staticmethod
    def exact(case, seed):
        s, rows = LatentAttention.prepare(case, seed), []
        for b, n in enumerate(LatentAttention.lengths(case)):
            c = s["cache"][s["table"][b].long()].flatten(0, 1)[:n].double()
            logits = torch.cat([s["q"][b].double() @ c.T * LatentAttention.SCALE, s["sink"].double()[:, None]], 1)
            rows.append(torch.softmax(logits, -1)[:, :-1] @ c)
        return torch.stack(rows)

    @staticmethod
    def work(case):
        tokens, L = sum(LatentAttention.lengths(case)), LatentAttention
        return {"bytes": 2 * L.RANK * (tokens + 2 * case["batch"] * case["heads"]), "flops": 4 * L.RANK * case["heads"] * tokens}

    @staticmethod
    def tolerance(case):
        return {"rel": 0.01, "max": 0.15}

    @staticmethod
    def draw(rng):
        batch = _log_int(rng, 1, 32)
        return {"batch": batch, "kv": _log_int(rng, 64, min(32768, 262144 // batch)), "heads": rng.choice((16, 32, 64)),
                "dtype": rng.choice(("bf16", "bf16", "f16"))}


# ---- mixture of experts -----------------------------------------------------------------------
# one layer: hidden size, intermediate size of an expert on this GPU; 128 experts, 8 per token
MOE = {"Qwen/Qwen3-30B-A3B": (2048, 768), "Qwen/Qwen3-235B-A22B, one of eight ranks": (4096, 192)}
EXPERTS, TOP = 128, 8


def _expert_work(case, weight_bytes):
    """An expert that gets a token is read; tokens spread over the experts as independent choices."""
    H, inter = MOE[case["layer"]]
    T = case["tokens"]
    used = EXPERTS * (1 - (1 - TOP / EXPERTS) ** T)
    return {"bytes": weight_bytes * 3 * H * inter * used + 4 * T * H, "flops": 6 * H * inter * TOP * T}


def _experts(x, ids, w, gate_up, down, quantize=lambda a: a):
    """The chosen experts' weighted sum, in 64 bits: ``gate_up(e)`` and ``down(e)`` give an expert's weights."""
    out = torch.zeros_like(x)
    for e in range(EXPERTS):
        tok, slot = torch.nonzero(ids == e, as_tuple=True)
        if tok.numel():
            g, u = (x[tok] @ gate_up(e).T).chunk(2, dim=1)
            out.index_add_(0, tok, quantize(_silu(g) * u) @ down(e).T * w[tok, slot, None])
    return out


class MoeLayer:
    """``TP_MoE`` on replicated tokens: router, both expert projections, the weighted sum over the chosen experts."""

    @staticmethod
    @functools.lru_cache(maxsize=1)
    def layer(name):
        H, inter = MOE[name]
        g = _generator(1)
        moe = TP_MoE(0, 1, None, TOP, True)
        # trained routers are sure of their first choices (and a near tie for the last place must not decide a token's result)
        moe._init_parameters(_normal(g, (EXPERTS, H), 6 * H ** -0.5), _normal(g, (EXPERTS, 2 * inter, H), H ** -0.5),
                             _normal(g, (EXPERTS, H, inter), inter ** -0.5))
        return moe

    @staticmethod
    def prepare(case, seed):
        return {"moe": MoeLayer.layer(case["layer"]), "x": _normal(_generator(seed), (case["tokens"], MOE[case["layer"]][0]))}

    @staticmethod
    def run(s):
        return s["moe"].dist_triton_AR_fwd(s["x"])

    @staticmethod
    def exact(case, seed):
        s = MoeLayer.prepare(case, seed)
        moe, x = s["moe"], s["x"].double()
        w, ids = torch.topk(torch.softmax(x @ moe.gate.double().T, -1), TOP, -1)
        return _experts(x, ids, w / w.sum(-1, keepdim=True), lambda e: moe.w_gate_up[e].double(), lambda e: moe.w_down[e].double())

    @staticmethod
    def work(case):
        return _expert_work(case, 2)

    @staticmethod
    def tolerance(case):
        return {"rel": 0.03, "max": 0.9}

    @staticmethod
    def draw(rng):
        return {"layer": rng.choice(sorted(MOE)), "tokens": _log_int(rng, 1, 8192)}


class Fp8Experts:
    """The expert block on block-scaled fp8 weights and activations, as an expert-parallel rank runs it on the tokens it received."""

    @staticmethod
    @functools.lru_cache(maxsize=1)
    def weights(name):
        H, inter = MOE[name]
        g = _generator(1)
        return (*quantize_fp8_weight_blocks(_normal(g, (EXPERTS, 2 * inter, H), H ** -0.5)),
                *quantize_fp8_weight_blocks(_normal(g, (EXPERTS, H, inter), inter ** -0.5)))

    @staticmethod
    def prepare(case, seed):
        g, T = _generator(seed), case["tokens"]
        x8, sx = quantize_fp8_rows(_normal(g, (T, MOE[case["layer"]][0])))
        logits = torch.randn(T, EXPERTS, device="cuda", generator=g) * 3
        w, ids = torch.topk(torch.softmax(logits, -1), TOP, -1)
        return {"x": x8, "scale": sx, "ids": ids.to(torch.int32), "w": w / w.sum(-1, keepdim=True), "weights": Fp8Experts.weights(case["layer"])}

    @staticmethod
    def run(s):
        up8, up_scale, down8, down_scale = s["weights"]
        up = grouped_gemm_fp8(s["x"], s["scale"], up8, up_scale, s["ids"])
        act, act_scale = ops.silu_mul_fp8(up)
        down = grouped_gemm_fp8(act, act_scale, down8, down_scale, s["ids"], a_per_pair=True, row_scale=s["w"])
        return reduce_topk(down, TOP)

    @staticmethod
    def exact(case, seed):
        s = Fp8Experts.prepare(case, seed)
        up8, up_scale, down8, down_scale = s["weights"]

        def dequantized(w8, scale, e):
            wide = scale[e].double().repeat_interleave(128, 0)[:w8.shape[1]].repeat_interleave(128, 1)
            return w8[e].double() * wide

        def quantized(a):
            blocks = a.view(a.shape[0], -1, 128)
            scale = blocks.abs().amax(-1, keepdim=True) / 448
            return ((blocks / scale).float().to(torch.float8_e4m3fn).double() * scale).view(a.shape)

        x = s["x"].double() * s["scale"].double().repeat_interleave(128, 1)
        return _experts(x, s["ids"], s["w"].double(), lambda e: dequantized(up8, up_scale, e), lambda e: dequantized(down8, down_scale, e), quantized)

    @staticmethod
    def work(case):
        return _expert_work(case, 1)

    @staticmethod
    def tolerance(case):
        return {"rel": 0.03, "max": 0.9}

    @staticmethod
    def draw(rng):
        return {"layer": "Qwen/Qwen3-30B-A3B", "tokens": _log_int(rng, 1, 8192)}


# ---- recurrent mixers -------------------------------------------------------------------------
class Recurrence:
    """``ops.wkv`` / ``ops.gated_delta``: the memories of a batch, advanced by the tokens of a prompt or by one token."""

    SIZES = {"wkv": ((32, 64), (64, 64)), "gated_delta": ((16, 128), (32, 128))}  # heads, channels
    EPS = 1e-6

    @staticmethod
    def prepare(case, seed):
        g, dtype = _generator(seed), DTYPES[case["dtype"]]
        B, S, H, D = case["batch"], case["tokens"], case["heads"], case["dim"]
        T, N = B * S, H * D
        s = {"kind": case["kind"], "start": _normal(g, (B, H, D, D), 1.0, torch.float32), "dim": D}
        s["memory"] = torch.empty_like(s["start"])
        if case["kind"] == "wkv":
            mixed = _normal(g, (T, 4 * N), 1.0, dtype)  # one projection of the shifted tokens
            s["rows"] = mixed.split(N, dim=1)
            s["z"] = _normal(g, (T, N), 0.5, dtype)
            s["w0"], s["u"] = _normal(g, (N,), 1.0, torch.float32, mean=-3.0), _normal(g, (N,), 0.5, torch.float32)
            s["gain"] = _normal(g, (N,), 0.1, torch.float32, mean=1.0)
        else:
            s["qk"] = _normal(g, (T, N), 1.0, dtype).split(N // 2, dim=1)  # two value heads to one key head
            s["v"], s["gate"] = _normal(g, (T, N), 1.0, dtype), _normal(g, (T, N), 1.0, dtype)
            s["ab"] = _normal(g, (T, 2 * H), 1.0, dtype).split(H, dim=1)
            s["a_log"], s["dt_bias"] = _normal(g, (H,), 0.5, torch.float32), _normal(g, (H,), 0.5, torch.float32, mean=-3.0)
            s["gain"] = _normal(g, (D,), 0.1, torch.float32, mean=1.0)
        return s

    @staticmethod
    def run(s):
        memory = s["memory"].copy_(s["start"])  # the sequences as they were before the call
        if s["kind"] == "wkv":
            out = ops.wkv(*s["rows"][:3], s["z"], s["rows"][3], s["w0"], s["u"], s["gain"], memory, s["dim"], s["dim"], Recurrence.EPS)
        else:
            out = ops.gated_delta(*s["qk"], s["v"], *s["ab"], s["gate"], s["a_log"], s["dt_bias"], s["gain"], memory, s["dim"], s["dim"],
                                  Recurrence.EPS)
        return {"out": out, "memory": memory}

    @staticmethod
    def exact(case, seed):
        s = Recurrence.prepare(case, seed)
        B, S, H, D = case["batch"], case["tokens"], case["heads"], case["dim"]
        M, outs = s["start"].double(), []
        if case["kind"] == "wkv":
            r, k, v, gate = (t.double().view(B, S, H, D) for t in s["rows"])
            decay = torch.exp(-torch.exp(s["z"].double() + s["w0"].double())).view(B, S, H, D)
            u, gain = s["u"].double().view(H, D), s["gain"].double().view(H, D)
            for t in range(S):
                kv = k[:, t, :, :, None] * v[:, t, :, None]
                outs.append(torch.einsum("bhd,bhde->bhe", r[:, t], M + u[..., None] * kv))
                M = decay[:, t, :, :, None] * M + kv
        else:
            q, k = (t.double().view(B, S, H // 2, D).repeat_interleave(2, 2) for t in s["qk"])
            q, k = (t / torch.sqrt(t.square().sum(-1, keepdim=True) + 1e-6) for t in (q, k))
            q, v, gate = q * D ** -0.5, s["v"].double().view(B, S, H, D), s["gate"].double().view(B, S, H, D)
            a, b = (t.double().view(B, S, H) for t in s["ab"])
            decay = torch.exp(-torch.exp(s["a_log"].double()) * F.softplus(a + s["dt_bias"].double()))
            step, gain = torch.sigmoid(b), s["gain"].double()
            for t in range(S):
                M = decay[:, t, :, None, None] * M
                d = step[:, t, :, None] * (v[:, t] - torch.einsum("bhd,bhde->bhe", k[:, t], M))
                M = M + k[:, t, :, :, None] * d[:, :, None]
                outs.append(torch.einsum("bhd,bhde->bhe", q[:, t], M))
        o = _rms(torch.stack(outs, 1), gain, Recurrence.EPS) * _silu(gate)
        return {"out": o.reshape(B * S, H * D), "memory": M}

    @staticmethod
    def work(case):
        T, H, D = case["batch"] * case["tokens"], case["heads"], case["dim"]
        wkv = case["kind"] == "wkv"
        rows = 6 if wkv else 4  # 16-bit rows of H * D values in and out
        return {"bytes": 2 * T * H * D * rows + 8 * case["batch"] * H * D * D, "flops": (5 if wkv else 7) * T * H * D * D}

    @staticmethod
    def tolerance(case):
        return {"rel": 0.01, "max": 0.15}

    @staticmethod
    def draw(rng):
        kind = rng.choice(("wkv", "gated_delta"))
        heads, dim = rng.choice(Recurrence.SIZES[kind])
        return {"kind": kind, "batch": _log_int(rng, 1, 8), "tokens": 1 if rng.random() < 0.25 else _log_int(rng, 16, 2048), "heads": heads,
                "dim": dim, "dtype": rng.choice(("bf16", "bf16", "f16"))}


# ---- 32-bit mode ------------------------------------------------------------------------------
class Mlp32:
    """The SwiGLU block of a model that runs in 32 bits (``TP_MLP``), as the replay of a trace uses it."""

    SIZES = {"sizilorn-1b": (2048, 5632), "sizilorn-7b": (4096, 11008)}

    @staticmethod
    @functools.lru_cache(maxsize=1)
    def layer(name):
        H, inter = Mlp32.SIZES[name]
        g, mlp = _generator(1), TP_MLP(0, 1)
        mlp._init_parameters(gate=_normal(g, (inter, H), H ** -0.5, torch.float32), up=_normal(g, (inter, H), H ** -0.5, torch.float32),
                             down=_normal(g, (H, inter), inter ** -0.5, torch.float32))
        return mlp

    @staticmethod
    def prepare(case, seed):
        return {"mlp": Mlp32.layer(case["model"]), "x": _normal(_generator(seed), (case["tokens"], Mlp32.SIZES[case["model"]][0]), 1.0, torch.float32)}

    @staticmethod
    def run(s):
        return s["mlp"].dist_triton_AR_fwd(s["x"])

    @staticmethod
    def exact(case, seed):
        s = Mlp32.prepare(case, seed)
        g, u = (s["x"].double() @ s["mlp"].gate_up_proj.double().T).chunk(2, dim=1)
        return (_silu(g) * u) @ s["mlp"].down_proj.double().T

    @staticmethod
    def work(case):
        H, inter = Mlp32.SIZES[case["model"]]
        T = case["tokens"]
        return {"bytes": 4 * (3 * H * inter + 2 * T * H), "flops": 6 * H * inter * T}

    @staticmethod
    def tolerance(case):
        return {"rel": 1e-5, "max": 1e-4}

    @staticmethod
    def draw(rng):
        return {"model": rng.choice(sorted(Mlp32.SIZES)), "tokens": _log_int(rng, 1, 1024)}


KINDS = {"decoder": Decoder, "prefill attention": PrefillAttention, "decode attention": DecodeAttention, "latent attention": LatentAttention,
         "moe": MoeLayer, "fp8 experts": Fp8Experts, "recurrence": Recurrence, "mlp 32": Mlp32}


def listed():
    qwen, shard, moe = "Qwen/Qwen3-8B", "Qwen3-32B-tp8-shard", "Qwen/Qwen3-30B-A3B"
    return [
        # one user's chat on one rank of a tensor-parallel group: every kernel is small, latency decides
        {"name": "decode 1", "of": "decoder", "model": shard, "batch": 1, "tokens": 1, "cached": 333},
        # a server's running batch: the headline benchmark's step, on a smaller model
        {"name": "decode 8", "of": "decoder", "model": qwen, "batch": 8, "tokens": 1, "cached": 2048},
        # three prompts of a chat, no size a multiple of a tile
        {"name": "prefill short", "of": "decoder", "model": qwen, "batch": 3, "tokens": 389, "cached": 0},
        # one long document
        {"name": "prefill long", "of": "decoder", "model": qwen, "batch": 1, "tokens": 16384, "cached": 0},
        # attention alone, over a pack of prompts of 1 K to 3 K tokens
        {"name": "attention pack", "of": "prefill attention", "sequences": 5, "mean": 2047, "heads": 64, "kv_heads": 8, "dtype": "bf16",
         "gated": False},
        # the decode attention of long contexts, where the cache's bytes decide
        {"name": "decode attention 32K", "of": "decode attention", "batch": 8, "kv": 32768, "heads": 32, "kv_heads": 8, "page": 64, "dtype": "bf16"},
        # latent attention of a short context: many heads share few bytes
        {"name": "latent attention 3K", "of": "latent attention", "batch": 8, "kv": 3000, "heads": 32, "dtype": "bf16"},
        # experts in a decode step (the weights' bytes decide) and in a prompt (the products do)
        {"name": "experts 24", "of": "moe", "layer": moe, "tokens": 24},
        {"name": "experts 4K", "of": "moe", "layer": moe, "tokens": 4099},
        {"name": "fp8 experts 2K", "of": "fp8 experts", "layer": moe, "tokens": 2048},
        # a recurrent mixer over prompts
        {"name": "recurrence prompts", "of": "recurrence", "kind": "wkv", "batch": 4, "tokens": 1500, "heads": 64, "dim": 64, "dtype": "bf16"},
        # a portion of a trace in 32 bits
        {"name": "feed-forward 32 bits", "of": "mlp 32", "model": "sizilorn-1b", "tokens": 100},
    ]


def draw(rng):
    of = rng.choice(sorted(KINDS))
    return {"of": of, **KINDS[of].draw(rng)}


def prepare(case, seed):
    return {"of": case["of"], "state": KINDS[case["of"]].prepare(case, seed)}


def run(state):
    return KINDS[state["of"]].run(state["state"])


def work(case):
    return KINDS[case["of"]].work(case)


def tolerance(case):
    return KINDS[case["of"]].tolerance(case)


def exact(case, seed):
    return KINDS[case["of"]].exact(case, seed)
