"""Decode GEMM whose tiles hold all of K, against the fp32 statement of the same chain."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N,K,swiglu", [
    (1, 8, 64, False),          # one granule, one k-block
    (8, 1280, 5120, False),     # a tile per SM or less, two stages of five k-blocks a warp
    (9, 1001, 192, False),      # the second half of the tokens, a ragged last tile, warps without a stage
    (16, 6144, 1088, False),
    (8, 1280, 4160, False),     # 65 k-blocks in stages of four: a ragged last stage
    (16, 3000, 4160, False), (5, 700, 704, True),
    (3, 60000, 128, False),     # several tiles per CTA
    (1, 3200, 5120, True), (8, 12288, 256, True), (16, 100, 320, True),
])
def test_gemm_rows(M, N, K, swiglu, dtype):
    from triton_distributed_b200 import ops
    torch.manual_seed(5)
    x = torch.randn(M, K, device="cuda").to(dtype)
    w = (torch.randn(N * (2 if swiglu else 1), K, device="cuda") * K ** -0.5).to(dtype)
    y = ops.gemm_rows(x, w, swiglu=swiglu)
    ref = x.double() @ w.double().T
    if swiglu:
        ref = torch.nn.functional.silu(ref[:, :N]) * ref[:, N:]
    # sums of K products of values around one in fp32, one rounding of the result
    eps = torch.finfo(dtype).eps
    torch.testing.assert_close(y.double(), ref, rtol=eps, atol=2e-5)
    for _ in range(20):  # the order of the sums is fixed, whatever order the boxes land in
        assert torch.equal(ops.gemm_rows(x, w, swiglu=swiglu, out_f32=True), y.float())
    if not swiglu:
        h = torch.randn(M, N, device="cuda").to(dtype)
        want = ref + h.double()
        ops.gemm_rows(x, w, out=h, residual=h)
        torch.testing.assert_close(h.double(), want, rtol=eps, atol=2e-5)


@pytest.mark.parametrize("M,N,K,swiglu", [(1, 1280, 5120, False), (8, 128, 64, False), (16, 3000, 4160, False), (5, 700, 704, True)])
def test_gemm_rows_norm(M, N, K, swiglu):
    from triton_distributed_b200 import ops
    torch.manual_seed(6)
    h = (torch.randn(M, K, device="cuda") * torch.logspace(-6, 6, M, device="cuda")[:, None]).bfloat16()
    gamma = (1 + torch.randn(K, device="cuda")).bfloat16()
    w = (torch.randn(N * (2 if swiglu else 1), K, device="cuda") * K ** -0.5).bfloat16()
    y = ops.gemm_rows(h, w, swiglu=swiglu, gamma=gamma, eps=1e-6)
    hd = h.double()
    scale = torch.rsqrt(hd.square().mean(-1, keepdim=True) + 1e-6)
    # the product of h and the gain is rounded to bf16, then everything is fp32 up to the result
    ref = ((hd * gamma.double()).to(torch.bfloat16).double() @ w.double().T) * scale
    if swiglu:
        ref = torch.nn.functional.silu(ref[:, :N]) * ref[:, N:]
    torch.testing.assert_close(y.double(), ref, rtol=2 ** -7, atol=2e-5)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N,K,swiglu", [(1, 130, 64, False), (8, 999, 4160, False), (13, 1280, 704, False), (16, 333, 1024, True)])
def test_gemm_rows_pitches(M, N, K, swiglu, dtype):
    """Rows of x, w, the result and the residual inside wider ones, through the entry that chooses the kernel; nothing beside them is
    written, and a token's result does not depend on the tokens beside it."""
    from triton_distributed_b200 import _lib, ops
    torch.manual_seed(8)
    rows = N * (2 if swiglu else 1)
    x = torch.randn(M + 1, K + 16, device="cuda").to(dtype)[1:, 8:K + 8]
    w = (torch.randn(rows, K + 24, device="cuda") * K ** -0.5).to(dtype)[:, 16:K + 16]
    wide = torch.full((M + 3, N + 5), 7.0, device="cuda", dtype=dtype)
    seen, call = [], _lib.call
    with pytest.MonkeyPatch.context() as m:
        m.setattr(_lib, "call", lambda name, *args: (seen.append(name), call(name, *args)))
        y = ops.gemm_skinny(x, w, wide[:M, 3:N + 3], swiglu=swiglu)
    assert seen == ["b200_gemm_rows"] and y.data_ptr() == wide[:M, 3:].data_ptr()
    ref = x.double() @ w.double().T
    if swiglu:
        ref = torch.nn.functional.silu(ref[:, :N]) * ref[:, N:]
    eps = torch.finfo(dtype).eps
    torch.testing.assert_close(y.double(), ref, rtol=eps, atol=2e-5)   # as in test_gemm_rows
    assert torch.equal(ops.gemm_rows(x[M // 2:M // 2 + 1], w, swiglu=swiglu)[0], y[M // 2])
    if not swiglu:
        h = torch.randn(M, N, device="cuda").to(dtype)
        wide[:M, 3:N + 3] = h
        ops.gemm_rows(x, w, out=wide[:M, 3:N + 3], residual=wide[:M, 3:N + 3])
        torch.testing.assert_close(wide[:M, 3:N + 3].double(), ref + h.double(), rtol=eps, atol=2e-5)
    assert torch.all(wide[M:] == 7.0) and torch.all(wide[:, :3] == 7.0) and torch.all(wide[:, N + 3:] == 7.0)


@pytest.mark.parametrize("settled", [False, True])
def test_gemm_rows_repeats_itself_in_chains(settled):
    """Launches of several sizes that start under one another, with another stream's work on the SMs: every result has the bits of the
    call alone, which is right against 64 bits."""
    from triton_distributed_b200 import ops
    torch.manual_seed(9)
    cases = []
    for M, N, K, gated, normed in [(1, 1280, 5120, False, True), (8, 592, 4096, False, False), (16, 128, 2048, False, False), (5, 3200, 1024, True, True),
                                   (16, 3000, 4160, False, False), (9, 8, 64, False, False)]:
        x, w = torch.randn(M, K).bfloat16(), (torch.randn(N * (2 if gated else 1), K) * K ** -0.5).bfloat16()
        gamma = (1 + torch.randn(K)).bfloat16() if normed else None
        ref = (x.double() * gamma.double()).bfloat16().double() @ w.double().T if normed else x.double() @ w.double().T   # on the host
        if normed:
            ref *= torch.rsqrt(x.double().square().mean(-1, keepdim=True) + 1e-6)
        if gated:
            ref = torch.nn.functional.silu(ref[:, :N]) * ref[:, N:]
        args = [t.cuda() if t is not None else None for t in (x, w, gamma)]
        cases.append((args, gated, ref))
    torch.cuda.synchronize()   # the operands are settled
    call = lambda a, gated: ops.gemm_rows(a[0], a[1], swiglu=gated, gamma=a[2], eps=1e-6, settled=settled)
    alone = [call(a, gated) for a, gated, _ in cases]
    for got, (_, _, ref) in zip(alone, cases):   # (as in test_gemm_rows_norm)
        torch.testing.assert_close(got.cpu().double(), ref, rtol=2 ** -7, atol=2e-5)
    side, busy = torch.cuda.Stream(), torch.randn(2048, 2048, device="cuda").bfloat16()
    torch.cuda.synchronize()
    wrong = torch.zeros(len(cases), dtype=torch.int32, device="cuda")
    for _ in range(20):
        with torch.cuda.stream(side):
            for _ in range(4):
                busy @ busy
        got = [[call(a, gated) for a, gated, _ in cases] for _ in range(10)]
        for ys in got:
            for i, y in enumerate(ys):
                wrong[i] += (y.view(torch.int16) != alone[i].view(torch.int16)).any()
    assert wrong.tolist() == [0] * len(cases)
    ops.check_pipeline_status()


def test_status_word_is_made_in_front_of_a_capture(monkeypatch):
    """A word that a capture made would be cleared by every replay, and read before the first."""
    from triton_distributed_b200 import ops
    x, w = torch.randn(8, 256, device="cuda").bfloat16(), torch.randn(512, 256, device="cuda").bfloat16()
    monkeypatch.setattr(ops, "_pipe_status", {})
    ops.reserve_skinny_scratch(x.device, 1, 1)
    words = dict(ops._pipe_status)
    assert len(words) == 1
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ops.gemm_skinny(x, w)
    assert ops._pipe_status == words
    words[x.device.index].fill_(3)
    graph.replay()
    with pytest.raises(RuntimeError):
        ops.check_pipeline_status()


def test_gemm_rows_refuses():
    from triton_distributed_b200 import _lib, ops
    x = torch.zeros(4, 128, device="cuda", dtype=torch.float16)
    w = torch.zeros(64, 128, device="cuda", dtype=torch.float16)
    with pytest.raises(_lib.NativeError):
        ops.gemm_rows(x, w, gamma=torch.ones(128, device="cuda", dtype=torch.float16), eps=1e-6)
    with pytest.raises(_lib.NativeError):
        ops.gemm_rows(x[:, :120], w[:, :120])
    with pytest.raises(_lib.NativeError):
        ops.gemm_rows(x.new_zeros(17, 128), w)
